// Retina-cluster decoding on sm_100a: the VELO front end for VPRetinaCluster banks (type 73),
// whose words already hold a cluster's column, row and fraction.  Replaces
// calculate_number_of_retinaclusters_each_sensor_pair, its prefix sum and decode_retinaclusters
// (device/velo/retinacluster_decoding/src/CalculateNumberOfRetinaClustersPerSensor.cu:12-48,
// DecodeRetinaClusters.cu:11-383) with two kernels and one scan of per-event totals:
//
//   retina_count_kernel   [N CTAs]  clusters per sensor (pair) of each event and the event's
//                                   total; the slice's first event writes the bank index
//   exclusive_scan_kernel           event bases from the totals
//   retina_decode_kernel  [N CTAs]  per event: the sensor offsets (prefix sum inside the CTA
//                                   plus the event base), the module-pair offsets, the clusters
//                                   decoded, keyed by (phi, id), ranked inside their module
//                                   pair and written to their sorted slot
//
// Outputs are the reference's: dev_each_sensor_pair_size, dev_offsets_each_sensor_pair_size,
// dev_retina_bank_index, dev_module_cluster_num, dev_offsets_module_pair_cluster (the search's
// dev_offsets_estimated_input_size) and the sorted cluster container.  The permutation is
// intermediate and stays in shared memory, the keys and the decoded hits in L2-resident scratch.
// Arithmetic in the reference's order and rounding, so every cluster is bit-identical.
#include "velo_kernels.cuh"

namespace velo {

  __device__ __forceinline__ unsigned retina_sensors(int version) { return (version == 2 || version == 3) ? n_sensors : n_sensors / 2; }

  struct RetinaBank {
    unsigned source_id, count, size, type;
    const uint32_t* word;
  };

  __device__ __forceinline__ unsigned retina_n_banks(const RawInput& in, unsigned ev)
  {
    return in.mep_layout ? mep_n_banks(in) : reinterpret_cast<const uint32_t*>(in.raw + in.offsets[ev])[0];
  }

  __device__ __forceinline__ RetinaBank retina_bank(const RawInput& in, unsigned ev, unsigned b)
  {
    const bool v23 = in.bank_version == 2 || in.bank_version == 3;
    if (in.mep_layout) {
      // MEPTools.h:55-205: the fragment starts with the bank data (no sourceID word)
      RetinaBank r;
      const uint32_t* frag = reinterpret_cast<const uint32_t*>(in.raw + mep_fragment_offset(in, ev, b));
      r.source_id = mep_source_id(in, b);
      r.count = v23 ? frag[0] : 0u;
      r.word = frag + (v23 ? 1 : 0);
      r.size = mep_bank_size(in, ev, b);
      r.type = mep_bank_type(in, ev, b);
      return r;
    }
    const char* blob = in.raw + in.offsets[ev];
    const uint32_t* w = reinterpret_cast<const uint32_t*>(blob);
    const unsigned n_banks = w[0];
    const char* payload = blob + 4 * (n_banks + 2);
    const uint32_t* bank = reinterpret_cast<const uint32_t*>(payload + w[1 + b]);
    RetinaBank r;
    r.source_id = bank[0];
    r.count = v23 ? bank[1] : 0u;
    r.word = bank + (v23 ? 2 : 1);
    r.size = bank_sizes(in, ev)[b];
    r.type = bank_types(in, ev)[b];
    return r;
  }

  // CalculateNumberOfRetinaClustersPerSensor.cu:12-48, plus the event total
  __global__ void __launch_bounds__(decode_threads) retina_count_kernel(RetinaParams p)
  {
    __shared__ unsigned warp_sums[33];
    const unsigned e = blockIdx.x, ev = e + p.in.event_start;
    const unsigned per_event = retina_sensors(p.in.bank_version);
    unsigned* size = p.each_sensor_pair_size + size_t(e) * per_event;
    for (unsigned s = threadIdx.x; s < per_event; s += blockDim.x)
      size[s] = 0;
    __syncthreads();
    const unsigned n_banks = retina_n_banks(p.in, ev);
    for (unsigned b = threadIdx.x; b < n_banks; b += blockDim.x) {
      const RetinaBank bank = retina_bank(p.in, ev, b);
      if (bank.type == bank_type_vp_retina) {
        const bool v23 = p.in.bank_version == 2 || p.in.bank_version == 3;
        const unsigned s = v23 ? bank.source_id : (bank.source_id & 0x1FFu);
        if (s < per_event) size[s] = v23 ? bank.count : bank.size / 4u;
        else set_error(p.status, err_input_capacity);
      }
      // the reference's block 0 writes every bank's number in bank order: the last wins
      if (e == 0 && (bank.source_id & 0x1FFu) < per_event) atomicMax(p.bank_index + (bank.source_id & 0x1FFu), b);
    }
    __syncthreads();
    unsigned part = 0;
    for (unsigned s = threadIdx.x; s < per_event; s += blockDim.x)
      part += size[s];
    unsigned total;
    block_exclusive_scan(part, warp_sums, &total);
    if (threadIdx.x == 0) p.event_total[e] = total;
  }

  struct RetinaCluster {
    uint32_t id;
    float x, y, z;
    int16_t phi;
    unsigned sensor;
  };

  // populate_retinacluster / populate_sorting_key (DecodeRetinaClusters.cu:80-160, 246-303)
  __device__ __forceinline__ RetinaCluster
  decode_word(const Geometry* g, const Constants& k, int version, unsigned source_id, uint32_t w)
  {
    RetinaCluster c;
    if (version == 2 || version == 3) c.sensor = source_id;
    else c.sensor = ((source_id & 0x1FFu) << 1) | ((w >> 22) & 0x1u);
    uint32_t cx, cy, or_fx, or_fy;
    float fx, fy;
    if (version == 2) {
      cx = (w >> 14) & 0x3FFu;
      fx = __fdiv_rn(__uint2float_rn((w >> 11) & 0x7u), 8.f);
      cy = (w >> 3) & 0xFFu;
      fy = __fdiv_rn(__uint2float_rn(w & 0x7FFu), 8.f);
      or_fx = 0;
      or_fy = 0;
    }
    else {
      cx = (w >> 12) & 0x3FFu;
      fx = __fdiv_rn(__uint2float_rn((w >> 10) & 0x3u), 4.f);
      cy = (w >> 2) & 0xFFu;
      fy = __fdiv_rn(__uint2float_rn(w & 0x3FFu), 4.f);
      or_fx = ((w >> 11) & 0x1u) | ((w >> 10) & 0x1u);
      or_fy = ((w >> 1) & 0x1u) | (w & 0x1u);
    }
    const unsigned sensor = c.sensor < n_sensors ? c.sensor : 0u;
    const float* ltg = g->ltg + 12 * sensor;
    const float local_x = column_local_x(g, cx) + fx * column_x_pitch(g, cx);
    const float local_y = (0.5f + fy) * 0.055f;
    c.x = __ldg(ltg + 0) * local_x + __ldg(ltg + 1) * local_y + __ldg(ltg + 9);
    c.y = __ldg(ltg + 3) * local_x + __ldg(ltg + 4) * local_y + __ldg(ltg + 10);
    c.z = __ldg(ltg + 6) * local_x + __ldg(ltg + 7) * local_y + __ldg(ltg + 11);
    c.id = lhcb_id((or_fx << 27) | (or_fy << 26) | channel_id(c.sensor, cx >> 8, cx & 0xFFu, cy));
    c.phi = hit_phi_16(k, c.x, c.y);
    return c;
  }

  // Where an event's clusters of sensor (pair) s lie: the bank comes from the bank index the slice's
  // first event wrote (as in the reference).
  struct SensorBank {
    const uint32_t* word;
    unsigned source_id;
    unsigned n; // words; retina_no_bank: the event has no such bank, retina_other_type: it is another one's
  };
  constexpr unsigned retina_no_bank = 0xFFFFFFFFu, retina_other_type = 0xFFFFFFFEu;

  __device__ __forceinline__ SensorBank sensor_bank(const RetinaParams& p, unsigned ev, unsigned s)
  {
    SensorBank r {nullptr, 0, retina_no_bank};
    const unsigned b = p.bank_index[s];
    if (b >= retina_n_banks(p.in, ev)) return r;
    const RetinaBank bank = retina_bank(p.in, ev, b);
    const bool v23 = p.in.bank_version == 2 || p.in.bank_version == 3;
    r.word = bank.word;
    r.source_id = bank.source_id;
    r.n = bank.type == bank_type_vp_retina ? min(v23 ? bank.count : bank.size / 4u, retina_other_type - 1) : retina_other_type;
    return r;
  }

  // binary_search_rightmost (BinarySearch.cuh:33-47)
  __device__ __forceinline__ unsigned rightmost(const unsigned* a, unsigned n, unsigned value)
  {
    int l = 0, r = int(n);
    while (l < r) {
      const int m = (l + r) / 2;
      if (a[m] > value) r = m;
      else l = m + 1;
    }
    return unsigned(r - 1);
  }

  // Rank buckets per module pair: the top 6 bits of the (signed) sort key, so that bucket order
  // is key order; about 1.3 clusters per bucket at nu = 7.6.
  constexpr unsigned rank_buckets = 64;
  constexpr unsigned rank_counters = n_module_pairs * rank_buckets;

  __device__ __forceinline__ unsigned key_bucket(int64_t key)
  {
    return static_cast<unsigned>(static_cast<int>(key >> 58) + 32);
  }

  // u16 counters packed two per 32-bit word; returns the previous value of counter b.
  __device__ __forceinline__ unsigned bump_u16(uint16_t* counters, unsigned b)
  {
    const unsigned shift = 16 * (b & 1u);
    const uint32_t old = atomicAdd(reinterpret_cast<uint32_t*>(counters) + (b >> 1), 1u << shift);
    return (old >> shift) & 0xFFFFu;
  }

  // The key (phi, id) a hit sorts by; a zero word's is the largest.
  __device__ __forceinline__ int64_t retina_key(uint32_t word, int16_t phi, uint32_t id)
  {
    return word != 0 ? static_cast<int64_t>((static_cast<uint64_t>(static_cast<uint16_t>(phi)) << 48) | id) : 0x7FFFFFFFFFFFFFFFll;
  }

  // Each cluster is decoded once, into a 16-byte record and its key in L2-resident scratch, and
  // written to the container in bucket order, so that neighbouring threads write neighbouring
  // places.  Capped for eight CTAs per SM (32 registers): 16 KB of bucket order plus about 8 KB
  // of counters, offsets and banks in shared memory allow that many.  16000 events of 2140
  // clusters: 0.85 ms; looking each word's bank up in the raw event twice, decoding it twice and
  // writing in bank order, 1.19.
  __global__ void __launch_bounds__(decode_threads, 8) retina_decode_kernel(RetinaParams p)
  {
    extern __shared__ __align__(16) unsigned char dsmem[];
    __shared__ unsigned so[n_sensors + 1]; // event-relative sensor offsets
    __shared__ unsigned mp_num[n_module_pairs], mp_zero[n_module_pairs];
    __shared__ unsigned warp_sums[33];
    __shared__ __align__(4) uint16_t bucket_end[rank_counters];
    __shared__ unsigned irregular;
    __shared__ SensorBank banks[n_sensors];
    const unsigned e = blockIdx.x, ev = e + p.in.event_start, n = p.in.n_events;
    const int version = p.in.bank_version;
    const unsigned per_event = retina_sensors(version);
    const unsigned step = per_event / n_module_pairs;
    const unsigned base = p.event_base[e];
    const unsigned T = p.event_base[n];
    if (T > p.cluster_capacity) {
      if (threadIdx.x == 0) set_error(p.status, err_input_capacity);
      return;
    }
    // sensor offsets: prefix sum of this event's sizes (per_event <= 208 < blockDim)
    const unsigned* size = p.each_sensor_pair_size + size_t(e) * per_event;
    const unsigned mine = threadIdx.x < per_event ? size[threadIdx.x] : 0u;
    unsigned total;
    const unsigned excl = block_exclusive_scan(mine, warp_sums, &total);
    if (threadIdx.x < per_event) {
      banks[threadIdx.x] = sensor_bank(p, ev, threadIdx.x);
      so[threadIdx.x] = excl;
      p.offsets_each_sensor_pair_size[size_t(e) * per_event + threadIdx.x] = base + excl;
    }
    if (threadIdx.x == 0) {
      so[per_event] = total;
      if (e == n - 1) p.offsets_each_sensor_pair_size[size_t(n) * per_event] = base + total;
      if (e == 0) p.offsets_module_pair_cluster[0] = 0;
      irregular = 0;
    }
    if (threadIdx.x < n_module_pairs) {
      mp_num[threadIdx.x] = 0;
      mp_zero[threadIdx.x] = 0;
    }
    for (unsigned i = threadIdx.x; i < rank_counters / 2; i += blockDim.x)
      reinterpret_cast<uint32_t*>(bucket_end)[i] = 0;
    __syncthreads();
    // populate_module_pair_offsets_and_sizes (DecodeRetinaClusters.cu:11-35)
    if (threadIdx.x < n_module_pairs) p.offsets_module_pair_cluster[e * n_module_pairs + threadIdx.x + 1] = base + so[(threadIdx.x + 1) * step];

    // the bucket order in shared memory when the event fits its capacity, else no buckets (the
    // full comparison)
    const bool in_smem = total <= p.smem_order_capacity;
    int64_t* keys = reinterpret_cast<int64_t*>(p.key_scratch) + base;
    uint4* hits = reinterpret_cast<uint4*>(p.hit_scratch) + base;
    uint16_t* order = reinterpret_cast<uint16_t*>(dsmem);
    const Geometry* g = p.geo;
    const Constants k = p.k;
    // velo_calculate_sorting_key (DecodeRetinaClusters.cu:162-244)
    for (unsigned c = threadIdx.x; c < total; c += blockDim.x) {
      const unsigned s = rightmost(so, per_event, c), index = c - so[s];
      const SensorBank& bank = banks[s];
      int64_t key = 0x7FFFFFFFFFFFFFFFll;
      bool counted = false;
      if (index < bank.n && bank.n < retina_other_type) {
        const uint32_t w = bank.word[index];
        const RetinaCluster cl = decode_word(g, k, version, bank.source_id, w);
        const unsigned mp = cl.sensor / 8;
        if (mp < n_module_pairs) {
          atomicAdd(w != 0 ? &mp_num[mp] : &mp_zero[mp], 1u);
          counted = mp == s / step;
        }
        key = retina_key(w, cl.phi, cl.id);
        hits[c] = make_uint4(__float_as_uint(cl.x), __float_as_uint(cl.y), __float_as_uint(cl.z), cl.id);
      }
      else if (bank.n != retina_other_type) {
        set_error(p.status, err_input_capacity); // no such bank, or fewer words than the event's counts
      }
      keys[c] = key;
      if (in_smem) {
        if (counted) bump_u16(bucket_end, (s / step) * rank_buckets + key_bucket(key));
        else irregular = 1; // a cluster the module-pair counts miss: rank by the full comparison
      }
    }
    __syncthreads();
    if (threadIdx.x < n_module_pairs) p.module_cluster_num[e * n_module_pairs + threadIdx.x] = mp_num[threadIdx.x];

    // velo_calculate_permutations + decode_retinaclusters_sorted (DecodeRetinaClusters.cu:37-78,
    // 305-383): a cluster's slot is its module pair's start plus the number of smaller keys of
    // the module pair.  When every cluster was counted in its module pair's (key) buckets, the
    // buckets are laid out in order by a scan of their counts, each cluster is placed in its
    // bucket, and its rank is the bucket's start plus the smaller keys of the same bucket.
    const bool bucketed = in_smem && !irregular;
    if (bucketed) {
      constexpr unsigned per = (rank_counters + decode_threads - 1) / decode_threads;
      unsigned v[per];
      unsigned sum = 0;
#pragma unroll
      for (unsigned q = 0; q < per; ++q) {
        const unsigned b = threadIdx.x * per + q;
        v[q] = b < rank_counters ? bucket_end[b] : 0u;
        sum += v[q];
      }
      unsigned all;
      unsigned run = block_exclusive_scan(sum, warp_sums, &all);
      __syncthreads(); // every count read before the starts overwrite them
#pragma unroll
      for (unsigned q = 0; q < per; ++q) {
        const unsigned b = threadIdx.x * per + q;
        if (b < rank_counters) bucket_end[b] = static_cast<uint16_t>(run); // start; the fill below ends it
        run += v[q];
      }
      __syncthreads();
      for (unsigned c = threadIdx.x; c < total; c += blockDim.x) {
        const unsigned s = rightmost(so, per_event, c);
        order[bump_u16(bucket_end, (s / step) * rank_buckets + key_bucket(keys[c]))] = static_cast<uint16_t>(c);
      }
      __syncthreads();
    }
    ClusterView out {p.container, T};
    auto write = [&](unsigned dst, const uint4& hit, int64_t key) {
      if (dst >= T) {
        set_error(p.status, err_cluster_capacity);
        return;
      }
      const float x = __uint_as_float(hit.x), y = __uint_as_float(hit.y);
      __stcs(&out.id(dst), hit.w);
      __stcs(&out.x(dst), x);
      __stcs(&out.y(dst), y);
      __stcs(&out.z(dst), __uint_as_float(hit.z));
      // a zero word's key does not hold its phi
      __stcs(&out.phi(dst), key != 0x7FFFFFFFFFFFFFFFll ? static_cast<int16_t>(key >> 48) : hit_phi_16(k, x, y));
    };
    if (bucketed) {
      unsigned mp = 0;
      for (unsigned q = threadIdx.x; q < total; q += blockDim.x) {
        const unsigned c = order[q];
        const int64_t key = keys[c];
        const uint4 hit = hits[c];
        while (q >= so[(mp + 1) * step]) ++mp;
        const unsigned b = mp * rank_buckets + key_bucket(key);
        const unsigned first = b ? bucket_end[b - 1] : 0u, last = bucket_end[b];
        unsigned position = first; // every cluster was counted: bucket order is event order
        for (unsigned i = first; i < last; ++i)
          position += key > keys[order[i]];
        write(base + position, hit, key);
      }
    }
    else {
      for (unsigned c = threadIdx.x; c < total; c += blockDim.x) {
        const unsigned s = rightmost(so, per_event, c), mp = s / step;
        if (c - so[s] >= banks[s].n || banks[s].n >= retina_other_type) continue;
        const unsigned start = so[mp * step];
        const int64_t key = keys[c];
        unsigned position = 0;
        const unsigned num = min(mp_num[mp] + mp_zero[mp], total - start);
        for (unsigned j = 0; j < num; ++j)
          position += (start + j != c) && key > keys[start + j];
        write(base + start + position, hits[c], key);
      }
    }
    // the event's records and keys are dead
    __syncthreads();
    discard_l2(hits, size_t(16) * total);
    discard_l2(keys, size_t(8) * total);
  }

} // namespace velo

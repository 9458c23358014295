// VELO super-pixel decoding on sm_100a: candidate counting and input-size estimate
// (velo_calculate_number_of_candidates + velo_estimate_input_size), masked clustering,
// phi and the sort by phi (velo_masked_clustering + velo_sort_by_phi), one event per CTA.
//
// The estimate kernel reads an event's super pixels once into shared memory, one thread per
// super pixel over the flattened bank list, sizes the event, and leaves an item per cluster to
// make: the isolated super pixels, and the pixel sums of the clusters that the candidates among
// the others grow into.  The clustering kernel turns the items into hits with every lane busy
// and sorts them; it needs neither the raw words nor a bank table.
// The neighbour scans of the reference (EstimateInputSize.cu:111-141,
// MaskedVeloClustering.cu:361-402) test the address of every super pixel of a bank against one
// range (four instructions each) and look closer at the few inside it.
//
// The sorted container is independent of the order in which clusters are produced
// (rank by (phi, id), SortByPhi.cu:104-122), so clusters are appended to their module
// pair with shared-memory atomics and ranked in place; no unsorted container is written.
#include "velo_kernels.cuh"

namespace velo {

  constexpr unsigned max_banks = 512;
  constexpr unsigned bank_hints = 512; // bank_of() hints, one per 32 SPs
  constexpr unsigned estimate_words = 3584; // SPs of an event that the estimate kernel holds in shared memory

  // ------------------------------------------------------------------------------------
  // Bank table of one event (ClusteringDefinitions.cuh:61-144)
  // ------------------------------------------------------------------------------------
  __device__ __forceinline__ unsigned bank_module_pair(unsigned source_id, int version)
  {
    return (version == 2 || version == 3) ? (source_id & 0x1FFu) / 8 : ((source_id & 0x1FFu) << 1) / 8;
  }

  // The words of an event: its own (Allen layout), or all of a MEP's, whose banks are scattered.
  struct EventWords {
    const uint32_t* w;
    unsigned n;           // words of the event (MEP: no bound)
    unsigned n_banks_raw; // as the event states it
    unsigned n_banks;     // at most max_banks
  };

  __device__ __forceinline__ EventWords event_words(const RawInput& in, unsigned ev)
  {
    EventWords r;
    if (in.mep_layout) {
      r.w = reinterpret_cast<const uint32_t*>(in.raw);
      r.n = 0xFFFFFFFFu;
      r.n_banks_raw = mep_n_banks(in);
    }
    else {
      const unsigned begin = in.offsets[ev];
      r.w = reinterpret_cast<const uint32_t*>(in.raw + begin);
      r.n = (in.offsets[ev + 1] - begin) / 4;
      r.n_banks_raw = r.n > 0 ? r.w[0] : 0u;
    }
    r.n_banks = min(r.n_banks_raw, max_banks);
    return r;
  }

  struct Bank {
    unsigned first;     // first SP word
    unsigned n_sp;      // SP words (any bank type), clamped to the event or the fragment
    unsigned stated;    // SP words as the bank states them
    unsigned source_id;
    bool velo;
    bool bad;           // the stated words do not fit
  };

  // Bank b < n_banks of an event.  A MEP fragment must start on a 4-byte boundary; its word
  // count is clamped to the bank size.
  __device__ __forceinline__ Bank event_bank(const RawInput& in, unsigned ev, const EventWords& e, unsigned b)
  {
    const bool v23 = in.bank_version == 2 || in.bank_version == 3;
    Bank r;
    r.bad = false;
    if (in.mep_layout) {
      const unsigned frag = mep_fragment_offset(in, ev, b);
      const unsigned size = mep_bank_size(in, ev, b);
      const unsigned type = mep_bank_type(in, ev, b);
      r.velo = type == bank_type_vp || type == bank_type_velo;
      r.source_id = mep_source_id(in, b);
      r.stated = r.n_sp = r.first = 0;
      if (frag & 3u) {
        r.bad = true;
      }
      else if (v23) {
        r.stated = size >= 4 ? e.w[frag / 4] : 0u;
        r.first = frag / 4 + 1;
        const unsigned room = size >= 4 ? size / 4 - 1 : 0u;
        r.bad = r.stated > room;
        r.n_sp = min(r.stated, room);
      }
      else {
        r.stated = r.n_sp = size / 4u;
        r.first = frag / 4;
      }
      return r;
    }
    const unsigned off = (1 + b < e.n) ? e.w[1 + b] : 0u;
    const unsigned w = 2 + e.n_banks_raw + off / 4;
    const unsigned type = bank_types(in, ev)[b];
    r.velo = type == bank_type_vp || type == bank_type_velo;
    r.source_id = w < e.n ? e.w[w] : 0u;
    if (v23) {
      r.stated = (w + 1 < e.n) ? e.w[w + 1] : 0u;
      r.first = w + 2;
    }
    else {
      r.stated = bank_sizes(in, ev)[b] / 4u;
      r.first = w + 1;
    }
    r.n_sp = r.stated;
    if (r.first > e.n) r.first = e.n;
    if (r.first + r.n_sp > e.n || r.first + r.n_sp < r.first) {
      r.bad = true;
      r.n_sp = e.n - r.first;
    }
    return r;
  }

  struct BankTable {
    unsigned n_banks;
    unsigned total_sp;
    unsigned count_total;          // SP words of VP/Velo banks as stated (reference: raw_bank.count or size / 4)
    unsigned words_off[max_banks]; // first SP word of the bank, in words from the event start
    unsigned flat[max_banks + 1];  // exclusive scan of the SP words over VP/Velo banks
    unsigned source_id[max_banks];
    // hint[k]: the bank holding flat SP k * 32 (entries up to total_sp / 32), where the searches
    // for an SP's bank start
    uint16_t hint[bank_hints];
  };

  // Fills the table; ends with a __syncthreads().
  __device__ void parse_banks(
    const RawInput& in, unsigned ev, const EventWords& e, BankTable& bt, unsigned* warp_sums, unsigned* status)
  {
    if (threadIdx.x == 0) {
      bt.count_total = 0;
      if (e.n_banks_raw > max_banks) set_error(status, err_input_capacity);
    }
    unsigned carry = 0, count = 0;
    for (unsigned base = 0; base < e.n_banks; base += blockDim.x) {
      const unsigned b = base + threadIdx.x;
      unsigned nsp_flat = 0;
      if (b < e.n_banks) {
        const Bank bank = event_bank(in, ev, e, b);
        if (bank.bad) set_error(status, err_input_capacity);
        if (bank.velo) {
          count += bank.stated;
          nsp_flat = bank.n_sp;
        }
        bt.words_off[b] = bank.first;
        bt.source_id[b] = bank.source_id;
      }
      unsigned total;
      const unsigned excl = block_exclusive_scan(nsp_flat, warp_sums, &total);
      if (b < e.n_banks) bt.flat[b] = carry + excl;
      carry += total;
    }
    count = __reduce_add_sync(0xFFFFFFFFu, count);
    if ((threadIdx.x & 31u) == 0 && count) atomicAdd(&bt.count_total, count);
    if (threadIdx.x == 0) {
      bt.n_banks = e.n_banks;
      bt.total_sp = carry;
      bt.flat[e.n_banks] = carry;
    }
    __syncthreads();
    for (unsigned b = threadIdx.x; b < e.n_banks; b += blockDim.x) {
      const unsigned hi = bt.flat[b + 1];
      for (unsigned k = (bt.flat[b] + 31) / 32; k < bank_hints && k * 32 < hi; ++k)
        bt.hint[k] = static_cast<uint16_t>(b);
    }
    __syncthreads();
  }

  // Adds each lane's v (0, 1 or 2) to its counter, from converged lanes: one atomic when all
  // lanes name the same counter.
  __device__ __forceinline__ void add_to_counter(unsigned* counters, unsigned key, unsigned v)
  {
    const unsigned lanes = __activemask(), leader = __ffs(lanes) - 1;
    if (__all_sync(lanes, key == __shfl_sync(lanes, key, leader))) {
      const unsigned sum = __popc(__ballot_sync(lanes, v > 0)) + __popc(__ballot_sync(lanes, v > 1));
      if ((threadIdx.x & 31u) == leader && sum) atomicAdd(counters + key, sum);
    }
    else if (v) {
      atomicAdd(counters + key, v);
    }
  }

  // Places for the converged lanes' items (v of 0, 1 or 2 each) behind *counter: one atomic per
  // warp.  Returns the place of a lane's first item; its second one lies at `second`.
  __device__ __forceinline__ unsigned append_items(unsigned* counter, unsigned v, unsigned& second)
  {
    const unsigned lanes = __activemask(), leader = __ffs(lanes) - 1, lane = threadIdx.x & 31u;
    const unsigned one = __ballot_sync(lanes, v > 0), two = __ballot_sync(lanes, v > 1);
    unsigned at = 0;
    if (lane == leader) at = atomicAdd(counter, static_cast<unsigned>(__popc(one) + __popc(two)));
    at = __shfl_sync(lanes, at, leader);
    const unsigned below = (1u << lane) - 1u;
    second = at + __popc(one) + __popc(two & below);
    return at + __popc(one & below);
  }

  __device__ __forceinline__ unsigned bank_of(const BankTable& bt, unsigned f)
  {
    // last bank b with flat[b] <= f < total_sp (banks with no SP share their start with the next)
    unsigned lo = 0, hi = bt.n_banks;
    while (hi - lo > 1) {
      const unsigned mid = (lo + hi) / 2;
      if (bt.flat[mid] <= f) lo = mid;
      else hi = mid;
    }
    return lo;
  }

  // bank_of() of the 32 consecutive SPs of a warp (f of lane 0 a multiple of 32, every lane of
  // the warp calls it): the lanes hold the starts of the banks behind the hint and bisect them
  // by shuffles.  Beyond the last SP the result is some bank.
  __device__ __forceinline__ unsigned bank_of_warp(const BankTable& bt, unsigned f)
  {
    const unsigned k = f / 32;
    const bool hinted = k < bank_hints && (f & ~31u) < bt.total_sp;
    const unsigned b0 = hinted ? bt.hint[k] : 0u;
    const unsigned next = b0 + 1 + (threadIdx.x & 31u);
    const unsigned start = next < bt.n_banks ? bt.flat[next] : 0xFFFFFFFFu;
    unsigned n = 0;
#pragma unroll
    for (unsigned step = 16; step >= 1; step /= 2)
      if (__shfl_sync(0xFFFFFFFFu, start, n + step - 1) <= f) n += step;
    if (!hinted || n == 31) return f < bt.total_sp ? bank_of(bt, f) : 0u;
    return b0 + n;
  }

  // ------------------------------------------------------------------------------------
  // Neighbour scans.  The reference visits every SP of the bank for every SP
  // (EstimateInputSize.cu:111-141) and every candidate (MaskedVeloClustering.cu:361-402).  The
  // SPs that can matter lie in one short range of addresses (column, then row), so the scan
  // only notes which SPs of the bank are in the range, a bit each, and the caller looks at
  // those: about one of the 12 to 24 SPs a bank holds, and a lane that has none does not wait
  // for the others at every SP.  (Against key-sorted bank copies searched by bisection, whose sort
  // compares every pair of a bank's SPs: estimate and clustering together 2.79 -> 2.10 ms for
  // 16000 events of 2540 SPs, 1.75 -> 1.06 ms for 2000 of 8200 SPs, version 4, 78 SPs per bank.)
  // ------------------------------------------------------------------------------------
  // visit(w) for the SPs among words[0, n) but words[self] with lo <= ((w >> 8) & key_mask) <= lo + span,
  // in order (self >= n: none left out).  Eight keys at a time: up to seven words behind the last
  // are read, and not used, when PAD says that they may be.
  template<bool PAD, typename Visit>
  __device__ __forceinline__ void scan_keys(
    const uint32_t* words, unsigned n, unsigned self, uint32_t lo, uint32_t span, uint32_t key_mask, Visit&& visit)
  {
    const uint32_t mask = key_mask << 8;
    lo <<= 8;
    span <<= 8;
    for (unsigned base = 0; base < n; base += 32) {
      const uint32_t* w = words + base;
      const unsigned count = min(n - base, 32u);
      uint32_t inside = 0;
      if constexpr (PAD) {
        for (unsigned j = 0; j < count; j += 8) {
          uint32_t eight = 0;
#pragma unroll
          for (unsigned q = 0; q < 8; ++q)
            if ((w[j + q] & mask) - lo <= span) eight |= 1u << q;
          inside |= eight << j;
        }
        inside &= 0xFFFFFFFFu >> (32u - count);
      }
      else {
#pragma unroll 4
        for (unsigned j = 0; j < count; ++j)
          inside |= ((w[j] & mask) - lo <= span ? 1u : 0u) << j;
      }
      if (self - base < 32u) inside &= ~(1u << (self - base));
      for (; inside; inside &= inside - 1)
        visit(w[__ffs(inside) - 1]);
    }
  }

  // ------------------------------------------------------------------------------------
  // Candidate search of a non-isolated SP (EstimateInputSize.cu:72-204).  Every SP of
  // the bank is a potential neighbour: the reference reads the current SP's own
  // no-neighbour bit instead of the other's (line 113), which is always 0 here.
  // Returns up to two candidate pixel codes: bit 8 set = present, bits 0..2 = pixel.
  // ------------------------------------------------------------------------------------
  // Neighbours of either sensor of a version 4 bank count (the reference compares bits 22:8 only).
  template<bool PAD>
  __device__ __forceinline__ uint32_t sp_candidates(uint32_t sp_word, const uint32_t* bank_words, unsigned n_sp, unsigned self)
  {
    const uint32_t sp_addr = (sp_word & 0x007FFF00u) >> 8;
    const uint32_t sp = sp_word & 0xFFu;
    uint32_t pixels = (sp & 0x0Fu) | ((sp & 0xF0u) << 2);
    const uint32_t row = sp_addr & 0x3Fu;
    // Addresses from one row below in the same column to one row above in the next (the SP itself
    // adds nothing); a row beyond the column's ends is another column's.
    scan_keys<PAD>(bank_words, n_sp, self, sp_addr - 1, 66, 0x7FFFu, [&](uint32_t ow) {
      const uint32_t ahead = ((ow & 0x007FFF00u) >> 8) - sp_addr;
      const bool above = row < 63 && (ahead == 1 || ahead == 65), below = row > 0 && (ahead == ~0u || ahead == 63);
      const bool next = ahead > 62 && ahead <= 65;
      uint32_t add = 0;
      if (above) add = next ? (ow & 0x01u) << 16 : ((ow & 0x01u) << 4) | ((ow & 0x10u) << 6);
      if (below) add = next ? (ow & 0x08u) << 8 : (ow & 0x80u) >> 2;
      if (ahead == 64) add = (ow & 0x0Fu) << 12;
      pixels |= add;
    });
    const uint32_t inside = pixels & 0x3CFu;
    const uint32_t mask = (inside << 1) | (inside << 5) | (inside << 6) | (inside << 7);
    const uint32_t working = mask & (~pixels);
    const uint32_t cand_tmp = (working >> 1) & (working >> 5) & (working >> 6) & (working >> 7);
    const uint32_t cands = cand_tmp & pixels;
    const uint32_t consolidated = (cands & 0x0Fu) | ((cands >> 2) & 0xF0u);
    const uint32_t first = consolidated & 0x33u;
    const uint32_t second = consolidated & 0xCCu;
    uint32_t r = 0;
    if (first) r |= 0x100u | (__clz(first) - 24);
    if (second) r |= (0x100u | (__clz(second) - 24)) << 16;
    return r;
  }

  __device__ __forceinline__ bool isolated_two_clusters(uint32_t sp)
  {
    const bool pattern_0 = (sp & 0x88u) && !(sp & 0x44u) && (sp & 0x33u);
    const bool pattern_1 = (sp & 0xCCu) && !(sp & 0x22u) && (sp & 0x11u);
    return pattern_0 || pattern_1;
  }

  // ------------------------------------------------------------------------------------
  // Mask clustering of one candidate (MaskedVeloClustering.cu:21-84, 290-496)
  // ------------------------------------------------------------------------------------
  __device__ __forceinline__ uint64_t make_8con_mask(uint64_t c)
  {
    return c | ((c & 0x7FFF7FFF7FFF7FFFull) << 1) | ((c & 0xFFFEFFFEFFFEFFFEull) << 15) | (c << 16) |
           ((c & 0xFFFCFFFCFFFCFFFCull) << 17) | ((c & 0xFFFEFFFEFFFEFFFEull) >> 1) |
           ((c & 0x7FFF7FFF7FFF7FFFull) >> 15) | (c >> 16) | ((c & 0x3FFF3FFF3FFF3FFFull) >> 17);
  }

  __device__ __forceinline__ uint64_t mask_east(uint64_t c)
  {
    const uint64_t m = c >> 48;
    return m | ((m & 0x7FFF7FFF7FFF7FFFull) << 1) | (m >> 1);
  }

  __device__ __forceinline__ uint64_t mask_west(uint64_t c)
  {
    const uint64_t m = c << 48;
    return m | (m << 1) | ((m & 0xFFFEFFFEFFFEFFFEull) >> 1);
  }

  struct PixelCluster {
    uint64_t pixels;
    uint32_t x, y, n;
  };

  __device__ __forceinline__ PixelCluster
  make_cluster(uint64_t map, uint64_t start, uint32_t col_lower, uint32_t row_lower)
  {
    uint64_t cur = 0, next = start;
    while (cur != next) {
      cur = next;
      next = map & make_8con_mask(cur);
    }
    // Sums over the pixels by bit planes of their positions (bit = 16 column + row).  Row 15
    // counts 15 here and nothing in the reference, which drops clusters that touch it.
    PixelCluster c;
    c.pixels = cur;
    const uint32_t lo = static_cast<uint32_t>(cur), hi = static_cast<uint32_t>(cur >> 32);
    const unsigned n_hi = __popc(hi);
    c.n = __popc(lo) + n_hi;
    c.x = col_lower * c.n + __popc(lo & 0xFFFF0000u) + __popc(hi & 0xFFFF0000u) + 2 * n_hi;
    auto plane = [&](uint32_t m) { return static_cast<unsigned>(__popc(lo & m) + __popc(hi & m)); };
    c.y = row_lower * c.n + plane(0xAAAAAAAAu) + 2 * plane(0xCCCCCCCCu) + 4 * plane(0xF0F0F0F0u) + 8 * plane(0xFF00FF00u);
    return c;
  }

  struct ClusterOut {
    uint32_t id;
    float x, y, z;
    int16_t phi;
  };

  __device__ __forceinline__ void
  local_to_global(const Geometry* g, const float* ltg, float local_x, float local_y, ClusterOut& o)
  {
    o.x = __ldg(ltg + 0) * local_x + __ldg(ltg + 1) * local_y + __ldg(ltg + 9);
    o.y = __ldg(ltg + 3) * local_x + __ldg(ltg + 4) * local_y + __ldg(ltg + 10);
    o.z = __ldg(ltg + 6) * local_x + __ldg(ltg + 7) * local_y + __ldg(ltg + 11);
  }

  // The cluster that a candidate grows into (MaskedVeloClustering.cu:290-459): its pixel count and
  // the sums of their columns and rows; n = 0: none (a cluster another candidate makes, one that
  // leaves the window, or, with bad set, no pixel at all).
  struct ClusterSums {
    uint32_t x, y, n;
    bool bad;
  };
  template<bool PAD>
  __device__ __forceinline__ ClusterSums grow_cluster(
    uint32_t sp_word, uint32_t start_loc, uint32_t sensor_number, const uint32_t* bank_words, unsigned n_sp, int version)
  {
    ClusterSums none {0, 0, 0, false};
    const uint32_t sp_addr = (sp_word & 0x007FFF00u) >> 8;
    const int32_t sp_row = static_cast<int32_t>(sp_addr & 0x3Fu);
    const int32_t sp_col = static_cast<int32_t>(sp_addr >> 6);

    uint32_t pa[5] = {0, 0, 0, 0, 0};
    const int32_t r_lo = sp_row - 2, r_hi = sp_row + 1;
    const int32_t c_lo = sp_col - 3, c_hi = sp_col + 1;
    const int32_t row_lower = r_lo * 4;
    const int32_t col_lower = c_lo * 2;
    // the window's SPs lie between its lowest and its highest address (version 4: with the
    // sensor bit above the address)
    const uint32_t key_mask = version > 3 ? 0xFFFFu : 0x7FFFu;
    const uint32_t sensor_key = version > 3 ? (sensor_number & 0x1u) << 15 : 0u;
    const uint32_t lowest = sensor_key + static_cast<uint32_t>(c_lo * 64 + r_lo);
    scan_keys<PAD>(bank_words, n_sp, 0xFFFFFFFFu, lowest, 4 * 64 + 3, key_mask, [&](uint32_t ow) {
      if ((((ow >> 8) & key_mask) ^ sensor_key) & 0x8000u) return;
      if (ow & 0x80000000u) return;
      const uint32_t oaddr = (ow & 0x007FFF00u) >> 8;
      const int32_t orow = static_cast<int32_t>(oaddr & 0x3Fu);
      const int32_t ocol = static_cast<int32_t>(oaddr >> 6);
      if (orow >= r_lo && orow <= r_hi && ocol >= c_lo && ocol <= c_hi) {
        const uint32_t osp = ow & 0xFFu;
        const int rel_row = orow - r_lo;
        const int rel_col = ocol - c_lo;
        const uint32_t bits = ((osp & 0x0Fu) << (4 * rel_row)) | ((osp & 0xF0u) << (12 + 4 * rel_row));
#pragma unroll
        for (int c = 0; c < 5; ++c)
          if (c == rel_col) pa[c] |= bits;
      }
    });

    const uint32_t rel_row0 = start_loc & 0x3u;
    const uint32_t rel_col0 = start_loc < 4 ? 1u : 0u;
    const uint32_t col = static_cast<uint32_t>(sp_col) * 2 + rel_col0;
    const uint64_t start = (static_cast<uint64_t>(0x01u << (11 - rel_row0)) << (16 * (col & 0x01u))) << 32;
    const uint64_t map = (static_cast<uint64_t>(pa[3]) << 32) | pa[2];
    const PixelCluster cl = make_cluster(map, start, static_cast<uint32_t>(col_lower + 4), static_cast<uint32_t>(row_lower));
    const uint64_t precedence = (mask_east(cl.pixels) & pa[4]) | (cl.pixels & (start ^ (0ull - start)));
    bool keep = precedence == 0 && !(cl.pixels & 0x8000800080008000ull) && !(cl.pixels & 0x0001000100010001ull);
    if (!keep) return none;
    uint32_t x = cl.x, y = cl.y, n = cl.n;
    if (cl.pixels & 0xFFFFull) {
      const uint64_t west_map = (static_cast<uint64_t>(pa[1]) << 32) | pa[0];
      const uint64_t west_start = mask_west(cl.pixels) & west_map;
      const PixelCluster ext =
        make_cluster(west_map, west_start, static_cast<uint32_t>(col_lower), static_cast<uint32_t>(row_lower));
      x += ext.x;
      y += ext.y;
      n += ext.n;
      keep = !(ext.pixels & 0x8000800080008000ull) && !(ext.pixels & 0xFFFFull) &&
             !(cl.pixels & 0x0001000100010001ull);
    }
    if (!keep) return none;
    // A candidate whose bank index names another bank (the reference's lookup of the bank by
    // sensor, when a slice holds more than one bank per sensor) can leave the start pixel
    // outside the map: no pixel, and the reference divides by zero.
    none.bad = n == 0;
    return n == 0 ? none : ClusterSums {x, y, n, false};
  }

  // The hit at the centroid of a candidate's cluster (MaskedVeloClustering.cu:461-496).
  __device__ __forceinline__ void
  candidate_cluster(const Geometry* g, const Constants& k, uint32_t sensor_number, uint32_t x, uint32_t y, uint32_t n, ClusterOut& o)
  {
    const float* ltg = g->ltg + 12 * sensor_number;
    // The integer centroids x / n and y / n are the truncated correctly rounded quotients: a
    // quotient below 1024 (columns < 768, rows < 256) with n < 32768 pixels is at least 1 / n
    // below the next integer, more than half an ulp, so rounding never reaches it.  The
    // fractions are the reference's fl(x / n) - cx (MaskedVeloClustering.cu:461-466).
    const float qx = __fdiv_rn(__uint2float_rn(x), __uint2float_rn(n));
    const float qy = __fdiv_rn(__uint2float_rn(y), __uint2float_rn(n));
    const uint32_t cx = __float2uint_rz(qx);
    const uint32_t cy = __float2uint_rz(qy);
    const float fx = qx - __uint2float_rn(cx);
    const float fy = qy - __uint2float_rn(cy);
    const uint32_t chip = cx >> 8;
    o.id = lhcb_id(channel_id(sensor_number, chip, cx & 0xFFu, cy));
    const float local_x = column_local_x(g, cx) + fx * column_x_pitch(g, cx);
    const float local_y = (__uint2float_rn(cy) + 0.5f + fy) * 0.055f;
    local_to_global(g, ltg, local_x, local_y, o);
    o.phi = hit_phi_16(k, o.x, o.y);
  }

  // Isolated SP through the lookup tables (MaskedVeloClustering.cu:131-288); which = 0/1.
  __device__ __forceinline__ void isolated_cluster(
    const Geometry* g,
    const Constants& k,
    uint32_t sp_word,
    unsigned source_id,
    int version,
    unsigned which,
    ClusterOut& o)
  {
    const bool v23 = version == 2 || version == 3;
    const bool bit23 = (sp_word & 0x800000u) != 0;
    const uint32_t pair = source_id & 0x1FFu;
    const uint32_t sensor_index = v23 ? source_id : (bit23 ? ((pair << 1) | 1u) : (pair << 1));
    const float* ltg = g->ltg + 12 * (v23 ? pair : (bit23 ? ((pair << 1) | 1u) : (pair << 1)));
    const uint32_t sp_addr = (sp_word & 0x007FFF00u) >> 8;
    const int32_t sp_row = static_cast<int32_t>(sp_addr & 0x3Fu);
    const int32_t sp_col = static_cast<int32_t>(sp_addr >> 6);
    const uint32_t sp = sp_word & 0xFFu;
    const uint32_t idx = __ldg(g->sp_patterns + sp);
    const uint32_t chip = static_cast<uint32_t>(sp_col) >> 7;
    const uint32_t row = which ? (idx >> 4) & 3u : idx & 3u;
    const uint32_t col = which ? (idx >> 6) & 1u : (idx >> 2) & 1u;
    const uint32_t cx = static_cast<uint32_t>(sp_col) * 2 + col;
    const uint32_t cy = static_cast<uint32_t>(sp_row) * 4 + row;
    o.id = lhcb_id(channel_id(sensor_index, chip, cx & 0xFFu, cy));
    const float fx = __ldg(g->sp_fx + sp * 2 + which);
    const float fy = __ldg(g->sp_fy + sp * 2 + which);
    const float local_x = column_local_x(g, cx) + fx * column_x_pitch(g, cx);
    const float local_y = (__uint2float_rn(cy) + 0.5f + fy) * 0.055f;
    local_to_global(g, ltg, local_x, local_y, o);
    o.phi = hit_phi_16(k, o.x, o.y);
  }

  constexpr unsigned estimate_queue = 1024; // SPs per chunk of the estimate (and queue entries)
  static_assert(estimate_queue % decode_threads == 0, "every lane takes the same number of SPs per chunk");

  // Items of the list an event leaves to the clustering kernel.  Isolated SP: its word's pattern,
  // address and (version 4) sensor bit, with the bank's sensor (pair) and which of its two
  // clusters: versions 2 and 3 which << 23 | sensor << 24, version 4 pair << 24 | which << 31.
  // Candidate's cluster: two words, the column sum | pixel count << 24 and the row sum | sensor << 24.
  // Bit 9 of a version 2 or 3 source ID, which the channel IDs of isolated SPs take over, has no room
  // here: the list has a bit per sensor for it (note_bit_9).
  __device__ __forceinline__ uint32_t isolated_item(uint32_t word, unsigned source_id, bool v23, unsigned which)
  {
    return v23 ? (word & 0x7FFFFFu) | (which << 23) | (source_id << 24) :
                 (word & 0xFFFFFFu) | ((source_id & 0x7Fu) << 24) | (which << 31);
  }

  // Notes in the list which sensors' banks have bit 9 of the source ID set; a sensor with banks of
  // both kinds takes the event its list.  masks: 16 words of shared memory.  Ends with a __syncthreads().
  __device__ __noinline__ void note_bit_9(const BankTable& bt, ItemList& list, unsigned& list_at, uint32_t* masks)
  {
    uint32_t *with = masks, *without = masks + 8;
    if (threadIdx.x < 16) masks[threadIdx.x] = 0;
    __syncthreads();
    for (unsigned b = threadIdx.x; b < bt.n_banks; b += blockDim.x) {
      const unsigned sensor = bt.source_id[b] & 0x1FFu;
      if (bt.flat[b] == bt.flat[b + 1] || sensor >= n_sensors) continue;
      atomicOr(((bt.source_id[b] & 0x200u) ? with : without) + sensor / 32, 1u << (sensor & 31u));
    }
    __syncthreads();
    if (threadIdx.x < 8) {
      list.bit_9[threadIdx.x] = with[threadIdx.x];
      if (with[threadIdx.x] & without[threadIdx.x]) list_at = no_item_list;
      if (threadIdx.x == 0) list.words |= 1u;
    }
    __syncthreads();
  }

  // ------------------------------------------------------------------------------------
  // estimate_kernel: dev_number_of_candidates, dev_velo_bank_index (as a max-reduced
  // key), dev_estimated_input_size and dev_module_candidate_num, and the clustering kernel's items.
  // ------------------------------------------------------------------------------------
  __device__ __forceinline__ void estimate_event(const EstimateParams& p, unsigned e)
  {
    __shared__ BankTable bt;
    __shared__ unsigned est_mp[n_module_pairs + 6]; // zeroed by the first warp
    __shared__ unsigned cand_count, isolated_count, grown_count;
    __shared__ unsigned warp_sums[33];
    __shared__ uint16_t queue[estimate_queue];
    __shared__ uint16_t candidates[2 * estimate_queue]; // SP in the chunk, pixel << 10
    __shared__ unsigned queue_count[2], chunk_candidates[2];
    __shared__ unsigned list_at;
    // the event's SPs in bank order, when they fit: the words, with the bank as its distance
    // from the hint (127: too far) in bits 24 to 30, which SPs do not use
    __shared__ uint32_t held[estimate_words + 8]; // (8: scans read on)

    const unsigned ev = e + p.in.event_start;
    const int version = p.in.bank_version;
    const bool v23 = version == 2 || version == 3;
    if (threadIdx.x < 32) est_mp[threadIdx.x] = 0;
    if (threadIdx.x == 0) cand_count = isolated_count = grown_count = 0;
    if (threadIdx.x < 2) queue_count[threadIdx.x] = chunk_candidates[threadIdx.x] = 0;

    const EventWords ew = event_words(p.in, ev);
    const uint32_t* words = ew.w;
    parse_banks(p.in, ev, ew, bt, warp_sums, p.status);
    const unsigned total_sp = bt.total_sp;
    const bool in_smem = total_sp <= estimate_words;
    if (in_smem) {
      for (unsigned f0 = 0; f0 < total_sp; f0 += blockDim.x) {
        const unsigned f = f0 + threadIdx.x;
        const unsigned b = bank_of_warp(bt, f);
        if (f < total_sp) {
          const uint32_t distance = min(b - bt.hint[f / 32], 127u);
          held[f] = (words[bt.words_off[b] + f - bt.flat[b]] & 0x80FFFFFFu) | (distance << 24);
        }
      }
    }
    // Room for the event's items, two words per SP: an event that finds none, or needs more,
    // hands over nothing.
    const unsigned room = 2 * total_sp;
    if (threadIdx.x == 0) {
      list_at = no_item_list;
      if (p.list_scratch != nullptr) {
        const unsigned at = atomicAdd(p.list_alloc, room);
        if (at <= p.list_capacity && room <= p.list_capacity - at) list_at = at;
        else atomicSub(p.list_alloc, room); // a smaller event may still fit
        p.lists[e].words = room;
      }
    }
    bool bit_9 = false;
    for (unsigned b = threadIdx.x; v23 && b < bt.n_banks; b += blockDim.x)
      bit_9 |= (bt.source_id[b] & 0x200u) != 0;
    if (__syncthreads_or(bit_9) && p.lists != nullptr) note_bit_9(bt, p.lists[e], list_at, warp_sums);
    uint32_t* list = list_at != no_item_list ? p.list_scratch + list_at : nullptr;

    // Three passes per chunk of SPs, so that the warps do not diverge between the isolated SPs
    // (about two thirds: one pattern test each), the neighbour scans of the others and the flood
    // fills of the candidates: pass 1 counts and lists the isolated SPs and queues the others,
    // pass 2 scans the queued SPs and queues their candidates, pass 3 grows the candidates'
    // clusters.  Counts are sums and the clustering sorts, so the order does not matter.
    auto sp_word = [&](unsigned f, unsigned& b) {
      if (in_smem) {
        const uint32_t w = held[f];
        const unsigned distance = (w >> 24) & 127u;
        b = distance < 127u ? bt.hint[f / 32] + distance : bank_of(bt, f);
        return w;
      }
      b = bank_of(bt, f);
      return words[bt.words_off[b] + f - bt.flat[b]];
    };
    for (unsigned chunk_base = 0, parity = 0; chunk_base < total_sp; chunk_base += estimate_queue, parity ^= 1u) {
      // (whole warps: f of lane 0 is a multiple of 32)
      for (unsigned f = chunk_base + threadIdx.x; (f & ~31u) < min(chunk_base + estimate_queue, total_sp); f += blockDim.x) {
        const unsigned lane = threadIdx.x & 31u;
        unsigned b = 0, clusters = 0, mp = 0, source_id = 0;
        uint32_t word = 0;
        bool other = false;
        if (f < total_sp) {
          word = sp_word(f, b);
          source_id = bt.source_id[b];
          mp = bank_module_pair(source_id, version);
          other = !(word & 0x80000000u);
          if (mp >= n_module_pairs) set_error(p.status, err_input_capacity);
          else if (!other) clusters = isolated_two_clusters(word & 0xFFu) ? 2u : 1u;
        }
        const unsigned one = __ballot_sync(0xFFFFFFFFu, clusters > 0), two = __ballot_sync(0xFFFFFFFFu, clusters > 1);
        const unsigned rest = __ballot_sync(0xFFFFFFFFu, other);
        // lanes 0 to 2 add to the three counters at once: the items, the queue, and the estimate of the
        // module pair when all isolated SPs of the warp lie in one
        const unsigned mp0 = __shfl_sync(0xFFFFFFFFu, mp, __ffs(one) - 1);
        const bool same = __all_sync(0xFFFFFFFFu, clusters == 0 || mp == mp0);
        const unsigned n_items = __popc(one) + __popc(two);
        unsigned* counter = lane == 0 ? &isolated_count : (lane == 1 ? &queue_count[parity] : est_mp + mp0);
        const unsigned n = lane == 1 ? __popc(rest) : n_items;
        unsigned at = 0;
        if (lane < (same && n_items ? 3u : 2u)) at = atomicAdd(counter, n);
        if (!same && clusters) atomicAdd(est_mp + mp, clusters);
        const unsigned first = __shfl_sync(0xFFFFFFFFu, at, 0), first_queued = __shfl_sync(0xFFFFFFFFu, at, 1);
        const unsigned below = (1u << lane) - 1u;
        if (other) queue[first_queued + __popc(rest & below)] = static_cast<uint16_t>(f - chunk_base);
        if (clusters && list != nullptr) {
          const unsigned k = first + __popc(one & below), k2 = first + __popc(one) + __popc(two & below);
          if (k < room) list[k] = isolated_item(word, source_id, v23, 0);
          if (clusters > 1 && k2 < room) list[k2] = isolated_item(word, source_id, v23, 1);
        }
      }
      __syncthreads();
      const unsigned n_queued = min(queue_count[parity], estimate_queue);
      if (threadIdx.x == 0) queue_count[parity ^ 1u] = 0;
      for (unsigned q = threadIdx.x; q < n_queued; q += blockDim.x) {
        const unsigned f = chunk_base + queue[q];
        unsigned b;
        const uint32_t word = sp_word(f, b);
        const unsigned at = bt.flat[b], source_id = bt.source_id[b];
        const unsigned n_sp = bt.flat[b + 1] - at;
        const uint32_t c = in_smem ? sp_candidates<true>(word, held + at, n_sp, f - at) :
                                     sp_candidates<false>(word, words + bt.words_off[b], n_sp, f - at);
        const unsigned add = ((c >> 8) & 1u) + ((c >> 24) & 1u);
        const unsigned mp = bank_module_pair(source_id, version);
        unsigned second;
        const unsigned first = append_items(&chunk_candidates[parity], add, second);
        if (add > 0)
          candidates[first] = static_cast<uint16_t>(queue[q] | (((c & 0x100u) ? c & 0x7u : (c >> 16) & 0x7u) << 10));
        if (add > 1) candidates[second] = static_cast<uint16_t>(queue[q] | (((c >> 16) & 0x7u) << 10));
        if (mp < n_module_pairs) add_to_counter(est_mp, mp, add);
        else set_error(p.status, err_input_capacity);
      }
      __syncthreads();
      const unsigned n_candidates = chunk_candidates[parity];
      if (threadIdx.x == 0) {
        chunk_candidates[parity ^ 1u] = 0;
        cand_count += n_candidates;
      }
      for (unsigned q = threadIdx.x; q < (list != nullptr ? n_candidates : 0u); q += blockDim.x) {
        const unsigned f = chunk_base + (candidates[q] & 0x3FFu);
        unsigned b;
        const uint32_t word = sp_word(f, b);
        const unsigned source_id = bt.source_id[b];
        if (bank_module_pair(source_id, version) >= n_module_pairs) continue; // flagged above
        // MaskedVeloClustering.cu:567-572: the candidate's bank is looked up by sensor
        const uint32_t sensor = v23 ? (source_id & 0x1FFu) : (((source_id & 0x1FFu) << 1) | ((word >> 23) & 0x1u));
        const unsigned b2 = static_cast<unsigned>(p.bank_index_key[sensor] & 0xFFFFFFFFull);
        ClusterSums c;
        if (b2 == b && in_smem) {
          const unsigned at = bt.flat[b];
          c = grow_cluster<true>(word, candidates[q] >> 10, sensor, held + at, bt.flat[b + 1] - at, version);
        }
        else {
          const unsigned index = f - bt.flat[b];
          Bank bank;
          bank.n_sp = 0;
          if (b2 < bt.n_banks) bank = event_bank(p.in, ev, ew, b2);
          if (index >= bank.n_sp) {
            set_error(p.status, err_input_capacity);
            continue;
          }
          const uint32_t* bank_words = words + bank.first;
          c = grow_cluster<false>(bank_words[index], candidates[q] >> 10, sensor, bank_words, bank.n_sp, version);
        }
        if (c.bad) set_error(p.status, err_bad_super_pixel);
        if (c.n > 0) {
          unsigned unused;
          const unsigned at = 2 * append_items(&grown_count, 1, unused);
          if (at + 2 <= room)
            *reinterpret_cast<uint2*>(list + (room - 2 - at)) = make_uint2(c.x | (c.n << 24), c.y | (sensor << 24));
        }
      }
      // the next chunk's first barrier comes before its candidates
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      const unsigned mine = threadIdx.x < n_module_pairs ? est_mp[threadIdx.x] : 0u;
      if (threadIdx.x < n_module_pairs) p.estimated_input_size[e * n_module_pairs + threadIdx.x] = mine;
      const unsigned sum = __reduce_add_sync(0xFFFFFFFFu, mine);
      if (threadIdx.x == 0) {
        p.event_estimate[e] = sum;
        p.number_of_candidates[e] = 2 * bt.count_total;
        p.module_candidate_num[e] = cand_count;
        if (p.lists != nullptr) {
          ItemList& l = p.lists[e];
          l.first = isolated_count + 2 * grown_count <= room ? list_at : no_item_list;
          l.isolated = isolated_count;
          l.grown = grown_count;
        }
      }
    }
  }

  // Issue-bound (80 % of the issue slots).  16000 events of 2540 SPs: 0.97 ms.  With scans of one key
  // at a time through a pointer to either memory, and the warp's places in list, queue and estimate
  // claimed one after the other, 1.06 (reading and parsing 0.14, pass 1 0.24, pass 2 0.37, pass 3
  // 0.31); without pass 3, when the clustering kernel took twice as long as now, 0.79.
  template<unsigned SM_THREADS>
  __global__ void __launch_bounds__(decode_threads, SM_THREADS / decode_threads) estimate_kernel(EstimateParams p)
  {
    for_each_event(p.queue, p.in.n_events, [&](unsigned e, unsigned) { estimate_event(p, e); });
  }
  template __global__ void estimate_kernel<2048>(EstimateParams p);
  template __global__ void estimate_kernel<few_decode_threads>(EstimateParams p);

  // ------------------------------------------------------------------------------------
  // cluster_sort_kernel
  // ------------------------------------------------------------------------------------
  __device__ __forceinline__ unsigned sort_bucket(int16_t phi) { return static_cast<unsigned>(phi + 32768) >> 9; }

  // u16 counters packed two per 32-bit word; returns the previous count of counter b.
  __device__ __forceinline__ uint16_t count_in_bucket(uint16_t* counters, unsigned b)
  {
    const unsigned shift = 16 * (b & 1u);
    const uint32_t old = atomicAdd(reinterpret_cast<uint32_t*>(counters) + (b >> 1), 1u << shift);
    return static_cast<uint16_t>(old >> shift);
  }

  // The clusters of an event as they are made (22 bytes each), in shared memory or in the event's
  // slice of the global staging buffer.
  struct StagedClusters {
    uint4* hit;        // x, y, z, id
    uint32_t* key;     // phi, module pair << 16
    uint16_t* members; // cluster indices in bucket order
    __device__ __forceinline__ StagedClusters(char* base, unsigned capacity)
    {
      hit = reinterpret_cast<uint4*>(base);
      key = reinterpret_cast<uint32_t*>(hit + capacity);
      members = reinterpret_cast<uint16_t*>(key + capacity);
    }
  };

  struct ClusterSortShared {
    unsigned region[n_module_pairs + 1]; // estimated start of each module pair, event-relative
    unsigned n_staged;
    unsigned warp_sums[33];
    uint32_t bit_9[8]; // of the event's item list
  };

  // Makes clusters and appends them to the event's staging.
  struct ClusterMaker {
    const ClusterSortParams& p;
    const StagedClusters& st;
    ClusterSortShared& s;
    uint16_t* counters;
    unsigned est_total;

    __device__ __forceinline__ void stage(const ClusterOut& o, unsigned mp) const
    {
      unsigned unused;
      const unsigned k = append_items(&s.n_staged, 1, unused);
      if (k < est_total) {
        st.hit[k] = make_uint4(__float_as_uint(o.x), __float_as_uint(o.y), __float_as_uint(o.z), o.id);
        st.key[k] = static_cast<uint16_t>(o.phi) | (mp << 16);
        count_in_bucket(counters, mp * sort_buckets + sort_bucket(o.phi));
      }
      else {
        set_error(p.status, err_cluster_capacity);
      }
    }
    __device__ __forceinline__ void isolated(uint32_t word, unsigned source_id, unsigned which) const
    {
      ClusterOut o;
      isolated_cluster(p.geo, p.k, word, source_id, p.in.bank_version, which, o);
      stage(o, bank_module_pair(source_id, p.in.bank_version));
    }
    __device__ __forceinline__ void grown(uint32_t x, uint32_t y, uint32_t n, uint32_t sensor) const
    {
      ClusterOut o;
      candidate_cluster(p.geo, p.k, sensor, x, y, n, o);
      stage(o, sensor / 8);
    }
  };

  // The clusters of an event without an item list (its list found no room, two clusters from
  // too many of its SPs, or a sensor with banks with and without bit 9 in the source ID): a thread per SP.  A warp takes
  // fallback_banks banks at a time, whose places its first lanes hold, and walks their SPs as one
  // run.  (4000 events of 2500 SPs without lists, the whole chain: 2.06 ms; with a thread per bank,
  // its SPs one after the other, 2.92; with lists 1.19.)
  constexpr unsigned fallback_banks = 8;

  __device__ __noinline__ void
  cluster_banks(const ClusterSortParams& p, char* stage_base, ClusterSortShared& s, uint16_t* counters, unsigned est_total, unsigned e)
  {
    const StagedClusters st {stage_base, est_total};
    const ClusterMaker m {p, st, s, counters, est_total};
    const unsigned ev = e + p.in.event_start;
    const EventWords ew = event_words(p.in, ev);
    const int version = p.in.bank_version;
    const bool v23 = version == 2 || version == 3;
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
    for (unsigned b0 = warp * fallback_banks; b0 < ew.n_banks; b0 += n_warps * fallback_banks) {
      unsigned n_sp = 0, at = 0, source_id = 0; // of bank b0 + lane
      if (lane < fallback_banks && b0 + lane < ew.n_banks) {
        const Bank bank = event_bank(p.in, ev, ew, b0 + lane);
        // a source id beyond the 26 module pairs: malformed input, flagged by estimate_kernel
        if (bank.velo && bank_module_pair(bank.source_id, version) < n_module_pairs) {
          n_sp = bank.n_sp;
          at = bank.first;
          source_id = bank.source_id;
        }
      }
      unsigned end = n_sp; // of the bank's SPs in the run
#pragma unroll
      for (unsigned o = 1; o < fallback_banks; o *= 2) {
        const unsigned t = __shfl_up_sync(0xFFFFFFFFu, end, o);
        if (lane >= o) end += t;
      }
      const unsigned run = __shfl_sync(0xFFFFFFFFu, end, fallback_banks - 1);
      for (unsigned r0 = 0; r0 < run; r0 += 32) {
        const unsigned r = r0 + lane;
        unsigned k = 0; // the lane that holds the SP's bank: the banks that end before it
#pragma unroll
        for (unsigned step = fallback_banks / 2; step >= 1; step /= 2)
          if (__shfl_sync(0xFFFFFFFFu, end, k + step - 1) <= r) k += step;
        const unsigned bank_n = __shfl_sync(0xFFFFFFFFu, n_sp, k), bank_source = __shfl_sync(0xFFFFFFFFu, source_id, k);
        const unsigned i = r - (__shfl_sync(0xFFFFFFFFu, end, k) - bank_n);
        const uint32_t* w = ew.w + __shfl_sync(0xFFFFFFFFu, at, k);
        if (r >= run) continue;
        const uint32_t word = w[i];
        if (word & 0x80000000u) {
          const unsigned clusters = isolated_two_clusters(word & 0xFFu) ? 2u : 1u;
          for (unsigned which = 0; which < clusters; ++which)
            m.isolated(word, bank_source, which);
          continue;
        }
        const uint32_t c = sp_candidates<false>(word, w, bank_n, i);
        if (c == 0) continue;
        const uint32_t sensor =
          v23 ? (bank_source & 0x1FFu) : (((bank_source & 0x1FFu) << 1) | ((word >> 23) & 0x1u));
        // MaskedVeloClustering.cu:567-572: the candidate's bank is looked up by sensor
        const unsigned b2 = static_cast<unsigned>(p.bank_index_key[sensor] & 0xFFFFFFFFull);
        Bank named;
        named.n_sp = 0;
        if (b2 < ew.n_banks) named = event_bank(p.in, ev, ew, b2);
        if (i >= named.n_sp) {
          set_error(p.status, err_input_capacity);
          continue;
        }
        const uint32_t* w2 = ew.w + named.first;
        for (unsigned which = 0; which < 2; ++which) {
          const uint32_t code = which ? (c >> 16) : c;
          if (!(code & 0x100u)) continue;
          const ClusterSums sums = grow_cluster<false>(w2[i], code & 0x7u, sensor, w2, named.n_sp, version);
          if (sums.bad) set_error(p.status, err_bad_super_pixel);
          if (sums.n > 0) m.grown(sums.x, sums.y, sums.n, sensor);
        }
      }
    }
  }

  template<unsigned THREADS>
  __device__ __forceinline__ void cluster_sort_event(const ClusterSortParams& p, unsigned e)
  {
    extern __shared__ __align__(128) unsigned char dsmem[];
    __shared__ ClusterSortShared s;

    const unsigned n = p.in.n_events;
    const unsigned base = p.event_base[e];
    const unsigned T = p.event_base[n];
    if (T > p.cluster_capacity) {
      // the slice needs more clusters than reserved: nothing is written
      if (threadIdx.x == 0) set_error(p.status, err_input_capacity);
      return;
    }
    if (threadIdx.x < 32) {
      const unsigned mp = threadIdx.x;
      const unsigned mine = mp < n_module_pairs ? p.estimated_input_size[e * n_module_pairs + mp] : 0u;
      unsigned incl = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (mp >= static_cast<unsigned>(o)) incl += t;
      }
      if (mp <= n_module_pairs) s.region[mp] = incl - mine;
      if (mp < n_module_pairs) p.offsets_estimated_input_size[e * n_module_pairs + mp] = base + incl - mine;
      if (mp == 0) s.n_staged = 0;
      if (e == n - 1 && mp == 0) p.offsets_estimated_input_size[n * n_module_pairs] = T;
    }
    uint16_t* bucket = reinterpret_cast<uint16_t*>(dsmem + cluster_sort_counter_offset(p.smem_cluster_capacity));
    for (unsigned i = threadIdx.x; i < sort_counters / 2; i += blockDim.x)
      reinterpret_cast<uint32_t*>(bucket)[i] = 0;
    __syncthreads();

    // Staging: shared memory when the event fits (always the smallest), else its slice of the
    // global staging buffer (24 bytes per estimated cluster), from a 16-byte boundary on.
    const unsigned est_total = s.region[n_module_pairs];
    const bool staged_in_smem = est_total <= p.smem_cluster_capacity;
    char* stage_base = staged_in_smem ? reinterpret_cast<char*>(dsmem) : p.staging + ((size_t(24) * base + 15) & ~size_t(15));
    const StagedClusters st {stage_base, est_total};

    const uint4 items = p.lists != nullptr ? *reinterpret_cast<const uint4*>(p.lists + e) : make_uint4(no_item_list, 0, 0, 0);
    const unsigned list_words = items.y & ~1u;
    if (items.x != no_item_list) {
      // the isolated SPs from the front, the candidates' clusters from the end
      const ClusterMaker make {p, st, s, bucket, est_total};
      const uint32_t* list = p.list_scratch + items.x;
      const bool v23 = p.in.bank_version == 2 || p.in.bank_version == 3, bit_9 = items.y & 1u;
      if (bit_9) {
        if (threadIdx.x < 8) s.bit_9[threadIdx.x] = p.lists[e].bit_9[threadIdx.x];
        __syncthreads();
      }
      for (unsigned q = threadIdx.x; q < items.z; q += blockDim.x) {
        const uint32_t item = __ldcs(list + q);
        unsigned source_id = item >> 24;
        if (bit_9) source_id |= ((s.bit_9[source_id / 32] >> (source_id & 31u)) & 1u) << 9;
        if (v23) make.isolated(item & 0x7FFFFFu, source_id, (item >> 23) & 1u);
        else make.isolated(item & 0xFFFFFFu, source_id & 0x7Fu, item >> 31);
      }
      const uint2* grown = reinterpret_cast<const uint2*>(list + list_words) - 1;
      for (unsigned q = threadIdx.x; q < items.w; q += blockDim.x) {
        const uint2 g = __ldcs(grown - q);
        make.grown(g.x & 0xFFFFFFu, g.y & 0xFFFFFFu, g.x >> 24, g.y >> 24);
      }
    }
    else {
      cluster_banks(p, stage_base, s, bucket, est_total, e);
    }
    __syncthreads();

    // Sort by (phi, id) inside each module pair (SortByPhi.cu:104-122).  The reference
    // ranks every pair of clusters; here clusters were counted into 128 phi buckets per
    // module pair while staged, so a scan of the counters places every bucket and a
    // cluster's rank is its bucket's start plus the number of smaller (phi, id) keys in the
    // same bucket - the same position as the reference's full count.
    const unsigned n_staged = min(s.n_staged, est_total);
    {
      // each thread owns `per` consecutive words of two counters: it sums them, and after the
      // scan turns them into starts in place (no other thread reads them in between)
      constexpr unsigned words = sort_counters / 2, per = (words + THREADS - 1) / THREADS;
      uint32_t* w = reinterpret_cast<uint32_t*>(bucket) + threadIdx.x * per;
      unsigned sum = 0;
#pragma unroll
      for (unsigned q = 0; q < per; ++q) {
        const uint32_t c = threadIdx.x * per + q < words ? w[q] : 0u;
        sum += (c & 0xFFFFu) + (c >> 16);
      }
      unsigned total;
      unsigned start = block_exclusive_scan(sum, s.warp_sums, &total);
#pragma unroll
      for (unsigned q = 0; q < per; ++q) {
        if (threadIdx.x * per + q < words) {
          const uint32_t c = w[q];
          w[q] = (start & 0xFFFFu) | ((start + (c & 0xFFFFu)) << 16);
          start += (c & 0xFFFFu) + (c >> 16);
        }
      }
    }
    __syncthreads();
    auto bucket_of_key = [&](uint32_t key) {
      return (key >> 16) * sort_buckets + sort_bucket(static_cast<int16_t>(key & 0xFFFFu));
    };
    // each cluster into its bucket; this moves a bucket's start to its end
    for (unsigned k = threadIdx.x; k < n_staged; k += blockDim.x)
      st.members[count_in_bucket(bucket, bucket_of_key(st.key[k]))] = static_cast<uint16_t>(k);
    __syncthreads();
    // In bucket order, which is output order up to the order inside a bucket: the threads of a
    // warp write neighbouring places of the container.
    auto bucket_begin = [&](unsigned b) { return b ? unsigned(bucket[b - 1]) : 0u; };
    ClusterView out {p.sorted_container, T};
    for (unsigned q = threadIdx.x; q < n_staged; q += blockDim.x) {
      const unsigned k = st.members[q];
      const uint32_t key = st.key[k];
      const uint4 hit = st.hit[k];
      const unsigned mp = key >> 16, b = bucket_of_key(key);
      const int16_t phi = static_cast<int16_t>(key & 0xFFFFu);
      const unsigned begin = bucket_begin(b), end = bucket[b];
      unsigned position = begin - bucket_begin(mp * sort_buckets);
      for (unsigned r = begin; r < end; ++r) {
        const unsigned j = st.members[r];
        const int16_t other = static_cast<int16_t>(st.key[j] & 0xFFFFu);
        position += phi > other || (phi == other && hit.w > st.hit[j].w);
      }
      if (position >= s.region[mp + 1] - s.region[mp]) {
        set_error(p.status, err_cluster_capacity);
        continue;
      }
      // written once here, read by the next kernel: streaming stores (evict first), which
      // leave L2 to the staging of the events in flight
      const unsigned dst = base + s.region[mp] + position;
      __stcs(&out.id(dst), hit.w);
      __stcs(&out.phi(dst), phi);
      __stcs(&out.x(dst), __uint_as_float(hit.x));
      __stcs(&out.y(dst), __uint_as_float(hit.y));
      __stcs(&out.z(dst), __uint_as_float(hit.z));
    }
    if (threadIdx.x < n_module_pairs) {
      const unsigned mp = threadIdx.x;
      const unsigned made = bucket[(mp + 1) * sort_buckets - 1] - bucket_begin(mp * sort_buckets);
      p.module_cluster_num[e * n_module_pairs + mp] = min(made, s.region[mp + 1] - s.region[mp]);
    }
    // the event's slices of the global staging and of the item list are dead
    __syncthreads();
    if (!staged_in_smem) discard_l2(stage_base, size_t(22) * est_total);
    if (items.x != no_item_list) discard_l2(p.list_scratch + items.x, size_t(4) * list_words);
  }

  // Issue- and latency-bound.  16000 events of 2540 SPs: 0.65 ms, of which making the clusters 0.2
  // and the sort 0.38; with the flood fills and the search for each SP's bank in this kernel, and
  // the clusters written out in the order they were staged, 1.31 ms.  Written out from a staging
  // without any order (a scattered store per value) the sort alone took 0.91 ms.
  // Capped for 2048 threads per SM (32 registers; 40 or 48 registers: 0.69, 0.71 ms).
  template<unsigned THREADS, unsigned SM_THREADS>
  __global__ void __launch_bounds__(THREADS, SM_THREADS / THREADS) cluster_sort_kernel(const __grid_constant__ ClusterSortParams p)
  {
    static_assert(THREADS == 128 || THREADS == 256, "block size");
    for_each_event(p.queue, p.in.n_events, [&](unsigned e, unsigned) { cluster_sort_event<THREADS>(p, e); });
  }
  template __global__ void cluster_sort_kernel<128, 2048>(const __grid_constant__ ClusterSortParams p);
  template __global__ void cluster_sort_kernel<256, 2048>(const __grid_constant__ ClusterSortParams p);
  template __global__ void cluster_sort_kernel<256, few_decode_threads>(const __grid_constant__ ClusterSortParams p);

  // Before the estimate kernel.  Block 0: the events of the slice by raw size, largest first (a
  // counting sort over 1024 size classes of 64 bytes; order within a class is arbitrary), when
  // order is given.  Block 1 + d: dev_velo_bank_index, as a max-reduced key, from event
  // d * stride: block 0 of the reference's velo_calculate_number_of_candidates (grid of
  // ceil(N / 256) blocks, one thread per event) handles events 0, stride, 2 stride, ... and the
  // last of them to write an entry wins.
  __global__ void __launch_bounds__(scan_threads)
  event_order_kernel(RawInput in, unsigned* order, unsigned stride, unsigned long long* bank_index_key)
  {
    if (blockIdx.x > 0) {
      const unsigned e = (blockIdx.x - 1) * stride;
      if (e >= in.n_events) return;
      const unsigned ev = e + in.event_start;
      const EventWords ew = event_words(in, ev);
      const unsigned long long key_hi = static_cast<unsigned long long>(e) << 32;
      for (unsigned b = threadIdx.x; b < ew.n_banks; b += blockDim.x) {
        const unsigned src = event_bank(in, ev, ew, b).source_id & 0x1FFu;
        if (in.bank_version > 3) {
          if ((src << 1) < n_sensors) atomicMax(bank_index_key + (src << 1), key_hi | b);
          if (((src << 1) | 1u) < n_sensors) atomicMax(bank_index_key + ((src << 1) | 1u), key_hi | b);
        }
        else if (src < n_sensors) {
          atomicMax(bank_index_key + src, key_hi | b);
        }
      }
      return;
    }
    if (order == nullptr) return;
    constexpr unsigned classes = 1024;
    __shared__ unsigned count[classes];
    __shared__ unsigned warp_sums[33];
    for (unsigned c = threadIdx.x; c < classes; c += blockDim.x)
      count[c] = 0;
    __syncthreads();
    auto size_class = [&](unsigned e) {
      const unsigned bytes = in.offsets[e + in.event_start + 1] - in.offsets[e + in.event_start];
      return classes - 1 - min(bytes / 64u, classes - 1); // descending size
    };
    if (in.mep_layout) {
      // no per-event blob sizes in a MEP: keep the events in order
      for (unsigned e = threadIdx.x; e < in.n_events; e += blockDim.x)
        order[e] = e;
      return;
    }
    for (unsigned e = threadIdx.x; e < in.n_events; e += blockDim.x)
      atomicAdd(&count[size_class(e)], 1u);
    __syncthreads();
    unsigned total;
    const unsigned mine = threadIdx.x < classes ? count[threadIdx.x] : 0u;
    const unsigned excl = block_exclusive_scan(mine, warp_sums, &total);
    __syncthreads();
    if (threadIdx.x < classes) count[threadIdx.x] = excl;
    __syncthreads();
    for (unsigned e = threadIdx.x; e < in.n_events; e += blockDim.x)
      order[atomicAdd(&count[size_class(e)], 1u)] = e;
  }

  // ------------------------------------------------------------------------------------
  // exclusive_scan_kernel: one CTA per job; out[0] = 0, out[i + 1] = sum(in[0..i])
  // (host_prefix_sum_t, HostPrefixSum.cpp:76-108, without the host round trip).
  // ------------------------------------------------------------------------------------
  __global__ void __launch_bounds__(scan_threads) exclusive_scan_kernel(ScanParams p)
  {
    __shared__ unsigned warp_sums[33];
    const ScanJob job = p.jobs[blockIdx.x];
    if (job.in == nullptr) return;
    unsigned carry = 0;
    constexpr unsigned per_thread = 4;
    const unsigned tile = blockDim.x * per_thread;
    for (unsigned t0 = 0; t0 < job.n; t0 += tile) {
      unsigned v[per_thread];
      unsigned s = 0;
#pragma unroll
      for (unsigned q = 0; q < per_thread; ++q) {
        const unsigned i = t0 + threadIdx.x * per_thread + q;
        v[q] = i < job.n ? job.in[i] : 0u;
        s += v[q];
      }
      unsigned total;
      unsigned excl = block_exclusive_scan(s, warp_sums, &total);
#pragma unroll
      for (unsigned q = 0; q < per_thread; ++q) {
        const unsigned i = t0 + threadIdx.x * per_thread + q;
        if (i < job.n) job.out[i] = carry + excl;
        excl += v[q];
      }
      carry += total;
    }
    if (threadIdx.x == 0) job.out[job.n] = carry;
  }

} // namespace velo

// search_by_triplet (seeding + forwarding) and the three-hit filter on sm_100a,
// one event per CTA.
//
// Reference: device/velo/search_by_triplet/src/SearchByTriplet.cu:110-609 (kernel,
// find_forward_candidate, track_seeding, track_forwarding) and
// ThreeHitTracksFilter.cu:48-169.
//
// Design.
//  * The event's sorted hits are staged once as 16-byte records (x, y, z, phi and the module
//    parity that forwarding needs), so that every hit a walk visits costs one vector load: in
//    shared memory, or for events above the shared-memory capacity (and in the tuned launch, every
//    event of a slice of more events than SMs) in a global scratch slice that stays in L2, through
//    the same code.
//  * Which hits are used is a bit per hit in shared memory (the reference's hit_used).
//  * Within a step every seed candidate (h1) and every track to follow is independent:
//    seeding only reads the used bits, forwarding only sets them, and each track to follow
//    owns its track.  Seeding finds the unused h1 by counting bits, a thread each picks its
//    h0 candidates out of the used bits around h1's phi, then a thread per (h0, h1) extrapolates
//    and walks the h2 window, and a shuffle reduction keeps the best (scatter, candidate
//    order) - the same choice as the reference's sequential loop.  Forwarding runs one thread
//    per track.
//  * Output slots (ring entries, track numbers, three-hit entries) are assigned by a
//    block-wide ordered scan in item order, which is the reference's sequential order, so
//    the track containers come out bit-identical to the reference CPU build.
//  * An entry of the ring of tracks to follow (2048 entries, as the reference) holds a seed's
//    three hits, or a track's last two hits, its number and its hit count, so that forwarding
//    reads nothing else of the track.  Tracks are written to dev_tracks as they grow.
//  * Leftmost binary searches over a module pair's phi go through a 128-bucket table plus a
//    short scan: same index, fewer loads.  A step reads the tables of three module pairs, and each
//    step builds the one it adds in the slot of the one it leaves.
#include <type_traits>

#include "velo_kernels.cuh"

namespace velo {

  // Ring entries.  Seed: its hits at bits 0, 16, 32.  Track: its last two hits at bits 0 and 16,
  // its number at bit 32 (one seed at most per hit: 16 bits hold it), its hit count at bit 48.
  // Both: skipped modules at bit 56, the seed flag at bit 63.
  constexpr uint64_t seed_flag = 1ull << 63;
  constexpr unsigned skipped_shift = 56;
  constexpr unsigned skipped_mask = 0x3Fu;
  constexpr unsigned hits_shift = 48;
  constexpr uint8_t flag_odd_module = 2;
  // Per CTA in shared memory: used bits of an event's first hits (larger events: global scratch),
  // phi of a module pair's hits (larger pairs: the staged records), ring entries per step
  constexpr unsigned used_capacity = 8192;
  constexpr unsigned phi_capacity = 256;
  constexpr unsigned near_entries = 192;
  constexpr unsigned seed_window_hits = 256; // hits of the middle module pair that are looked over at once
  constexpr unsigned seed_slots = 512;       // (h0, h1) doublets in flight

  struct ModulePair {
    unsigned hit_start;
    unsigned hit_num;
    float z[2];
    unsigned table; // slot of its bucket table: the module pair's index % 3
  };

  struct SearchShared {
    alignas(16) unsigned scan_sums[2][32]; // double-buffered warp totals of the block scans (0 past the last warp)
    unsigned track_hits;       // sum of hitsNum over the >= 4 hit tracks
    // counters only reported (thread 0 keeps them): atomics::local_number_of_hits, the unused
    // h1 met by the seeding (seed candidates), the candidates whose h0 and h2 windows were
    // searched (the gate let through)
    unsigned local_hits, candidates, searched;
    uint32_t used[used_capacity / 32 + 1];
    // bucket tables and phi values of the three module pairs a step reads, filled one per step
    uint16_t bucket[3][n_buckets + 1];
    int16_t phi[3][phi_capacity];
    // the event's module pairs, last first: a step's three are mps[25 - first] onwards
    ModulePair mps[n_module_pairs];
    // the seeding's h1, and their h0 candidates in pendulum order (4 or 8 places each)
    unsigned seed_before[9];         // the window's hits to search before each of its words, and all
    uint32_t seed_bits[8];           // those words
    unsigned n_h0;                   // unused hits of the previous module pair
    uint16_t seed_h1[seed_slots / 4];
    uint16_t seed_h0[seed_slots];
  };
  struct SearchSharedGated : SearchShared {
    uint32_t pass[seed_window_hits / 32]; // the window's unused hits that the gate lets through
  };

  // A staged hit, unpacked from its 16-byte record.
  struct Hit {
    float x, y, z;
    int16_t phi;
    unsigned flags;
  };

  // The event's staged hits: one 16-byte record per hit (x, y, z as fp32 bits, then phi in
  // bits 0-15 and the flags in bits 16-23 of the fourth word), so that a candidate costs
  // one vector load instead of one load per field.
  struct Hits {
    uint4* r;
    __device__ __forceinline__ Hit operator[](unsigned i) const
    {
      const uint4 v = r[i];
      return Hit {__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), static_cast<int16_t>(v.w & 0xFFFFu),
                  (v.w >> 16) & 0xFFu};
    }
    __device__ __forceinline__ int16_t phi(unsigned i) const { return reinterpret_cast<const int16_t*>(r + i)[6]; }
  };

  // The used bits of an event's hits, one word more than they fill.
  struct UsedBits {
    uint32_t* w;
    __device__ __forceinline__ bool operator[](unsigned i) const { return (w[i >> 5] >> (i & 31u)) & 1u; }
    __device__ __forceinline__ void set(unsigned i) const { atomicOr(w + (i >> 5), 1u << (i & 31u)); }
    // the unused hits among [i, i + 32) as a word
    __device__ __forceinline__ uint32_t unused(unsigned i) const
    {
      return ~__funnelshift_r(w[i >> 5], w[(i >> 5) + 1], i & 31u);
    }
  };

  // The ring of tracks to follow.  A step reads the entries that the step before appended and
  // appends its own, so only two generations are alive: with NEAR, the first entries of each
  // lie in shared memory, the others (and without NEAR all of them) in the ring proper.
  template<bool NEAR>
  struct Ring {
    uint64_t* ring;
    uint64_t* near_ring;  // [2][near_entries]
    unsigned begin;       // first entry of the generation being appended
    unsigned parity;      // its half of near_ring
    __device__ __forceinline__ uint64_t& at(unsigned i, unsigned first, unsigned half) const
    {
      if (NEAR && i - first < near_entries) return near_ring[half * near_entries + (i - first)];
      return ring[i % max_tracks_to_follow];
    }
    __device__ __forceinline__ uint64_t& append(unsigned i) const { return at(i, begin, parity); }
    __device__ __forceinline__ void next_generation(unsigned ttf)
    {
      begin = ttf;
      parity ^= 1u;
    }
  };

  // Bits of a word below bit n (n may be 32 or more).
  __device__ __forceinline__ uint32_t low_bits(uint32_t v, unsigned n) { return n < 32 ? v & ((1u << n) - 1u) : v; }

  // Position of the set bit of rank r (r < popc(v)).
  __device__ __forceinline__ unsigned select_bit(uint32_t v, unsigned r)
  {
    unsigned at = 0;
#pragma unroll
    for (unsigned step = 16; step >= 1; step /= 2) {
      const unsigned c = __popc(v & ((1u << step) - 1u));
      if (r >= c) {
        r -= c;
        v >>= step;
        at += step;
      }
    }
    return at;
  }

  // The pendulum around p0 in [0, n] (SearchByTriplet.cu:351-370): step 0 is p0, step 2d - 1 is
  // p0 + d, step 2d is p0 - d, for steps below n, each position wrapping once.  As offsets from p0
  // the visit order is 0, +1, -1, +2, ...: two words of unused hits, upwards and downwards from p0,
  // hold 32 offsets at a time, and the next candidate is the nearer of their lowest bits, the
  // upward one first.
  struct Pendulum {
    unsigned start, n, p0;
    uint32_t up, down; // bit k: p0 + base + k; p0 - base - k
    unsigned base;
    __device__ __forceinline__ Pendulum(unsigned hit_start, unsigned hit_num, unsigned center) :
      start(hit_start), n(hit_num), p0(center < hit_num ? center : 0u), up(0), down(0), base(0u - 32u)
    {}
    __device__ __forceinline__ void load(const UsedBits& used)
    {
      base += 32;
      // offsets up to n / 2 upwards and (n - 1) / 2 downwards are visited
      const unsigned s = p0 + base < n ? p0 + base : p0 + base - n;
      up = low_bits(used.unused(start + s), n - s);
      if (n - s < 32) up |= used.unused(start) << (n - s);
      up = base <= n / 2 ? low_bits(up, n / 2 + 1 - base) : 0u;
      const unsigned t = p0 >= base ? p0 - base : p0 + n - base;
      if (t >= 31) {
        down = __brev(used.unused(start + t - 31));
      }
      else {
        const uint32_t end = n >= 32 ? used.unused(start + n - 32) : used.unused(start) << (32 - n);
        down = (__brev(used.unused(start) << (31 - t))) | (__brev(end) << (t + 1));
      }
      down = base <= (n - 1) / 2 ? low_bits(down, (n - 1) / 2 + 1 - base) : 0u;
      if (base == 0) down &= ~1u; // offset 0 is the upward word's
    }
    // The next candidate's position; there is one (the caller knows the number of unused hits).
    __device__ __forceinline__ unsigned next(const UsedBits& used)
    {
      while ((up | down) == 0 && base + 32u <= n)
        load(used);
      const int u = up ? __ffs(up) - 1 : 32;
      const int d = down ? __ffs(down) - 1 : 32;
      int pos = static_cast<int>(p0);
      if (u <= d) {
        pos += static_cast<int>(base) + u;
        up &= up - 1;
      }
      else {
        pos -= static_cast<int>(base) + d;
        down &= down - 1;
      }
      return static_cast<unsigned>(pos < 0 ? pos + int(n) : (pos >= int(n) ? pos - int(n) : pos));
    }
  };

  // The first h2 of the circular window walk: start % n (0 for an empty module pair), without
  // a division for start in [0, n], leftmost()'s range.
  __device__ __forceinline__ unsigned first_candidate(int16_t start, unsigned n)
  {
    const unsigned x = static_cast<unsigned>(start);
    return x < n ? x : (x == n || n == 0 ? 0u : x % n);
  }

  // leftmost() over a module pair's hits, through the phi values of its table slot when they fit.
  __device__ __forceinline__ int leftmost_hit(const SearchShared& s, const Hits& h, const ModulePair& m, int16_t value)
  {
    unsigned i = s.bucket[m.table][bucket_of(value)];
    if (m.hit_num <= phi_capacity) {
      while (i < m.hit_num && s.phi[m.table][i] < value)
        ++i;
    }
    else {
      while (i < m.hit_num && h.phi(m.hit_start + i) < value)
        ++i;
    }
    return static_cast<int>(i);
  }

  // The event's counters that place items (the reference's dev_atomics_velo and track
  // count), kept in registers: every thread holds the same values and advances them by scan
  // totals.
  struct Counters {
    unsigned ttf;      // atomics::tracks_to_follow
    unsigned n_three;  // atomics::number_of_three_hit_tracks
    unsigned n_tracks; // dev_number_of_velo_tracks
    unsigned scan_parity;
  };

  // The block-wide part of an exclusive scan, with a single barrier: warp totals go to one
  // of two buffers, alternating per call, so a call never overwrites totals still being
  // read.  incl: the warp-inclusive sum of v.
  __device__ __forceinline__ unsigned scan_block(SearchShared& s, Counters& c, unsigned incl, unsigned v, unsigned& total)
  {
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
    unsigned* buf = s.scan_sums[c.scan_parity];
    c.scan_parity ^= 1u;
    if (lane == 31) buf[warp] = incl;
    __syncthreads();
    unsigned before = 0, all = 0;
    if (n_warps <= 4) { // one vector read of the four totals (those past the last warp stay 0)
      const uint4 t = *reinterpret_cast<const uint4*>(buf);
      all = t.x + t.y + t.z + t.w;
      before = (warp > 0 ? t.x : 0u) + (warp > 1 ? t.y : 0u) + (warp > 2 ? t.z : 0u);
    }
    else {
      for (unsigned w = 0; w < n_warps; ++w) {
        const unsigned t = buf[w];
        before += w < warp ? t : 0u;
        all += t;
      }
    }
    total = all;
    return before + incl - v;
  }

  // Block-wide exclusive scan of up to three 0/1 flags packed at bits 0, S1 and S2 (each field
  // wide enough for a block total), the warp part by ballots.
  template<unsigned NF, unsigned S1 = 16, unsigned S2 = 32>
  __device__ __forceinline__ unsigned scan_flags(SearchShared& s, Counters& c, bool f0, bool f1, bool f2, unsigned& total)
  {
    const unsigned le = 0xFFFFFFFFu >> (31u - (threadIdx.x & 31u)); // this lane and those below
    unsigned incl = __popc(__ballot_sync(0xFFFFFFFFu, f0) & le);
    unsigned v = f0 ? 1u : 0u;
    if constexpr (NF > 1) {
      incl |= static_cast<unsigned>(__popc(__ballot_sync(0xFFFFFFFFu, f1) & le)) << S1;
      v |= (f1 ? 1u : 0u) << S1;
    }
    if constexpr (NF > 2) {
      incl |= static_cast<unsigned>(__popc(__ballot_sync(0xFFFFFFFFu, f2) & le)) << S2;
      v |= (f2 ? 1u : 0u) << S2;
    }
    return scan_block(s, c, incl, v, total);
  }

  __device__ __forceinline__ bool phi_outside(int16_t phi, int16_t extrapolated, int16_t tol)
  {
    const int16_t diff = static_cast<int16_t>(phi - extrapolated);
    const int16_t abs_diff = static_cast<int16_t>(diff < 0 ? -diff : diff);
    return abs_diff > tol;
  }

  struct Extrapolation {
    int start;   // first h2 candidate (find_forward_candidate, SearchByTriplet.cu:272-292)
    int16_t phi; // extrapolated phi
  };

  __device__ __forceinline__ Extrapolation extrapolate(
    const Constants& k,
    const SearchShared& s,
    const Hits& h,
    const ModulePair& next,
    float h0x,
    float h0y,
    float tx,
    float ty,
    float dz)
  {
    const float predx = tx * dz;
    const float predy = ty * dz;
    const float xp = h0x + predx;
    const float yp = h0y + predy;
    Extrapolation x;
    x.phi = hit_phi_16(k, xp, yp);
    const int16_t lo = static_cast<int16_t>(x.phi - static_cast<int16_t>(k.phi_tolerance_i16));
    // find_forward_candidate returns the index as int16
    x.start = static_cast<int16_t>(leftmost_hit(s, h, next, lo));
    return x;
  }

  // Seeding over the current module pair (SearchByTriplet.cu:298-446).  Phase A, one thread per
  // unused h1: its rank among the window's unused hits names it (a bisection over the counts of
  // the words of bits), and the pendulum its h0 candidates; every h1 has the same
  // number of them, the unused hits of the previous module pair or n_candidates.  Phase B, one
  // thread per (h0, h1) doublet: the h2 window; the doublets of an h1 are neighbouring lanes,
  // whose shuffle reduction keeps the best (scatter, candidate order), the reference's
  // sequential choice, and a scan queues the seeds in h1 order.  Counting by one warp for all, and
  // the pendulum by words of bits to its end instead of step by step where the first words hold too
  // few unused hits, made the search 2.36 -> 2.31 ms for 16000 events and 235 -> 214 us for 10
  // (an extra barrier costs 2 us of the former).
  // GATED kernels take the learned seed gate (gate, event-relative, or null): an unused h1
  // whose gate byte is 0 is not searched; and, for training, record each unused h1's
  // outcome (outcome: 1 no seed, 2 seed; null = off).
  template<bool GATED, typename Shared, typename RingT>
  __device__ __forceinline__ void seeding(
    Shared& s,
    const RingT& ring,
    Counters& cnt,
    const Constants& k,
    const Hits& h,
    const UsedBits& used,
    const ModulePair* md,
    unsigned n_candidates,
    const uint8_t* gate,
    uint8_t* outcome)
  {
    const ModulePair &prev = md[0], &cur = md[1], &next = md[2];
    const unsigned lane = threadIdx.x & 31u;
    const int16_t tol = static_cast<int16_t>(k.phi_tolerance_i16);
    const unsigned places_log = n_candidates > 4 ? 3 : 2;
    for (unsigned w0 = 0; w0 < cur.hit_num; w0 += seed_window_hits) {
      const unsigned n_window = min(seed_window_hits, cur.hit_num - w0);
      const unsigned first = cur.hit_start + w0;
      if constexpr (GATED) {
        if (gate != nullptr) {
          for (unsigned i = threadIdx.x; i < (n_window + 31u) / 32u * 32u; i += blockDim.x) {
            const uint32_t pass = __ballot_sync(0xFFFFFFFFu, i < n_window && !used[first + i] && gate[first + i] != 0);
            if (lane == 0) s.pass[i / 32] = pass;
          }
          __syncthreads();
        }
      }
      // One warp counts for all (barriers cost less than every warp's share of this): the
      // window's unused hits, 32 per lane, and those of the previous module pair
      if (threadIdx.x < 32) {
        static_assert(seed_window_hits == 256, "8 words");
        uint32_t word = 32 * lane < n_window ? low_bits(used.unused(first + 32 * lane), n_window - 32 * lane) : 0u;
        if constexpr (GATED) {
          const unsigned unused = __reduce_add_sync(0xFFFFFFFFu, __popc(word));
          if (lane == 0) {
            s.local_hits += unused;
            s.candidates += unused;
          }
          if (gate != nullptr) word = 32 * lane < n_window ? s.pass[lane] : 0u;
        }
        unsigned before = __popc(word);
#pragma unroll
        for (unsigned o = 1; o < 8; o *= 2) {
          const unsigned t = __shfl_up_sync(0xFFFFFFFFu, before, o);
          if (lane >= o) before += t;
        }
        if (lane < 8) {
          s.seed_before[lane + 1] = before;
          s.seed_bits[lane] = word;
        }
        unsigned n_h0 = 0;
        for (unsigned i = 32 * lane; i < prev.hit_num; i += 1024)
          n_h0 += __popc(low_bits(used.unused(prev.hit_start + i), prev.hit_num - i));
        n_h0 = __reduce_add_sync(0xFFFFFFFFu, n_h0);
        if (lane == 0) {
          s.seed_before[0] = 0;
          s.n_h0 = n_h0;
        }
      }
      __syncthreads();
      const unsigned n_h1 = s.seed_before[8], n_h0 = min(s.n_h0, n_candidates);
      const unsigned per_chunk = min(blockDim.x, seed_slots >> places_log);
      for (unsigned c0 = 0; c0 < n_h1; c0 += per_chunk) {
        const unsigned n_chunk = min(per_chunk, n_h1 - c0);
        // Phase A
        if (threadIdx.x < n_chunk) {
          {
            const unsigned rank = c0 + threadIdx.x;
            unsigned at = 0; // the last word with no more than rank hits before it
#pragma unroll
            for (unsigned step = 4; step >= 1; step /= 2)
              if (s.seed_before[at + step] <= rank) at += step;
            const unsigned h1 = first + 32 * at + select_bit(s.seed_bits[at], rank - s.seed_before[at]);
            s.seed_h1[threadIdx.x] = static_cast<uint16_t>(h1);
            if (n_h0 > 0) {
              Pendulum pendulum(prev.hit_start, prev.hit_num, static_cast<unsigned>(leftmost_hit(s, h, prev, h.phi(h1))));
              for (unsigned c = 0; c < n_h0; ++c)
                s.seed_h0[(threadIdx.x << places_log) + c] = static_cast<uint16_t>(prev.hit_start + pendulum.next(used));
            }
          }
        }
        __syncthreads();
        // Phase B
        for (unsigned q0 = 0; q0 < n_chunk << places_log; q0 += blockDim.x) {
          const unsigned q = q0 + threadIdx.x, i = q >> places_log, c = q & ((1u << places_log) - 1u);
          float best_fit = k.max_scatter;
          unsigned best = 0, best_c = c; // best: h0 | h2 << 16
          unsigned h1 = 0;
          if (i < n_chunk && c < n_h0) {
            h1 = s.seed_h1[i];
            const unsigned h0 = s.seed_h0[q];
            const Hit a = h[h0], b = h[h1];
            const float td = __frcp_rn(b.z - a.z);
            const float tx = (b.x - a.x) * td;
            const float ty = (b.y - a.y) * td;
            const Extrapolation f = extrapolate(k, s, h, next, a.x, a.y, tx, ty, next.z[0] - prev.z[0]);
            // circular walk from the candidate: index (start + j) % n without a division per step
            unsigned idx = first_candidate(f.start, next.hit_num);
            for (unsigned j = 0; j < next.hit_num; ++j, idx = (idx + 1 == next.hit_num) ? 0u : idx + 1) {
              const unsigned h2 = next.hit_start + idx;
              const Hit d = h[h2];
              if (phi_outside(d.phi, f.phi, tol)) break;
              const float dz = d.z - a.z;
              const float dx = (a.x + tx * dz) - d.x;
              const float dy = (a.y + ty * dz) - d.y;
              const float scatter = dx * dx + dy * dy;
              if (scatter < best_fit && !used[h2]) {
                best_fit = scatter;
                best = h0 | (h2 << 16);
              }
            }
          }
          for (unsigned o = 1; o < 1u << places_log; o *= 2) {
            const float of = __shfl_xor_sync(0xFFFFFFFFu, best_fit, o);
            const unsigned oc = __shfl_xor_sync(0xFFFFFFFFu, best_c, o);
            const unsigned ob = __shfl_xor_sync(0xFFFFFFFFu, best, o);
            if (of < best_fit || (of == best_fit && oc < best_c)) {
              best_fit = of;
              best_c = oc;
              best = ob;
            }
          }
          const bool first_lane = c == 0 && i < n_chunk;
          const bool ok = first_lane && best_fit < k.max_scatter;
          if (GATED && outcome != nullptr && first_lane) outcome[s.seed_h1[i]] = ok ? 2 : 1;
          unsigned n_seeds;
          const unsigned excl = scan_flags<1>(s, cnt, ok, false, false, n_seeds);
          if (ok) {
            ring.append(cnt.ttf + excl) =
              seed_flag | uint64_t(best & 0xFFFFu) | (uint64_t(h1 & 0xFFFFu) << 16) | (uint64_t(best >> 16) << 32);
          }
          cnt.ttf += n_seeds;
        }
      }
      if (threadIdx.x == 0) {
        if (!GATED) {
          s.local_hits += n_h1;
          s.candidates += n_h1;
        }
        s.searched += n_h1;
      }
      if (w0 + seed_window_hits < cur.hit_num) __syncthreads(); // the window's words are read
    }
  }

  // Forwarding of the tracks to follow (SearchByTriplet.cu:451-609), one thread per track.  The
  // hits the >= 4 hit tracks gained are added to the thread's track_hits.
  template<typename Shared, typename RingT>
  __device__ __forceinline__ void forwarding(
    Shared& s,
    const RingT& ring,
    Counters& cnt,
    const Constants& k,
    const Hits& h,
    const UsedBits& used,
    const ModulePair& next,
    unsigned prev_ttf,
    unsigned diff_ttf,
    TrackHits* tracks,
    unsigned track_limit,
    TrackletHits* three_hit,
    unsigned& track_hits,
    unsigned* status)
  {
    const int16_t tol = static_cast<int16_t>(k.phi_tolerance_i16);
    for (unsigned c0 = 0; c0 < diff_ttf; c0 += blockDim.x) {
      const unsigned kk = c0 + threadIdx.x;
      const bool active = kk < diff_ttf;
      uint64_t entry = 0;
      unsigned h0n = 0, h1n = 0;
      bool is_seed = false, found = false;
      unsigned best_h2 = 0;
      if (active) {
        entry = ring.at(prev_ttf + kk, prev_ttf, ring.parity ^ 1u);
        is_seed = (entry & seed_flag) != 0;
        const unsigned pair = static_cast<unsigned>(is_seed ? entry >> 16 : entry);
        h0n = pair & 0xFFFFu;
        h1n = pair >> 16;
        const Hit a = h[h0n], b = h[h1n];
        const unsigned odd = (a.flags & flag_odd_module) ? 1u : 0u;
        const float td = __frcp_rn(b.z - a.z);
        const float tx = (b.x - a.x) * td;
        const float ty = (b.y - a.y) * td;
        float best_fit = k.max_scatter;
        const Extrapolation f = extrapolate(k, s, h, next, a.x, a.y, tx, ty, next.z[odd] - a.z);
        unsigned idx = first_candidate(f.start, next.hit_num);
        for (unsigned j = 0; j < next.hit_num; ++j, idx = (idx + 1 == next.hit_num) ? 0u : idx + 1) {
          const unsigned h2 = next.hit_start + idx;
          const Hit c = h[h2];
          if (phi_outside(c.phi, f.phi, tol)) break;
          const float dz = c.z - a.z;
          const float dx = (a.x + tx * dz) - c.x;
          const float dy = (a.y + ty * dz) - c.y;
          const float scatter = dx * dx + dy * dy;
          if (scatter < best_fit) {
            best_fit = scatter;
            best_h2 = h2;
            found = true;
          }
        }
      }
      const unsigned nh = is_seed ? 3u : static_cast<unsigned>(entry >> hits_shift) & 0x1Fu;
      const unsigned skipped = static_cast<unsigned>(entry >> skipped_shift) & skipped_mask;
      const bool new_track = active && found && is_seed;
      const bool enqueue =
        active && ((found && nh + 1 < max_track_size) || (!found && skipped < k.max_skipped_modules));
      const bool three = active && !found && !(skipped < k.max_skipped_modules) && is_seed;
      unsigned total;
      const unsigned excl =
        scan_flags<3, 10, 20>(s, cnt, new_track, enqueue, three, total);
      if (active) {
        if (found) {
          used.set(best_h2);
          unsigned track_number = static_cast<unsigned>(entry >> 32) & 0xFFFFu;
          if (is_seed) {
            const unsigned t0 = static_cast<unsigned>(entry) & 0xFFFFu;
            used.set(t0);
            used.set(h0n);
            used.set(h1n);
            track_number = cnt.n_tracks + (excl & 0x3FFu);
            if (track_number < track_limit) {
              TrackHits& t = tracks[track_number];
              t.hits[0] = static_cast<uint16_t>(t0);
              t.hits[1] = static_cast<uint16_t>(h0n);
              t.hits[2] = static_cast<uint16_t>(h1n);
              t.hits[3] = static_cast<uint16_t>(best_h2);
              t.hits_num = 4;
            }
            else {
              set_error(status, err_track_capacity);
            }
          }
          else if (track_number < track_limit) {
            tracks[track_number].hits[nh] = static_cast<uint16_t>(best_h2);
            tracks[track_number].hits_num = static_cast<uint8_t>(nh + 1);
          }
          track_hits += is_seed ? 4u : 1u;
          entry = uint64_t(h1n) | (uint64_t(best_h2 & 0xFFFFu) << 16) | (uint64_t(track_number & 0xFFFFu) << 32) |
                  (uint64_t(nh + 1) << hits_shift);
        }
        else {
          // requeued as it is, with skipped + 1
          entry = (entry & ~(uint64_t(skipped_mask) << skipped_shift)) |
                  (uint64_t((skipped + 1) & skipped_mask) << skipped_shift);
        }
        if (enqueue) ring.append(cnt.ttf + ((excl >> 10) & 0x3FFu)) = entry;
        if (three) {
          const unsigned slot = cnt.n_three + ((excl >> 20) & 0x3FFu);
          if (slot < track_limit) {
            three_hit[slot] = TrackletHits {
              {static_cast<uint16_t>(entry & 0xFFFFu), static_cast<uint16_t>(h0n), static_cast<uint16_t>(h1n)}};
          }
          else {
            set_error(status, err_track_capacity);
          }
        }
      }
      cnt.n_tracks += total & 0x3FFu;
      cnt.ttf += (total >> 10) & 0x3FFu;
      cnt.n_three += (total >> 20) & 0x3FFu;
    }
  }

  // ThreeHitTracksFilter.cu:48-107
  __device__ __forceinline__ float means_square_fit_chi2(const Hit (&r)[3])
  {
    const float w = 6400.f;
    float s0, sx, sz, sxz, sz2, u0, uy, uz, uyz, uz2;
    s0 = sx = sz = sxz = sz2 = 0.0f;
    u0 = uy = uz = uyz = uz2 = 0.0f;
#pragma unroll
    for (unsigned i = 0; i < 3; ++i) {
      const float x = r[i].x, y = r[i].y, z = r[i].z;
      const float wx_t_x = w * x, wx_t_z = w * z;
      s0 += w;
      sx += wx_t_x;
      sz += wx_t_z;
      sxz += wx_t_x * z;
      sz2 += wx_t_z * z;
      const float wy_t_y = w * y, wy_t_z = w * z;
      u0 += w;
      uy += wy_t_y;
      uz += wy_t_z;
      uyz += wy_t_y * z;
      uz2 += wy_t_z * z;
    }
    const float dens = __fdiv_rn(1.0f, sz2 * s0 - sz * sz);
    const float state_tx = (sxz * s0 - sx * sz) * dens;
    const float state_x = (sx * sz2 - sxz * sz) * dens;
    const float denu = __fdiv_rn(1.0f, uz2 * u0 - uz * uz);
    const float state_ty = (uyz * u0 - uy * uz) * denu;
    const float state_y = (uy * uz2 - uyz * uz) * denu;
    float chi2 = 0.0f;
#pragma unroll
    for (unsigned i = 0; i < 3; ++i) {
      const float z = r[i].z;
      const float x = state_x + state_tx * z;
      const float y = state_y + state_ty * z;
      const float dx = x - r[i].x;
      const float dy = y - r[i].y;
      chi2 += dx * dx * w + dy * dy * w;
    }
    return chi2 * 0.5f;
  }

  // The event's module pairs into shared memory, last first (threads 0-25; a barrier follows).
  __device__ __forceinline__ void module_pairs(
    ModulePair* mps, const Geometry* g, const unsigned* start, const unsigned* num, unsigned hit_offset)
  {
    const unsigned mp = threadIdx.x;
    if (mp < n_module_pairs) {
      ModulePair& m = mps[n_module_pairs - 1 - mp];
      m.hit_start = start[mp] - hit_offset;
      m.hit_num = num[mp];
      m.z[0] = __ldg(g->module_zs + 2 * mp);
      m.z[1] = __ldg(g->module_zs + 2 * mp + 1);
      m.table = mp % 3;
    }
  }

  // The phi values of a module pair into its slot, then its bucket table from them (barriers between
  // the two and after; a larger pair's table from the records).
  __device__ __forceinline__ void load_phi(SearchShared& s, const Hits& h, const ModulePair& m)
  {
    if (m.hit_num <= phi_capacity)
      for (unsigned i = threadIdx.x; i < m.hit_num; i += blockDim.x)
        s.phi[m.table][i] = h.phi(m.hit_start + i);
  }
  __device__ __forceinline__ void build_table(SearchShared& s, const Hits& h, const ModulePair& m)
  {
    if (m.hit_num <= phi_capacity) {
      const int16_t* phi = s.phi[m.table];
      build_bucket_table_of(s.bucket[m.table], [phi](unsigned j) { return phi[j]; }, 0, m.hit_num);
    }
    else {
      build_bucket_table_of(s.bucket[m.table], [h](unsigned j) { return h.phi(j); }, m.hit_start, m.hit_num);
    }
  }

  // Seeding, forwarding and the tail of one event over staged hits (used bits clear):
  // SearchByTriplet.cu:165-264.  Returns the event's counters; the track containers hold
  // its tracks and three-hit tracks, s.track_hits the hits of the former.
  template<bool GATED, typename Shared, typename RingT>
  __device__ __forceinline__ Counters search_pass(
    const SearchParams& p,
    Shared& s,
    RingT& ring,
    const Constants& k,
    const Hits& h,
    const UsedBits& used,
    const unsigned* start,
    const unsigned* num,
    unsigned hit_offset,
    TrackHits* tracks,
    unsigned track_limit,
    TrackletHits* three_hit,
    const uint8_t* gate,
    uint8_t* outcome)
  {
    if (threadIdx.x == 0) s.track_hits = s.candidates = s.searched = 0;
    if (threadIdx.x < 64) s.scan_sums[threadIdx.x >> 5][threadIdx.x & 31u] = 0;
    Counters cnt {0, 0, 0, 0};
    module_pairs(s.mps, p.geo, start, num, hit_offset);
    __syncthreads();
    unsigned first = n_module_pairs - 1;
    const ModulePair* md = s.mps;
    for (unsigned i = 0; i < 2; ++i)
      load_phi(s, h, md[i]);
    __syncthreads();
    for (unsigned i = 0; i < 2; ++i)
      build_table(s, h, md[i]);

    // One step per module pair first = 25 ... 2 (the first without forwarding), with a single
    // copy of the seeding code.
    unsigned last_ttf = 0, track_hits = 0;
    const unsigned window = GATED && gate != nullptr && p.seed_window ? p.seed_window : 4u;
    for (;;) {
      // module pair first - 2 takes the slot of first + 1, last read by the previous step's
      // seeding before its last barrier
      load_phi(s, h, md[2]);
      __syncthreads();
      build_table(s, h, md[2]);
      const bool forward = first < n_module_pairs - 1;
      const unsigned prev_ttf = last_ttf;
      if (forward) {
        last_ttf = cnt.ttf;
        ring.next_generation(cnt.ttf);
      }
      if (threadIdx.x == 0) s.local_hits = 0;
      __syncthreads(); // ring entries of the last seeding, the new bucket table
      if (forward) {
        forwarding(
          s, ring, cnt, k, h, used, md[2], prev_ttf, last_ttf - prev_ttf, tracks, track_limit, three_hit, track_hits,
          p.status);
        // The ring holds 2048 entries; beyond that the reference overwrites entries it has
        // not read yet, an order-dependent outcome this kernel does not reproduce.
        if (threadIdx.x == 0 && cnt.ttf - prev_ttf > max_tracks_to_follow) set_error(p.status, err_ttf_overflow);
        __syncthreads(); // used bits set by forwarding
      }
      seeding<GATED>(s, ring, cnt, k, h, used, md, forward ? window : 8u, gate, outcome);
      if (forward && threadIdx.x == 0 && cnt.ttf - last_ttf > max_tracks_to_follow) set_error(p.status, err_ttf_overflow);
      if (--first <= 1) break;
      ++md;
    }
    track_hits = __reduce_add_sync(0xFFFFFFFFu, track_hits);
    if ((threadIdx.x & 31u) == 0) atomicAdd(&s.track_hits, track_hits);
    __syncthreads(); // ring entries of the last seeding

    // Tail: seeds still in flight become three-hit tracks (SearchByTriplet.cu:247-264)
    const unsigned diff = cnt.ttf - last_ttf;
    for (unsigned c0 = 0; c0 < diff; c0 += blockDim.x) {
      const unsigned kk = c0 + threadIdx.x;
      uint64_t entry = 0;
      bool seed = false;
      if (kk < diff) {
        entry = ring.append(last_ttf + kk);
        seed = (entry & seed_flag) != 0;
      }
      unsigned total;
      const unsigned excl = scan_flags<1>(s, cnt, seed, false, false, total);
      if (seed) {
        const unsigned slot = cnt.n_three + excl;
        if (slot < track_limit) {
          three_hit[slot] = TrackletHits {{static_cast<uint16_t>(entry & 0xFFFFu),
                                           static_cast<uint16_t>((entry >> 16) & 0xFFFFu),
                                           static_cast<uint16_t>((entry >> 32) & 0xFFFFu)}};
        }
        else {
          set_error(p.status, err_track_capacity);
        }
      }
      cnt.n_three += total;
    }
    return cnt;
  }

  template<bool SMEM, bool GATED, typename Shared, typename RingT>
  __device__ __forceinline__ void
  search_event(const SearchParams& p, Shared& s, RingT ring, unsigned char* dsmem, unsigned e)
  {
    const unsigned n = p.n_events;
    const unsigned* start = p.offsets_estimated_input_size + e * n_module_pairs;
    const unsigned* num = p.module_cluster_num + e * n_module_pairs;
    const unsigned hit_offset = start[0];
    const unsigned n_hits = start[n_module_pairs] - hit_offset;
    const unsigned T = *p.total_clusters;
    const Constants k = p.k;
    if (T > p.cluster_capacity) return; // flagged by the clustering kernel
    if (n_hits > 65536u && threadIdx.x == 0) set_error(p.status, err_hits_per_event);

    // Track container size as SearchByTriplet.cu:23-27 computes it on the host.
    const float by_clusters = __uint2float_rn(T) * 0.34f;
    const unsigned track_container_size = by_clusters < __uint2float_rn(n * minimum_container_size) ?
                                            n * minimum_container_size :
                                            static_cast<unsigned>(by_clusters);
    const unsigned container = min(track_container_size, p.track_capacity);
    if (track_container_size > p.track_capacity && e == 0 && threadIdx.x == 0) set_error(p.status, err_input_capacity);
    const unsigned to = track_offset(p.offsets_estimated_input_size, e);
    const unsigned to_next = e + 1 < n ? track_offset(p.offsets_estimated_input_size, e + 1) : container;
    // Tracks may spill past the event's slice exactly as in the reference (no bound
    // there); writes stay inside the container and the spill is flagged.
    const unsigned track_limit = container > to ? container - to : 0u;
    TrackHits* tracks = p.tracks + to;
    TrackletHits* three_hit = p.three_hit_tracks + to;

    // Stage the hits as 16-byte records: shared memory when they fit (SMEM), else the
    // event's global slice (16 bytes per estimated hit).  All unused.
    const Hits h {SMEM ? reinterpret_cast<uint4*>(dsmem) : reinterpret_cast<uint4*>(p.hit_scratch) + hit_offset};
    const UsedBits used {n_hits <= used_capacity ? s.used :
                                                   reinterpret_cast<uint32_t*>(p.used_scratch + size_t(24) * hit_offset)};
    for (unsigned i = threadIdx.x; i <= (n_hits + 31u) / 32u; i += blockDim.x)
      used.w[i] = 0;
    {
      const ClusterView g {const_cast<char*>(p.sorted_container), T};
      // read once: streaming loads (evict first), which leave L2 to the staged hits
      for (unsigned i = threadIdx.x; i < n_hits; i += blockDim.x) {
        const unsigned gi = hit_offset + i;
        const unsigned module = ((__ldcs(&g.id(gi)) & 0x3FC0000u) >> 18) / 4;
        const unsigned flags = (module & 1u) ? flag_odd_module : 0u;
        h.r[i] = make_uint4(__float_as_uint(__ldcs(&g.x(gi))), __float_as_uint(__ldcs(&g.y(gi))),
                            __float_as_uint(__ldcs(&g.z(gi))), static_cast<uint16_t>(__ldcs(&g.phi(gi))) | (flags << 16));
      }
    }

    // Learned mode: the gate of the event's seed candidates, unless the fraction it lets
    // through falls outside the model's bounds, in which case the plain search runs
    unsigned mode = seed_mode_plain;
    const uint8_t* gate = nullptr;
    if (GATED && p.seed_gate != nullptr) {
      const unsigned cand = p.gate_stats[2 * e], kept = p.gate_stats[2 * e + 1];
      const float frac = cand > 0 ? __fdiv_rn(__uint2float_rn(kept), __uint2float_rn(cand)) : 1.0f;
      if (frac >= p.kept_lo && frac <= p.kept_hi) {
        gate = p.seed_gate + hit_offset;
        mode = seed_mode_learned;
      }
      else {
        mode = seed_mode_fallback;
      }
    }
    uint8_t* outcome = GATED && p.h1_outcome != nullptr ? p.h1_outcome + hit_offset : nullptr;
    Counters cnt = search_pass<GATED>(
      p, s, ring, k, h, used, start, num, hit_offset, tracks, track_limit, three_hit, gate, outcome);
    if (p.seed_stats != nullptr && threadIdx.x == 0) {
      p.seed_stats[3 * e] = s.candidates;
      p.seed_stats[3 * e + 1] = s.searched;
      p.seed_stats[3 * e + 2] = mode;
    }

    if (threadIdx.x == 0) {
      unsigned* atomics = p.atomics_velo + 3 * e;
      atomics[0] = cnt.n_three;
      atomics[1] = cnt.ttf;
      atomics[2] = s.local_hits;
      p.number_of_velo_tracks[e] = cnt.n_tracks;
      if (cnt.n_tracks > to_next - to) set_error(p.status, err_track_capacity);
    }
    {
      uint8_t* g_used = reinterpret_cast<uint8_t*>(p.hit_used) + hit_offset;
      for (unsigned i = threadIdx.x; i < n_hits; i += blockDim.x)
        g_used[i] = used[i];
    }
    __syncthreads();

    // Three-hit filter (ThreeHitTracksFilter.cu:109-130), input order preserved
    const unsigned n_in = min(cnt.n_three, track_limit);
    TrackletHits* out = p.three_hit_tracks_output + to;
    unsigned filter_count = 0;
    for (unsigned c0 = 0; c0 < n_in; c0 += blockDim.x) {
      const unsigned i = c0 + threadIdx.x;
      bool keep = false;
      TrackletHits t {};
      if (i < n_in) {
        t = three_hit[i];
        if (!used[t.hits[0]] && !used[t.hits[1]] && !used[t.hits[2]]) {
          const Hit r[3] = {h[t.hits[0]], h[t.hits[1]], h[t.hits[2]]};
          keep = means_square_fit_chi2(r) < k.max_chi2;
        }
      }
      unsigned total;
      const unsigned excl = scan_flags<1>(s, cnt, keep, false, false, total);
      if (keep) out[filter_count + excl] = t;
      filter_count += total;
    }
    if (threadIdx.x == 0) {
      p.number_of_three_hit_tracks_output[e] = filter_count;
      p.event_track_hits[e] = s.track_hits + 3 * filter_count;
    }
    // the staged hits are dead (the filter's last scan is a barrier after the last read)
    if (!SMEM) discard_l2(h.r, size_t(16) * n_hits);
  }

  // One instantiation per (block size, ring place); the chain launches the one its launch
  // configuration names (autotuned).  Events whose hits fit the shared-memory capacity run the
  // shared-memory body, the others the global-scratch body.  The ring of tracks to follow (2048
  // entries, 16 KiB) sits in shared memory, or with RING = 1 in this CTA's slice of a global
  // scratch (persistent launches only: the slice is the CTA's index) behind near_entries of each
  // step in shared memory, which leaves room for more resident CTAs per SM.
  // Issue-bound.  Register-capped for 2048 threads per SM (32 registers): with the hits staged
  // through L2 shared memory does not limit the CTAs per SM, and the resident events hide more
  // latency than the cap costs (16000 events: 2.36 ms; twelve CTAs per SM at 40 registers 2.51,
  // eight at 64 registers 2.83).  Slices that eight CTAs per SM hold take 64 registers (128
  // threads with global rings: 1000 events 437 -> 384 us, 10 events 245 -> 235 us).  The seeding by
  // used bits, against used flags in the hit records, an index of the unused hits and a packed list
  // of doublets per step (ten barriers a step instead of five): 3.01 -> 2.36 ms, 10 events 313 ->
  // 245 us.
  template<unsigned THREADS, unsigned RING, bool GATED>
  __device__ __forceinline__ void search_events(const SearchParams& p)
  {
    extern __shared__ __align__(128) unsigned char dsmem[];
    __shared__ std::conditional_t<GATED, SearchSharedGated, SearchShared> s;
    __shared__ uint64_t near_ring[RING ? 2 * near_entries : max_tracks_to_follow];
    const Ring<RING != 0> ring {RING ? p.ring_scratch + size_t(blockIdx.x) * max_tracks_to_follow : near_ring, near_ring, 0, 0};
    for_each_event(p.queue, p.n_events, [&](unsigned e, unsigned) {
      const unsigned* start = p.offsets_estimated_input_size + e * n_module_pairs;
      const unsigned n_hits = start[n_module_pairs] - start[0];
      if (n_hits <= p.smem_hit_capacity) search_event<true, GATED>(p, s, ring, dsmem, e);
      else search_event<false, GATED>(p, s, ring, dsmem, e);
    });
  }

  template<unsigned THREADS, unsigned RING, unsigned SM_THREADS>
  __global__ void __launch_bounds__(THREADS, SM_THREADS / THREADS) search_by_triplet_kernel(SearchParams p)
  {
    search_events<THREADS, RING, false>(p);
  }

  // The learned search: the seeding behind the seed gate (with seed_gate null, the plain
  // search, recording each seed candidate's outcome when h1_outcome is set).  Capped like the plain
  // kernel, though it spills more at 32 registers (244 bytes of stores and 344 of loads against 44 and
  // 84): 4000 events 0.63 ms, the plain search 0.65.
  template<unsigned THREADS, unsigned RING, unsigned SM_THREADS>
  __global__ void __launch_bounds__(THREADS, SM_THREADS / THREADS) search_by_triplet_gated_kernel(SearchParams p)
  {
    search_events<THREADS, RING, true>(p);
  }

#define VELO_SEARCH_CONFIG(T, R)                                                  \
  template __global__ void search_by_triplet_kernel<T, R, 2048>(SearchParams p);  \
  template __global__ void search_by_triplet_gated_kernel<T, R, 2048>(SearchParams p);
  VELO_SEARCH_CONFIGS(VELO_SEARCH_CONFIG)
#undef VELO_SEARCH_CONFIG
  template __global__ void search_by_triplet_kernel<128, 1, few_events_threads>(SearchParams p);
  template __global__ void search_by_triplet_gated_kernel<128, 1, few_events_threads>(SearchParams p);

} // namespace velo

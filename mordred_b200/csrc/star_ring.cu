// star_ring.cu — the fused star query for calls with at least one probe: the form mb_star_query
// and the SSB and engine entry points run by default (see star.cuh for the plan; star_impl.cuh
// holds the tile-staged kernels that remain for filter-aggregates and explicit launch shapes).
//
// Most rows of a star query end at the first one or two probes, so only the columns every
// row needs are streamed: the filters, the keys of the leading probes with a presence bitmap
// in shared memory, and the key of the first probe after those. Each warp works alone:
//   * slices of 256 rows arrive by bulk copies in the warp's own two buffers, so that no
//     warp waits for another and a slice is on its way while one is worked on;
//   * dense part: 8 rows a lane, filters and bitmaps into a bit mask a lane;
//   * the survivors are compacted and the first table probe runs over full lanes, two rows a
//     lane, its loads in flight under the next slice's dense part; the rows it keeps — row
//     number and payload — go to the warp's ring in shared memory;
//   * 32 rows of the ring at a time, one a lane, take the rest of the pipeline: the remaining
//     keys and the aggregate columns are gathered from the fact columns (all at once), the
//     remaining tables are probed (all at once), and the sums go to a shared-memory group array
//     flushed once per CTA, to L2 atomics, or to a scalar.
// The kernels before it staged every column of every row and ran the later probes and the
// aggregate for the few rows each 256-row slice had left. 120,000,000 rows, kernel alone: Query B
// 614 -> 341 us, Query A 457 -> 350; the engine's group-by over 23 cached segments 159 -> 103;
// Query B over 1,000,000 rows 24 -> 16.
// What bounds it: instruction issue together with the trips to L2 (52 to 61 % issue-active, 32
// warps an SM; 2.0 to 2.6 warp instructions a row against 2.8 to 3.9), not DRAM (9.3 bytes a row
// for Query A, 14.1 for Query B, 2.8 to 4.3 TB/s). What it leaves of the SM's 256 KB as L1 counts:
// the scattered loads in flight sit there, and a bitmap of one byte a slot (120 KB more shared
// memory) took Query B to 486 us. One CTA an SM with 32 warps: 18 warps are as good for Query A,
// 30 and more for Query B.
// Selection, payloads, sums and status bits equal the sequential chain's: presence is combined
// probe by probe in order, a probe the bitmaps settled is present for every row that passes
// them, and sums are integers.
#include "star_impl.cuh"

namespace mb {

constexpr int kRingMaxWarps = 32;
constexpr int kRingItems = 8;               // rows a lane
constexpr int kRingRows = 32 * kRingItems;  // rows per slice
constexpr int kRingRound = 64;              // survivors a round probes (two a lane)
constexpr int kRingCap = 64;                // rows a ring holds

struct __align__(16) RingWarp {
  int2 ring[kRingCap];       // first probe's payload, row of the call
  uint16_t off[kRingRows];   // survivors: their rows within the slice
  uint64_t bar[2];
  // followed by the two buffers: [2][P.r_nst][kRingRows]
};
__host__ __device__ constexpr int ring_warp_bytes(int nst) {
  return static_cast<int>(sizeof(RingWarp)) + 2 * nst * kRingRows * 4;
}

// lo, hi = the word of slot h >= 0 of a table if `on` (0 when absent), else left alone. Only the
// loads, under opposite predicates: nothing waits for them before their first use.
__device__ __forceinline__ void ring_word(const int* ht, bool key_layout, int h, bool on, unsigned& lo, unsigned& hi) {
  asm volatile(
      "{\n\t.reg .pred k, v;\n\t"
      "setp.eq.u32 k, %4, 1;\n\t"
      "setp.eq.u32 v, %4, 2;\n\t"
      "@k ld.global.u32 %0, [%2];\n\t"
      "@v ld.global.v2.u32 {%0, %1}, [%3];\n\t}"
      : "+r"(lo), "+r"(hi)
      : "l"(ht + h), "l"(ht + 2ll * h), "r"(!on ? 0u : key_layout ? 1u : 2u));
}
// The payload in a word, as probe_round's.
__device__ __forceinline__ int ring_payload(int layout, unsigned lo, unsigned hi) {
  return static_cast<int>(layout == MB_HT_KEY_VAL ? hi : layout == MB_HT_VAL_OFF ? lo : 0u);
}

// Adds a row to the groups: `hh` its group index, val its value; keys written for the first
// row of a group (per CTA with shared-memory groups). key(q): payload of sparse position q.
template <class Key>
__device__ __forceinline__ void ring_add(const StarPlan& P, unsigned hh, int val, int ns, unsigned long long* s_sum,
                                         uint32_t* s_touch, bool& bad_group, Key key) {
  int h = static_cast<int>(hh);
  if (hh >= static_cast<unsigned>(P.total_val)) h = slow_mod(h, P.total_val);
  if (h < 0) {
    bad_group = true;
    return;
  }
  bool keys = P.res_layout != MB_RES_DENSE;
  if (P.gmode == kGroupSmem) {
    smem_add_i64(&s_sum[h], val);
    const uint32_t bit = 1u << (h & 31);
    keys = !(s_touch[h >> 5] & bit) && !(atomicOr(&s_touch[h >> 5], bit) & bit) && keys;
  } else {
    atomicAdd(group_sum_ptr(P, h), static_cast<unsigned long long>(static_cast<long long>(val)));
  }
  if (!keys) return;
  int* res = static_cast<int*>(P.res) + static_cast<long long>(P.res_layout == MB_RES_ENGINE6 ? 6 : 4) * h;
#pragma unroll
  for (int q = 0; q < MB_MAX_PROBES; ++q) {
    if (q >= ns) break;
    const int rs = P.p_res_slot[P.sp_ord[q]];
    if (rs >= 0) res[rs] = key(q);
  }
}

// Bits of `v` table words: a bitmap holds slot s at bit 31 - s % 32, so that a shift left by s
// puts it at the top and a funnel shift moves it into the lane's mask; bit `slots` is 0 and
// stands for every key outside [key_min, key_min + 2 * slots).
__device__ __forceinline__ void ring_stage_bitmap(const StarPlan& P, int p, uint32_t* bm, int warp, int nwarps, int lane) {
  const int slots = P.p_slots[p], words = P.p_bm_words[p];
  if (P.p_presence[p] != nullptr) {
    const int given = (slots + 31) / 32;
    const uint32_t tail = slots % 32 != 0 ? (1u << (slots % 32)) - 1u : kFull;
    for (int w = warp * 32 + lane; w < words; w += nwarps * 32) {
      uint32_t v = 0u;
      if (w < given) v = static_cast<uint32_t>(ld_word(reinterpret_cast<const int*>(P.p_presence[p]) + w));
      if (w == given - 1) v &= tail;
      bm[w] = __brev(v);
    }
    return;
  }
  const int* ht = P.p_ht[p];
  const bool aligned = aligned16_dev(ht);
  if (P.p_layout[p] == MB_HT_KEY) {
    // 128 slots a warp step, four a lane: the ballots over slots 4l + e interleave
#pragma unroll 4
    for (int w0 = 4 * warp; w0 < words; w0 += 4 * nwarps) {
      const int h = w0 * 32 + 4 * lane;
      int4 t = make_int4(0, 0, 0, 0);
      if (aligned && h + 3 < slots) {
        t = ld_word4(ht + h);
      } else {
        if (h < slots) t.x = ld_word(ht + h);
        if (h + 1 < slots) t.y = ld_word(ht + h + 1);
        if (h + 2 < slots) t.z = ld_word(ht + h + 2);
        if (h + 3 < slots) t.w = ld_word(ht + h + 3);
      }
      // lane l's nibble in slot order, then eight lanes' nibbles into a word
      uint32_t nib = (t.x != 0 ? 8u : 0u) | (t.y != 0 ? 4u : 0u) | (t.z != 0 ? 2u : 0u) | (t.w != 0 ? 1u : 0u);
      uint32_t word = nib << (28 - 4 * (lane & 7));
      word |= __shfl_xor_sync(kFull, word, 1);
      word |= __shfl_xor_sync(kFull, word, 2);
      word |= __shfl_xor_sync(kFull, word, 4);
      if ((lane & 7) == 0 && w0 + (lane >> 3) < words) bm[w0 + (lane >> 3)] = word;
    }
  } else {
    // 64 slots of 8 bytes a warp step, two a lane, sixteen lanes' pairs into a word
#pragma unroll 4
    for (int w0 = 2 * warp; w0 < words; w0 += 2 * nwarps) {
      const int h = w0 * 32 + 2 * lane;
      bool even = false, odd = false;
      if (aligned && h + 1 < slots) {
        const int4 t = ld_word4(ht + 2ll * h);
        even = (t.x | t.y) != 0;
        odd = (t.z | t.w) != 0;
      } else {
        if (h < slots) even = ld_word2(ht + 2ll * h) != 0ull;
        if (h + 1 < slots) odd = ld_word2(ht + 2ll * h + 2) != 0ull;
      }
      uint32_t word = ((even ? 2u : 0u) | (odd ? 1u : 0u)) << (30 - 2 * (lane & 15));
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) word |= __shfl_xor_sync(kFull, word, o);
      if ((lane & 15) == 0 && w0 + (lane >> 4) < words) bm[w0 + (lane >> 4)] = word;
    }
  }
}

// NFC filters (-1: P.nf), NDC leading bitmap probes (-1: P.n_dense), K: a table probe follows
// them and runs before the ring (sparse position 0).
template <int NFC, int NDC, bool K>
__global__ void __launch_bounds__(kRingMaxWarps * 32, 1) star_ring_kernel(const __grid_constant__ StarPlan P) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ unsigned long long s_red[2 * kRingMaxWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int nst = P.r_nst;
  unsigned char* mine = smem + P.smem_list_off + warp * ring_warp_bytes(nst);
  RingWarp& w = *reinterpret_cast<RingWarp*>(mine);
  int* stage = reinterpret_cast<int*>(mine + sizeof(RingWarp));
  unsigned long long* s_sum = reinterpret_cast<unsigned long long*>(smem + P.smem_groups_off);
  uint32_t* s_touch = reinterpret_cast<uint32_t*>(smem + P.smem_groups_off + 8 * P.total_val);
  const int nf = NFC >= 0 ? NFC : P.nf, nd = NDC >= 0 ? NDC : P.n_dense;
  const int ns = P.np - P.sparse_p0;  // sparse_p0: bitmap probes settled by their bit
  const unsigned bias = static_cast<unsigned>(P.group_bias) + P.dense_bias;
  const bool two_cols = P.agg_op == MB_AGG_SUB || P.agg_op == MB_AGG_MUL;
  // the aggregate columns are gathered with the remaining keys, unless two or more tables can
  // still drop the row: then only for the rows they leave
  const bool early = (K ? ns - 1 - (nd - P.sparse_p0) : 0) <= 1;
  // fewer than 2^32 rows: rows and slices count in 32 bits
  const unsigned rows = static_cast<unsigned>(P.n);
  const int nslices = static_cast<int>((P.n + kRingRows - 1) / kRingRows);
  // consecutive slices per CTA (its warps interleaved): a warp changes segment rarely
  const int per = (nslices + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
  const int s_end = min(nslices, (static_cast<int>(blockIdx.x) + 1) * per);
  const uint64_t policy = l2_policy_evict_first();
  const uint32_t below = (1u << lane) - 1u;
  Accum A;
  bool failed = false;

  // lane c < nst copies staged column c: its column at the current segment
  const int* my_col = lane < nst ? P.col[P.r_col[lane]] : nullptr;
  const int* my_src = my_col;
  int cur_vseg = -1;
  auto start = [&](int s, int buf) {
    const unsigned r0 = static_cast<unsigned>(s) * kRingRows;
    unsigned at = r0;
    if (P.gpu_cache != nullptr) {
      const int vseg = static_cast<int>(r0 >> P.seg_shift);
      if (vseg != cur_vseg) {
        cur_vseg = vseg;
        const int seg = P.seg_group ? static_cast<int>(P.seg_group[vseg])
                                    : static_cast<int>((P.start_offset + r0) >> P.seg_shift);
        if (lane < nst) my_src = P.gpu_cache + (static_cast<long long>(__ldg(my_col + seg)) << P.seg_shift);
      }
      at = r0 & ((1u << P.seg_shift) - 1u);
    }
    if (rows - r0 >= kRingRows) {
      if (lane < nst) {
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(&w.bar[buf], kRingRows * 4);
        bulk_g2s(stage + (buf * nst + lane) * kRingRows, my_src + at, kRingRows * 4, &w.bar[buf], policy);
      }
    } else {
      const int have = static_cast<int>(rows - r0);
      for (int c = 0; c < nst; ++c) {
        const int* src = reinterpret_cast<const int*>(
            __shfl_sync(kFull, static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(my_src)), c));
        for (int r = lane; r < have; r += 32) stage[(buf * nst + c) * kRingRows + r] = __ldg(src + at + r);
      }
      __syncwarp();
    }
  };

  wait_for_predecessor();
  if (lane == 0) {
    mbar_init(&w.bar[0], nst);
    mbar_init(&w.bar[1], nst);
    mbar_fence_init();
  }
  __syncwarp();
  int s = static_cast<int>(blockIdx.x) * per + warp;
  if (s < s_end) start(s, 0);
  if (s + nwarps < s_end) start(s + nwarps, 1);
  if (P.gmode == kGroupSmem) {
    for (int g = tid; g < P.total_val; g += blockDim.x) s_sum[g] = 0;
    for (int i = tid; i < (P.total_val + 31) / 32; i += blockDim.x) s_touch[i] = 0;
  }
  for (int p = 0; p < nd; ++p)
    ring_stage_bitmap(P, p, reinterpret_cast<uint32_t*>(smem + P.p_bm_off[p]), warp, nwarps, lane);
  __syncthreads();

  int held = 0;  // rows in the ring
  // the round of the first table probe in flight: its table words (0: no survivor) and rows
  unsigned plo[2] = {0, 0}, phi[2] = {0, 0};
  int prow[2] = {0, 0};
  for (uint32_t it = 0;; ++it, s += nwarps) {
    const bool drain = s >= s_end || failed;  // one more step after the last slice empties the ring
    const int buf = it & 1;
    const int* st = stage + buf * nst * kRingRows;
    int cnt = 0;
    if (!drain) {
      const unsigned left = rows - static_cast<unsigned>(s) * kRingRows;
      uint32_t sel = (1u << kRingItems) - 1u;
      if (left >= kRingRows) {
        const bool ok = mbar_wait_bounded(&w.bar[buf], (it >> 1) & 1u);
        if (!__all_sync(kFull, ok)) failed = true;
      } else {
        sel = 0;
#pragma unroll
        for (int i = 0; i < kRingItems; ++i)
          if (static_cast<unsigned>(((i >> 2) * 32 + lane) * 4 + (i & 3)) < left) sel |= 1u << i;
      }
      if (failed) sel = 0;
      // ---- dense part: bit j * 4 + e of the lane's mask is row (j * 32 + lane) * 4 + e ----
      int v[kRingItems];
      auto load = [&](int c) {
#pragma unroll
        for (int j = 0; j < kRingItems / 4; ++j) {
          const int4 q = lds128(st + c * kRingRows + (j * 32 + lane) * 4);
          v[4 * j] = q.x;
          v[4 * j + 1] = q.y;
          v[4 * j + 2] = q.z;
          v[4 * j + 3] = q.w;
        }
      };
#pragma unroll
      for (int f = 0; f < MB_MAX_FILTERS; ++f) {
        if (f >= nf) break;
        if (P.count_after == f) A.cnt += __popc(sel);
        load(P.r_fcol[f]);
        const int mode = P.f_mode[f], c1 = P.f_c1[f], c2 = P.f_c2[f];
        if (mode == MB_FILTER_BETWEEN) {
          // c1 <= x <= c2  <=>  (unsigned)(x - c1) <= (unsigned)(c2 - c1), for c1 <= c2
          const unsigned span = static_cast<unsigned>(c2) - static_cast<unsigned>(c1);
          if (c2 < c1) sel = 0;
#pragma unroll
          for (int i = 0; i < kRingItems; ++i)
            if (static_cast<unsigned>(v[i]) - static_cast<unsigned>(c1) > span) sel &= ~(1u << i);
        } else {
#pragma unroll
          for (int i = 0; i < kRingItems; ++i)
            if (!pass_filter(v[i], mode, c1, c2)) sel &= ~(1u << i);
        }
      }
      if (P.count_after >= nf) A.cnt += __popc(sel);
#pragma unroll
      for (int p = 0; p < MB_MAX_PROBES; ++p) {
        if (p >= nd) break;
        load(P.r_pcol[p]);
        const uint32_t* bm = reinterpret_cast<const uint32_t*>(smem + P.p_bm_off[p]);
        const unsigned slots = static_cast<unsigned>(P.p_slots[p]), kmin = static_cast<unsigned>(P.p_kmin[p]);
        uint32_t m = 0, top = 0;
#pragma unroll
        for (int i = kRingItems - 1; i >= 0; --i) {
          const unsigned d = static_cast<unsigned>(v[i]) - kmin;
          const unsigned h = min(min(d, d - slots), slots);  // d, one range down, or `slots`
          top = max(top, h);
          m = __funnelshift_l(bm[h >> 5] << (h & 31), m, 1);
        }
        if (top == slots) {
          // some key needs the division (or lies below key_min)
#pragma unroll 1
          for (int i = 0; i < kRingItems; ++i) {
            if (!((sel >> i) & 1u)) continue;
            const int h = pht_slot(st[P.r_pcol[p] * kRingRows + ((i >> 2) * 32 + lane) * 4 + (i & 3)], P.p_slots[p],
                                   P.p_kmin[p]);
            if (h < 0) A.bad_probe = true;
            m &= ~(1u << i);
            if (h >= 0 && ((bm[h >> 5] << (h & 31)) >> 31)) m |= 1u << i;
          }
        }
        sel &= m;
      }
      // ---- compaction: a ballot per item gives the survivors' places ----
#pragma unroll
      for (int i = 0; i < kRingItems; ++i) {
        const bool on = (sel >> i) & 1u;
        const uint32_t b = __ballot_sync(kFull, on);
        if (on) w.off[cnt + __popc(b & below)] = static_cast<uint16_t>((i >> 2) * 128 + lane * 4 + (i & 3));
        cnt += __popc(b);
      }
      __syncwarp();
    }
    int base = 0;
    do {
      // ---- the round probed last: its survivors to the ring ----
      const bool ok0 = (plo[0] | phi[0]) != 0u, ok1 = (plo[1] | phi[1]) != 0u;
      const uint32_t b0 = __ballot_sync(kFull, ok0), b1 = __ballot_sync(kFull, ok1);
      const int add = __popc(b0) + __popc(b1);
      bool pushed = add == 0;
      while (true) {
        if (!pushed && held + add <= kRingCap) {
          const int layout = K ? P.p_layout[P.sp_ord[0]] : MB_HT_KEY;
          if (ok0) w.ring[held + __popc(b0 & below)] = make_int2(ring_payload(layout, plo[0], phi[0]), prow[0]);
          if (ok1)
            w.ring[held + __popc(b0) + __popc(b1 & below)] = make_int2(ring_payload(layout, plo[1], phi[1]), prow[1]);
          held += add;
          pushed = true;
          __syncwarp();
        }
        if (!(held >= 32 || (held > 0 && (drain || !pushed)))) break;
        // ---- the rest of the pipeline for the last rows of the ring, one a lane ----
        const int n = held < 32 ? held : 32;
        held -= n;
        bool live = lane < n;
        const int2 entry = w.ring[held + (live ? lane : 0)];
        const long long r = static_cast<unsigned>(entry.y);
        int gv[MB_MAX_PROBES], a0 = 0, a1 = 0;
#pragma unroll
        for (int q = 0; q < MB_MAX_PROBES; ++q) gv[q] = 0;
        if (K) gv[0] = entry.x;
        constexpr int kQ0 = K ? 1 : 0;
        int seg = 0;
        const int* in_seg = nullptr;
        if (P.gpu_cache == nullptr) {
#pragma unroll
          for (int q = kQ0; q < MB_MAX_PROBES; ++q)
            if (q < ns) gv[q] = gather_ld(P.col[P.p_col[P.sp_ord[q]]] + r);
          if (early) {
            a0 = gather_ld(P.col[P.a_col[0]] + r);
            if (two_cols) a1 = gather_ld(P.col[P.a_col[1]] + r);
          }
        } else {
          const long long vseg = r >> P.seg_shift;
          seg = P.seg_group ? static_cast<int>(P.seg_group[vseg])
                                      : static_cast<int>((P.start_offset + r) >> P.seg_shift);
          in_seg = P.gpu_cache + (r & ((1ll << P.seg_shift) - 1));
#pragma unroll
          for (int q = kQ0; q < MB_MAX_PROBES; ++q)
            if (q < ns) gv[q] = __ldg(P.col[P.p_col[P.sp_ord[q]]] + seg);
          if (early) {
            a0 = __ldg(P.col[P.a_col[0]] + seg);
            if (two_cols) a1 = __ldg(P.col[P.a_col[1]] + seg);
          }
#pragma unroll
          for (int q = kQ0; q < MB_MAX_PROBES; ++q)
            if (q < ns) gv[q] = gather_ld(in_seg + (static_cast<long long>(gv[q]) << P.seg_shift));
          if (early) {
            a0 = gather_ld(in_seg + (static_cast<long long>(a0) << P.seg_shift));
            if (two_cols) a1 = gather_ld(in_seg + (static_cast<long long>(a1) << P.seg_shift));
          }
        }
        unsigned lo[MB_MAX_PROBES], hi[MB_MAX_PROBES];
        bool below_min[MB_MAX_PROBES];
#pragma unroll
        for (int q = kQ0; q < MB_MAX_PROBES; ++q) {
          lo[q] = hi[q] = 0;
          below_min[q] = false;
          if (q < ns) {
            const int p = P.sp_ord[q];
            const int h = pht_slot(gv[q], P.p_slots[p], P.p_kmin[p]);
            below_min[q] = h < 0;
            ring_word(P.p_ht[p], P.p_layout[p] == MB_HT_KEY, h, h >= 0, lo[q], hi[q]);
          }
        }
#pragma unroll
        for (int q = kQ0; q < MB_MAX_PROBES; ++q) {
          if (q >= ns) continue;
          if (live && below_min[q]) A.bad_probe = true;
          live = live && (lo[q] | hi[q]) != 0u;
          gv[q] = ring_payload(P.p_layout[P.sp_ord[q]], lo[q], hi[q]);
        }
        if (live) {
          if (P.count_after < 0) ++A.cnt;
          if (!early) {
            if (P.gpu_cache == nullptr) {
              a0 = gather_ld(P.col[P.a_col[0]] + r);
              if (two_cols) a1 = gather_ld(P.col[P.a_col[1]] + r);
            } else {
              a0 = __ldg(P.col[P.a_col[0]] + seg);
              if (two_cols) a1 = __ldg(P.col[P.a_col[1]] + seg);
              a0 = gather_ld(in_seg + (static_cast<long long>(a0) << P.seg_shift));
              if (two_cols) a1 = gather_ld(in_seg + (static_cast<long long>(a1) << P.seg_shift));
            }
          }
          const unsigned u0 = static_cast<unsigned>(a0), u1 = static_cast<unsigned>(a1);
          const int val = static_cast<int>(P.agg_op == MB_AGG_SUM ? u0 : P.agg_op == MB_AGG_SUB ? u0 - u1 : u0 * u1);
          if (P.gmode == kGroupScalar) {
            A.acc += static_cast<unsigned long long>(static_cast<long long>(val));
          } else {
            unsigned hh = bias;
#pragma unroll
            for (int q = 0; q < MB_MAX_PROBES; ++q)
              if (q < ns)
                hh += (static_cast<unsigned>(gv[q]) - static_cast<unsigned>(P.p_min[P.sp_ord[q]])) *
                      static_cast<unsigned>(P.p_mul[P.sp_ord[q]]);
            ring_add(P, hh, val, ns, s_sum, s_touch, A.bad_group, [&](int q) { return gv[q]; });
          }
        }
        __syncwarp();  // the rows are read before others take their places
      }
      // ---- the next round of the first table probe: entries base + r * 32 + lane of the
      // survivors (an absent one reads row 0). Its table words are looked at when the next
      // round begins, after the next slice's dense part where this was the slice's last ----
      plo[0] = phi[0] = plo[1] = phi[1] = 0;
      if (!drain) {
        int row[2], key[2];
        bool ok[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int e = base + r * 32 + lane;
          ok[r] = e < cnt;
          row[r] = ok[r] ? w.off[e] : 0;
          key[r] = K ? st[P.r_kcol * kRingRows + row[r]] : 0;
        }
        if (base + kRingRound >= cnt) {
          __syncwarp();  // the buffer has been read: another slice may land on it
          if (s + 2 * nwarps < s_end && !failed) start(s + 2 * nwarps, buf);
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          prow[r] = static_cast<int>(static_cast<unsigned>(s) * kRingRows + static_cast<unsigned>(row[r]));
          if (K) {
            const int p = P.sp_ord[0];
            const int h = pht_slot(key[r], P.p_slots[p], P.p_kmin[p]);
            if (h < 0 && ok[r]) A.bad_probe = true;
            ring_word(P.p_ht[p], P.p_layout[p] == MB_HT_KEY, h, ok[r] && h >= 0, plo[r], phi[r]);
          } else {
            plo[r] = ok[r] ? 1u : 0u;
          }
        }
      }
      base += kRingRound;
    } while (base < cnt);
    if (drain) break;
  }
  if (failed) {
    // no copy may land after the CTA is gone: give the ones in flight another (bounded) while
    mbar_wait_bounded(&w.bar[0], 0);
    mbar_wait_bounded(&w.bar[0], 1);
    mbar_wait_bounded(&w.bar[1], 0);
    mbar_wait_bounded(&w.bar[1], 1);
    set_status(P.status, MB_STATUS_TIMEOUT);
  }
  if (A.bad_probe) set_status(P.status, MB_STATUS_PROBE_RANGE);
  if (A.bad_group) set_status(P.status, MB_STATUS_GROUP_RANGE);

  // ---- publish -------------------------------------------------------------------
  unsigned long long acc = A.acc, cnt = A.cnt;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    acc += __shfl_down_sync(kFull, acc, o);
    cnt += __shfl_down_sync(kFull, cnt, o);
  }
  if (lane == 0) {
    s_red[warp] = acc;
    s_red[kRingMaxWarps + warp] = cnt;
  }
  __syncthreads();
  if (tid == 0) {
    unsigned long long ta = 0, tc = 0;
    for (int i = 0; i < nwarps; ++i) {
      ta += s_red[i];
      tc += s_red[kRingMaxWarps + i];
    }
    if (P.gmode == kGroupScalar && ta != 0) atomicAdd(static_cast<unsigned long long*>(P.res), ta);
    if (P.count != nullptr && tc != 0) {
      if (P.count32)
        atomicAdd(static_cast<int*>(P.count), static_cast<int>(tc));
      else
        atomicAdd(static_cast<unsigned long long*>(P.count), tc);
    }
  }
  if (P.gmode == kGroupSmem) {
    for (int g = tid; g < P.total_val; g += blockDim.x)
      if ((s_touch[g >> 5] >> (g & 31)) & 1u) atomicAdd(group_sum_ptr(P, g), s_sum[g]);
  }
}

// [filters: 0, any][leading bitmap probes: 0, 1, any][table probe before the ring]
static const KernelFn kRing[2][3][2] = {
    {{star_ring_kernel<0, 0, false>, star_ring_kernel<0, 0, true>},
     {star_ring_kernel<0, 1, false>, star_ring_kernel<0, 1, true>},
     {star_ring_kernel<0, -1, false>, star_ring_kernel<0, -1, true>}},
    {{star_ring_kernel<-1, 0, false>, star_ring_kernel<-1, 0, true>},
     {star_ring_kernel<-1, 1, false>, star_ring_kernel<-1, 1, true>},
     {star_ring_kernel<-1, -1, false>, star_ring_kernel<-1, -1, true>}}};

int ring_init_device(const DeviceState& ds) {
  for (const auto& of_filters : kRing)
    for (const auto& of_dense : of_filters)
      for (KernelFn fn : of_dense)
        if (cudaFuncSetAttribute(reinterpret_cast<const void*>(fn), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 ds.max_smem_optin - 2048) != cudaSuccess)
          return MB_ERR_CUDA;
  return MB_OK;
}

int launch_ring(StarPlan& P, int group_mode, const DeviceState& ds, cudaStream_t stream) {
  // Leading probes decided by a bitmap: given by the caller, or derived by every CTA from a table
  // it reads whole — a small one, and not for a handful of rows. A call with the first probe
  // (40,000 slots) derived against looked up in L2 row by row: Query A over 120,000,000 rows 361
  // against 865 us, Query B 375 and 954; the engine's group-by (8-byte slots) over 23 segments 137
  // and 238. Key tables gain at every size measured, down to 2 rows a slot (four probes, 80,000
  // rows: 11.2 and 13.5 us), tables of 8-byte slots up to 20,000 slots likewise (three probes that
  // keep 20 %, 160,000 rows, 20,000 slots: 10.8 and 12.5), 40,000 of them from some 32 rows a slot
  // on (1,000,000 rows 15.3 and 14.0, 1,300,000 rows 18.4 and 21.4).
  P.n_dense = P.sparse_p0 = 0;
  P.dense_bias = 0;
  int off = 0;
  if (P.res_layout == MB_RES_SCALAR)
    P.gmode = kGroupScalar;
  else if (group_mode == 2 || P.total_val > kSmemGroupMax)
    P.gmode = kGroupGlobal;
  else
    P.gmode = kGroupSmem;
  P.smem_groups_off = off;
  if (P.gmode == kGroupSmem) off += (8 * P.total_val + 4 * ((P.total_val + 31) / 32) + 15) / 16 * 16;
  int bm_total = 0;
  int read[MB_MAX_PROBES], nread = 0;  // bitmap probes whose payload somebody reads
  for (int p = 0; p < P.np; ++p) {
    P.p_bm_off[p] = -1;
    P.p_bm_words[p] = 0;
    if (P.n_dense < p) continue;
    const int bytes = (P.p_slots[p] / 32 + 1) * 4;  // slots 0 .. p_slots (the last one absent)
    const int derive_max = P.p_layout[p] == MB_HT_KEY ? 8 * kBitmapSmemMaxBytes : kBitmapDeriveMaxSlots8;
    const int rows_a_slot = P.p_layout[p] == MB_HT_KEY || P.p_slots[p] <= 20'000 ? 4 : 32;
    const bool have = P.p_presence[p] != nullptr || (P.p_slots[p] <= derive_max && P.n / rows_a_slot >= P.p_slots[p]);
    if (!have || bytes > kBitmapSmemMaxBytes + 4 || bm_total + bytes > kBitmapSmemTotalBytes) continue;
    P.p_bm_off[p] = off + bm_total;
    P.p_bm_words[p] = bytes / 4;
    bm_total += (bytes + 15) / 16 * 16;
    P.n_dense = p + 1;
    // one whose payload nobody reads is settled by its bit, wherever it stands: its group term is
    // a constant (24,000,000 rows, a date table before a 40,000-slot key table and a third probe:
    // 82 us with a fifth of the rows kept by each and 607 with all of them kept when the key table
    // was looked up again, now 79 and 414; the tile kernels 182 and 514)
    if (P.p_layout[p] == MB_HT_KEY || (P.p_mul[p] == 0 && P.p_res_slot[p] < 0)) {
      ++P.sparse_p0;
      P.dense_bias += (0u - static_cast<unsigned>(P.p_min[p])) * static_cast<unsigned>(P.p_mul[p]);
    } else {
      read[nread++] = p;
    }
  }
  off = (off + bm_total + 127) / 128 * 128;
  P.smem_list_off = off;
  // visiting order of the others: chain order, except that the first probe without a bitmap
  // leads (the bitmap probes are read for their payloads only); it runs before the ring
  const bool key = P.n_dense < P.np;
  int ns = 0;
  if (key) P.sp_ord[ns++] = P.n_dense;
  for (int i = 0; i < nread; ++i) P.sp_ord[ns++] = read[i];
  for (int p = P.n_dense + 1; p < P.np; ++p) P.sp_ord[ns++] = p;
  // staged columns
  P.r_nst = 0;
  auto staged = [&](int c) {
    for (int i = 0; i < P.r_nst; ++i)
      if (P.r_col[i] == c) return i;
    P.r_col[P.r_nst] = c;
    return P.r_nst++;
  };
  for (int f = 0; f < P.nf; ++f) P.r_fcol[f] = staged(P.f_col[f]);
  for (int p = 0; p < P.n_dense; ++p) P.r_pcol[p] = staged(P.p_col[p]);
  P.r_kcol = key ? staged(P.p_col[P.sp_ord[0]]) : 0;
  // one CTA an SM with as many warps as their buffers leave room for (also where fewer
  // have a slice: they help to derive the bitmaps — as many warps as slices took 13.9 against 11.9 us
  // for four probes over 600,000 rows); short calls spread over the SMs first
  const int budget = ds.max_smem_optin - 2048 - static_cast<int>(2 * kRingMaxWarps * sizeof(unsigned long long));
  int warps = (budget - off) / ring_warp_bytes(P.r_nst);
  if (warps > kRingMaxWarps) warps = kRingMaxWarps;
  if (warps < 4) return MB_ERR_SIZE;
  const long long nslices = (P.n + kRingRows - 1) / kRingRows;
  long long blocks = (nslices + 3) / 4;
  if (blocks > ds.num_sms) blocks = ds.num_sms;
  P.smem_total = off + warps * ring_warp_bytes(P.r_nst);
  const KernelFn fn = kRing[P.nf > 0 ? 1 : 0][P.n_dense > 1 ? 2 : P.n_dense][key ? 1 : 0];
  if (launch_dependent(fn, static_cast<int>(blocks), warps * 32, static_cast<size_t>(P.smem_total), stream, P) !=
      cudaSuccess)
    return MB_ERR_LAUNCH;
  note_launches(1);
  return MB_OK;
}

}  // namespace mb

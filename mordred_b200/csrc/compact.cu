// compact.cu — selection with compaction: the rows of a fact range (or of an input
// offset list) that pass a query's filters and probes, written out as an offset list of
// physical rows plus, per probe, the dimension offset or payload the probe found.
//
// This is the handoff of CPU/GPU split execution: when a query's filters and probes run
// on the GPU but its aggregation runs on the CPU (or the other way round), the survivors
// cross PCIe as offset lists (src/gpudb/CPUGPUProcessing.cu:60-144 switch_device_fact).
// Restates the reference's compaction kernels filter_GPU2/3, filter_probe_GPU2/3 and
// probe_GPU2/3 (src/gpudb/GPUProcessing.h:496-925, 1174-1383), which scan per block and
// take one atomicAdd on the output cursor per block; here a warp takes one for each 64 rows it
// has queued (contiguous rows) or for the survivors among 32 rows (listed rows, small segments),
// so the list order is not deterministic (it never is in the reference either) while its set of
// rows is.
//
// Probe outputs per layout: MB_HT_VAL_OFF (engine builds) — present when the row word
// ht[2h+1] != 0, output ht[2h+1] - 1, the dimension row (BlockLibrary.cuh:9-33);
// MB_HT_KEY_VAL — present when the 8-byte slot != 0, output the payload; MB_HT_KEY —
// present when ht[h] != 0, output 0.
#include "common.cuh"

namespace mb {

struct SelPlan {
  long long n;               // virtual rows, or entries of in_rows
  const int* in_rows;        // physical-row input list (list form), or null
  const int* in_dim[4];      // list form: dimension offsets passed through to dim slots not probed here
  int nf;
  const int* fcol[MB_MAX_FILTERS];
  int fmode[MB_MAX_FILTERS], fc1[MB_MAX_FILTERS], fc2[MB_MAX_FILTERS];
  int np;
  const int* pkey[MB_MAX_PROBES];
  const int* pht[MB_MAX_PROBES];
  int pslots[MB_MAX_PROBES], pkmin[MB_MAX_PROBES], playout[MB_MAX_PROBES];
  int slot_src[4];           // output dim slot j <- probe index, or -1: pass in_dim[j] through
  int* dim_out[4];
  int* lo_off;
  int* total;
  long long capacity;        // entries the output lists hold
  const int* gpu_cache;      // segment addressing (column fields are slot-index arrays)
  const short* seg_group;
  long long start_offset;
  int seg_shift;
  unsigned int* status;
  // sliced kernel: rows a slice, whether the columns read ahead allow 16-byte loads, and the
  // words of the first probe's presence bitmap (0: none)
  int slice_rows;
  int vec;
  int bm_words;
};

__device__ __forceinline__ bool sel_pass(int x, int mode, int c1, int c2) {
  return mode == MB_FILTER_BETWEEN ? (x >= c1 && x <= c2) : mode == MB_FILTER_EQ ? x == c1 : (x == c1 || x == c2);
}

// ---- contiguous rows: slices of 512 ------------------------------------------------------
// A warp takes slices of 512 consecutive rows, 16 a lane (of 64 to 256 in short calls). The columns every row needs — the
// filters, and the first probe's key where its table is small enough for a presence bitmap
// in shared memory (derived once per CTA) — arrive by bulk copies into the warp's own buffer,
// and so does the key of the first probe after those while at least one row in 16 of the
// warp's last slice came to it (its 32-byte sectors would nearly all be fetched anyway, at a
// DRAM latency per round). The dense part turns the columns into a bit mask a lane; the
// survivors are compacted and the remaining probes' table loads (and later key gathers) run
// over full lanes, two rows a lane, each only for the rows the probes before it left (for every
// row of a round, 24,000,000 rows, a 1,000,000-slot table that keeps 5 % and a date table took 245
// us, and 163 now; one row a lane 194). The next slice's copies go out as soon as the last
// round's keys are in registers, to land under its table loads and the output. Rows
// that pass everything wait in the warp's queue and leave 64 at a time: one atomicAdd on the
// list cursor and full 128-byte stores per 64 rows; a probe the bitmap decided reads its
// output there.
// 24,000,000 rows with a date filter and two probes: 85 us, bound by instruction issue and the
// L2 trips of a round (1.9 warp instructions a row, 51 % issue; DRAM 293 MB, 3.4 TB/s). One
// row a lane with every load behind a branch, and an atomic per 32 rows: 8.8 warp
// instructions a row, 448 us.
constexpr int kSelMaxWarps = 32;          // one CTA an SM: the bitmap is derived once an SM
constexpr int kSelItems = 16;             // rows a lane
constexpr int kSelRows = 32 * kSelItems;  // rows per slice, at most
constexpr int kSelRound = 64;             // survivors probed at a time (two a lane)
constexpr int kSelQueue = 2 * kSelRound;  // rows a warp's output queue holds
constexpr int kSelBitmapMaxSlots = 65536;

template <int NC>
struct __align__(16) SelWarp {
  int stage[NC > 0 ? NC : 1][kSelRows];   // the slice's staged columns
  int q[1 + MB_MAX_PROBES][kSelQueue];    // physical row, probe outputs (the bitmap probe's key)
  const int* col[2][8];                   // columns at the current and the next slice's segment: filters, probe keys
  uint16_t off[kSelRows];                 // survivors: their rows within the slice
  uint64_t bar;
};

// The word(s) of slot h (>= 0): present, and the probe's output.
__device__ __forceinline__ bool sel_lookup(const int* ht, int layout, int h, int& out) {
  if (layout == MB_HT_KEY_VAL) {
    const unsigned long long s = ld_word2(ht + 2ll * h);
    out = static_cast<int>(s >> 32);
    return s != 0;
  }
  const int w = ld_word(layout == MB_HT_KEY ? ht + h : ht + 2ll * h + 1);
  out = layout == MB_HT_KEY ? 0 : w - 1;
  return w != 0;
}

// lo, hi = the word(s) of slot h >= 0 that tell a row's presence and output, if `on` (else left
// alone): only the loads, so that nothing waits for them before their first use.
__device__ __forceinline__ void sel_word(const int* ht, int layout, int h, bool on, unsigned& lo, unsigned& hi) {
  asm volatile(
      "{\n\t.reg .pred k, v;\n\t"
      "setp.eq.u32 k, %4, 1;\n\t"
      "setp.eq.u32 v, %4, 2;\n\t"
      "@k ld.global.u32 %0, [%2];\n\t"
      "@v ld.global.v2.u32 {%0, %1}, [%3];\n\t}"
      : "+r"(lo), "+r"(hi)
      : "l"(layout == MB_HT_KEY ? ht + h : ht + 2ll * h + 1), "l"(ht + 2ll * h),
        "r"(!on ? 0u : layout == MB_HT_KEY_VAL ? 2u : 1u));
}

// Writes `n` (<= 64) queued rows to the output lists.
template <bool BM, class W>
__device__ __forceinline__ void sel_flush(const SelPlan& P, const W& w, int n, int lane, bool& overflow) {
  int b0 = 0;
  if (lane == 0) b0 = atomicAdd(P.total, n);
  b0 = __shfl_sync(0xffffffffu, b0, 0);
#pragma unroll
  for (int r = 0; r < kSelRound / 32; ++r) {
    const int e = r * 32 + lane;
    if (e >= n) continue;
    const long long pos = static_cast<long long>(b0) + e;
    if (pos >= P.capacity) {
      overflow = true;
      continue;
    }
    P.lo_off[pos] = w.q[0][e];
#pragma unroll
    for (int j = 0; j < MB_MAX_PROBES; ++j) {
      if (P.dim_out[j] == nullptr) continue;
      const int src = P.slot_src[j];
      int v = src >= 0 ? w.q[1 + src][e] : 0;
      if (BM && src == 0) sel_lookup(P.pht[0], P.playout[0], pht_slot(v, P.pslots[0], P.pkmin[0]), v);
      P.dim_out[j][pos] = v;
    }
  }
}

// Staged columns: NF filters, then (BM) the key of the first probe, which is decided by the
// bitmap, then (K) the key of the first probe after that. The bitmap holds slot s at bit 31 - s % 32, so that a shift left by s puts it at
// the top and a funnel shift moves it into the lane's mask; its bit `slots` is 0 and stands
// for every key outside [key_min, key_min + 2 * slots), which one check per slice catches.
template <int NF, bool BM, bool K>
__global__ void __launch_bounds__(kSelMaxWarps * 32, 1) select_slices_kernel(const __grid_constant__ SelPlan P) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int ND = NF + (BM ? 1 : 0);  // columns of the dense part
  constexpr int NC = ND + (K ? 1 : 0);
  constexpr int kFirst = BM ? 1 : 0;     // the first probe of the sparse part
  using W = SelWarp<NC>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  W& w = reinterpret_cast<W*>(smem)[warp];
  uint32_t* bm = reinterpret_cast<uint32_t*>(smem + nwarps * sizeof(W));
  const int rows = P.slice_rows;
  const long long nslices = (P.n + rows - 1) / rows;
  // consecutive slices per CTA (its warps interleaved): a warp changes segment rarely
  const long long per = (nslices + gridDim.x - 1) / gridDim.x;
  const long long s_end = min(nslices, (blockIdx.x + 1) * per);
  const uint64_t policy = l2_policy_evict_first();
  bool bad_probe = false, overflow = false, failed = false;
  int queued = 0;
  uint32_t parity = 0;  // of the barrier's next phase
  bool in_flight = false, staged = true;  // `staged`: the slice started last has its key K
  int tab = 0;          // pointer table of the slice located last
  long long tab_vseg = -1, tab_seg = 0;      // its segment in the call, and the table's
  long long phys0 = 0, idx0 = 0;             // physical row and column index of its first row

  // Locate slice s and start its copies (or, where they do not apply, load it).
  auto start = [&](long long s) {
    const long long r0 = s * rows;
    const bool list = P.seg_group != nullptr;
    const long long v0 = list ? r0 : P.start_offset + r0;
    const long long vseg = P.gpu_cache == nullptr ? 0 : v0 >> P.seg_shift;
    if (vseg != tab_vseg) {
      tab ^= 1;  // the other table still serves the slice being worked on
      tab_vseg = vseg;
      tab_seg = list ? P.seg_group[vseg] : vseg;
      if (lane < P.nf + P.np) {
        const int* c = lane < P.nf ? P.fcol[lane] : P.pkey[lane - P.nf];
        w.col[tab][lane] =
            P.gpu_cache == nullptr ? c : P.gpu_cache + (static_cast<long long>(__ldg(c + tab_seg)) << P.seg_shift);
      }
    }
    idx0 = P.gpu_cache == nullptr ? r0 : v0 & ((1ll << P.seg_shift) - 1);
    phys0 = P.gpu_cache == nullptr ? v0 : (tab_seg << P.seg_shift) + idx0;
    __syncwarp();
    if (NC == 0) return;
    in_flight = P.vec && r0 + rows <= P.n && (ND > 0 || staged);
    if (in_flight) {
      if (lane == 0) {
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(&w.bar, (staged ? NC : ND) * rows * 4);
#pragma unroll
        for (int c = 0; c < NC; ++c)
          if (c < ND || staged) bulk_g2s(w.stage[c], w.col[tab][c] + idx0, rows * 4, &w.bar, policy);
      }
    } else {
      const int have = static_cast<int>(min(static_cast<long long>(rows), P.n - r0));
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int* col = w.col[tab][c] + idx0;
        for (int r = lane; r < have && (c < ND || staged); r += 32) w.stage[c][r] = __ldg(col + r);
      }
      __syncwarp();
    }
  };

  wait_for_predecessor();
  if (lane == 0) {
    mbar_init(&w.bar, 1);
    mbar_fence_init();
  }
  __syncwarp();
  long long s = blockIdx.x * per + warp;
  if (s < s_end) start(s);
  if (BM) {
    // slot s of the first probe's table is present when its word (VAL_OFF: the row word) is
    // nonzero; a warp folds 64 consecutive slots into two words: a lane loads two slots (16
    // bytes of an 8-byte-slot table), and the ballots over even and odd slots interleave
    const int* ht = P.pht[0];
    const int slots = P.pslots[0], layout = P.playout[0];
    auto present = [&](int h) {
      if (h >= slots) return false;
      return layout == MB_HT_KEY       ? ld_word(ht + h) != 0
             : layout == MB_HT_VAL_OFF ? ld_word(ht + 2ll * h + 1) != 0
                                       : ld_word2(ht + 2ll * h) != 0ull;
    };
    const bool pairs = layout != MB_HT_KEY && (reinterpret_cast<uintptr_t>(ht) & 15u) == 0;
#pragma unroll 8
    for (int word = 2 * warp; word < P.bm_words; word += 2 * nwarps) {
      const int h = word * 32 + 2 * lane;
      bool even, odd;
      if (pairs && h + 1 < slots) {
        const int4 t = ld_word4(ht + 2ll * h);
        even = layout == MB_HT_VAL_OFF ? t.y != 0 : (t.x | t.y) != 0;
        odd = layout == MB_HT_VAL_OFF ? t.w != 0 : (t.z | t.w) != 0;
      } else {
        even = present(h);
        odd = present(h + 1);
      }
      const uint32_t be = __ballot_sync(0xffffffffu, even), bo = __ballot_sync(0xffffffffu, odd);
      if (lane < 2 && word + lane < P.bm_words) {
        auto spread = [](uint32_t x) {  // bit i of the low half to bit 2i
          x = (x | (x << 8)) & 0x00ff00ffu;
          x = (x | (x << 4)) & 0x0f0f0f0fu;
          x = (x | (x << 2)) & 0x33333333u;
          return (x | (x << 1)) & 0x55555555u;
        };
        bm[word + lane] = __brev(spread((be >> (16 * lane)) & 0xffffu) | (spread((bo >> (16 * lane)) & 0xffffu) << 1));
      }
    }
    __syncthreads();
  }
  for (; s < s_end; s += nwarps) {
    const long long phys = phys0, idx = idx0;
    const bool staged_now = staged;
    const int* const* cols = w.col[tab];
    const int have = static_cast<int>(min(static_cast<long long>(rows), P.n - s * rows));
    if (NC > 0 && in_flight) {
      const bool ok = mbar_wait_bounded(&w.bar, parity);
      parity ^= 1u;
      if (!__all_sync(0xffffffffu, ok)) {
        failed = true;
        break;
      }
    }
    // ---- dense part: bit j * 4 + e of the lane's mask is row (j * 32 + lane) * 4 + e ----
    uint32_t sel = (1u << kSelItems) - 1u;
    if (have < kSelRows) {
      sel = 0;
#pragma unroll
      for (int i = 0; i < kSelItems; ++i)
        if (((i >> 2) * 32 + lane) * 4 + (i & 3) < have) sel |= 1u << i;
    }
    int v[kSelItems];
    auto load = [&](int c) {
#pragma unroll
      for (int j = 0; j < kSelItems / 4; ++j) {
        const int4 q = lds128(&w.stage[c][(j * 32 + lane) * 4]);
        v[4 * j] = q.x;
        v[4 * j + 1] = q.y;
        v[4 * j + 2] = q.z;
        v[4 * j + 3] = q.w;
      }
    };
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      load(f);
      const int mode = P.fmode[f], c1 = P.fc1[f], c2 = P.fc2[f];
      if (mode == MB_FILTER_BETWEEN) {
        // c1 <= x <= c2  <=>  (unsigned)(x - c1) <= (unsigned)(c2 - c1), for c1 <= c2
        const unsigned span = static_cast<unsigned>(c2) - static_cast<unsigned>(c1);
        if (c2 < c1) sel = 0;
#pragma unroll
        for (int i = 0; i < kSelItems; ++i)
          if (static_cast<unsigned>(v[i]) - static_cast<unsigned>(c1) > span) sel &= ~(1u << i);
      } else {
#pragma unroll
        for (int i = 0; i < kSelItems; ++i)
          if (!sel_pass(v[i], mode, c1, c2)) sel &= ~(1u << i);
      }
    }
    if (BM) {
      load(NF);
      const unsigned slots = static_cast<unsigned>(P.pslots[0]), kmin = static_cast<unsigned>(P.pkmin[0]);
      uint32_t m = 0, top = 0;
#pragma unroll
      for (int i = kSelItems - 1; i >= 0; --i) {
        const unsigned d = static_cast<unsigned>(v[i]) - kmin;
        const unsigned h = min(min(d, d - slots), slots);  // d, one range down, or `slots`
        top = max(top, h);
        m = __funnelshift_l(bm[h >> 5] << (h & 31), m, 1);
      }
      if (top == slots) {
        // some key needs the division (or lies below key_min)
#pragma unroll 1
        for (int i = 0; i < kSelItems; ++i) {
          if (!((sel >> i) & 1u)) continue;
          const int h = pht_slot(w.stage[NF][((i >> 2) * 32 + lane) * 4 + (i & 3)], P.pslots[0], P.pkmin[0]);
          if (h < 0) bad_probe = true;
          m &= ~(1u << i);
          if (h >= 0 && ((bm[h >> 5] << (h & 31)) >> 31)) m |= 1u << i;
        }
      }
      sel &= m;
    }
    // ---- compaction: lane by lane, positions from a warp prefix sum ----
    int incl = __popc(sel);
    const int own = incl;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    const int cnt = __shfl_sync(0xffffffffu, incl, 31);
    staged = cnt >= rows / 16;
    uint16_t* at = w.off + (incl - own);
    while (sel) {
      const int i = __ffs(sel) - 1;
      sel &= sel - 1;
      *at++ = static_cast<uint16_t>((i >> 2) * 128 + lane * 4 + (i & 3));
    }
    __syncwarp();
    // ---- sparse part: rounds of 64 survivors, entries base + r * 32 + lane (an absent one
    // reads row 0). Each candidate's words go to queue position queued + r * 32 + lane, from
    // where the rows that pass every probe close up ----
    int base = 0;
    do {
      const bool two = cnt - base > 32;
      int row[2], h[2];
      bool ok[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int e = base + r * 32 + lane;
        ok[r] = e < cnt;
        row[r] = ok[r] ? w.off[e] : 0;
        h[r] = 0;
      }
      int* q = &w.q[0][queued + lane];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        if (r == 1 && !two) break;
        q[r * 32] = static_cast<int>(phys) + row[r];
        if (BM) q[kSelQueue + r * 32] = w.stage[NF][row[r]];  // its key: looked up on the way out
        if (K) h[r] = staged_now ? w.stage[ND][row[r]] : gather_ld(cols[NF + kFirst] + idx + row[r]);
      }
      if (base + kSelRound >= cnt) {
        __syncwarp();  // the buffer has been read: the next slice may land on it
        if (s + nwarps < s_end) start(s + nwarps);
        if (cnt == 0) break;
      }
      if (K) {
#pragma unroll 1
        for (int p = kFirst; p < P.np; ++p) {
          const int layout = P.playout[p], slots = P.pslots[p], kmin = P.pkmin[p];
          const int* ht = P.pht[p];
          if (p > kFirst) {
            if (!__any_sync(0xffffffffu, ok[0] || ok[1])) break;
            const int* col = cols[NF + p] + idx;
#pragma unroll
            for (int r = 0; r < 2; ++r) h[r] = ok[r] ? gather_ld(col + row[r]) : 0;
          }
          unsigned lo[2] = {0, 0}, hi[2] = {0, 0};
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            h[r] = pht_slot(h[r], slots, kmin);
            if (h[r] < 0 && ok[r]) bad_probe = true;
            ok[r] = ok[r] && h[r] >= 0;
            sel_word(ht, layout, h[r], ok[r], lo[r], hi[r]);
          }
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            ok[r] = (lo[r] | hi[r]) != 0;
            if (ok[r])
              q[(1 + p) * kSelQueue + r * 32] =
                  layout == MB_HT_KEY_VAL ? static_cast<int>(hi[r]) : layout == MB_HT_KEY ? 0 : static_cast<int>(lo[r]) - 1;
          }
        }
      }
      const uint32_t b0 = __ballot_sync(0xffffffffu, ok[0]), b1 = __ballot_sync(0xffffffffu, ok[1]);
      base += kSelRound;
      if ((b0 | b1) == 0) continue;
      const uint32_t below = (1u << lane) - 1u;
      const int to0 = queued + __popc(b0 & below), to1 = queued + __popc(b0) + __popc(b1 & below);
#pragma unroll 1
      for (int j = 0; j <= P.np; ++j) {
        const int v0 = q[j * kSelQueue], v1 = q[j * kSelQueue + 32];
        __syncwarp();
        if (ok[0]) w.q[j][to0] = v0;
        if (ok[1]) w.q[j][to1] = v1;
      }
      queued += __popc(b0) + __popc(b1);
      __syncwarp();
      if (queued >= kSelRound) {
        sel_flush<BM>(P, w, kSelRound, lane, overflow);
        __syncwarp();
        // the rows beyond the first 64 move to the front
        queued -= kSelRound;
#pragma unroll
        for (int r = 0; r < kSelRound / 32; ++r)
          if (r * 32 + lane < queued)
            for (int j = 0; j <= P.np; ++j) w.q[j][r * 32 + lane] = w.q[j][kSelRound + r * 32 + lane];
        __syncwarp();
      }
    } while (base < cnt);
    __syncwarp();
  }
  if (failed) {
    mbar_wait_bounded(&w.bar, parity ^ 1u);  // no copy may land after the CTA is gone
    set_status(P.status, MB_STATUS_TIMEOUT);
  }
  if (queued > 0) sel_flush<BM>(P, w, queued, lane, overflow);
  if (bad_probe) set_status(P.status, MB_STATUS_PROBE_RANGE);
  if (overflow) set_status(P.status, MB_STATUS_OVERFLOW);
}

// ---- listed rows, and segments the slices do not divide: one row a lane at a time ----------
template <int ITEMS>
__global__ void __launch_bounds__(256) select_kernel(const __grid_constant__ SelPlan P) {
  const int lane = threadIdx.x & 31;
  const long long gwarp = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5;
  const long long nwarps = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  const long long S = 1ll << P.seg_shift;
  bool bad_probe = false, overflow = false;
  for (long long base = gwarp * 32 * ITEMS; base < P.n; base += nwarps * 32 * ITEMS) {
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
      const long long i = base + it * 32 + lane;
      bool ok = i < P.n;
      long long phys = 0, idx = 0;  // physical row; column index (plain) or in-segment offset
      int seg = 0;
      if (ok) {
        if (P.in_rows) {
          phys = P.in_rows[i];
        } else if (P.gpu_cache && P.seg_group) {
          phys = (static_cast<long long>(P.seg_group[i >> P.seg_shift]) << P.seg_shift) + (i & (S - 1));
        } else {
          phys = P.start_offset + i;
        }
        if (P.gpu_cache) {
          seg = static_cast<int>(phys >> P.seg_shift);
          idx = phys & (S - 1);
        } else {
          idx = phys - P.start_offset;
        }
      }
      auto load = [&](const int* col) -> int {
        if (P.gpu_cache) return __ldg(P.gpu_cache + (static_cast<long long>(__ldg(col + seg)) << P.seg_shift) + idx);
        return __ldg(col + idx);
      };
      for (int f = 0; f < P.nf; ++f)
        if (ok) ok = sel_pass(load(P.fcol[f]), P.fmode[f], P.fc1[f], P.fc2[f]);
      int outv[MB_MAX_PROBES] = {0, 0, 0, 0};
      for (int p = 0; p < P.np; ++p) {
        if (!ok) break;
        const int h = pht_slot(load(P.pkey[p]), P.pslots[p], P.pkmin[p]);
        if (h < 0) {
          bad_probe = true;
          ok = false;
          break;
        }
        const int* ht = P.pht[p];
        if (P.playout[p] == MB_HT_KEY) {
          ok = ld_word(ht + h) != 0;
        } else if (P.playout[p] == MB_HT_VAL_OFF) {
          const int w = ld_word(ht + 2ll * h + 1);
          ok = w != 0;
          outv[p] = w - 1;
        } else {
          const unsigned long long s = ld_word2(ht + 2ll * h);
          ok = s != 0;
          outv[p] = static_cast<int>(s >> 32);
        }
      }
      const unsigned m = __ballot_sync(0xffffffffu, ok);
      if (m == 0) continue;
      int b0 = 0;
      if (lane == 0) b0 = atomicAdd(P.total, __popc(m));
      b0 = __shfl_sync(0xffffffffu, b0, 0);
      if (!ok) continue;
      const long long pos = static_cast<long long>(b0) + __popc(m & ((1u << lane) - 1u));
      if (pos >= P.capacity) {
        overflow = true;
        continue;
      }
      P.lo_off[pos] = static_cast<int>(phys);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (P.dim_out[j] == nullptr) continue;
        const int src = P.slot_src[j];
        P.dim_out[j][pos] = src >= 0 ? outv[src] : (P.in_dim[j] ? P.in_dim[j][i] : 0);
      }
    }
  }
  if (bad_probe) set_status(P.status, MB_STATUS_PROBE_RANGE);
  if (overflow) set_status(P.status, MB_STATUS_OVERFLOW);
}

using SelFn = void (*)(SelPlan);
#define MB_SELECT_VARIANTS(NF) \
  {select_slices_kernel<NF, false, false>, select_slices_kernel<NF, false, true>, \
   select_slices_kernel<NF, true, false>, select_slices_kernel<NF, true, true>}
// [filters][2 * bitmap + key]
static const SelFn kSlices[MB_MAX_FILTERS + 1][4] = {MB_SELECT_VARIANTS(0), MB_SELECT_VARIANTS(1),
                                                     MB_SELECT_VARIANTS(2), MB_SELECT_VARIANTS(3)};
static int warp_bytes(int nc) {
  static const int kBytes[MB_MAX_FILTERS + 3] = {sizeof(SelWarp<0>), sizeof(SelWarp<1>), sizeof(SelWarp<2>),
                                                 sizeof(SelWarp<3>), sizeof(SelWarp<4>), sizeof(SelWarp<5>)};
  return kBytes[nc];
}

int select_init_device(const DeviceState& ds) {
  for (const auto& of_filters : kSlices)
    for (SelFn fn : of_filters)
      if (cudaFuncSetAttribute(reinterpret_cast<const void*>(fn), cudaFuncAttributeMaxDynamicSharedMemorySize,
                               ds.max_smem_optin) != cudaSuccess)
        return MB_ERR_CUDA;
  return MB_OK;
}

static int launch_slices(SelPlan& P, const DeviceState& ds, cudaStream_t st) {
  // The first probe goes to a bitmap when its table is small and enough rows are to be read:
  // every CTA reads the whole table once, to save a scattered load (a cycle of the SM's load path
  // and an L2 trip) per row. A 40,000-slot table of 8-byte slots, a filter and a second probe:
  // 24,000,000 rows 96 against 376 us. Its cost shows below some 32 rows a slot: 800,000 rows, each
  // probe keeping 5, 20, 50 and 100 %, 21, 22, 26 and 34 us with it and 17, 18, 19 and 24 without;
  // 1,300,000 rows 20, 22, 28 and 42 against 22, 25, 26 and 36.
  const bool bm = P.np > 0 && P.pslots[0] <= kSelBitmapMaxSlots && P.n / 32 >= P.pslots[0];
  const bool key = P.np > (bm ? 1 : 0);
  const int nc = P.nf + (bm ? 1 : 0) + (key ? 1 : 0);
  P.bm_words = bm ? P.pslots[0] / 32 + 1 : 0;  // slots 0 .. pslots (the last one absent)
  P.vec = 1;
  if (P.gpu_cache != nullptr) {
    P.vec = aligned16(P.gpu_cache) ? 1 : 0;
  } else {
    for (int f = 0; f < P.nf; ++f) P.vec = P.vec && aligned16(P.fcol[f]);
    for (int p = 0; p < P.np && p < nc - P.nf; ++p) P.vec = P.vec && aligned16(P.pkey[p]);
  }
  // as many warps as their buffers leave room for
  int warps = (ds.max_smem_optin - 4 * P.bm_words) / warp_bytes(nc);
  if (warps > kSelMaxWarps) warps = kSelMaxWarps;
  // Smaller slices while every one of them still has a warp of its own: a slice's rounds run one
  // after the other. 300,000 rows (the call above, no bitmap, all rows kept) 14.3 us, 500,000 18; 24
  // and 30 with the bitmap, 36 with slices of 512 as well; one row a lane 17 and 23.
  P.slice_rows = kSelRows;
  const long long at_once = static_cast<long long>(warps) * ds.num_sms;
  while (P.slice_rows > 64 && (P.n + P.slice_rows / 2 - 1) / (P.slice_rows / 2) <= at_once) P.slice_rows /= 2;
  const long long nslices = (P.n + P.slice_rows - 1) / P.slice_rows;
  long long blocks = (nslices + 3) / 4;
  if (blocks > ds.num_sms) blocks = ds.num_sms;
  const int smem = warps * warp_bytes(nc) + 4 * P.bm_words;
  if (launch_dependent(kSlices[P.nf][2 * (bm ? 1 : 0) + (key ? 1 : 0)], static_cast<int>(blocks), warps * 32,
                       static_cast<size_t>(smem), st, P) != cudaSuccess)
    return MB_ERR_LAUNCH;
  note_launches(1);
  return MB_OK;
}

static int launch_select(SelPlan& P, cudaStream_t st) {
  if (P.n == 0) return MB_OK;
  if (P.n < 0 || P.lo_off == nullptr || P.total == nullptr || P.capacity < 0) return MB_ERR_ARG;
  if (P.gpu_cache == nullptr && P.seg_group != nullptr) return MB_ERR_ARG;
  for (int f = 0; f < P.nf; ++f)
    if (P.fcol[f] == nullptr || P.fmode[f] < MB_FILTER_EQ || P.fmode[f] > MB_FILTER_EQ_OR_EQ) return MB_ERR_ARG;
  for (int p = 0; p < P.np; ++p) {
    if (P.pkey[p] == nullptr || P.pht[p] == nullptr || P.pslots[p] <= 0) return MB_ERR_ARG;
    if (P.playout[p] < MB_HT_KEY || P.playout[p] > MB_HT_VAL_OFF) return MB_ERR_ARG;
    if (P.playout[p] != MB_HT_KEY && !aligned8(P.pht[p])) return MB_ERR_ALIGN;
  }
  int err = MB_OK;
  DeviceState* ds = current_device_state(&err);
  if (ds == nullptr) return err;
  P.status = ds->status;
  const long long S = 1ll << P.seg_shift;
  if (P.in_rows == nullptr &&
      (P.gpu_cache == nullptr || (S % kSelRows == 0 && (P.seg_group != nullptr || P.start_offset % kSelRows == 0))))
    return launch_slices(P, *ds, st);
  constexpr int kItems = 4, kThreads = 256;
  const long long per_block = static_cast<long long>(kThreads) * kItems;
  long long blocks = (P.n + per_block - 1) / per_block;
  if (blocks > static_cast<long long>(ds->num_sms) * 8) blocks = static_cast<long long>(ds->num_sms) * 8;
  select_kernel<kItems><<<static_cast<int>(blocks), kThreads, 0, st>>>(P);
  if (cudaGetLastError() != cudaSuccess) return MB_ERR_LAUNCH;
  note_launches(1);
  return MB_OK;
}

static void engine_filters(SelPlan& P, const mb_filterArgsGPU* f) {
  if (f == nullptr) return;
  if (f->filter_idx1) {
    P.fcol[P.nf] = f->filter_idx1;
    P.fmode[P.nf] = f->mode1;
    P.fc1[P.nf] = f->compare1;
    P.fc2[P.nf++] = f->compare2;
  }
  if (f->filter_idx2) {
    P.fcol[P.nf] = f->filter_idx2;
    P.fmode[P.nf] = f->mode2;
    P.fc1[P.nf] = f->compare3;
    P.fc2[P.nf++] = f->compare4;
  }
}

// Engine probes, dimension slots 1..4 = supplier, customer, part, date, over VAL_OFF tables.
static void engine_probes(SelPlan& P, const mb_probeArgsGPU* q) {
  for (int j = 0; j < 4; ++j) P.slot_src[j] = -1;
  if (q == nullptr) return;
  const int* keys[4] = {q->key_idx1, q->key_idx2, q->key_idx3, q->key_idx4};
  const int* hts[4] = {q->ht1, q->ht2, q->ht3, q->ht4};
  const int lens[4] = {q->dim_len1, q->dim_len2, q->dim_len3, q->dim_len4};
  const int mins[4] = {q->min_key1, q->min_key2, q->min_key3, q->min_key4};
  for (int j = 0; j < 4; ++j) {
    if (keys[j] == nullptr || hts[j] == nullptr) continue;
    P.pkey[P.np] = keys[j];
    P.pht[P.np] = hts[j];
    P.pslots[P.np] = lens[j];
    P.pkmin[P.np] = mins[j];
    P.playout[P.np] = MB_HT_VAL_OFF;
    P.slot_src[j] = P.np++;
  }
}

static void engine_out(SelPlan& P, const mb_offsetGPU* out, const mb_offsetGPU* in) {
  P.lo_off = out ? out->lo_off : nullptr;
  int* const outs[4] = {out ? out->dim_off1 : nullptr, out ? out->dim_off2 : nullptr, out ? out->dim_off3 : nullptr,
                        out ? out->dim_off4 : nullptr};
  const int* const ins[4] = {in ? in->dim_off1 : nullptr, in ? in->dim_off2 : nullptr, in ? in->dim_off3 : nullptr,
                             in ? in->dim_off4 : nullptr};
  for (int j = 0; j < 4; ++j) {
    P.dim_out[j] = outs[j];
    P.in_dim[j] = ins[j];
  }
}

static int engine_select(const int* gpuCache, const mb_offsetGPU* in_off, const mb_filterArgsGPU* f,
                         const mb_probeArgsGPU* q, const mb_offsetGPU* out_off, int num_tuples, int* total,
                         int start_offset, const short* segment_group, cudaStream_t st) {
  if (num_tuples == 0) return MB_OK;
  if (gpuCache == nullptr || out_off == nullptr || num_tuples < 0) return MB_ERR_ARG;
  if (in_off != nullptr && in_off->lo_off == nullptr) return MB_ERR_ARG;
  SelPlan P = {};
  P.n = num_tuples;
  P.in_rows = in_off ? in_off->lo_off : nullptr;
  engine_filters(P, f);
  engine_probes(P, q);
  engine_out(P, out_off, in_off);
  P.capacity = num_tuples;
  P.total = total;
  P.gpu_cache = gpuCache;
  P.seg_group = in_off ? nullptr : segment_group;
  P.start_offset = in_off ? 0 : start_offset;
  P.seg_shift = 20;  // SEGMENT_SIZE = 1,048,576 (src/gpudb/common.h:73)
  return launch_select(P, st);
}

}  // namespace mb

using namespace mb;

extern "C" int mb_star_select(const mb_star_args* a, const int* in_rows, int64_t num_in, int* lo_off,
                              int* const* dim_off, int64_t capacity, int* total, mb_stream_t stream) {
  if (a == nullptr) return MB_ERR_ARG;
  if (a->num_filters < 0 || a->num_filters > MB_MAX_FILTERS || a->num_probes < 0 || a->num_probes > MB_MAX_PROBES)
    return MB_ERR_ARG;
  SelPlan P = {};
  P.n = in_rows ? num_in : a->num_rows;
  P.in_rows = in_rows;
  P.nf = a->num_filters;
  for (int f = 0; f < P.nf; ++f) {
    P.fcol[f] = a->filter[f].col;
    P.fmode[f] = a->filter[f].mode;
    P.fc1[f] = a->filter[f].c1;
    P.fc2[f] = a->filter[f].c2;
  }
  P.np = a->num_probes;
  for (int p = 0; p < 4; ++p) P.slot_src[p] = p < P.np ? p : -1;
  for (int p = 0; p < P.np; ++p) {
    P.pkey[p] = a->probe[p].fkey;
    P.pht[p] = a->probe[p].ht;
    P.pslots[p] = a->probe[p].num_slots;
    P.pkmin[p] = a->probe[p].key_min;
    P.playout[p] = a->probe[p].layout;
    P.dim_out[p] = dim_off ? dim_off[p] : nullptr;
  }
  P.lo_off = lo_off;
  P.total = total;
  P.capacity = capacity;
  P.gpu_cache = a->gpu_cache;
  P.seg_group = a->gpu_cache ? a->segment_group : nullptr;
  P.start_offset = a->start_offset;
  if (a->gpu_cache) {
    if (a->segment_size <= 0 || (a->segment_size & (a->segment_size - 1)) != 0) return MB_ERR_ARG;
    P.seg_shift = __builtin_ctz(static_cast<unsigned>(a->segment_size));
  }
  return launch_select(P, static_cast<cudaStream_t>(stream));
}

extern "C" int mb_filter_GPU2(const int* gpuCache, const mb_filterArgsGPU* fargs, const mb_offsetGPU* out_off,
                              int num_tuples, int* total, int start_offset, const short* segment_group,
                              mb_stream_t stream) {
  return engine_select(gpuCache, nullptr, fargs, nullptr, out_off, num_tuples, total, start_offset, segment_group,
                       static_cast<cudaStream_t>(stream));
}

extern "C" int mb_filter_probe_GPU2(const int* gpuCache, const mb_filterArgsGPU* fargs,
                                    const mb_probeArgsGPU* pargs, const mb_offsetGPU* out_off, int num_tuples,
                                    int* total, int start_offset, const short* segment_group, mb_stream_t stream) {
  return engine_select(gpuCache, nullptr, fargs, pargs, out_off, num_tuples, total, start_offset, segment_group,
                       static_cast<cudaStream_t>(stream));
}

extern "C" int mb_probe_GPU2(const int* gpuCache, const mb_probeArgsGPU* pargs, const mb_offsetGPU* out_off,
                             int num_tuples, int* total, int start_offset, const short* segment_group,
                             mb_stream_t stream) {
  return engine_select(gpuCache, nullptr, nullptr, pargs, out_off, num_tuples, total, start_offset, segment_group,
                       static_cast<cudaStream_t>(stream));
}

extern "C" int mb_filter_GPU3(const int* gpuCache, const mb_offsetGPU* in_off, const mb_filterArgsGPU* fargs,
                              const mb_offsetGPU* out_off, int num_tuples, int* total, mb_stream_t stream) {
  return engine_select(gpuCache, in_off, fargs, nullptr, out_off, num_tuples, total, 0, nullptr,
                       static_cast<cudaStream_t>(stream));
}

extern "C" int mb_filter_probe_GPU3(const int* gpuCache, const mb_offsetGPU* in_off, const mb_filterArgsGPU* fargs,
                                    const mb_probeArgsGPU* pargs, const mb_offsetGPU* out_off, int num_tuples,
                                    int* total, mb_stream_t stream) {
  return engine_select(gpuCache, in_off, fargs, pargs, out_off, num_tuples, total, 0, nullptr,
                       static_cast<cudaStream_t>(stream));
}

extern "C" int mb_probe_GPU3(const int* gpuCache, const mb_offsetGPU* in_off, const mb_probeArgsGPU* pargs,
                             const mb_offsetGPU* out_off, int num_tuples, int* total, mb_stream_t stream) {
  return engine_select(gpuCache, in_off, nullptr, pargs, out_off, num_tuples, total, 0, nullptr,
                       static_cast<cudaStream_t>(stream));
}

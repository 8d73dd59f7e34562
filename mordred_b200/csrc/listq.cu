// listq.cu — the fused star pipeline over an offset list: the rows a previous operator
// selected (on the GPU by mb_star_select, or on the CPU) arrive as a list of physical fact
// rows, possibly with the dimension rows earlier joins matched them with, and are
// filtered, probed, grouped and aggregated here.
//
// Restates the offset-list ("GPU3") forms of the engine's fused kernels:
//   filter_probe_group_by_GPU3  src/gpudb/GPUProcessing.h:157-273
//   probe_group_by_GPU3         GPUProcessing.h:393-494
//   groupByGPU                  GPUProcessing.h:1385-1470
//   aggregationGPU              GPUProcessing.h:1472-1524
//   probe_aggr_GPU3             GPUProcessing.h:1610-1673
//   filter_probe_aggr_GPU3      GPUProcessing.h:1778-1846
// Row k of the call reads every fact column at the physical row rows[k] (through the
// segment cache: gpuCache[col_idx[row >> 20] << 20 | row & (2^20 - 1)], BlockLibrary.cuh:
// 543-592); a probe either looks the row's key up in a hash table, or — layout MB_HT_PASS —
// takes the group value an earlier join found: the dimension column `ht` read at the
// dimension row fkey[k] (BlockReadFilteredOffset, BlockLibrary.cuh:484-541).
//
// The rows of a list are gathers, not a stream, so the kernel is bound by how many loads it
// has in flight and how long its chain of dependent ones is. A thread keeps kListItems
// entries and runs them through straight-line rounds (every load of a round goes out before
// one is used): the entries' rows; the filters; the first table probe; then the remaining
// probes of its survivors — and, when that is one table at most, the aggregate columns with
// them; at last the passed-through group values and the aggregates. Outcomes are combined
// probe by probe in the chain's order, so selection and status bits equal the sequential
// chain's. Group accumulation is the star kernel's: 64-bit sums in a shared-memory group
// array flushed once per CTA, or L2 atomics for large group arrays; scalars reduced per CTA.
// 2,000,003 entries over 24,000,000 rows (segment cache, two table probes, one passed-through
// value): one entry at a time behind branches 127 us; in rounds 76 us; with the 64-byte fetches
// of gather_ld about 69 (74 a call, from 140). Its entries lie 12 rows apart, so the four
// gathered columns come in nearly whole (340 MB, 52 us at the copy rate).
#include <cstring>
#include <type_traits>

#include "star.cuh"

namespace mb {

// Two entries a thread at three CTAs an SM is what the registers carry without spilling
// (2,000,003 entries, plain gathers: 81 us a call; 4 entries at 3 CTAs 113 us and 2 at 4 CTAs 93 us, both
// spilling; 4 at 2 CTAs 80 us, but 133 against 123 us for 4.8 M entries).
constexpr int kListItems = 2;
constexpr int kListThreads = 256;
constexpr int kListCtas = 3;

struct ListPlan {
  long long n;
  const int* rows;  // physical fact rows, or null: row k is virtual row k
  int nf;
  const int* f_col[MB_MAX_FILTERS];
  int f_mode[MB_MAX_FILTERS], f_c1[MB_MAX_FILTERS], f_c2[MB_MAX_FILTERS];
  int np;
  const int* p_key[MB_MAX_PROBES];
  const int* p_ht[MB_MAX_PROBES];
  int p_slots[MB_MAX_PROBES], p_kmin[MB_MAX_PROBES], p_layout[MB_MAX_PROBES];
  int p_min[MB_MAX_PROBES], p_mul[MB_MAX_PROBES], p_res_slot[MB_MAX_PROBES];
  const int* a_col[2];
  int agg_op;
  int total_val, group_bias, res_layout;
  void* res;
  unsigned long long* count;
  int count_after;
  int gmode;
  const int* gpu_cache;
  const short* seg_group;
  long long start_offset;
  int seg_shift;
  unsigned int* status;
};

__device__ __forceinline__ bool list_pass(int x, int mode, int c1, int c2) {
  if (mode == MB_FILTER_BETWEEN) return x >= c1 && x <= c2;
  if (mode == MB_FILTER_EQ) return x == c1;
  return x == c1 || x == c2;
}

__device__ __forceinline__ unsigned long long* list_sum_ptr(const ListPlan& P, int h) {
  if (P.res_layout == MB_RES_ENGINE6)
    return reinterpret_cast<unsigned long long*>(static_cast<int*>(P.res) + 6 * h + 4);
  if (P.res_layout == MB_RES_CRYSTAL4)
    return reinterpret_cast<unsigned long long*>(static_cast<int*>(P.res) + 4 * h + 2);
  return static_cast<unsigned long long*>(P.res) + h;
}

// SEG: segment-cache addressing (gpu_cache set).
template <bool SEG>
__global__ void __launch_bounds__(kListThreads, kListCtas) list_kernel(const __grid_constant__ ListPlan P) {
  constexpr int R = kListItems;
  using Index = std::conditional_t<SEG, int, long long>;  // in-segment row, or row of the column
  extern __shared__ __align__(16) unsigned char lsmem[];
  __shared__ unsigned long long s_red[2 * kListThreads / 32];
  unsigned long long* s_sum = reinterpret_cast<unsigned long long*>(lsmem);
  uint32_t* s_touch = reinterpret_cast<uint32_t*>(lsmem + 8 * P.total_val);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  wait_for_predecessor();
  if (P.gmode == kGroupSmem) {
    for (int g = tid; g < P.total_val; g += kListThreads) s_sum[g] = 0;
    for (int w = tid; w < (P.total_val + 31) / 32; w += kListThreads) s_touch[w] = 0;
  }
  __syncthreads();
  unsigned long long acc = 0, cnt = 0;
  bool bad_probe = false, bad_group = false;
  // the first table probe; a second round follows it, with the aggregate columns when it
  // holds one table at most
  int first = 0, later_tables = 0;
  while (first < P.np && P.p_layout[first] == MB_HT_PASS) ++first;
  for (int p = first + 1; p < P.np; ++p) later_tables += P.p_layout[p] != MB_HT_PASS ? 1 : 0;
  const bool early_aggr = later_tables <= 1;
  const bool two_cols = P.agg_op == MB_AGG_SUB || P.agg_op == MB_AGG_MUL;
  const long long stride = static_cast<long long>(gridDim.x) * kListThreads;
  for (long long base = blockIdx.x * static_cast<long long>(kListThreads) * R + tid; base < P.n; base += stride * R) {
    // ---- entries k = base + i * kListThreads: their rows ----
    int seg[R];
    Index idx[R];
    unsigned sel = 0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const long long k = base + static_cast<long long>(i) * kListThreads;
      seg[i] = idx[i] = 0;
      if (k < P.n) {
        sel |= 1u << i;
        if (P.rows) {
          idx[i] = ld_word(P.rows + k);
        } else {
          idx[i] = static_cast<Index>(SEG ? k & ((1ll << P.seg_shift) - 1) : k);
          if (SEG)
            seg[i] = P.seg_group ? static_cast<int>(P.seg_group[k >> P.seg_shift])
                                 : static_cast<int>((P.start_offset + k) >> P.seg_shift);
        }
      }
    }
    if (SEG && P.rows) {
#pragma unroll
      for (int i = 0; i < R; ++i) {
        seg[i] = static_cast<int>(idx[i] >> P.seg_shift);  // physical rows index the slot arrays directly
        idx[i] &= (1 << P.seg_shift) - 1;
      }
    }
    // a column at the entries in `of` (0 elsewhere)
    auto load = [&](const int* col, unsigned of, int (&v)[R]) {
      if (SEG) {
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = (of >> i) & 1u ? __ldg(col + seg[i]) : 0;
#pragma unroll
        for (int i = 0; i < R; ++i)
          v[i] = (of >> i) & 1u ? gather_ld(P.gpu_cache + (static_cast<long long>(v[i]) << P.seg_shift) + idx[i]) : 0;
      } else {
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = (of >> i) & 1u ? gather_ld(col + idx[i]) : 0;
      }
    };
    // ---- filters ----
#pragma unroll
    for (int f = 0; f < MB_MAX_FILTERS; ++f) {
      if (f >= P.nf) break;
      if (P.count_after == f) cnt += __popc(sel);
      int v[R];
      load(P.f_col[f], sel, v);
#pragma unroll
      for (int i = 0; i < R; ++i)
        if (!list_pass(v[i], P.f_mode[f], P.f_c1[f], P.f_c2[f])) sel &= ~(1u << i);
    }
    if (P.count_after >= P.nf) cnt += __popc(sel);
    // ---- probes: gv[p] = the payload, or the dimension row of a passed-through value ----
    int gv[MB_MAX_PROBES][R], a0[R], a1[R];
#pragma unroll
    for (int p = 0; p < MB_MAX_PROBES; ++p)
#pragma unroll
      for (int i = 0; i < R; ++i) gv[p][i] = 0;
#pragma unroll
    for (int i = 0; i < R; ++i) a0[i] = a1[i] = 0;
    auto round = [&](auto in_round) {
      unsigned long long sv[MB_MAX_PROBES][R];
      unsigned range_bad[MB_MAX_PROBES];
#pragma unroll
      for (int p = 0; p < MB_MAX_PROBES; ++p) {
        range_bad[p] = 0;
        if (p >= P.np || !in_round(p)) continue;
        if (P.p_layout[p] == MB_HT_PASS) {
#pragma unroll
          for (int i = 0; i < R; ++i)
            if ((sel >> i) & 1u) gv[p][i] = ld_word(P.p_key[p] + base + static_cast<long long>(i) * kListThreads);
        } else {
          load(P.p_key[p], sel, gv[p]);
        }
      }
#pragma unroll
      for (int p = 0; p < MB_MAX_PROBES; ++p) {
        if (p >= P.np || !in_round(p)) continue;
        const int layout = P.p_layout[p], slots = P.p_slots[p];
        if (layout == MB_HT_PASS) {
#pragma unroll
          for (int i = 0; i < R; ++i)
            if (gv[p][i] < 0 || gv[p][i] >= slots) range_bad[p] |= 1u << i;
          continue;
        }
        const int* ht = P.p_ht[p];
        int h[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
          h[i] = pht_slot(gv[p][i], slots, P.p_kmin[p]);
          if (h[i] < 0) {
            range_bad[p] |= 1u << i;
            h[i] = 0;
          }
        }
        const unsigned of = sel & ~range_bad[p];
        if (layout == MB_HT_KEY) {
#pragma unroll
          for (int i = 0; i < R; ++i) sv[p][i] = (of >> i) & 1u ? static_cast<unsigned>(ld_word(ht + h[i])) : 0u;
        } else {
#pragma unroll
          for (int i = 0; i < R; ++i) sv[p][i] = (of >> i) & 1u ? ld_word2(ht + 2ll * h[i]) : 0ull;
        }
      }
#pragma unroll
      for (int p = 0; p < MB_MAX_PROBES; ++p) {
        if (p >= P.np || !in_round(p)) continue;
        if (sel & range_bad[p]) bad_probe = true;
        sel &= ~range_bad[p];
        const int layout = P.p_layout[p];
        if (layout == MB_HT_PASS) continue;
#pragma unroll
        for (int i = 0; i < R; ++i) {
          if (sv[p][i] == 0) sel &= ~(1u << i);
          gv[p][i] = layout == MB_HT_KEY_VAL   ? static_cast<int>(sv[p][i] >> 32)
                     : layout == MB_HT_VAL_OFF ? static_cast<int>(static_cast<unsigned>(sv[p][i]))
                                               : 0;
        }
      }
    };
    if (P.np > 0) {
      round([&](int p) { return p <= first; });
      if (early_aggr) {
        load(P.a_col[0], sel, a0);
        if (two_cols) load(P.a_col[1], sel, a1);
      }
      round([&](int p) { return p > first; });
    }
    if (P.count_after < 0) cnt += __popc(sel);
    if (!early_aggr || P.np == 0) {
      load(P.a_col[0], sel, a0);
      if (two_cols) load(P.a_col[1], sel, a1);
    }
    // ---- passed-through group values: the dimension column at the listed dimension row ----
#pragma unroll
    for (int p = 0; p < MB_MAX_PROBES; ++p) {
      if (p >= P.np) break;
      if (P.p_layout[p] != MB_HT_PASS) continue;
      const int* col = P.p_ht[p];
      if (SEG) {
        int slot[R];
#pragma unroll
        for (int i = 0; i < R; ++i) slot[i] = (sel >> i) & 1u ? __ldg(col + (gv[p][i] >> P.seg_shift)) : 0;
#pragma unroll
        for (int i = 0; i < R; ++i)
          if ((sel >> i) & 1u)
            gv[p][i] = __ldg(P.gpu_cache + (static_cast<long long>(slot[i]) << P.seg_shift) +
                             (gv[p][i] & ((1 << P.seg_shift) - 1)));
      } else {
#pragma unroll
        for (int i = 0; i < R; ++i)
          if ((sel >> i) & 1u) gv[p][i] = __ldg(col + gv[p][i]);
      }
    }
    // ---- aggregate ----
#pragma unroll
    for (int i = 0; i < R; ++i) {
      if (!((sel >> i) & 1u)) continue;
      const unsigned u0 = static_cast<unsigned>(a0[i]), u1 = static_cast<unsigned>(a1[i]);
      const int val = static_cast<int>(P.agg_op == MB_AGG_SUM           ? u0
                                       : P.agg_op == MB_AGG_MUL_PAYLOAD ? u0 * static_cast<unsigned>(gv[0][i])
                                       : P.agg_op == MB_AGG_SUB         ? u0 - u1
                                                                        : u0 * u1);
      const unsigned long long w = static_cast<unsigned long long>(static_cast<long long>(val));
      if (P.gmode == kGroupScalar) {
        acc += w;
        continue;
      }
      unsigned hh = static_cast<unsigned>(P.group_bias);
#pragma unroll
      for (int p = 0; p < MB_MAX_PROBES; ++p)
        if (p < P.np)
          hh += (static_cast<unsigned>(gv[p][i]) - static_cast<unsigned>(P.p_min[p])) * static_cast<unsigned>(P.p_mul[p]);
      int h = static_cast<int>(hh);
      if (hh >= static_cast<unsigned>(P.total_val)) h = slow_mod(h, P.total_val);
      if (h < 0) {
        bad_group = true;
        continue;
      }
      bool keys = P.res_layout != MB_RES_DENSE;
      if (P.gmode == kGroupSmem) {
        smem_add_i64(&s_sum[h], val);
        const uint32_t bit = 1u << (h & 31);
        keys = !(s_touch[h >> 5] & bit) && !(atomicOr(&s_touch[h >> 5], bit) & bit) && keys;
      } else {
        atomicAdd(list_sum_ptr(P, h), w);
      }
      if (!keys) continue;
      int* res = static_cast<int*>(P.res) + static_cast<long long>(P.res_layout == MB_RES_ENGINE6 ? 6 : 4) * h;
#pragma unroll
      for (int p = 0; p < MB_MAX_PROBES; ++p)
        if (p < P.np && P.p_res_slot[p] >= 0) res[P.p_res_slot[p]] = gv[p][i];
    }
  }
  if (bad_probe) set_status(P.status, MB_STATUS_PROBE_RANGE);
  if (bad_group) set_status(P.status, MB_STATUS_GROUP_RANGE);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    acc += __shfl_down_sync(0xffffffffu, acc, o);
    cnt += __shfl_down_sync(0xffffffffu, cnt, o);
  }
  if (lane == 0) {
    s_red[warp] = acc;
    s_red[kListThreads / 32 + warp] = cnt;
  }
  __syncthreads();
  if (tid == 0) {
    unsigned long long ta = 0, tc = 0;
    for (int w = 0; w < kListThreads / 32; ++w) {
      ta += s_red[w];
      tc += s_red[kListThreads / 32 + w];
    }
    if (P.gmode == kGroupScalar && ta != 0) atomicAdd(static_cast<unsigned long long*>(P.res), ta);
    if (P.count != nullptr && tc != 0) atomicAdd(P.count, tc);
  }
  if (P.gmode == kGroupSmem) {
    for (int g = tid; g < P.total_val; g += kListThreads)
      if ((s_touch[g >> 5] >> (g & 31)) & 1u) atomicAdd(list_sum_ptr(P, g), s_sum[g]);
  }
}

int list_init_device(const DeviceState& ds) {
  for (auto fn : {list_kernel<false>, list_kernel<true>})
    if (cudaFuncSetAttribute(reinterpret_cast<const void*>(fn), cudaFuncAttributeMaxDynamicSharedMemorySize,
                             ds.max_smem_optin - 2048) != cudaSuccess)
      return MB_ERR_CUDA;
  return MB_OK;
}

int launch_list(const mb_star_args* a, cudaStream_t stream, const DeviceState* ds) {
  ListPlan P;
  memset(&P, 0, sizeof(P));
  P.n = a->num_rows;
  P.rows = a->rows;
  P.nf = a->num_filters;
  for (int f = 0; f < P.nf; ++f) {
    const mb_filter& F = a->filter[f];
    if (F.col == nullptr || F.mode < MB_FILTER_EQ || F.mode > MB_FILTER_EQ_OR_EQ) return MB_ERR_ARG;
    P.f_col[f] = F.col;
    P.f_mode[f] = F.mode;
    P.f_c1[f] = F.c1;
    P.f_c2[f] = F.c2;
  }
  P.np = a->num_probes;
  for (int p = 0; p < P.np; ++p) {
    const mb_probe& Q = a->probe[p];
    if (Q.fkey == nullptr || Q.ht == nullptr || Q.num_slots <= 0) return MB_ERR_ARG;
    if (Q.layout < MB_HT_KEY || Q.layout > MB_HT_PASS) return MB_ERR_ARG;
    if ((Q.layout == MB_HT_KEY_VAL || Q.layout == MB_HT_VAL_OFF) && !aligned8(Q.ht)) return MB_ERR_ALIGN;
    const int rs = Q.res_slot;
    if (rs >= 0 && ((a->res_layout == MB_RES_ENGINE6 && rs > 3) || (a->res_layout == MB_RES_CRYSTAL4 && rs > 1)))
      return MB_ERR_ARG;
    P.p_key[p] = Q.fkey;
    P.p_ht[p] = Q.ht;
    P.p_slots[p] = Q.num_slots;
    P.p_kmin[p] = Q.key_min;
    P.p_layout[p] = Q.layout;
    P.p_min[p] = Q.min_val;
    P.p_mul[p] = Q.unique_val;
    P.p_res_slot[p] = (a->res_layout == MB_RES_ENGINE6 || a->res_layout == MB_RES_CRYSTAL4) ? rs : -1;
  }
  if (a->agg_op == MB_AGG_MUL_PAYLOAD && (P.np < 1 || P.p_layout[0] == MB_HT_KEY)) return MB_ERR_ARG;
  P.a_col[0] = a->aggr[0];
  P.a_col[1] = a->aggr[1];
  P.agg_op = a->agg_op;
  P.total_val = a->res_layout == MB_RES_SCALAR ? 1 : a->total_val;
  P.group_bias = a->group_bias;
  P.res_layout = a->res_layout;
  P.res = a->res;
  P.count = a->count;
  P.count_after = a->count_after < 0 ? -1 : a->count_after;
  P.status = ds->status;
  if (a->gpu_cache != nullptr) {
    const int ss = a->segment_size;
    if (ss <= 0 || (ss & (ss - 1)) != 0) return MB_ERR_ARG;
    P.gpu_cache = a->gpu_cache;
    P.seg_group = a->rows ? nullptr : a->segment_group;
    P.start_offset = a->start_offset;
    P.seg_shift = __builtin_ctz(static_cast<unsigned>(ss));
  }
  int smem = 0;
  if (P.res_layout == MB_RES_SCALAR) {
    P.gmode = kGroupScalar;
  } else if (a->group_mode != 2 && P.total_val <= kSmemGroupMax) {
    P.gmode = kGroupSmem;
    smem = 8 * P.total_val + 4 * ((P.total_val + 31) / 32);
  } else {
    if (a->group_mode == 1) return MB_ERR_SIZE;
    P.gmode = kGroupGlobal;
  }
  const long long per_block = static_cast<long long>(kListThreads) * kListItems;
  long long blocks = (P.n + per_block - 1) / per_block;
  const long long cap = static_cast<long long>(ds->num_sms) * kListCtas;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  const auto fn = P.gpu_cache != nullptr ? list_kernel<true> : list_kernel<false>;
  if (launch_dependent(fn, static_cast<int>(blocks), kListThreads, static_cast<size_t>(smem), stream, P) != cudaSuccess)
    return MB_ERR_LAUNCH;
  note_launches(1);
  return MB_OK;
}

}  // namespace mb

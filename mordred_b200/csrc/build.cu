// build.cu — perfect-hash builds over (filtered) dimension tables.
//
//  MB_HT_KEY      atomicCAS(&ht[h], 0, key)                       crystal/join.cuh:167-206
//  MB_HT_KEY_VAL  atomicCAS(&ht[2h], 0, key); ht[2h+1] = val      crystal/join.cuh:236-279
//  MB_HT_VAL_OFF  atomicCAS(&ht[2h], 0, val) if val; ht[2h+1] = row+1
//                                                                 BlockLibrary.cuh:594-715
// with h = (key - key_min) % num_slots (crystal/join.cuh:3). Dimension tables are small
// (<= 1 M rows), so a build is one wave of a plain kernel and its launch counts as much as
// its work: mb_build_tables clears and builds a query's tables in two launches. A build can
// also fill a presence bitmap that the fused probe stages in shared memory.
#include "common.cuh"
#include "star.cuh"

namespace mb {

__device__ __forceinline__ bool build_pass(int x, int mode, int c1, int c2) {
  if (mode == MB_FILTER_BETWEEN) return x >= c1 && x <= c2;
  if (mode == MB_FILTER_EQ) return x == c1;
  return x == c1 || x == c2;
}

constexpr int kBuildThreads = 256;
constexpr int kBuildItems = 4;  // rows a thread (8: Query B over 1 M rows 32.6 us, 4: 31.4)

struct BuildPlan {
  const int* filter;   // column / cache-slot index array, or null
  int mode, c1, c2;
  const int* key;
  const int* val;      // or null
  long long n;
  int* ht;
  int slots, kmin, layout;
  uint32_t* presence;
  const int* gpu_cache;
  const short* seg_group;
  long long start_offset;
  int seg_shift;
  unsigned int* status;
  const int* rows;     // optional list of dimension rows to build from (build_GPU3 forms)
  int* min_out;        // optional key range of the rows passing the filter (minmax forms)
  int* max_out;
  int val_min, val_max;  // where each warp's range starts (the reference's block start values)
};

__device__ __forceinline__ long long build_row_index(const BuildPlan& B, long long r, int* seg_out) {
  if (B.rows != nullptr) {
    // a listed dimension row: the physical row, through its own segment's slot
    const long long d = ld_word(B.rows + r);
    if (B.gpu_cache == nullptr) {
      *seg_out = 0;
      return d;
    }
    *seg_out = static_cast<int>(d >> B.seg_shift);
    return d & ((1ll << B.seg_shift) - 1);
  }
  if (B.gpu_cache == nullptr) {
    *seg_out = 0;
    return r;
  }
  const long long vseg = r >> B.seg_shift;
  *seg_out = B.seg_group ? static_cast<int>(B.seg_group[vseg])
                         : static_cast<int>((B.start_offset + r) >> B.seg_shift);
  return r & ((1ll << B.seg_shift) - 1);
}

__device__ __forceinline__ int build_load(const BuildPlan& B, const int* col, int seg, long long idx) {
  if (B.gpu_cache == nullptr) return col[idx];
  return B.gpu_cache[(static_cast<long long>(col[seg]) << B.seg_shift) + idx];
}

struct BuildRange {
  int kmin, kmax;
  bool bad = false;
};

// Row r's key (and payload v) into the table.
__device__ __forceinline__ void build_row(const BuildPlan& B, long long rowid, int key, int v, BuildRange& R) {
  R.kmin = key < R.kmin ? key : R.kmin;
  R.kmax = key > R.kmax ? key : R.kmax;
  const int h = pht_slot(key, B.slots, B.kmin);
  if (h < 0) {
    R.bad = true;
    return;
  }
  bool present;
  if (B.layout == MB_HT_KEY) {
    atomicCAS(B.ht + h, 0, key);
    present = key != 0;
  } else if (B.layout == MB_HT_KEY_VAL) {
    atomicCAS(B.ht + 2ll * h, 0, key);
    B.ht[2ll * h + 1] = v;
    present = key != 0 || v != 0;
  } else {
    // engine layout: the row id is the dimension row's position in the table, stored +1 so
    // 0 stays "empty"
    if (B.val != nullptr) atomicCAS(B.ht + 2ll * h, 0, v);
    B.ht[2ll * h + 1] = static_cast<int>(rowid + 1);
    present = true;
  }
  if (B.presence != nullptr && present) atomicOr(B.presence + (h >> 5), 1u << (h & 31));
}

__device__ __forceinline__ void build_publish(const BuildPlan& B, BuildRange R) {
  if (R.bad) set_status(B.status, MB_STATUS_PROBE_RANGE);
  if (B.min_out != nullptr) {
    // every warp folds its range in, starting from (val_max, val_min) as the reference's
    // blocks do (GPUProcessing.h:1052,1101-1110)
    const int kmin = __reduce_min_sync(0xffffffffu, R.kmin), kmax = __reduce_max_sync(0xffffffffu, R.kmax);
    if ((threadIdx.x & 31) == 0) {
      atomicMin(B.min_out, kmin);
      atomicMax(B.max_out, kmax);
    }
  }
}

// Dimension rows through the segment cache, or listed ones: a row a thread at a time.
__global__ void __launch_bounds__(kBuildThreads) build_kernel(const __grid_constant__ BuildPlan B) {
  allow_dependent();
  wait_for_predecessor();
  BuildRange R{B.val_max, B.val_min};
  for (long long r = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; r < B.n;
       r += static_cast<long long>(gridDim.x) * blockDim.x) {
    int seg;
    const long long idx = build_row_index(B, r, &seg);
    if (B.filter != nullptr && !build_pass(build_load(B, B.filter, seg, idx), B.mode, B.c1, B.c2)) continue;
    const int key = build_load(B, B.key, seg, idx);
    const int v = B.val != nullptr ? build_load(B, B.val, seg, idx) : 0;
    // the row's position in the table (segment * segment_size + in-segment offset, or the
    // listed row)
    const long long rowid = B.rows != nullptr       ? static_cast<long long>(ld_word(B.rows + r))
                            : B.gpu_cache == nullptr ? B.start_offset + r
                                                     : (static_cast<long long>(seg) << B.seg_shift) + idx;
    build_row(B, rowid, key, v, R);
  }
  build_publish(B, R);
}

// Contiguous dimension columns: kBuildItems consecutive rows a thread in 16-byte loads, filter,
// key and payload all in flight together. A build is a launch and one wave of dependent
// loads: the engine's four builds and their clears take 33 us in a stream, against 45 row by row
// behind the filter and without overlapped set-up.
__device__ __forceinline__ void build_chunk(const BuildPlan& B, long long block, long long blocks) {
  auto aligned = [](const int* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  const bool vec = aligned(B.key) && (B.filter == nullptr || aligned(B.filter)) && (B.val == nullptr || aligned(B.val));
  BuildRange R{B.val_max, B.val_min};
  for (long long r0 = (block * kBuildThreads + threadIdx.x) * kBuildItems; r0 < B.n;
       r0 += blocks * kBuildThreads * kBuildItems) {
    int f[kBuildItems], k[kBuildItems], v[kBuildItems];
    auto load = [&](const int* col, int (&x)[kBuildItems]) {
      if (col == nullptr) {
#pragma unroll
        for (int i = 0; i < kBuildItems; ++i) x[i] = 0;
      } else if (vec && r0 + kBuildItems <= B.n) {
#pragma unroll
        for (int j = 0; j < kBuildItems / 4; ++j) {
          const int4 q = __ldg(reinterpret_cast<const int4*>(col + r0) + j);
          x[4 * j] = q.x;
          x[4 * j + 1] = q.y;
          x[4 * j + 2] = q.z;
          x[4 * j + 3] = q.w;
        }
      } else {
#pragma unroll
        for (int i = 0; i < kBuildItems; ++i) x[i] = r0 + i < B.n ? __ldg(col + r0 + i) : 0;
      }
    };
    load(B.filter, f);
    load(B.key, k);
    load(B.val, v);
#pragma unroll
    for (int i = 0; i < kBuildItems; ++i) {
      if (r0 + i >= B.n || (B.filter != nullptr && !build_pass(f[i], B.mode, B.c1, B.c2))) continue;
      build_row(B, B.start_offset + r0 + i, k[i], v[i], R);
    }
  }
  build_publish(B, R);
}

__global__ void __launch_bounds__(kBuildThreads) build_columns_kernel(const __grid_constant__ BuildPlan B) {
  allow_dependent();
  wait_for_predecessor();
  build_chunk(B, blockIdx.x, gridDim.x);
}

// All tables of a query in one launch: table t takes blocks [first[t], first[t + 1]).
struct BuildMany {
  int count;
  int first[MB_MAX_TABLE_BUILDS + 1];
  BuildPlan b[MB_MAX_TABLE_BUILDS];
};
__global__ void __launch_bounds__(kBuildThreads) build_many_kernel(const __grid_constant__ BuildMany M) {
  allow_dependent();
  wait_for_predecessor();
  const int blk = static_cast<int>(blockIdx.x);
  int t = 0;
  while (t + 1 < M.count && blk >= M.first[t + 1]) ++t;
  build_chunk(M.b[t], blk - M.first[t], M.first[t + 1] - M.first[t]);
}

// Zeroes up to 2 * MB_MAX_TABLE_BUILDS + 1 ranges of 32-bit words, by the blocks of one grid.
struct ZeroMany {
  int count;
  long long words[2 * MB_MAX_TABLE_BUILDS + 1];
  int* at[2 * MB_MAX_TABLE_BUILDS + 1];
};
__global__ void __launch_bounds__(kBuildThreads) zero_many_kernel(const __grid_constant__ ZeroMany Z) {
  allow_dependent();
  wait_for_predecessor();
  const long long t = blockIdx.x * static_cast<long long>(kBuildThreads) + threadIdx.x;
  const long long threads = static_cast<long long>(gridDim.x) * kBuildThreads;
  for (int i = 0; i < Z.count; ++i) {
    int* p = Z.at[i];
    // single words up to a 16-byte boundary and after the last one
    const long long head = min(Z.words[i], static_cast<long long>((16u - (reinterpret_cast<uintptr_t>(p) & 15u)) & 15u) / 4);
    const long long quads = (Z.words[i] - head) / 4, tail = head + 4 * quads;
    for (long long q = t; q < quads; q += threads) reinterpret_cast<int4*>(p + head)[q] = make_int4(0, 0, 0, 0);
    if (t < head) p[t] = 0;
    if (tail + t < Z.words[i]) p[tail + t] = 0;
  }
}

static int launch_build(BuildPlan& B, cudaStream_t stream) {
  int err = MB_OK;
  DeviceState* ds = current_device_state(&err);
  if (ds == nullptr) return err;
  B.status = ds->status;
  if (B.n <= 0) return MB_OK;
  const bool columns = B.rows == nullptr && B.gpu_cache == nullptr;
  const long long per_block = static_cast<long long>(kBuildThreads) * (columns ? kBuildItems : 1);
  long long blocks = (B.n + per_block - 1) / per_block;
  const long long cap = static_cast<long long>(ds->num_sms) * 8;
  if (blocks > cap) blocks = cap;
  if (launch_dependent(columns ? build_columns_kernel : build_kernel, static_cast<int>(blocks), kBuildThreads, 0, stream,
                       B) != cudaSuccess)
    return MB_ERR_LAUNCH;
  note_launches(1);
  return MB_OK;
}

}  // namespace mb

using namespace mb;

extern "C" int mb_build_pht(const int* filter_col, int filter_mode, int c1, int c2, const int* dim_key,
                            const int* dim_val, int num_tuples, int* ht, int num_slots, int key_min,
                            uint32_t* presence, mb_stream_t stream) {
  if (num_tuples == 0) return MB_OK;
  if (dim_key == nullptr || ht == nullptr || num_tuples < 0 || num_slots <= 0) return MB_ERR_ARG;
  if (filter_col != nullptr && (filter_mode < MB_FILTER_EQ || filter_mode > MB_FILTER_EQ_OR_EQ)) return MB_ERR_ARG;
  if (dim_val != nullptr && !aligned8(ht)) return MB_ERR_ALIGN;
  BuildPlan B = {};
  B.filter = filter_col;
  B.mode = filter_mode;
  B.c1 = c1;
  B.c2 = c2;
  B.key = dim_key;
  B.val = dim_val;
  B.n = num_tuples;
  B.ht = ht;
  B.slots = num_slots;
  B.kmin = key_min;
  B.layout = dim_val != nullptr ? MB_HT_KEY_VAL : MB_HT_KEY;
  B.presence = presence;
  return launch_build(B, static_cast<cudaStream_t>(stream));
}

extern "C" int mb_build_tables(const mb_table_build* builds, int num_builds, int* zero, int64_t zero_words,
                               mb_stream_t stream) {
  if (num_builds < 0 || num_builds > MB_MAX_TABLE_BUILDS || (num_builds > 0 && builds == nullptr)) return MB_ERR_ARG;
  if (zero_words < 0 || (zero_words > 0 && zero == nullptr)) return MB_ERR_ARG;
  BuildPlan plan[MB_MAX_TABLE_BUILDS] = {};
  int count = 0;
  ZeroMany Z = {};
  auto clear = [&](void* p, long long words) {
    if (words == 0) return;
    Z.at[Z.count] = static_cast<int*>(p);
    Z.words[Z.count++] = words;
  };
  clear(zero, zero_words);
  for (int t = 0; t < num_builds; ++t) {
    const mb_table_build& b = builds[t];
    if (b.ht == nullptr || b.num_tuples < 0 || b.num_slots <= 0 || (b.num_tuples > 0 && b.dim_key == nullptr))
      return MB_ERR_ARG;
    if (b.filter_col != nullptr && (b.filter_mode < MB_FILTER_EQ || b.filter_mode > MB_FILTER_EQ_OR_EQ))
      return MB_ERR_ARG;
    if (b.dim_val != nullptr && !aligned8(b.ht)) return MB_ERR_ALIGN;
    clear(b.ht, (b.dim_val != nullptr ? 2ll : 1ll) * b.num_slots);
    if (b.presence != nullptr) clear(b.presence, (b.num_slots + 31ll) / 32);
    if (b.num_tuples == 0) continue;
    BuildPlan& B = plan[count++];
    B.filter = b.filter_col;
    B.mode = b.filter_mode;
    B.c1 = b.c1;
    B.c2 = b.c2;
    B.key = b.dim_key;
    B.val = b.dim_val;
    B.n = b.num_tuples;
    B.ht = b.ht;
    B.slots = b.num_slots;
    B.kmin = b.key_min;
    B.layout = b.dim_val != nullptr ? MB_HT_KEY_VAL : MB_HT_KEY;
    B.presence = b.presence;
  }
  int err = MB_OK;
  DeviceState* ds = current_device_state(&err);
  if (ds == nullptr) return err;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (Z.count > 0) {
    long long most = 0;
    for (int i = 0; i < Z.count; ++i) most = Z.words[i] > most ? Z.words[i] : most;
    long long blocks = (most / 4 + kBuildThreads - 1) / kBuildThreads;
    const long long cap = static_cast<long long>(ds->num_sms) * 8;
    blocks = blocks < 1 ? 1 : blocks > cap ? cap : blocks;
    if (launch_dependent(zero_many_kernel, static_cast<int>(blocks), kBuildThreads, 0, st, Z) != cudaSuccess)
      return MB_ERR_LAUNCH;
    note_launches(1);
  }
  // all of them together, but a build into memory that an earlier one writes after that one
  auto shares = [](const BuildPlan& x, const BuildPlan& y) {
    auto meet = [](const void* p, long long pw, const void* q, long long qw) {  // of pw and qw words
      const uintptr_t a = reinterpret_cast<uintptr_t>(p), b = reinterpret_cast<uintptr_t>(q);
      return a != 0 && b != 0 && a < b + 4 * static_cast<uintptr_t>(qw) && b < a + 4 * static_cast<uintptr_t>(pw);
    };
    const long long xt = (x.layout == MB_HT_KEY ? 1ll : 2ll) * x.slots, xb = (x.slots + 31ll) / 32;
    const long long yt = (y.layout == MB_HT_KEY ? 1ll : 2ll) * y.slots, yb = (y.slots + 31ll) / 32;
    return meet(x.ht, xt, y.ht, yt) || meet(x.ht, xt, y.presence, yb) || meet(x.presence, xb, y.ht, yt) ||
           meet(x.presence, xb, y.presence, yb);
  };
  for (int t = 0; t < count;) {
    BuildMany M = {};
    for (; t < count; ++t) {
      bool after = false;
      for (int o = 0; o < M.count; ++o) after = after || shares(plan[t], M.b[o]);
      if (after) break;
      BuildPlan& B = M.b[M.count];
      B = plan[t];
      B.status = ds->status;
      const long long per_block = static_cast<long long>(kBuildThreads) * kBuildItems;
      M.first[M.count + 1] = M.first[M.count] + static_cast<int>((B.n + per_block - 1) / per_block);
      ++M.count;
    }
    if (launch_dependent(build_many_kernel, M.first[M.count], kBuildThreads, 0, st, M) != cudaSuccess)
      return MB_ERR_LAUNCH;
    note_launches(1);
  }
  return MB_OK;
}

extern "C" int mb_join_build(const int* dim_key, const int* dim_val, int num_tuples, int* hash_table,
                             int num_slots, mb_stream_t stream) {
  if (dim_val == nullptr) return MB_ERR_ARG;
  return mb_build_pht(nullptr, 0, 0, 0, dim_key, dim_val, num_tuples, hash_table, num_slots, 0, nullptr, stream);
}

// The engine builds (VAL_OFF layout): build_GPU2 / build_GPU_minmax over a segment range,
// build_GPU3 / build_GPU_minmax2 over a list of dimension rows (dim_off), the minmax forms
// also folding the key range into *min_out / *max_out.
static int engine_build(const int* gpuCache, const int* dim_off, const mb_filterArgsGPU* fargs,
                        const mb_buildArgsGPU* bargs, int num_tuples, int* hash_table, int start_offset,
                        const short* segment_group, int* min_out, int* max_out, mb_stream_t stream) {
  if (num_tuples == 0) return MB_OK;
  if (bargs == nullptr || bargs->key_idx == nullptr || hash_table == nullptr || num_tuples < 0 ||
      bargs->num_slots <= 0)
    return MB_ERR_ARG;
  if ((min_out == nullptr) != (max_out == nullptr)) return MB_ERR_ARG;
  if (!aligned8(hash_table)) return MB_ERR_ALIGN;
  // the list forms take no filter (GPUProcessing.h:1018, cudaAssert(fargs.filter_idx1 == NULL))
  if (dim_off != nullptr && fargs != nullptr && fargs->filter_idx1 != nullptr) return MB_ERR_ARG;
  BuildPlan B = {};
  B.rows = dim_off;
  B.min_out = min_out;
  B.max_out = max_out;
  B.val_min = bargs->val_min;
  B.val_max = bargs->val_max;
  if (fargs != nullptr && fargs->filter_idx1 != nullptr) {
    if (fargs->mode1 < MB_FILTER_EQ || fargs->mode1 > MB_FILTER_EQ_OR_EQ) return MB_ERR_ARG;
    B.filter = fargs->filter_idx1;
    B.mode = fargs->mode1;
    B.c1 = fargs->compare1;
    B.c2 = fargs->compare2;
  }
  B.key = bargs->key_idx;
  B.val = bargs->val_idx;
  B.n = num_tuples;
  B.ht = hash_table;
  B.slots = bargs->num_slots;
  B.kmin = bargs->val_min;
  B.layout = MB_HT_VAL_OFF;
  B.gpu_cache = gpuCache;
  B.seg_group = dim_off != nullptr ? nullptr : segment_group;
  B.start_offset = dim_off != nullptr ? 0 : start_offset;
  B.seg_shift = 20;  // SEGMENT_SIZE = 1,048,576 (src/gpudb/common.h:73)
  return launch_build(B, static_cast<cudaStream_t>(stream));
}

extern "C" int mb_build_GPU2(const int* gpuCache, const mb_filterArgsGPU* fargs, const mb_buildArgsGPU* bargs,
                             int num_tuples, int* hash_table, int start_offset, const short* segment_group,
                             mb_stream_t stream) {
  return engine_build(gpuCache, nullptr, fargs, bargs, num_tuples, hash_table, start_offset, segment_group, nullptr,
                      nullptr, stream);
}

extern "C" int mb_build_GPU3(const int* gpuCache, const int* dim_off, const mb_filterArgsGPU* fargs,
                             const mb_buildArgsGPU* bargs, int num_tuples, int* hash_table, mb_stream_t stream) {
  if (dim_off == nullptr) return MB_ERR_ARG;
  return engine_build(gpuCache, dim_off, fargs, bargs, num_tuples, hash_table, 0, nullptr, nullptr, nullptr, stream);
}

extern "C" int mb_build_GPU_minmax(const int* gpuCache, const mb_filterArgsGPU* fargs, const mb_buildArgsGPU* bargs,
                                   int num_tuples, int* hash_table, int* min_global, int* max_global,
                                   int start_offset, const short* segment_group, mb_stream_t stream) {
  if (min_global == nullptr || max_global == nullptr) return MB_ERR_ARG;
  return engine_build(gpuCache, nullptr, fargs, bargs, num_tuples, hash_table, start_offset, segment_group,
                      min_global, max_global, stream);
}

extern "C" int mb_build_GPU_minmax2(const int* gpuCache, const int* dim_off, const mb_filterArgsGPU* fargs,
                                    const mb_buildArgsGPU* bargs, int num_tuples, int* hash_table, int* min_global,
                                    int* max_global, mb_stream_t stream) {
  if (dim_off == nullptr || min_global == nullptr || max_global == nullptr) return MB_ERR_ARG;
  return engine_build(gpuCache, dim_off, fargs, bargs, num_tuples, hash_table, 0, nullptr, min_global, max_global,
                      stream);
}

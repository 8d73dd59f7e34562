// batch.cu — batched multi-query star execution (see mb_batch_run in mordred_b200.h).
//
// A batch of up to 256 queries is answered by one scan of the fact table:
//   * a producer warp streams fact tiles (the union of the columns the batch reads) into
//     a ring of shared-memory stages with 1-D bulk copies (cp.async.bulk, no multicast);
//   * per row, each needed dimension is looked up once in its packed attribute table (PAT,
//     one 32-bit word per hash slot: bit 31 present, attribute fields below) and the word
//     replaces the key in the stage; in small batches only while some query left for the row
//     reads that dimension;
//   * predicates are evaluated for all queries at once: tables built per batch map an
//     attribute's value — or the values of several attributes with small domains together —
//     to the bitmask of queries accepting it (queries that do not constrain an attribute
//     accept every value), and a table over the 16 dimension-presence patterns does the
//     same for the dimensions each query needs; a row ANDs one mask per table and visits
//     only the queries left set;
//   * queries that add the same expression to the same group index form a class (the forms
//     of one template). Class by class, the (row, query) pairs a warp finds go to a list in
//     shared memory and are aggregated 32 pairs at a time, one per lane: value, keys and
//     group come from fields that are the same for all lanes, the destination from a
//     16-byte record of the query — its scalar or shared-memory group array (flushed once
//     per CTA) or its group array in L2. Queries beyond the four largest classes are
//     aggregated from a 32-byte descriptor of their own.
// What bounds it: instruction issue, with the shared-memory pipe behind it (mask reads, match
// lists, the sums' atomics): 64 and 60 % issue-active at 256 and 24 queries. With a descriptor
// read for every match and a mask table for every attribute, the form before, the warps issued
// 80 instructions a row for 256 queries and 23 for 24; now 69 and 15. 256 queries over 60 M rows
// 6,940 -> 5,230 us a call, over 20 M date-sorted rows 2,500 -> 1,650; 24 queries over a
// date-sorted chunk of 75 M rows 3,130 -> 1,950.
// A query's result equals its lone run through mb_star_query with filtered hash tables:
// with unique dimension keys, "the key is in the filtered table" is "the row's
// attributes pass the filter", and the payload is the attribute itself; sums are
// integers, so the order of additions cannot change a bit.
#include <algorithm>
#include <climits>
#include <cstddef>
#include <cstring>
#include <mutex>
#include <vector>

#include "common.cuh"

namespace mb {

constexpr unsigned kFullMask = 0xffffffffu;
constexpr int kBatchStages = 8;
constexpr int kMaxPredFields = 8;
constexpr int kMaskWordsMax = MB_BATCH_MAX_QUERIES / 32;
constexpr int kSmemTableMaxEntries = 512;  // predicate tables up to this many values sit in shared memory
constexpr int kCombineMaxEntries = 320;    // entries of a table that combines several small attributes
constexpr int kMaxComponents = 4;          // attributes a table combines
constexpr int kMaxClasses = 4;
// Shared memory the default group placement fills at most: what is left of the SM's 256 KB is L1,
// and the dimension lookups of every row miss it — with 28 KB of L1 few can be in flight. 256
// queries over 20 M rows, group arrays up to 32 KB (60 KB of L1) 1.84 ms, 64 KB and more 2.20;
// date-sorted 1.73 and 2.05.
constexpr int kSmemBesideL1 = 195 * 1024;
constexpr int kMatchListCap = 512;         // pairs of one class a consumer warp collects before aggregating
constexpr int kColPad = 4;                 // words between staged columns: the same row of two columns
                                           // falls in different banks (and stays 16-byte aligned)
constexpr int kMaxStageCols = MB_NUM_FACT_COLS + 1;
constexpr int kMaxBreakpoints = 768;       // range end points of wide attributes, over all of them
constexpr int kMaxBuckets = 2048;          // bucket index entries per wide attribute
constexpr int kScalarCopies = 4;           // shared-memory copies of each scalar sum, one per lane mod 4:
                                           // rows of one date (a date-sorted table) match the same
                                           // scalar queries, and same-word atomics of one warp serialise

// Field codes inside the kernel address staged columns: (stage column << 11) | (shift << 6) | width.
// Aggregation descriptor of one query (32 bytes, shared memory). The group index is
// k0*kmul0 + k1*kmul1 + bias in 32-bit wrapping arithmetic, which equals
// (k0 - kmin0)*kmul0 + (k1 - kmin1)*kmul1 with bias = -(kmin0*kmul0 + kmin1*kmul1); an
// absent key has multiplier 0. Scalars are one-group arrays.
struct __align__(16) AQ {
  uint16_t a0, a1, k0, k1;  // stage field codes
  unsigned kmul0, kmul1, bias;
  int total;                // groups (1 for a scalar)
  int soff;                 // shared-memory byte offset of the 64-bit sums; < 0: sums by L2
                            // atomics, and soff <= -2 puts the keys' touch bitmap at -soff - 2
  int flags;                // bits 0-1 agg op, bit 2 CRYSTAL4 keys, bits 3-4 number of keys,
                            // bit 5 a scalar kept in kScalarCopies words (lane mod 4 adds to
                            // its own), bits 8-16 its family's group stride, bits 17-25 its
                            // place in it
};
// A family is a set of queries with the same group count whose shared-memory sums are
// interleaved group-major: the sum of group g of the family's j-th query lies at
// base + 8 * (g * stride + j) (soff = base + 8 * j), so the matches of one row — same
// group, neighbouring queries — hit neighbouring words rather than banks at random. The
// stride is the member count rounded up to an odd number: matches of one query to
// different groups (rows of one date on a date-sorted table match the same queries) then
// fall in different bank pairs, where an even stride that is a multiple of 16 would put
// them all in one. The members' touch bitmaps follow the sums:
// base + 8 * total * stride + 4 * words * j. A query alone is a family of one.
__device__ __forceinline__ int aq_family(const AQ& A) { return (A.flags >> 8) & 0x1ff; }
__device__ __forceinline__ int aq_member(const AQ& A) { return (A.flags >> 17) & 0x1ff; }
static_assert(sizeof(AQ) == 32, "aggregation descriptor size");

// What a match of a query needs when its class supplies value, group and keys (16 bytes,
// shared memory).
struct __align__(16) QD {
  int soff;    // shared-memory byte offset of the sums; < 0: at s_addr[query]
  int stride;  // bytes between the sums of neighbouring groups
  int touch;   // >= 0: shared-memory byte offset of the key touch bitmap; -1: no keys to
               // write; -2: written on every match
  int pad;
};
static_assert(sizeof(QD) == 16, "match record size");

// Per-query descriptor in the launch parameters (96 bytes).
struct BQ {
  AQ a;
  uint8_t np, res_layout, pad[2];
  uint16_t pf[MB_BATCH_MAX_PREDS];  // row-schema field codes of the predicates
  int plo[MB_BATCH_MAX_PREDS], phi[MB_BATCH_MAX_PREDS];
  int pad2;
  void* res;
};
static_assert(sizeof(BQ) == 96, "descriptor size");

// A field of a staged row: word offset of its column in the stage, shift, mask.
struct Field {
  int word, shift;
  unsigned mask;
};

// An attribute the batch constrains, and its part in a table of query masks. A table covers
// one attribute or several with few values, and holds one mask per combination of their
// indexes (the sum of index * mul). An attribute's index is its value less `min`, or its
// interval when interval-coded, or one more than the last of these for every value outside
// the queries' hull (which no query constraining the attribute accepts).
// Interval coding of a wide attribute (hull wider than kSmemTableMaxEntries values): the
// queries' range end points cut the hull into nint intervals on which every query's verdict
// is constant; the table holds one mask per interval. A value v (relative to min) is in
// interval i when bp[i] <= v < bp[i+1]; bucket v >> bkt_shift of a shared-memory index gives
// the interval of the bucket's first value, and a short forward scan over the end points
// finishes the search.
struct Attr {
  Field f;
  int code, scode;         // row-schema and stage field codes
  int min, n;              // hull
  int nint, bp_off, bkt_shift;
  int bps_off, bkt_off;    // shared-memory byte offsets of end points and bucket index
  int mul;
  int last;                // 1: the last attribute of its table, which the fields below describe
  int ent, smem_off;       // entries; byte offset in shared memory, -1: in the workspace
  long long goff;          // word offset in the workspace
};

// A dimension the batch reads: where its key and its word lie in the stage, its table, and
// per query whether the row must exist (need) and whether the query reads the word at all.
struct Dim {
  int d, key_word, word;
  int slots, kmin;
  const unsigned* pat;
  unsigned need[kMaskWordsMax], use[kMaskWordsMax];
};

// What the queries of a class share (see AQ).
struct Class {
  Field a0, a1, k0, k1;
  unsigned kmul0, kmul1, bias;
  int total, op, scalar, two_keys;
};

struct BatchPlan {
  long long n, nfull;
  int ncols;                       // staged fact columns
  const int* col[MB_NUM_FACT_COLS];
  int cidx[13];                    // row-schema column -> stage column (-1: absent)
  int stage_dim[kMaxStageCols];    // stage column -> dimension whose word it holds (-1: fact column)
  int ndims;
  Dim dim[4];
  int nq, nwords;
  // The attributes some query constrains: those of fact columns first (nfact), then those of
  // dimension words; attributes that share a table are neighbours.
  int nfields, nfact;
  Attr at[kMaxPredFields];
  int bp[kMaxBreakpoints];
  unsigned pres_mask[16][kMaskWordsMax];
  unsigned all[kMaskWordsMax];
  int ncls, others;                // classes; 1: some queries belong to none
  Class cls[kMaxClasses];
  unsigned cls_mask[kMaxClasses + 1][kMaskWordsMax];  // ... the last: queries without a class
  unsigned* tables;                // workspace
  long long table_entries;
  int stages, stage_words;
  int smem_acc_off, smem_aq_off, smem_qd_off, smem_res_off, smem_addr_off, smem_pres_off, smem_list_off;
  int acc_words;                   // 8-byte scalar words (kScalarCopies per scalar query)
  int smem_groups_off, smem_groups_words, smem_stage_off;
  unsigned int* status;
  // segment-cache addressing: col[c] is a per-segment slot array into gpu_cache
  const int* gpu_cache;
  const short* seg_group;
  int seg_shift;
  BQ q[MB_BATCH_MAX_QUERIES];
};
static_assert(sizeof(BatchPlan) < 32000, "launch parameter limit");

// (key - kmin) % slots: keys within two table lengths of kmin without a division.
__device__ __forceinline__ int bslot(int key, int slots, int kmin) {
  const unsigned d = static_cast<unsigned>(key) - static_cast<unsigned>(kmin), n = static_cast<unsigned>(slots);
  const unsigned h = min(d, d - n);
  return h < n ? static_cast<int>(h) : slow_mod(static_cast<int>(d), slots);
}

// Physical tile of scan position t (CTA b takes positions b, b + G, b + 2G, ...). The
// first kTileRegions * Q tiles (Q = nfull / kTileRegions) are visited column-major over
// kTileRegions regions of the table, so the tiles the grid holds at one moment lie in
// different regions rather than side by side. On a table sorted by date, side-by-side
// tiles share a date: every SM would then add into the same queries' group records (the
// same year's) at once, while the regions spread those updates over the table's years.
// Every CTA still sees every region, so the work stays balanced.
constexpr long long kTileRegions = 16;
__device__ __forceinline__ long long tile_order(long long t, long long nfull) {
  const long long q = nfull / kTileRegions;
  if (t >= q * kTileRegions) return t;
  return (t % kTileRegions) * q + t / kTileRegions;
}

__device__ __forceinline__ int field_value(int v, int code) {
  const int width = code & 63;
  const unsigned shift = (code >> 6) & 31;
  const unsigned mask = width >= 32 ? 0xffffffffu : (1u << width) - 1u;
  return static_cast<int>((static_cast<unsigned>(v) >> shift) & mask);
}

// Stage column c, row r, read from global memory (direct, or through the segment cache).
__device__ __forceinline__ int batch_load(const BatchPlan& P, int c, long long r) {
  if (P.gpu_cache == nullptr) return __ldg(P.col[c] + r);
  const long long vseg = r >> P.seg_shift;
  const int seg = P.seg_group ? static_cast<int>(P.seg_group[vseg]) : static_cast<int>(vseg);
  return __ldg(P.gpu_cache + (static_cast<long long>(__ldg(P.col[c] + seg)) << P.seg_shift) +
               (r & ((1ll << P.seg_shift) - 1)));
}

__device__ __forceinline__ void bmbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ AQ load_aq(const AQ* s_aq, int qi) {
  const uint4* p = reinterpret_cast<const uint4*>(s_aq + qi);
  const uint4 x = p[0], y = p[1];
  AQ a;
  a.a0 = static_cast<uint16_t>(x.x);
  a.a1 = static_cast<uint16_t>(x.x >> 16);
  a.k0 = static_cast<uint16_t>(x.y);
  a.k1 = static_cast<uint16_t>(x.y >> 16);
  a.kmul0 = x.z;
  a.kmul1 = x.w;
  a.bias = y.x;
  a.total = static_cast<int>(y.y);
  a.soff = static_cast<int>(y.z);
  a.flags = static_cast<int>(y.w);
  return a;
}

// The 32-bit value a match adds (sign-extended to 64 bits by the caller), as the
// single-query path computes it: SUM a0, SUB a0 - a1, MUL a0 * a1 (wrapping).
template <class Get>
__device__ __forceinline__ unsigned batch_value(const AQ& A, Get get) {
  const unsigned v0 = static_cast<unsigned>(get(A.a0)), v1 = static_cast<unsigned>(get(A.a1));
  const int op = A.flags & 3;
  return op == MB_AGG_SUM ? v0 : op == MB_AGG_SUB ? v0 - v1 : v0 * v1;
}

// Add one (row, query) match: `get(code)` reads a field of the row.
template <class Get>
__device__ __forceinline__ void batch_match(const AQ& A, void* const* s_res, int qi, Get get, unsigned char* smem,
                                            bool& bad_group) {
  const unsigned u = batch_value(A, get);
  const unsigned long long w = static_cast<unsigned long long>(static_cast<long long>(static_cast<int>(u)));
  const int k0 = get(A.k0), k1 = get(A.k1);
  const unsigned hh = static_cast<unsigned>(k0) * A.kmul0 + static_cast<unsigned>(k1) * A.kmul1 + A.bias;
  int g = static_cast<int>(hh);
  if (hh >= static_cast<unsigned>(A.total)) {
    g %= A.total;
    if (g < 0) {
      bad_group = true;
      return;
    }
  }
  const bool c4 = (A.flags >> 2) & 1;
  if (A.soff >= 0) {
    const int fam = aq_family(A), j = aq_member(A);
    const int copy = (A.flags >> 5) & 1 ? static_cast<int>(threadIdx.x & (kScalarCopies - 1)) : 0;
    smem_add_i64(reinterpret_cast<unsigned long long*>(smem + A.soff) + g * fam + copy, static_cast<int>(u));
    if (!c4) return;
    // the first row of a group in this CTA writes the group's keys
    uint32_t* s_touch = reinterpret_cast<uint32_t*>(smem + A.soff - 8 * j + 8 * A.total * fam) +
                        j * ((A.total + 31) >> 5);
    const uint32_t bit = 1u << (g & 31);
    if ((s_touch[g >> 5] & bit) || (atomicOr(&s_touch[g >> 5], bit) & bit)) return;
  } else {
    void* res = s_res[qi];
    atomicAdd(c4 ? reinterpret_cast<unsigned long long*>(static_cast<int*>(res) + 4 * g + 2)
                 : static_cast<unsigned long long*>(res) + g,
              w);
    if (!c4) return;
    if (A.soff <= -2) {
      // keys once per CTA and group: the group records are few lines that every SM updates
      uint32_t* s_touch = reinterpret_cast<uint32_t*>(smem + (-A.soff - 2));
      const uint32_t bit = 1u << (g & 31);
      if ((s_touch[g >> 5] & bit) || (atomicOr(&s_touch[g >> 5], bit) & bit)) return;
    }
  }
  int* res = static_cast<int*>(s_res[qi]);
  const int nk = (A.flags >> 3) & 3;
  if (nk > 1)
    *reinterpret_cast<int2*>(res + 4 * g) = make_int2(k0, k1);  // one 8-byte store (16-byte records)
  else if (nk > 0)
    res[4 * g] = k0;
}

__device__ __forceinline__ int field_of(const int* row, const Field& f) {
  return static_cast<int>((static_cast<unsigned>(row[f.word]) >> f.shift) & f.mask);
}

// Index of a value among attribute A's table indexes (see Attr).
__device__ __forceinline__ int attr_index(const BatchPlan& P, const Attr& A, int value, const unsigned char* smem) {
  const unsigned v = static_cast<unsigned>(value) - static_cast<unsigned>(A.min);
  const unsigned n = static_cast<unsigned>(A.n);
  if (A.nint == 0) return static_cast<int>(min(v, n));
  if (v >= n) return A.nint;
  const int* bp = reinterpret_cast<const int*>(smem + A.bps_off);
  int e = reinterpret_cast<const uint16_t*>(smem + A.bkt_off)[v >> A.bkt_shift];
  while (e + 1 < A.nint && bp[e + 1] <= static_cast<int>(v)) ++e;
  return e;
}

// m &= entry e of the table that attribute A closes. Entries of eight words lie in two arrays
// of four, so that the 16-byte loads of neighbouring entries fall in different banks.
template <int NWM>
__device__ __forceinline__ void and_entry(const BatchPlan& P, const Attr& A, int e, const unsigned char* smem,
                                          unsigned (&m)[NWM]) {
  const unsigned* base = A.smem_off >= 0 ? reinterpret_cast<const unsigned*>(smem + A.smem_off) : P.tables + A.goff;
  if constexpr (NWM >= 4) {
#pragma unroll
    for (int h = 0; h < NWM / 4; ++h) {
      const uint4 u = *reinterpret_cast<const uint4*>(base + 4 * (h * A.ent + e));
      m[4 * h] &= u.x;
      m[4 * h + 1] &= u.y;
      m[4 * h + 2] &= u.z;
      m[4 * h + 3] &= u.w;
    }
  } else if constexpr (NWM == 2) {
    const uint2 u = *reinterpret_cast<const uint2*>(base + 2 * e);
    m[0] &= u.x;
    m[1] &= u.y;
  } else {
    m[0] &= base[e];
  }
}

// The masks of GR rows (row r at stage pointer row + 32 r) ANDed with the tables over fact
// columns (DIMS false) or over dimension words.
template <int NWM, int GR, bool DIMS>
__device__ __forceinline__ void and_tables(const BatchPlan& P, const int* row, const unsigned char* smem,
                                           unsigned (&m)[GR][NWM]) {
  int e[GR];
#pragma unroll
  for (int r = 0; r < GR; ++r) e[r] = 0;
#pragma unroll
  for (int i = 0; i < kMaxPredFields; ++i) {
    if (i >= (DIMS ? P.nfields : P.nfact)) break;
    if (DIMS && i < P.nfact) continue;
    const Attr& A = P.at[i];
#pragma unroll
    for (int r = 0; r < GR; ++r) e[r] += attr_index(P, A, field_of(row + 32 * r, A.f), smem) * A.mul;
    if (A.last) {
#pragma unroll
      for (int r = 0; r < GR; ++r) {
        and_entry<NWM>(P, A, e[r], smem, m[r]);
        e[r] = 0;
      }
    }
  }
}

template <int NCW, int ITEMS, int NWM>
__global__ void __launch_bounds__((NCW + 1) * 32, 1) batch_kernel(const __grid_constant__ BatchPlan P) {
  constexpr int WROWS = 32 * ITEMS;
  constexpr int TILE = NCW * WROWS;
  constexpr int CS = TILE + kColPad;  // stage column stride (words)
  constexpr int NWARPS = NCW + 1;
  // rows a lane works on at a time: their table lookups are in flight together and their
  // matches share the aggregation passes (as many as eight mask words in registers allow)
  constexpr int GR = ITEMS * NWM <= 8 ? ITEMS : NWM >= 8 ? 1 : 8 / NWM;
  static_assert(ITEMS % GR == 0, "whole groups of rows");
  // with one or two mask words a row often runs out of queries on its fact columns: it then
  // looks up a dimension only if a query that reads it is left
  constexpr bool LAZY = NWM <= 2;
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty = full + kBatchStages;
  AQ* s_aq = reinterpret_cast<AQ*>(smem + P.smem_aq_off);
  QD* s_qd = reinterpret_cast<QD*>(smem + P.smem_qd_off);
  void** s_res = reinterpret_cast<void**>(smem + P.smem_res_off);
  unsigned char** s_addr = reinterpret_cast<unsigned char**>(smem + P.smem_addr_off);
  unsigned* s_pres = reinterpret_cast<unsigned*>(smem + P.smem_pres_off);
  int* stage_base = reinterpret_cast<int*>(smem + P.smem_stage_off);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int S = P.stages;

  wait_for_predecessor();  // the mask kernel, or the batch before
  // ---- set-up: accumulators, descriptors, masks, small tables, barriers ------------
  {
    unsigned long long* s_acc = reinterpret_cast<unsigned long long*>(smem + P.smem_acc_off);
    for (int w = tid; w < P.acc_words; w += NWARPS * 32) s_acc[w] = 0;
    for (int q = tid; q < P.nq; q += NWARPS * 32) {
      const BQ& Q = P.q[q];
      const AQ A = Q.a;
      const bool c4 = (A.flags >> 2) & 1;
      const int nk = (A.flags >> 3) & 3;
      s_aq[q] = A;
      s_res[q] = Q.res;
      s_addr[q] = static_cast<unsigned char*>(Q.res) + (c4 ? 8 : 0);
      QD d;
      d.soff = A.soff >= 0 ? A.soff : -1;
      d.stride = A.soff < 0 ? (c4 ? 16 : 8) : (A.flags >> 5) & 1 ? 8 : 8 * aq_family(A);
      d.touch = !c4 || nk == 0 ? -1
                : A.soff >= 0  ? A.soff - 8 * aq_member(A) + 8 * A.total * aq_family(A) +
                                    4 * ((A.total + 31) >> 5) * aq_member(A)
                : A.soff <= -2 ? -A.soff - 2
                               : -2;
      d.pad = 0;
      s_qd[q] = d;
    }
    for (int w = tid; w < 16 * kMaskWordsMax; w += NWARPS * 32) s_pres[w] = (&P.pres_mask[0][0])[w];
    unsigned* g = reinterpret_cast<unsigned*>(smem + P.smem_groups_off);
    for (int w = tid; w < P.smem_groups_words; w += NWARPS * 32) g[w] = 0;
    for (int f = 0; f < P.nfields; ++f) {
      const Attr& A = P.at[f];
      if (A.last && A.smem_off >= 0) {
        unsigned* dst = reinterpret_cast<unsigned*>(smem + A.smem_off);
        const unsigned* src = P.tables + A.goff;
        for (int w = tid; w < A.ent * NWM; w += NWARPS * 32) dst[w] = src[w];
      }
      int* bp = reinterpret_cast<int*>(smem + A.bps_off);
      for (int i = tid; i < A.nint; i += NWARPS * 32) bp[i] = P.bp[A.bp_off + i];
    }
  }
  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], NCW);
    }
    mbar_fence_init();
  }
  __syncthreads();
  // bucket indexes of the interval-coded attributes: the interval of each bucket's first value
  for (int f = 0; f < P.nfields; ++f) {
    const Attr& A = P.at[f];
    if (A.nint == 0) continue;
    const int* bp = reinterpret_cast<const int*>(smem + A.bps_off);
    uint16_t* bkt = reinterpret_cast<uint16_t*>(smem + A.bkt_off);
    const int nb = ((A.n - 1) >> A.bkt_shift) + 1;
    for (int b = tid; b < nb; b += NWARPS * 32) {
      const int v0 = b << A.bkt_shift;
      int lo = 0, hi = A.nint - 1;  // bp[0] = 0 <= v0: find the last bp[i] <= v0
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (bp[mid] <= v0)
          lo = mid;
        else
          hi = mid - 1;
      }
      bkt[b] = static_cast<uint16_t>(lo);
    }
  }
  __syncthreads();

  const long long G = gridDim.x, b = blockIdx.x;
  const long long my_tiles = P.nfull > b ? (P.nfull - 1 - b) / G + 1 : 0;
  bool failed = false, bad_probe = false, bad_group = false;

  if (warp == 0) {
    if (lane == 0) {
      const uint64_t policy = l2_policy_evict_first();
      long long k = 0;
      int s = 0;
      uint32_t phase = 0;
      for (; k < my_tiles; ++k) {
        if (k >= S && !mbar_wait_bounded(&empty[s], phase ^ 1u)) {
          failed = true;
          break;
        }
        const long long r0 = tile_order(b + k * G, P.nfull) * static_cast<long long>(TILE);
        int* dst = stage_base + s * P.stage_words;
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(&full[s], static_cast<uint32_t>(P.ncols) * TILE * 4u);
        if (P.gpu_cache == nullptr) {
          for (int c = 0; c < P.ncols; ++c) bulk_g2s(dst + c * CS, P.col[c] + r0, TILE * 4, &full[s], policy);
        } else {
          // through the segment cache: a tile that crosses a segment boundary is copied in
          // two pieces (row offsets are multiples of 4, so every piece is 16-byte aligned)
          const long long S = 1ll << P.seg_shift;
          for (int done = 0; done < TILE;) {
            const long long r = r0 + done;
            const long long vseg = r >> P.seg_shift;
            const int seg = P.seg_group ? static_cast<int>(P.seg_group[vseg]) : static_cast<int>(vseg);
            const long long in = r & (S - 1);
            const int take = static_cast<int>(S - in < TILE - done ? S - in : TILE - done);
            // all slots first (their loads in flight together), then the ordered copies
            int slot[MB_NUM_FACT_COLS];
#pragma unroll
            for (int c = 0; c < MB_NUM_FACT_COLS; ++c)
              if (c < P.ncols) slot[c] = P.col[c][seg];
#pragma unroll
            for (int c = 0; c < MB_NUM_FACT_COLS; ++c)
              if (c < P.ncols)
                bulk_g2s(dst + c * CS + done, P.gpu_cache + (static_cast<long long>(slot[c]) << P.seg_shift) + in,
                         static_cast<uint32_t>(take) * 4u, &full[s], policy);
            done += take;
          }
        }
        if (++s == S) {
          s = 0;
          phase ^= 1u;
        }
      }
      for (long long j = (k > S ? k - S : 0); j < k; ++j)
        if (!mbar_wait_bounded(&full[j % S], static_cast<uint32_t>((j / S) & 1))) failed = true;
    }
  } else {
    const int cw = warp - 1;
    uint16_t* mlist = reinterpret_cast<uint16_t*>(smem + P.smem_list_off) + cw * kMatchListCap;
    int s = 0;
    uint32_t phase = 0;
    for (long long k = 0; k < my_tiles; ++k) {
      const bool ok = mbar_wait_bounded(&full[s], phase);
      if (!__all_sync(kFullMask, ok)) {
        failed = true;
        break;
      }
      int* wst = stage_base + s * P.stage_words + cw * WROWS;
#pragma unroll 1
      for (int i0 = 0; i0 < ITEMS; i0 += GR) {
        // ---- the queries accepting each row (lane l has rows i0 * 32 + l, + 32, ...) ----
        int* row = wst + i0 * 32 + lane;
        unsigned m[GR][NWM];
#pragma unroll
        for (int r = 0; r < GR; ++r)
#pragma unroll
          for (int w = 0; w < NWM; ++w) m[r][w] = P.all[w];
        auto look_up = [&](unsigned (&word)[GR][4]) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int r = 0; r < GR; ++r) word[r][j] = 0;
            if (j >= P.ndims) continue;
            const Dim& D = P.dim[j];
#pragma unroll
            for (int r = 0; r < GR; ++r) {
              const int h = bslot(row[32 * r + D.key_word], D.slots, D.kmin);
              bool want = true;
              if constexpr (LAZY) {
                want = false;
#pragma unroll
                for (int w = 0; w < NWM; ++w) want = want || (m[r][w] & D.use[w]) != 0;
              }
              if (h < 0)
                bad_probe = true;
              else if (want)
                word[r][j] = static_cast<unsigned>(ld_word(reinterpret_cast<const int*>(D.pat) + h));
            }
          }
        };
        auto keep_words = [&](const unsigned (&word)[GR][4]) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (j >= P.ndims) break;
#pragma unroll
            for (int r = 0; r < GR; ++r) row[32 * r + P.dim[j].word] = static_cast<int>(word[r][j]);
          }
        };
        if constexpr (LAZY) {
          and_tables<NWM, GR, false>(P, row, smem, m);
          unsigned word[GR][4];
          look_up(word);
          keep_words(word);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (j >= P.ndims) break;
#pragma unroll
            for (int r = 0; r < GR; ++r)
#pragma unroll
              for (int w = 0; w < NWM; ++w) m[r][w] &= word[r][j] >> 31 ? kFullMask : ~P.dim[j].need[w];
          }
        } else {
          unsigned word[GR][4];
          look_up(word);
          and_tables<NWM, GR, false>(P, row, smem, m);  // while the words are on their way
          keep_words(word);
#pragma unroll
          for (int r = 0; r < GR; ++r) {
            unsigned pres = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (j < P.ndims) pres |= (word[r][j] >> 31) << P.dim[j].d;
#pragma unroll
            for (int q = 0; q < NWM; q += 4) {
              const uint4 u = *reinterpret_cast<const uint4*>(s_pres + pres * kMaskWordsMax + q);
              m[r][q] &= u.x;
              m[r][q + 1] &= u.y;
              m[r][q + 2] &= u.z;
              m[r][q + 3] &= u.w;
            }
          }
        }
        and_tables<NWM, GR, true>(P, row, smem, m);
        // ---- class by class: list the matches, aggregate them (one copy of the code for all
        // classes: unrolled over them it no longer fits the instruction cache) ----
#pragma unroll 1
        for (int c = 0; c <= kMaxClasses; ++c) {
          if (c < kMaxClasses ? c >= P.ncls : !P.others) continue;
          int mine = 0;
#pragma unroll
          for (int w = 0; w < NWM; ++w) {
            const unsigned of = P.cls_mask[c][w];
#pragma unroll
            for (int r = 0; r < GR; ++r) mine += __popc(m[r][w] & of);
          }
          if (!__any_sync(kFullMask, mine != 0)) continue;
          int up_to = mine;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFullMask, up_to, o);
            if (lane >= o) up_to += y;
          }
          const int total = __shfl_sync(kFullMask, up_to, 31);
          if (total > kMatchListCap) {
            // more matches than the list holds: lane by lane
#pragma unroll 1
            for (int k = 0; k < GR * NWM; ++k) {
              unsigned bits = 0;
#pragma unroll
              for (int r = 0; r < GR; ++r)
#pragma unroll
                for (int w = 0; w < NWM; ++w)
                  if (k == r * NWM + w) bits = m[r][w] & P.cls_mask[c][w];
              const int* mrow = row + 32 * (k / NWM);
              auto get = [&](int code) { return field_value(mrow[(code >> 11) * CS], code); };
              while (bits) {
                const int qi = (k % NWM) * 32 + __ffs(bits) - 1;
                bits &= bits - 1;
                batch_match(load_aq(s_aq, qi), s_res, qi, get, smem, bad_group);
              }
            }
            __syncwarp();
            continue;
          }
          uint16_t* at = mlist + (up_to - mine);
#pragma unroll
          for (int w = 0; w < NWM; ++w) {
            const unsigned of = P.cls_mask[c][w];
            if (of == 0) continue;
#pragma unroll
            for (int r = 0; r < GR; ++r) {
              unsigned bits = m[r][w] & of;
              while (bits) {
                const int qi = w * 32 + __ffs(bits) - 1;
                bits &= bits - 1;
                *at++ = static_cast<uint16_t>((((i0 + r) * 32 + lane) << 8) | qi);
              }
            }
          }
          __syncwarp();
          for (int base = 0; base < total; base += 32) {
            if (base + lane >= total) continue;
            const unsigned pair = mlist[base + lane];
            const int qi = static_cast<int>(pair & 255u);
            const int* mrow = wst + (pair >> 8);
            if (c == kMaxClasses) {
              auto get = [&](int code) { return field_value(mrow[(code >> 11) * CS], code); };
              batch_match(load_aq(s_aq, qi), s_res, qi, get, smem, bad_group);
              continue;
            }
            const Class& C = P.cls[c < kMaxClasses ? c : 0];
            const unsigned v0 = static_cast<unsigned>(field_of(mrow, C.a0)), v1 = static_cast<unsigned>(field_of(mrow, C.a1));
            const int v = static_cast<int>(C.op == MB_AGG_SUM ? v0 : C.op == MB_AGG_SUB ? v0 - v1 : v0 * v1);
            const QD D = s_qd[qi];
            if (C.scalar) {
              smem_add_i64(reinterpret_cast<unsigned long long*>(smem + D.soff) + (lane & (kScalarCopies - 1)), v);
              continue;
            }
            const int k0 = field_of(mrow, C.k0), k1 = field_of(mrow, C.k1);
            const unsigned hh = static_cast<unsigned>(k0) * C.kmul0 + static_cast<unsigned>(k1) * C.kmul1 + C.bias;
            int g = static_cast<int>(hh);
            if (hh >= static_cast<unsigned>(C.total)) {
              g = slow_mod(g, C.total);
              if (g < 0) {
                bad_group = true;
                continue;
              }
            }
            if (D.soff >= 0)
              smem_add_i64(reinterpret_cast<unsigned long long*>(smem + D.soff + g * D.stride), v);
            else
              atomicAdd(reinterpret_cast<unsigned long long*>(s_addr[qi] + static_cast<long long>(g) * D.stride),
                        static_cast<unsigned long long>(static_cast<long long>(v)));
            if (D.touch == -1) continue;
            if (D.touch >= 0) {
              // the first row of a group in this CTA writes the group's keys
              uint32_t* touch = reinterpret_cast<uint32_t*>(smem + D.touch) + (g >> 5);
              const uint32_t bit = 1u << (g & 31);
              if ((*touch & bit) || (atomicOr(touch, bit) & bit)) continue;
            }
            int* out = static_cast<int*>(s_res[qi]) + 4ll * g;
            if (C.two_keys)
              *reinterpret_cast<int2*>(out) = make_int2(k0, k1);  // one 8-byte store (16-byte records)
            else
              *out = k0;
          }
          __syncwarp();
        }
      }
      __syncwarp();
      if (lane == 0) bmbar_arrive(&empty[s]);
      if (++s == S) {
        s = 0;
        phase ^= 1u;
      }
    }
    // ---- remainder rows, one per thread, straight from global memory ------------
    if (!failed) {
      for (long long r = P.nfull * TILE + b * (NCW * 32) + (tid - 32); r < P.n; r += G * (NCW * 32)) {
        int dimw[4] = {0, 0, 0, 0};
        uint32_t pr = 0;
        for (int j = 0; j < P.ndims; ++j) {
          const int d = P.dim[j].d;
          const int h = bslot(batch_load(P, P.dim[j].key_word / CS, r), P.dim[j].slots, P.dim[j].kmin);
          if (h < 0) {
            bad_probe = true;
            continue;
          }
          dimw[d] = ld_word(reinterpret_cast<const int*>(P.dim[j].pat) + h);
          pr |= (static_cast<unsigned>(dimw[d]) >> 31) << d;
        }
        auto get = [&](int code) {
          const int c = code >> 11;
          const int d = P.stage_dim[c];
          return field_value(d >= 0 ? dimw[d] : batch_load(P, c, r), code);
        };
        unsigned m[NWM];
#pragma unroll
        for (int w = 0; w < NWM; ++w) m[w] = s_pres[pr * kMaskWordsMax + w];
        int e = 0;
        for (int f = 0; f < P.nfields; ++f) {
          const Attr& A = P.at[f];
          e += attr_index(P, A, get(A.scode), smem) * A.mul;
          if (A.last) {
            and_entry<NWM>(P, A, e, smem, m);
            e = 0;
          }
        }
#pragma unroll
        for (int w = 0; w < NWM; ++w) {
          unsigned bits = m[w];
          while (bits) {
            const int qi = w * 32 + __ffs(bits) - 1;
            bits &= bits - 1;
            batch_match(load_aq(s_aq, qi), s_res, qi, get, smem, bad_group);
          }
        }
      }
    }
  }

  if (failed) set_status(P.status, MB_STATUS_TIMEOUT);
  if (bad_probe) set_status(P.status, MB_STATUS_PROBE_RANGE);
  if (bad_group) set_status(P.status, MB_STATUS_GROUP_RANGE);
  __syncthreads();
  // ---- fold this CTA's scalars and shared-memory group arrays into the results -------
  // (a zero partial is skipped: adding it changes nothing)
  for (int q = 0; q < P.nq; ++q) {
    const AQ A = s_aq[q];
    if (A.soff < 0) continue;
    const unsigned long long* s_sum = reinterpret_cast<const unsigned long long*>(smem + A.soff);
    const bool c4 = (A.flags >> 2) & 1;
    const int fam = aq_family(A);
    const bool copies = (A.flags >> 5) & 1;
    for (int g = tid; g < A.total; g += NWARPS * 32) {
      unsigned long long v = s_sum[g * fam];
      if (copies)
        for (int k = 1; k < kScalarCopies; ++k) v += s_sum[k];
      if (v == 0) continue;
      atomicAdd(c4 ? reinterpret_cast<unsigned long long*>(static_cast<int*>(s_res[q]) + 4 * g + 2)
                   : static_cast<unsigned long long*>(s_res[q]) + g,
                v);
    }
  }
}

// The tables' entries. Entry e of a table, word w holds bit (q - 32w) for every query q that
// accepts the entry's values: every one of its predicates on the table's attributes holds
// there (no value outside an attribute's hull passes a predicate on it). A warp takes 32
// entries of one table and one word: lane l knows the values of the l-th entry and the ranges
// of the l-th query, and entry by entry the values are broadcast and the verdicts balloted
// (256 queries: 13.8 us, 24 queries: 8.4; each thread walking all queries' descriptors: 70 and 8.5).
__global__ void batch_mask_kernel(const __grid_constant__ BatchPlan P, int tasks) {
  const int lane = threadIdx.x & 31;
  allow_dependent();
  wait_for_predecessor();
  for (int task = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; task < tasks; task += (gridDim.x * blockDim.x) >> 5) {
    int rest = task, first = 0, last = 0;  // the table's attributes
    for (;; first = last + 1) {
      last = first;
      while (!P.at[last].last) ++last;
      const int of_table = (P.at[last].ent + 31) / 32 * P.nwords;
      if (rest < of_table) break;
      rest -= of_table;
    }
    const int w = rest % P.nwords;
    const int e = rest / P.nwords * 32 + lane;
    // lane's query: its range on each attribute (all its predicates on one hold together)
    const int qi = 32 * w + lane;
    int lo[kMaxComponents], hi[kMaxComponents];
    unsigned constrains = 0;
#pragma unroll
    for (int c = 0; c < kMaxComponents; ++c) {
      lo[c] = INT_MIN;
      hi[c] = INT_MAX;
    }
    if (qi < P.nq) {
      const BQ& Q = P.q[qi];
      for (int p = 0; p < Q.np; ++p) {
        const int code = Q.pf[p], plo = Q.plo[p], phi = Q.phi[p];
#pragma unroll
        for (int c = 0; c < kMaxComponents; ++c)
          if (first + c <= last && code == P.at[first + c].code) {
            lo[c] = max(lo[c], plo);
            hi[c] = min(hi[c], phi);
            constrains |= 1u << c;
          }
      }
    }
    // lane's entry: the attributes' values (an interval's verdicts are those of its first value)
    int x[kMaxComponents];
    unsigned outside = 0;
#pragma unroll
    for (int c = 0; c < kMaxComponents; ++c) {
      x[c] = 0;
      if (first + c > last) continue;
      const Attr& A = P.at[first + c];
      const int n = A.nint > 0 ? A.nint : A.n;
      const int i = e / A.mul % (n + 1);
      if (i == n) outside |= 1u << c;
      x[c] = A.min + (A.nint > 0 && i < n ? P.bp[A.bp_off + i] : i);
    }
    unsigned bits = 0;
    for (int j = 0; j < 32; ++j) {
      const unsigned out = __shfl_sync(kFullMask, outside, j);
      bool ok = qi < P.nq && (out & constrains) == 0;
#pragma unroll
      for (int c = 0; c < kMaxComponents; ++c) {
        if (first + c > last) break;
        const int v = __shfl_sync(kFullMask, x[c], j);
        ok = ok && (!((constrains >> c) & 1u) || (v >= lo[c] && v <= hi[c]));
      }
      const unsigned b = __ballot_sync(kFullMask, ok);
      if (lane == j) bits = b;
    }
    const Attr& A = P.at[last];
    if (e < A.ent) {
      const long long at = P.nwords == 8 ? 4ll * ((w >> 2) * A.ent + e) + (w & 3) : static_cast<long long>(e) * P.nwords + w;
      P.tables[A.goff + at] = bits;
    }
  }
}

// ---- PAT build -----------------------------------------------------------------------
__global__ void pat_build_kernel(const int* key, int n, int kmin, int slots, const int* a0, int f0, const int* a1, int f1,
                                 const int* a2, int f2, unsigned* words, unsigned* status) {
  bool bad_slot = false, bad_attr = false;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int h = bslot(key[i], slots, kmin);
    if (h < 0) {
      bad_slot = true;
      continue;
    }
    unsigned w = 0x80000000u;
    const int* attrs[3] = {a0, a1, a2};
    const int fields[3] = {f0, f1, f2};
    for (int k = 0; k < 3; ++k) {
      if (attrs[k] == nullptr) continue;
      const int width = fields[k] & 63, shift = (fields[k] >> 6) & 31;
      const unsigned v = static_cast<unsigned>(attrs[k][i]);
      if (width < 32 && (v >> width) != 0) {
        bad_attr = true;
        continue;
      }
      w |= v << shift;
    }
    words[h] = w;
  }
  if (bad_slot) set_status(status, MB_STATUS_PROBE_RANGE);
  if (bad_attr) set_status(status, MB_STATUS_GROUP_RANGE);
}

// ---- host ----------------------------------------------------------------------------
using BatchFn = void (*)(BatchPlan);
struct BatchVariant {
  int warps, items, nwm;
  BatchFn fn;
};
#define MB_BATCH_VARIANTS(W, I) \
  {W, I, 1, batch_kernel<W, I, 1>}, {W, I, 2, batch_kernel<W, I, 2>}, {W, I, 4, batch_kernel<W, I, 4>}, \
      {W, I, 8, batch_kernel<W, I, 8>}
// (consumer warps, rows per lane per stage): more warps per CTA hide more latency; fewer
// rows per lane keep their stage ring small enough for that
static const BatchVariant kBatchVariants[] = {
    MB_BATCH_VARIANTS(8, 4), MB_BATCH_VARIANTS(16, 4), MB_BATCH_VARIANTS(16, 2),
    MB_BATCH_VARIANTS(24, 1), MB_BATCH_VARIANTS(24, 2), MB_BATCH_VARIANTS(30, 1),
};

static bool field_ok(int code) {
  const int col = code >> 11, width = code & 63, shift = (code >> 6) & 31;
  return col >= 0 && col <= MB_COL_DIM_D && width >= 1 && width <= 32 && (width == 32 || shift + width <= 32) &&
         code < 65536;
}

int batch_init_device(const DeviceState& ds) {
  for (const BatchVariant& v : kBatchVariants)
    if (cudaFuncSetAttribute(reinterpret_cast<const void*>(v.fn), cudaFuncAttributeMaxDynamicSharedMemorySize,
                             ds.max_smem_optin - 2048) != cudaSuccess)
      return MB_ERR_CUDA;
  return MB_OK;
}

// Fill everything but the shared-memory layout; returns MB_OK or an error.
// `sizing`: only what the workspace size needs (the queries keep the caller's order).
static int plan_batch(const mb_batch_args* a, BatchPlan& P, bool sizing) {
  if (a == nullptr || a->num_queries < 1 || a->num_queries > MB_BATCH_MAX_QUERIES || a->queries == nullptr)
    return MB_ERR_ARG;
  if (a->num_rows < 0) return MB_ERR_ARG;
  memset(&P, 0, offsetof(BatchPlan, q));  // the queries' descriptors are cleared one by one below
  P.n = a->num_rows;
  P.nq = a->num_queries;
  // mask words per entry, rounded to 1, 2, 4 or 8 so table entries stay 16-byte aligned
  const int words = (P.nq + 31) / 32;
  P.nwords = words <= 1 ? 1 : words <= 2 ? 2 : words <= 4 ? 4 : 8;
  bool fact_used[MB_NUM_FACT_COLS] = {false};
  unsigned dims_used = 0;
  auto note_field = [&](int code) -> bool {
    if (!field_ok(code)) return false;
    const int col = code >> 11;
    if (col < MB_NUM_FACT_COLS) {
      if (a->fact[col] == nullptr) return false;
      fact_used[col] = true;
    } else {
      dims_used |= 1u << (col - MB_COL_DIM_S);
    }
    return true;
  };
  // row-schema codes of the aggregation fields, converted to stage codes below
  int af[MB_BATCH_MAX_QUERIES][2], kf[MB_BATCH_MAX_QUERIES][2];
  unsigned req[MB_BATCH_MAX_QUERIES];  // dims_required
  for (int qi = 0; qi < P.nq; ++qi) {
    const mb_batch_query& q = a->queries[qi];
    BQ& d = P.q[qi];
    d = BQ{};
    if (q.num_preds < 0 || q.num_preds > MB_BATCH_MAX_PREDS || q.num_keys < 0 || q.num_keys > 2) return MB_ERR_ARG;
    if (q.agg_op < MB_AGG_SUM || q.agg_op > MB_AGG_MUL || q.res == nullptr) return MB_ERR_ARG;
    if (q.res_layout != MB_RES_SCALAR && q.res_layout != MB_RES_CRYSTAL4 && q.res_layout != MB_RES_DENSE)
      return MB_ERR_ARG;
    if (q.res_layout != MB_RES_SCALAR && q.total_val <= 0) return MB_ERR_ARG;
    if (!aligned8(q.res)) return MB_ERR_ALIGN;
    if (q.dims_required < 0 || q.dims_required > 15) return MB_ERR_ARG;
    const int nk = q.res_layout == MB_RES_SCALAR ? 0 : q.num_keys;
    d.np = static_cast<uint8_t>(q.num_preds);
    d.res_layout = static_cast<uint8_t>(q.res_layout);
    dims_used |= static_cast<unsigned>(q.dims_required);
    for (int p = 0; p < q.num_preds; ++p) {
      if (!note_field(q.pred_field[p])) return MB_ERR_ARG;
      d.pf[p] = static_cast<uint16_t>(q.pred_field[p]);
      d.plo[p] = q.pred_lo[p];
      d.phi[p] = q.pred_hi[p];
    }
    for (int k = 0; k < (q.agg_op == MB_AGG_SUM ? 1 : 2); ++k)
      if (!note_field(q.agg_field[k])) return MB_ERR_ARG;
    af[qi][0] = q.agg_field[0];
    af[qi][1] = q.agg_op == MB_AGG_SUM ? q.agg_field[0] : q.agg_field[1];
    for (int k = 0; k < nk; ++k)
      if (!note_field(q.key_field[k])) return MB_ERR_ARG;
    // an absent key reads the first aggregation field and weighs it by 0
    kf[qi][0] = nk > 0 ? q.key_field[0] : af[qi][0];
    kf[qi][1] = nk > 1 ? q.key_field[1] : af[qi][0];
    AQ& A = d.a;
    A.kmul0 = nk > 0 ? static_cast<unsigned>(q.key_mul[0]) : 0u;
    A.kmul1 = nk > 1 ? static_cast<unsigned>(q.key_mul[1]) : 0u;
    A.bias = 0u - ((nk > 0 ? static_cast<unsigned>(q.key_min[0]) * A.kmul0 : 0u) +
                   (nk > 1 ? static_cast<unsigned>(q.key_min[1]) * A.kmul1 : 0u));
    A.total = q.res_layout == MB_RES_SCALAR ? 1 : q.total_val;
    A.soff = -1;
    A.flags = q.agg_op | ((q.res_layout == MB_RES_CRYSTAL4 ? 1 : 0) << 2) | (nk << 3) |
              ((q.res_layout == MB_RES_SCALAR ? 1 : 0) << 5) | (1 << 8);
    d.res = q.res;
    req[qi] = static_cast<unsigned>(q.dims_required);
  }
  // Constrained attributes, the hull of the ranges on each, and interval coding, which goes to
  // wide attributes in the order the caller's queries first name them: before the queries are
  // renumbered, so that sizing the workspace and running the batch plan the same tables.
  Attr attr[kMaxPredFields] = {};
  int hmin[kMaxPredFields], hmax[kMaxPredFields];
  bool has[kMaxPredFields] = {false};
  for (int qi = 0; qi < P.nq; ++qi) {
    const BQ& d = P.q[qi];
    for (int p = 0; p < d.np; ++p) {
      int f = 0;
      while (f < P.nfields && attr[f].code != d.pf[p]) ++f;
      if (f == P.nfields) {
        if (P.nfields == kMaxPredFields) return MB_ERR_SIZE;
        attr[P.nfields++].code = d.pf[p];
      }
      if (d.plo[p] > d.phi[p]) continue;  // an empty range accepts nothing, inside or outside the hull
      if (!has[f]) {
        hmin[f] = d.plo[p];
        hmax[f] = d.phi[p];
        has[f] = true;
      } else {
        hmin[f] = d.plo[p] < hmin[f] ? d.plo[p] : hmin[f];
        hmax[f] = d.phi[p] > hmax[f] ? d.phi[p] : hmax[f];
      }
    }
  }
  int nbp = 0;
  for (int f = 0; f < P.nfields; ++f) {
    Attr& A = attr[f];
    const long long n = has[f] ? static_cast<long long>(hmax[f]) - hmin[f] + 1 : 1;
    if (n > 65536) return MB_ERR_SIZE;  // attribute ranges wider than 65,536 values
    A.min = has[f] ? hmin[f] : 0;
    A.n = static_cast<int>(n);
    if (n > kSmemTableMaxEntries) {
      // interval coding: end points lo and hi + 1 of every non-empty range on f, and 0; the
      // hull has at most 65,536 values, so a bit per value sorts them
      uint64_t at[65536 / 64] = {0};
      at[0] = 1;
      for (int qi = 0; qi < P.nq; ++qi) {
        const BQ& d = P.q[qi];
        for (int p = 0; p < d.np; ++p) {
          if (d.pf[p] != A.code || d.plo[p] > d.phi[p]) continue;
          const long long lo = static_cast<long long>(d.plo[p]) - A.min;
          const long long hi1 = static_cast<long long>(d.phi[p]) + 1 - A.min;
          at[lo / 64] |= 1ull << (lo % 64);
          if (hi1 < n) at[hi1 / 64] |= 1ull << (hi1 % 64);
        }
      }
      int np = 0;
      for (int i = 0; i < (A.n + 63) / 64; ++i) np += __builtin_popcountll(at[i]);
      if (nbp + np <= kMaxBreakpoints) {
        int* bp = P.bp + nbp;
        for (int i = 0; i < (A.n + 63) / 64; ++i)
          for (uint64_t w = at[i]; w != 0; w &= w - 1) *bp++ = 64 * i + __builtin_ctzll(w);
        A.nint = np;
        A.bp_off = nbp;
        nbp += np;
        int shift = 0;
        while ((static_cast<long long>(kMaxBuckets) << shift) < n) ++shift;
        A.bkt_shift = shift;
      }
    }
  }
  // Classes: queries that add the same expression to the same group index, most members
  // first. The queries are renumbered class by class, so that a class's bits share few words.
  int cls_of[MB_BATCH_MAX_QUERIES], first_of[MB_BATCH_MAX_QUERIES], members[MB_BATCH_MAX_QUERIES], nfound = 0;
  for (int qi = 0; qi < P.nq && !sizing; ++qi) {
    auto same = [&](int o) {
      const AQ &A = P.q[qi].a, &C = P.q[o].a;
      return af[qi][0] == af[o][0] && af[qi][1] == af[o][1] && kf[qi][0] == kf[o][0] && kf[qi][1] == kf[o][1] &&
             A.kmul0 == C.kmul0 && A.kmul1 == C.kmul1 && A.bias == C.bias && A.total == C.total && A.flags == C.flags;
    };
    int c = 0;
    while (c < nfound && !same(first_of[c])) ++c;
    if (c == nfound) {
      first_of[nfound] = qi;
      members[nfound++] = 0;
    }
    ++members[c];
    cls_of[qi] = c;
  }
  if (!sizing) {
    int rank[MB_BATCH_MAX_QUERIES], order[MB_BATCH_MAX_QUERIES], next[kMaxClasses + 1] = {0};
    for (int c = 0; c < nfound; ++c) rank[c] = kMaxClasses;
    for (int i = 0; i < kMaxClasses && i < nfound; ++i) {
      int best = -1;
      for (int c = 0; c < nfound; ++c)
        if (rank[c] == kMaxClasses && (best < 0 || members[c] > members[best])) best = c;
      rank[best] = i;
    }
    for (int qi = 0; qi < P.nq; ++qi) {
      cls_of[qi] = rank[cls_of[qi]];
      for (int c = cls_of[qi] + 1; c <= kMaxClasses; ++c) ++next[c];
    }
    for (int qi = 0; qi < P.nq; ++qi) order[next[cls_of[qi]]++] = qi;
    P.ncls = nfound < kMaxClasses ? nfound : kMaxClasses;
    P.others = nfound > kMaxClasses ? 1 : 0;
    std::vector<BQ> q0(P.q, P.q + P.nq);
    std::vector<int> from(6 * P.nq);
    for (int qi = 0; qi < P.nq; ++qi) {
      int* f = &from[6 * qi];
      f[0] = af[qi][0], f[1] = af[qi][1], f[2] = kf[qi][0], f[3] = kf[qi][1];
      f[4] = static_cast<int>(req[qi]), f[5] = cls_of[qi];
    }
    for (int qi = 0; qi < P.nq; ++qi) {
      const int* f = &from[6 * order[qi]];
      P.q[qi] = q0[order[qi]];
      af[qi][0] = f[0], af[qi][1] = f[1], kf[qi][0] = f[2], kf[qi][1] = f[3];
      req[qi] = static_cast<unsigned>(f[4]), cls_of[qi] = f[5];
      P.cls_mask[cls_of[qi]][qi / 32] |= 1u << (qi % 32);
      P.all[qi / 32] |= 1u << (qi % 32);
    }
  }
  if (!sizing) {
    unsigned by_req[16][kMaskWordsMax] = {{0}};
    unsigned seen = 0;
    for (int qi = 0; qi < P.nq; ++qi) {
      by_req[req[qi]][qi / 32] |= 1u << (qi % 32);
      seen |= 1u << req[qi];
    }
    for (unsigned pm = 0; pm < 16; ++pm)
      for (unsigned r = 0; r < 16; ++r)
        if (((seen >> r) & 1u) && (pm & r) == r)
          for (int w = 0; w < P.nwords; ++w) P.pres_mask[pm][w] |= by_req[r][w];
  }

  // dimensions: their keys are staged, their words overwrite the key columns (the date
  // word gets its own column because orderdate is also a field)
  static const int kKeyCol[4] = {MB_COL_SUPPKEY, MB_COL_CUSTKEY, MB_COL_PARTKEY, MB_COL_ORDERDATE};
  for (int d = 0; d < 4; ++d) {
    if (!(dims_used & (1u << d))) continue;
    if (a->dim[d].words == nullptr || a->dim[d].slots <= 0 || a->fact[kKeyCol[d]] == nullptr) return MB_ERR_ARG;
    fact_used[kKeyCol[d]] = true;
  }
  for (int c = 0; c < 13; ++c) P.cidx[c] = -1;
  for (int c = 0; c < kMaxStageCols; ++c) P.stage_dim[c] = -1;
  if (a->gpu_cache != nullptr) {
    const int ss = a->segment_size;
    if (ss < 4 || (ss & (ss - 1)) != 0) return MB_ERR_ARG;
    if (!aligned16(a->gpu_cache)) return MB_ERR_ALIGN;
    P.gpu_cache = a->gpu_cache;
    P.seg_group = a->segment_group;
    P.seg_shift = __builtin_ctz(static_cast<unsigned>(ss));
  } else if (a->segment_group != nullptr) {
    return MB_ERR_ARG;
  }
  for (int c = 0; c < MB_NUM_FACT_COLS; ++c) {
    if (!fact_used[c]) continue;
    if (P.gpu_cache == nullptr && !aligned16(a->fact[c])) return MB_ERR_ALIGN;
    P.cidx[c] = P.ncols;
    P.col[P.ncols++] = a->fact[c];
  }
  for (int d = 0; d < 4; ++d) {
    if (!(dims_used & (1u << d))) continue;
    Dim& D = P.dim[P.ndims++];
    const int key_stage = P.cidx[kKeyCol[d]];
    const int word_stage = d == 3 ? P.ncols : key_stage;
    P.cidx[MB_COL_DIM_S + d] = word_stage;
    P.stage_dim[word_stage] = d;
    D.d = d;
    D.key_word = key_stage;  // columns here; word offsets once the tile is known
    D.word = word_stage;
    D.pat = a->dim[d].words;
    D.slots = a->dim[d].slots;
    D.kmin = a->dim[d].key_min;
  }
  // a dimension word that replaces its key makes that key unavailable as a field
  auto uses_key = [&](int code) {
    const int col = code >> 11;
    for (int t = 0; t < 3; ++t)
      if ((dims_used & (1u << t)) && col == kKeyCol[t]) return true;
    return false;
  };
  for (int qi = 0; qi < P.nq; ++qi) {
    const BQ& d = P.q[qi];
    for (int p = 0; p < d.np; ++p)
      if (uses_key(d.pf[p])) return MB_ERR_ARG;
    for (int k = 0; k < 2; ++k)
      if (uses_key(af[qi][k]) || uses_key(kf[qi][k])) return MB_ERR_ARG;
  }
  // stage codes
  auto scode = [&](int code) { return (P.cidx[code >> 11] << 11) | (code & 0x7ff); };
  for (int f = 0; f < P.nfields; ++f) attr[f].scode = scode(attr[f].code);
  for (int qi = 0; qi < P.nq; ++qi) {
    AQ& A = P.q[qi].a;
    A.a0 = static_cast<uint16_t>(scode(af[qi][0]));
    A.a1 = static_cast<uint16_t>(scode(af[qi][1]));
    A.k0 = static_cast<uint16_t>(scode(kf[qi][0]));
    A.k1 = static_cast<uint16_t>(scode(kf[qi][1]));
  }
  // Position among the batch's dimensions of the one a field reads, -1 for a fact column.
  int pos_of[MB_NUM_FACT_COLS + 4];
  for (int& p : pos_of) p = -1;
  for (int j = 0; j < P.ndims; ++j) pos_of[MB_COL_DIM_S + P.dim[j].d] = j;
  auto dim_pos = [&](int code) { return pos_of[code >> 11]; };
  for (int qi = 0; qi < P.nq && !sizing; ++qi) {
    const unsigned bit = 1u << (qi % 32);
    const int w = qi / 32;
    auto uses = [&](int code) {
      const int j = dim_pos(code);
      if (j >= 0) P.dim[j].use[w] |= bit;
    };
    for (int j = 0; j < P.ndims; ++j)
      if ((req[qi] >> P.dim[j].d) & 1u) {
        P.dim[j].need[w] |= bit;
        P.dim[j].use[w] |= bit;
      }
    for (int p = 0; p < P.q[qi].np; ++p) uses(P.q[qi].pf[p]);
    for (int k = 0; k < 2; ++k) {
      uses(af[qi][k]);
      uses(kf[qi][k]);
    }
  }
  // Tables: fact attributes among themselves and dimension attributes among themselves share
  // one while the product of their index counts stays small (fewer lookups and ANDs per row
  // for a few KB of shared memory).
  auto of_dim = [&](int f) { return dim_pos(attr[f].code) >= 0; };
  auto indexes = [&](int f) { return (attr[f].nint > 0 ? attr[f].nint : attr[f].n) + 1; };
  int order[kMaxPredFields];
  for (int f = 0; f < P.nfields; ++f) order[f] = f;
  std::stable_sort(order, order + P.nfields, [&](int x, int y) {
    return of_dim(x) != of_dim(y) ? of_dim(x) < of_dim(y) : indexes(x) > indexes(y);
  });
  int tab[kMaxPredFields], ntabs = 0, t_ent[kMaxPredFields], t_n[kMaxPredFields];
  bool t_dim[kMaxPredFields];
  for (int i = 0; i < P.nfields; ++i) {
    const int f = order[i];
    int t = 0;
    while (t < ntabs && !(t_dim[t] == of_dim(f) && t_n[t] < kMaxComponents &&
                          static_cast<long long>(t_ent[t]) * indexes(f) <= kCombineMaxEntries))
      ++t;
    if (t == ntabs) {
      t_dim[t] = of_dim(f);
      t_ent[t] = 1;
      t_n[t] = 0;
      ++ntabs;
    }
    attr[f].mul = t_ent[t];
    t_ent[t] *= indexes(f);
    ++t_n[t];
    tab[f] = t;
  }
  std::stable_sort(order, order + P.nfields, [&](int x, int y) { return tab[x] < tab[y]; });
  long long entries = 0;
  for (int i = 0; i < P.nfields; ++i) {
    const int f = order[i];
    Attr& A = P.at[i];
    A = attr[f];
    if (!of_dim(f)) P.nfact = i + 1;
    A.last = i + 1 == P.nfields || tab[order[i + 1]] != tab[f] ? 1 : 0;
    if (!A.last) continue;
    A.ent = t_ent[tab[f]];
    A.goff = entries * P.nwords;
    entries += A.ent;
  }
  P.table_entries = entries;
  return MB_OK;
}

static size_t workspace_bytes(const BatchPlan& P) { return static_cast<size_t>(P.table_entries) * P.nwords * 4; }

}  // namespace mb

using namespace mb;

extern "C" int mb_pat_build(const int* dim_key, int num_rows, int key_min, int slots, const int* attr0, int field0,
                            const int* attr1, int field1, const int* attr2, int field2, unsigned int* words,
                            mb_stream_t stream) {
  if (num_rows == 0) return MB_OK;
  if (dim_key == nullptr || words == nullptr || num_rows < 0 || slots <= 0) return MB_ERR_ARG;
  if ((attr0 && !field_ok(field0)) || (attr1 && !field_ok(field1)) || (attr2 && !field_ok(field2))) return MB_ERR_ARG;
  int err = MB_OK;
  DeviceState* ds = current_device_state(&err);
  if (ds == nullptr) return err;
  int blocks = (num_rows + 255) / 256;
  if (blocks > ds->num_sms * 8) blocks = ds->num_sms * 8;
  pat_build_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(dim_key, num_rows, key_min, slots, attr0,
                                                                          field0, attr1, field1, attr2, field2, words,
                                                                          ds->status);
  if (cudaGetLastError() != cudaSuccess) return MB_ERR_LAUNCH;
  note_launches(1);
  return MB_OK;
}

extern "C" size_t mb_batch_workspace_bytes(const mb_batch_args* a) {
  static BatchPlan P;  // large; host-side scratch for sizing only
  static std::mutex mu;
  std::lock_guard<std::mutex> lk(mu);
  if (plan_batch(a, P, true) != MB_OK) return 0;
  return workspace_bytes(P);
}

extern "C" int mb_batch_run(const mb_batch_args* a, mb_stream_t stream) {
  BatchPlan* Pp = new BatchPlan;  // ~25 KB of launch parameters, kept off the host stack
  struct Free {
    BatchPlan* p;
    ~Free() { delete p; }
  } guard{Pp};
  BatchPlan& P = *Pp;
  int e = plan_batch(a, P, false);
  if (e != MB_OK) return e;
  if (P.n == 0) return MB_OK;
  if (workspace_bytes(P) > 0 &&
      (a->workspace == nullptr || a->workspace_bytes < workspace_bytes(P) || !aligned16(a->workspace)))
    return a->workspace == nullptr || a->workspace_bytes < workspace_bytes(P) ? MB_ERR_SIZE : MB_ERR_ALIGN;
  P.tables = static_cast<unsigned*>(a->workspace);
  int err = MB_OK;
  DeviceState* ds = current_device_state(&err);
  if (ds == nullptr) return err;
  P.status = ds->status;

  // Defaults: up to 64 queries a row has few matches and the work per row decides, so a lane
  // takes two rows at a time (24 queries over 75 M rows: 768x2 1.76 ms, 960x1 2.22, 768x1
  // 2.52) unless an SM gets one tile at most, which half the rows finish sooner (24 queries over
  // 113,000 rows: 768x1 36 us, 768x2 40; over 150,000: 42 and 40; over less than a tile's 1,536 rows,
  // read without the ring, 37 and 31); above, the match lists are full anyway and one more warp a scheduler hides more
  // (120 queries over 20 M rows: 960x1 1.10 ms, 768x1 1.20, 768x2 1.33; 256 queries, with
  // group arrays filling the shared memory: 2.21, 2.30, 2.21). A call that sets one of the
  // two gets 768 threads or one row for the other.
  const bool by_size = a->threads == 0 && a->items_per_thread == 0;
  int threads = a->threads ? a->threads : by_size && P.nwords > 2 ? 960 : 768;
  const bool one_tile = P.n >= 2 * 768 && P.n <= 768ll * ds->num_sms;
  int items = a->items_per_thread ? a->items_per_thread : by_size && P.nwords <= 2 && !one_tile ? 2 : 1;
  auto variant = [&]() -> const BatchVariant* {
    for (const BatchVariant& v : kBatchVariants)
      if (v.warps * 32 == threads && v.items == items && v.nwm == P.nwords) return &v;
    return nullptr;
  };
  int stages = a->stages ? a->stages : 2;
  if (variant() == nullptr || stages < 2 || stages > kBatchStages) return MB_ERR_ARG;

  // shared memory: barriers | scalars | aggregation descriptors | match records | result
  // pointers | sum addresses | presence masks | predicate tables | match lists | small
  // group arrays | stage ring
  int off = 2 * kBatchStages * 8;
  int nscalar = 0;
  for (int qi = 0; qi < P.nq; ++qi) nscalar += P.q[qi].res_layout == MB_RES_SCALAR ? 1 : 0;
  P.smem_acc_off = off;
  P.acc_words = kScalarCopies * nscalar;
  off += 8 * P.acc_words;
  off = (off + 15) / 16 * 16;
  P.smem_aq_off = off;
  off += static_cast<int>(sizeof(AQ)) * P.nq;
  P.smem_qd_off = off;
  off += static_cast<int>(sizeof(QD)) * P.nq;
  P.smem_res_off = off;
  off += 8 * P.nq;
  P.smem_addr_off = off;
  off += 8 * P.nq;
  off = (off + 15) / 16 * 16;
  P.smem_pres_off = off;
  off += 16 * kMaskWordsMax * 4;
  const int budget = ds->max_smem_optin - 2048;
  const int stage_cols = P.ncols + (P.ndims && P.dim[P.ndims - 1].d == 3 ? 1 : 0);
  const int tables_off = off;
  bool in_smem[kMaxPredFields];
  for (int f = 0; f < P.nfields; ++f)  // single attributes with too many values and end points stay in the workspace
    in_smem[f] = P.at[f].last && (P.at[f].nint > 0 || P.at[f].ent <= kSmemTableMaxEntries + 1);
  auto place_tables = [&] {
    off = tables_off;
    for (int f = 0; f < P.nfields; ++f) {
      Attr& A = P.at[f];
      if (A.nint > 0) {
        A.bps_off = off;
        off += (A.nint * 4 + 15) / 16 * 16;
        A.bkt_off = off;
        off += ((((A.n - 1) >> A.bkt_shift) + 1) * 2 + 15) / 16 * 16;
      }
      A.smem_off = in_smem[f] ? off : -1;
      if (in_smem[f]) off += (A.ent * P.nwords * 4 + 15) / 16 * 16;
    }
  };
  place_tables();
  auto fits = [&](int st) {
    const int lists = threads / 32 * kMatchListCap * 2;
    return (off + lists + 127) / 128 * 128 + st * stage_cols * (threads * items + kColPad) * 4 <= budget;
  };
  // What does not fit takes less, at the cost of speed: a default launch the smaller shape, then
  // the largest tables stay in the workspace too, until the launch fits.
  if (by_size && !fits(2)) threads = 768, items = 1;
  while (!fits(2)) {
    int most = -1;
    for (int f = 0; f < P.nfields; ++f)
      if (in_smem[f] && (most < 0 || P.at[f].ent > P.at[most].ent)) most = f;
    if (most < 0) return MB_ERR_SIZE;
    in_smem[most] = false;
    place_tables();
  }
  while (!fits(stages)) --stages;
  P.smem_list_off = off;
  off += (threads / 32) * kMatchListCap * 2;

  const BatchVariant* var = variant();
  const int tile = threads * items;
  P.nfull = P.n / tile;
  // stage word offsets
  auto field = [&](int code) {
    const int width = code & 63;
    return Field{(code >> 11) * (tile + kColPad), (code >> 6) & 31, width >= 32 ? 0xffffffffu : (1u << width) - 1u};
  };
  for (int f = 0; f < P.nfields; ++f) P.at[f].f = field(P.at[f].scode);
  for (int j = 0; j < P.ndims; ++j) {
    P.dim[j].key_word *= tile + kColPad;
    P.dim[j].word *= tile + kColPad;
  }
  for (int c = 0; c < P.ncls; ++c) {
    int qi = 0;  // its first query
    while (!((P.cls_mask[c][qi / 32] >> (qi % 32)) & 1u)) ++qi;
    const AQ& A = P.q[qi].a;
    P.cls[c] = {field(A.a0), field(A.a1), field(A.k0), field(A.k1), A.kmul0, A.kmul1, A.bias,
                A.total, A.flags & 3, (A.flags >> 5) & 1, ((A.flags >> 3) & 3) > 1 ? 1 : 0};
  }
  P.stage_words = stage_cols * (tile + kColPad);
  auto total_smem = [&](int base, int st) { return (base + 127) / 128 * 128 + st * P.stage_words * 4; };
  P.stages = stages;
  // scalars accumulate in their shared-memory words (kScalarCopies each)
  for (int qi = 0, k = 0; qi < P.nq; ++qi)
    if (P.q[qi].res_layout == MB_RES_SCALAR) {
      P.q[qi].a.soff = P.smem_acc_off + 8 * kScalarCopies * k++;
    }
  // small group arrays (<= 1,024 groups) to shared memory, smallest first, within the budget
  P.smem_groups_off = off;
  int groups_bytes = 0;
  const int group_cap = a->smem_group_bytes < 0 ? 131072 : a->smem_group_bytes;
  const int group_budget = a->smem_group_bytes < 0 && budget > kSmemBesideL1 ? kSmemBesideL1 : budget;
  // shared memory kept for the touch bitmaps of the small-array queries that end up with
  // L2 sums (below): a few bytes each, and without one such a query writes its keys on
  // every match
  int touch_reserve = 0;
  for (int qi = 0; qi < P.nq; ++qi) {
    const AQ& A = P.q[qi].a;
    if (P.q[qi].res_layout != MB_RES_SCALAR && ((A.flags >> 2) & 1) && A.total <= 1024)
      touch_reserve += (4 * ((A.total + 31) / 32) + 15) / 16 * 16;
  }
  // queries with the same group count form a family (group-major interleaved sums); as
  // many members as fit, smallest group counts first, and of a family the queries that most
  // rows can match: its share of the values its predicates' attributes have in this batch.
  // Sums by L2 atomics of a query that matches often meet on a few lines. 256 queries over 40 M
  // rows, three draws: the first queries that fit 5.13, 4.00 and 4.88 ms, the widest ones
  // 3.53, 3.49 and 4.24.
  float share[MB_BATCH_MAX_QUERIES];
  for (int qi = 0; qi < P.nq; ++qi) {
    const BQ& Q = P.q[qi];
    share[qi] = 1.0f;
    for (int k = 0; k < Q.np; ++k)
      for (int f = 0; f < P.nfields; ++f) {
        if (P.at[f].code != Q.pf[k]) continue;
        const long long width = static_cast<long long>(Q.phi[k]) - Q.plo[k] + 1;
        share[qi] *= width > 0 ? static_cast<float>(width) / static_cast<float>(P.at[f].n > 0 ? P.at[f].n : 1) : 0.0f;
      }
  }
  for (;;) {
    int total = 0;
    for (int qi = 0; qi < P.nq; ++qi) {
      const AQ& A = P.q[qi].a;
      if (P.q[qi].res_layout == MB_RES_SCALAR || A.soff >= 0 || A.total > 1024 || (A.flags & (1 << 30))) continue;
      if (total == 0 || A.total < total) total = A.total;
    }
    if (total == 0) break;
    const int words = (total + 31) / 32;
    auto fam_bytes = [&](int k) { return (8 * total * (k | 1) + 4 * words * k + 15) / 16 * 16; };
    int members = 0;
    for (int qi = 0; qi < P.nq; ++qi) {
      const AQ& A = P.q[qi].a;
      if (P.q[qi].res_layout == MB_RES_SCALAR || A.soff >= 0 || A.total != total) continue;
      if (groups_bytes + fam_bytes(members + 1) > group_cap ||
          total_smem(off + groups_bytes + fam_bytes(members + 1) + touch_reserve, stages) > group_budget)
        break;
      ++members;
    }
    short by_share[MB_BATCH_MAX_QUERIES];
    bool chosen[MB_BATCH_MAX_QUERIES] = {};
    int candidates = 0;
    for (int qi = 0; qi < P.nq; ++qi) {
      const AQ& A = P.q[qi].a;
      if (P.q[qi].res_layout != MB_RES_SCALAR && A.soff < 0 && A.total == total)
        by_share[candidates++] = static_cast<short>(qi);
    }
    std::stable_sort(by_share, by_share + candidates, [&](short x, short y) { return share[x] > share[y]; });
    for (int i = 0; i < members; ++i) chosen[by_share[i]] = true;
    int j = 0;
    for (int qi = 0; qi < P.nq; ++qi) {
      AQ& A = P.q[qi].a;
      if (P.q[qi].res_layout == MB_RES_SCALAR || A.soff >= 0 || A.total != total) continue;
      if (chosen[qi]) {
        A.soff = off + groups_bytes + 8 * j;
        A.flags = (A.flags & 0xff) | ((members | 1) << 8) | (j << 17);
        ++j;
      } else {
        A.flags |= 1 << 30;  // no room: sums by L2 atomics (marked so the search moves on)
      }
    }
    if (members > 0) groups_bytes += fam_bytes(members);  // a family without room takes none
  }
  for (int qi = 0; qi < P.nq; ++qi) P.q[qi].a.flags &= ~(1 << 30);
  // queries left with L2 sums that write keys, and few groups (a few hot result lines),
  // get a touch bitmap in shared memory where it fits (smallest group counts first), so
  // they write their keys once per CTA and group; with many groups the stores spread out
  // and cost less than the test
  for (int pass_total = 1; pass_total <= 1024; pass_total *= 2) {
    for (int qi = 0; qi < P.nq; ++qi) {
      AQ& A = P.q[qi].a;
      if (A.soff != -1 || !((A.flags >> 2) & 1) || A.total > pass_total || A.total <= pass_total / 2) continue;
      const int bytes = (4 * ((A.total + 31) / 32) + 15) / 16 * 16;
      if (total_smem(off + groups_bytes + bytes, stages) > budget) continue;
      A.soff = -(off + groups_bytes) - 2;
      groups_bytes += bytes;
    }
  }
  P.smem_groups_words = groups_bytes / 4;
  P.smem_stage_off = (off + groups_bytes + 127) / 128 * 128;
  const int smem = total_smem(off + groups_bytes, stages);

  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (P.table_entries > 0) {
    long long tasks = 0;  // warps' worth: 32 entries of a table, one word
    for (int f = 0; f < P.nfields; ++f) tasks += P.at[f].last ? (P.at[f].ent + 31) / 32 * P.nwords : 0;
    long long blocks = (tasks + 3) / 4;
    if (blocks > ds->num_sms * 8) blocks = ds->num_sms * 8;
    if (launch_dependent(batch_mask_kernel, static_cast<int>(blocks), 128, 0, st, P, static_cast<int>(tasks)) !=
        cudaSuccess)
      return MB_ERR_LAUNCH;
    note_launches(1);
  }
  int grid = a->grid;
  if (grid <= 0) {
    // 16 warps or more leave registers for one CTA an SM; only the 8-warp shapes have to ask
    int per_sm = 1;
    if (threads < 512 &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, var->fn, threads + 32, smem) != cudaSuccess)
      return MB_ERR_CUDA;
    grid = ds->num_sms * (per_sm < 1 ? 1 : per_sm);
  }
  long long want = P.nfull > 0 ? P.nfull : (P.n + threads - 1) / threads;
  if (want < 1) want = 1;
  if (grid > want) grid = static_cast<int>(want);
  if (launch_dependent(var->fn, grid, threads + 32, static_cast<size_t>(smem), st, P) != cudaSuccess)
    return MB_ERR_LAUNCH;
  note_launches(1);
  return MB_OK;
}

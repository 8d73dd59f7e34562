// mlp.cu — the learned planner's cost model: a 24 -> 64 -> 64 -> 2 ReLU MLP (5,890
// fp32 parameters) that maps a (query, segment) feature vector to the predicted log CPU
// ms and log GPU ms of running the segment on each device. Forward, backward and Adam
// are hand-written kernels; the reference plans with an analytic bandwidth model
// instead (src/gpudb/CostModel.cu:283-440), which stays as the fallback.
//
// Parameter layout (one flat fp32 array): W1[24][64], b1[64], W2[64][64], b2[64],
// W3[64][2], b3[2]; W[i][j] is input i -> unit j. SIMT fp32 on purpose: the planner's
// predictions and gradients keep fp32 products and sums (a tensor-core split would not),
// so the roofline is the fp32 FMA rate, 148 SMs x 128 lanes x 2 x 1.965 GHz = 74.4 TFLOP/s.
// The kernels' pointers are not __restrict__: parameters and gradients are written by the kernel
// before, which may still run when a dependent launch begins, and const __restrict__ would have
// them read by non-coherent loads.
#include <cmath>

#include "common.cuh"

namespace mb {

constexpr int kIn = MB_MLP_IN, kHid = MB_MLP_HIDDEN, kOut = MB_MLP_OUT;
constexpr int kW1 = 0, kB1 = kW1 + kIn * kHid, kW2 = kB1 + kHid, kB2 = kW2 + kHid * kHid, kW3 = kB2 + kHid,
              kB3 = kW3 + kHid * kOut, kParams = kB3 + kOut;
static_assert(kParams == MB_MLP_PARAMS, "parameter count");
static_assert(kHid == 64 && kOut == 2 && kIn % 4 == 0, "thread tilings below");

// ---- forward -------------------------------------------------------------------------
// One warp takes 8 * S samples through all three layers on its own (no CTA barrier in the
// loop): a lane holds 16 units x S samples of a layer in registers as packed pairs of units,
// so a step of the inner product is 8 * S packed fp32x2 FMAs against S + 16 words from shared
// memory. Shared memory delivers 128 bytes a cycle to the lanes whether or not they share an
// address, so the tile has to be that large: at S = 8 a step is 24 wavefronts against 32
// cycles of FMA. 1,700,000 samples: 360 us, 54 TFLOP/s (8 units x 8 samples a lane with the
// weights stored as ready pairs, 24 wavefronts against 16 cycles: 526 us; one FMA per two
// shared loads, the form before: 3,738 us). Samples and
// the hidden layer are kept row by row (sample i * 8 + sg of lane group sg, rows padded so
// that the groups fall in different banks) and read four inputs at a time; the next tile's
// inputs arrive by cp.async under the second layer. Every unit's sum runs over its inputs in
// order, with the bias first; the output layer sums a lane's sixteen units, then its four
// lanes by a transposing butterfly.
constexpr int kFwdWarps = 8;
constexpr int kFwdXRow = kIn + 4, kFwdHRow = kHid + 4;  // padded rows, 16-byte multiples
template <int S>
struct FwdSmem {
  float w1[kIn * kHid], w2[kHid * kHid], w3[kHid * kOut];
  float b1[kHid], b2[kHid], b3[4];
  float x[kFwdWarps][8 * S * kFwdXRow];
  float h[kFwdWarps][8 * S * kFwdHRow];
};

__device__ __forceinline__ unsigned long long ffma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}

// acc[i][p] = biases of unit pair p + sums over K inputs, for sample 8 i of `in` (its rows
// start at the lane's group): pair p = units 16 (p / 2) + 4 ug + 2 (p % 2), + 1. `w` and
// `bias` point at the lane's first unit.
template <int K, int ROW, int S>
__device__ __forceinline__ void fwd_layer(const float* in, const float* w, const float* bias,
                                          unsigned long long (&acc)[S][8]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(bias + q * 16);
#pragma unroll
    for (int i = 0; i < S; ++i) {
      acc[i][2 * q] = b.x;
      acc[i][2 * q + 1] = b.y;
    }
  }
#pragma unroll 1
  for (int k = 0; k < K; k += 4) {
    float4 v[S];
#pragma unroll
    for (int i = 0; i < S; ++i) v[i] = *reinterpret_cast<const float4*>(in + i * 8 * ROW + k);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      unsigned long long xx[S];
#pragma unroll
      for (int i = 0; i < S; ++i) {
        const float f = e == 0 ? v[i].x : e == 1 ? v[i].y : e == 2 ? v[i].z : v[i].w;
        xx[i] = pack2(f, f);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const ulonglong2 wv = *reinterpret_cast<const ulonglong2*>(w + (k + e) * kHid + q * 16);
#pragma unroll
        for (int i = 0; i < S; ++i) {
          acc[i][2 * q] = ffma2(wv.x, xx[i], acc[i][2 * q]);
          acc[i][2 * q + 1] = ffma2(wv.y, xx[i], acc[i][2 * q + 1]);
        }
      }
    }
  }
}

template <int S>
__global__ void __launch_bounds__(kFwdWarps * 32, 1) mlp_forward_kernel(const float* params, const float* x,
                                                                       int batch, float* y) {
  extern __shared__ __align__(16) unsigned char raw[];
  FwdSmem<S>& s = *reinterpret_cast<FwdSmem<S>*>(raw);
  constexpr int kTile = 8 * S;  // samples per warp
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ug = lane & 3, sg = lane >> 2;
  float* xs = s.x[warp];
  float* hs = s.h[warp];
  const bool vec = (reinterpret_cast<uintptr_t>(x) & 15u) == 0, vec_y = (reinterpret_cast<uintptr_t>(y) & 7u) == 0;
  const long long tiles = (static_cast<long long>(batch) + kTile - 1) / kTile;
  const long long step = static_cast<long long>(gridDim.x) * kFwdWarps;
  // a tile's inputs: kTile rows of 24 floats, six 16-byte pieces a row (rows past the batch
  // keep what they hold: their outputs are not written)
  auto fetch = [&](long long tile) {
    const long long r0 = tile * kTile;
    const float* src = x + r0 * kIn;
    const int have = batch - r0 < kTile ? static_cast<int>(batch - r0) : kTile;
#pragma unroll
    for (int c = lane; c < kTile * kIn / 4; c += 32) {
      const int b = c / (kIn / 4), part = c % (kIn / 4);
      if (b >= have) continue;
      float* dst = xs + b * kFwdXRow + part * 4;
      const float* from = src + b * kIn + part * 4;
      if (vec) {
        cp_async16(dst, from);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) dst[e] = from[e];
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  wait_for_predecessor();
  long long tile = blockIdx.x + static_cast<long long>(gridDim.x) * warp;
  for (int i = lane; i < kTile * kFwdXRow; i += 32) xs[i] = 0.f;
  __syncwarp();
  if (tile < tiles) fetch(tile);
#pragma unroll
  for (int i = 0; i < kIn * kHid / (kFwdWarps * 32); ++i)
    s.w1[i * kFwdWarps * 32 + tid] = params[kW1 + i * kFwdWarps * 32 + tid];
#pragma unroll
  for (int i = 0; i < kHid * kHid / (kFwdWarps * 32); ++i)
    s.w2[i * kFwdWarps * 32 + tid] = params[kW2 + i * kFwdWarps * 32 + tid];
  if (tid < kHid) {
    s.b1[tid] = params[kB1 + tid];
    s.b2[tid] = params[kB2 + tid];
  }
  if (tid < kHid * kOut) s.w3[tid] = params[kW3 + tid];
  if (tid < kOut) s.b3[tid] = params[kB3 + tid];
  __syncthreads();
  for (; tile < tiles; tile += step) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    unsigned long long acc[S][8];
    fwd_layer<kIn, kFwdXRow, S>(xs + sg * kFwdXRow, s.w1 + ug * 4, s.b1 + ug * 4, acc);
    __syncwarp();  // the inputs have been read: the next tile's may land on them
    if (tile + step < tiles) fetch(tile + step);
#pragma unroll
    for (int i = 0; i < S; ++i)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float4 v;
        unpack2(acc[i][2 * q], v.x, v.y);
        unpack2(acc[i][2 * q + 1], v.z, v.w);
        v.x = fmaxf(v.x, 0.f);
        v.y = fmaxf(v.y, 0.f);
        v.z = fmaxf(v.z, 0.f);
        v.w = fmaxf(v.w, 0.f);
        *reinterpret_cast<float4*>(hs + (i * 8 + sg) * kFwdHRow + q * 16 + ug * 4) = v;
      }
    __syncwarp();
    fwd_layer<kHid, kFwdHRow, S>(hs + sg * kFwdHRow, s.w2 + ug * 4, s.b2 + ug * 4, acc);
    // output layer: this lane's sixteen units, both outputs of its S samples
    float o[S][kOut];
#pragma unroll
    for (int i = 0; i < S; ++i) o[i][0] = o[i][1] = 0.f;
#pragma unroll
    for (int p = 0; p < 8; ++p) {
      const float4 w = *reinterpret_cast<const float4*>(s.w3 + ((p >> 1) * 16 + ug * 4 + (p & 1) * 2) * kOut);
#pragma unroll
      for (int i = 0; i < S; ++i) {
        float h0, h1;
        unpack2(acc[i][p], h0, h1);
        h0 = fmaxf(h0, 0.f);
        h1 = fmaxf(h1, 0.f);
        o[i][0] = fmaf(h1, w.z, fmaf(h0, w.x, o[i][0]));
        o[i][1] = fmaf(h1, w.w, fmaf(h0, w.y, o[i][1]));
      }
    }
    // transposing butterfly over the four unit lanes: each step halves the samples a lane
    // keeps (or, once it keeps one, just adds)
    int first = 0;
    int kept = S;
#pragma unroll
    for (int bit = 2; bit >= 1; bit >>= 1) {
      const bool up = ug & bit;
      if (kept > 1) {
        kept >>= 1;
#pragma unroll
        for (int i = 0; i < kept; ++i)
#pragma unroll
          for (int c = 0; c < kOut; ++c) {
            const float keep = up ? o[i + kept][c] : o[i][c];
            const float give = up ? o[i][c] : o[i + kept][c];
            o[i][c] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
          }
        first += up ? kept : 0;
      } else {
#pragma unroll
        for (int c = 0; c < kOut; ++c) o[0][c] += __shfl_xor_sync(0xffffffffu, o[0][c], bit);
      }
    }
#pragma unroll
    for (int i = 0; i < (S >= 4 ? S / 4 : 1); ++i) {
      const long long r = tile * kTile + (first + i) * 8 + sg;
      if (r >= batch || (S == 2 && (ug & 1))) continue;
      const float y0 = o[i][0] + s.b3[0], y1 = o[i][1] + s.b3[1];
      if (vec_y) {
        *reinterpret_cast<float2*>(y + r * kOut) = make_float2(y0, y1);
      } else {
        y[r * kOut] = y0;
        y[r * kOut + 1] = y1;
      }
    }
    __syncwarp();  // the hidden layer is read before the next tile's is written
  }
}

// ---- backward ------------------------------------------------------------------------
// A CTA takes tiles of T samples: it recomputes the forward pass, forms dL/dy = (y - t) / B
// for the loss 1/(2B) * sum (y - t)^2, propagates it through the ReLUs and sums the tiles'
// weight gradients in registers; one round of fp32 atomics per CTA adds them into the
// global gradient (so summation order, and the last bits, vary from run to run). A training
// step is latency alone (256 samples are 8 MFLOP): small tiles spread it over more SMs,
// each thread keeps T / 4 samples of one unit, activations are read four inputs at a time,
// and W2 has a 65-word row so that the pass back through it walks distinct banks. 256
// samples: 5.6 us (before, 8 CTAs of 32 samples, 32-way conflicts on W2's columns and an
// atomic per tile: 38.2 us).
constexpr int kBwdThreads = 256;
constexpr int kW2Row = kHid + 1;
template <int T>
struct BwdSmem {
  float w1[kIn * kHid];
  float w2[kHid * kW2Row];
  float b1[kHid], b2[kHid], w3[kHid * kOut], b3[4];
  alignas(16) float x[T][kIn];
  alignas(16) float h1[T][kHid];
  alignas(16) float h2[T][kHid];
  alignas(16) float d1[T][kHid];
  alignas(16) float d2[T][kHid];
  float dy[T][kOut];
};

template <int T>
__global__ void __launch_bounds__(kBwdThreads) mlp_backward_kernel(const float* params, const float* x,
                                                                   const float* target, int batch, float* grads,
                                                                   float* loss_sum) {
  extern __shared__ __align__(16) unsigned char raw[];
  BwdSmem<T>& s = *reinterpret_cast<BwdSmem<T>*>(raw);
  constexpr int NS = T / 4;  // samples a thread computes in each layer
  constexpr int kWarps = kBwdThreads / 32;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int j = tid & (kHid - 1), b0 = (tid >> 6) * NS;
  allow_dependent();
  wait_for_predecessor();
#pragma unroll
  for (int i = 0; i < kIn * kHid / kBwdThreads; ++i) s.w1[i * kBwdThreads + tid] = params[kW1 + i * kBwdThreads + tid];
#pragma unroll
  for (int i = 0; i < kHid * kHid / kBwdThreads; ++i)
    s.w2[(i * 4 + (tid >> 6)) * kW2Row + j] = params[kW2 + i * kBwdThreads + tid];
  if (tid < kHid) {
    s.b1[tid] = params[kB1 + tid];
    s.b2[tid] = params[kB2 + tid];
  }
  if (tid < kHid * kOut) s.w3[tid] = params[kW3 + tid];
  if (tid < kOut) s.b3[tid] = params[kB3 + tid];

  const float inv_b = 1.f / static_cast<float>(batch);
  // gradient entries of this thread: W2[16 (tid / 64) + i][j], W1[6 (tid / 64) + i][j], one
  // of W3, b1, b2 (gs), and for two threads one of b3 (gb3)
  constexpr int G2 = kHid / 4, G1 = kIn / 4;
  float g2[G2], g1[G1], gs = 0.f, gb3 = 0.f, loss = 0.f;
#pragma unroll
  for (int i = 0; i < G2; ++i) g2[i] = 0.f;
#pragma unroll
  for (int i = 0; i < G1; ++i) g1[i] = 0.f;
  for (int r0 = blockIdx.x * T; r0 < batch; r0 += gridDim.x * T) {
    const int nt = min(T, batch - r0);
    __syncthreads();  // weights staged / the previous tile's gradients read
    for (int i = tid; i < T * kIn; i += kBwdThreads)
      (&s.x[0][0])[i] = i < nt * kIn ? x[static_cast<long long>(r0) * kIn + i] : 0.f;
    __syncthreads();
    float a[NS];
#pragma unroll
    for (int b = 0; b < NS; ++b) a[b] = s.b1[j];
#pragma unroll
    for (int k = 0; k < kIn; k += 4) {
      const float w0 = s.w1[k * kHid + j], w1 = s.w1[(k + 1) * kHid + j], w2 = s.w1[(k + 2) * kHid + j],
                  w3 = s.w1[(k + 3) * kHid + j];
#pragma unroll
      for (int b = 0; b < NS; ++b) {
        const float4 v = *reinterpret_cast<const float4*>(&s.x[b0 + b][k]);
        a[b] = fmaf(v.w, w3, fmaf(v.z, w2, fmaf(v.y, w1, fmaf(v.x, w0, a[b]))));
      }
    }
#pragma unroll
    for (int b = 0; b < NS; ++b) s.h1[b0 + b][j] = fmaxf(a[b], 0.f);
    __syncthreads();
#pragma unroll
    for (int b = 0; b < NS; ++b) a[b] = s.b2[j];
#pragma unroll 4
    for (int k = 0; k < kHid; k += 4) {
      const float w0 = s.w2[k * kW2Row + j], w1 = s.w2[(k + 1) * kW2Row + j], w2 = s.w2[(k + 2) * kW2Row + j],
                  w3 = s.w2[(k + 3) * kW2Row + j];
#pragma unroll
      for (int b = 0; b < NS; ++b) {
        const float4 v = *reinterpret_cast<const float4*>(&s.h1[b0 + b][k]);
        a[b] = fmaf(v.w, w3, fmaf(v.z, w2, fmaf(v.y, w1, fmaf(v.x, w0, a[b]))));
      }
    }
#pragma unroll
    for (int b = 0; b < NS; ++b) s.h2[b0 + b][j] = fmaxf(a[b], 0.f);
    __syncthreads();
    // outputs, loss and dL/dy: a warp a sample
    for (int b = warp; b < T; b += kWarps) {
      const float ha = s.h2[b][lane], hb = s.h2[b][lane + 32];
      float y0 = fmaf(hb, s.w3[2 * lane + 64], ha * s.w3[2 * lane]);
      float y1 = fmaf(hb, s.w3[2 * lane + 65], ha * s.w3[2 * lane + 1]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        y0 += __shfl_xor_sync(0xffffffffu, y0, o);
        y1 += __shfl_xor_sync(0xffffffffu, y1, o);
      }
      if (lane < kOut) {
        float d = 0.f;
        if (b < nt) {
          d = (lane == 0 ? y0 + s.b3[0] : y1 + s.b3[1]) - target[static_cast<long long>(r0 + b) * kOut + lane];
          loss += d * d;
        }
        s.dy[b][lane] = d * inv_b;
      }
    }
    __syncthreads();
    // dL/dh2 (through the second ReLU)
#pragma unroll
    for (int b = 0; b < NS; ++b) {
      const float g = fmaf(s.dy[b0 + b][1], s.w3[2 * j + 1], s.dy[b0 + b][0] * s.w3[2 * j]);
      s.d2[b0 + b][j] = s.h2[b0 + b][j] > 0.f ? g : 0.f;
      a[b] = 0.f;
    }
    __syncthreads();
    // dL/dh1 (through the first ReLU): this thread's unit j of the first layer
#pragma unroll 4
    for (int k = 0; k < kHid; k += 4) {
      const float w0 = s.w2[j * kW2Row + k], w1 = s.w2[j * kW2Row + k + 1], w2 = s.w2[j * kW2Row + k + 2],
                  w3 = s.w2[j * kW2Row + k + 3];
#pragma unroll
      for (int b = 0; b < NS; ++b) {
        const float4 v = *reinterpret_cast<const float4*>(&s.d2[b0 + b][k]);
        a[b] = fmaf(v.w, w3, fmaf(v.z, w2, fmaf(v.y, w1, fmaf(v.x, w0, a[b]))));
      }
    }
#pragma unroll
    for (int b = 0; b < NS; ++b) s.d1[b0 + b][j] = s.h1[b0 + b][j] > 0.f ? a[b] : 0.f;
    __syncthreads();
    // the tile's weight gradients, summed over its samples in order
#pragma unroll 2
    for (int b = 0; b < nt; ++b) {
      const float e2 = s.d2[b][j], e1 = s.d1[b][j];
#pragma unroll
      for (int i = 0; i < G2; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(&s.h1[b][(tid >> 6) * G2 + i]);
        g2[i] = fmaf(v.x, e2, g2[i]);
        g2[i + 1] = fmaf(v.y, e2, g2[i + 1]);
        g2[i + 2] = fmaf(v.z, e2, g2[i + 2]);
        g2[i + 3] = fmaf(v.w, e2, g2[i + 3]);
      }
#pragma unroll
      for (int i = 0; i < G1; ++i) g1[i] = fmaf(s.x[b][(tid >> 6) * G1 + i], e1, g1[i]);
      if (tid < 2 * kHid)
        gs = fmaf(s.h2[b][tid >> 1], s.dy[b][tid & 1], gs);
      else
        gs += tid < 3 * kHid ? e1 : e2;
      if (tid < kOut) gb3 += s.dy[b][tid];
    }
  }
  auto add = [&](int i, float g) {
    if (g != 0.f) atomicAdd(grads + i, g);
  };
#pragma unroll
  for (int i = 0; i < G2; ++i) add(kW2 + ((tid >> 6) * G2 + i) * kHid + j, g2[i]);
#pragma unroll
  for (int i = 0; i < G1; ++i) add(kW1 + ((tid >> 6) * G1 + i) * kHid + j, g1[i]);
  add(tid < 2 * kHid ? kW3 + tid : tid < 3 * kHid ? kB1 + j : kB2 + j, gs);
  if (tid < kOut) add(kB3 + tid, gb3);
  if (loss_sum != nullptr) {
    loss += __shfl_xor_sync(0xffffffffu, loss, 1);
    if (lane == 0 && loss != 0.f) atomicAdd(loss_sum, 0.5f * loss);
  }
}

__global__ void mlp_adam_kernel(float* params, const float* grads, float* m, float* v, int n, float lr, float beta1,
                                float beta2, float eps, float bc1, float bc2, float weight_decay) {
  allow_dependent();
  wait_for_predecessor();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float g = grads[i] + weight_decay * params[i];
    const float mi = beta1 * m[i] + (1.f - beta1) * g;
    const float vi = beta2 * v[i] + (1.f - beta2) * g * g;
    m[i] = mi;
    v[i] = vi;
    params[i] -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
  }
}

// Backward tiles: 8 samples while that gives at most half of the SMs one (a training step:
// latency), else 32 — every CTA's partial gradient is one more fp32 rounding in each sum, and
// at 1,000 to 4,096 samples both take a step of the same length (23 us, launches).
constexpr int kBwdSmall = 8, kBwdLarge = 32;
// Forward samples a lane: 2 while tiles of 16 give every warp of the chip at most one (18,944
// samples: 11.1 us a call; the tiles of 64 that 18,945 take: 14.3 us, and a batch of 64 would
// wait for one warp's 64), else 8.
constexpr int kFwdSmall = 2, kFwdLarge = 8;

// Both kernels need more than the default 48 KB of shared memory: opt in, per device.
int mlp_init_device(const DeviceState&) {
  auto opt_in = [](const void* fn, size_t bytes) {
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  };
  if (opt_in(reinterpret_cast<const void*>(mlp_forward_kernel<kFwdSmall>), sizeof(FwdSmem<kFwdSmall>)) != cudaSuccess ||
      opt_in(reinterpret_cast<const void*>(mlp_forward_kernel<kFwdLarge>), sizeof(FwdSmem<kFwdLarge>)) != cudaSuccess ||
      opt_in(reinterpret_cast<const void*>(mlp_backward_kernel<kBwdSmall>), sizeof(BwdSmem<kBwdSmall>)) != cudaSuccess ||
      opt_in(reinterpret_cast<const void*>(mlp_backward_kernel<kBwdLarge>), sizeof(BwdSmem<kBwdLarge>)) != cudaSuccess)
    return MB_ERR_CUDA;
  return MB_OK;
}

}  // namespace mb

using namespace mb;

extern "C" int mb_mlp_forward(const float* params, const float* x, int batch, float* y, mb_stream_t stream) {
  if (batch == 0) return MB_OK;
  if (params == nullptr || x == nullptr || y == nullptr || batch < 0) return MB_ERR_ARG;
  int err = MB_OK;
  DeviceState* ds = current_device_state(&err);
  if (ds == nullptr) return err;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool small = batch <= 8 * kFwdSmall * kFwdWarps * ds->num_sms;
  const int tile = 8 * (small ? kFwdSmall : kFwdLarge);
  const long long tiles = (static_cast<long long>(batch) + tile - 1) / tile;
  const int grid = static_cast<int>(tiles < ds->num_sms ? tiles : ds->num_sms);
  const auto fn = small ? mlp_forward_kernel<kFwdSmall> : mlp_forward_kernel<kFwdLarge>;
  const size_t smem = small ? sizeof(FwdSmem<kFwdSmall>) : sizeof(FwdSmem<kFwdLarge>);
  if (launch_dependent(fn, grid, kFwdWarps * 32, smem, st, params, x, batch, y) != cudaSuccess) return MB_ERR_LAUNCH;
  note_launches(1);
  return MB_OK;
}

extern "C" int mb_mlp_backward(const float* params, const float* x, const float* target, int batch, float* grads,
                               float* loss_sum, mb_stream_t stream) {
  if (batch == 0) return MB_OK;
  if (params == nullptr || x == nullptr || target == nullptr || grads == nullptr || batch < 0) return MB_ERR_ARG;
  int err = MB_OK;
  DeviceState* ds = current_device_state(&err);
  if (ds == nullptr) return err;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool small = batch <= kBwdSmall * (ds->num_sms / 2);
  const int tile = small ? kBwdSmall : kBwdLarge;
  const long long tiles = (static_cast<long long>(batch) + tile - 1) / tile;
  const int grid = static_cast<int>(tiles < ds->num_sms ? tiles : ds->num_sms);
  const auto fn = small ? mlp_backward_kernel<kBwdSmall> : mlp_backward_kernel<kBwdLarge>;
  const size_t smem = small ? sizeof(BwdSmem<kBwdSmall>) : sizeof(BwdSmem<kBwdLarge>);
  if (launch_dependent(fn, grid, kBwdThreads, smem, st, params, x, target, batch, grads, loss_sum) != cudaSuccess)
    return MB_ERR_LAUNCH;
  note_launches(1);
  return MB_OK;
}

extern "C" int mb_mlp_adam(float* params, const float* grads, float* m, float* v, int n, float lr, float beta1,
                           float beta2, float eps, int step, float weight_decay, mb_stream_t stream) {
  if (n == 0) return MB_OK;
  if (params == nullptr || grads == nullptr || m == nullptr || v == nullptr || n < 0 || step < 1) return MB_ERR_ARG;
  // bias corrections 1 - beta^step, computed on the host in double
  const float bc1 = static_cast<float>(1.0 - std::pow(static_cast<double>(beta1), step));
  const float bc2 = static_cast<float>(1.0 - std::pow(static_cast<double>(beta2), step));
  int blocks = (n + 255) / 256;
  if (blocks > 1024) blocks = 1024;
  if (launch_dependent(mlp_adam_kernel, blocks, 256, 0, static_cast<cudaStream_t>(stream), params, grads, m, v, n, lr,
                       beta1, beta2, eps, bc1, bc2, weight_decay) != cudaSuccess)
    return MB_ERR_LAUNCH;
  note_launches(1);
  return MB_OK;
}

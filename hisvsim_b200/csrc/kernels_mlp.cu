// K7: the learned cost model's network, forward, backward and Adam, in FP32.
// One block handles 64 samples at a time with the whole parameter set, the
// activations of its samples and its gradient accumulators in shared memory
// (about 160 KB); gradients leave as per-block partials that a second kernel
// sums in a fixed order, so training is deterministic.
#include "internal.h"

namespace hisv {
namespace {

constexpr int H = kMlpHidden;
constexpr int SB = kMlpSamples;
constexpr int LDH = H + 1;  // odd row strides: no shared-memory bank conflicts
constexpr int kThreads = 256;

struct Offs {  // flat parameter offsets (global layout)
  int w1, b1, w2, b2, w3, b3, w4, b4, P;
  __host__ __device__ explicit Offs(int in) {
    w1 = 0;
    b1 = w1 + H * in;
    w2 = b1 + H;
    b2 = w2 + H * H;
    w3 = b2 + H;
    b3 = w3 + H * H;
    w4 = b3 + H;
    b4 = w4 + H;
    P = b4 + 1;
  }
};

// shared-memory image of the parameters: weight rows padded to odd strides
struct SParams {
  float *w1, *b1, *w2, *b2, *w3, *b3, *w4, *b4;
  int ld1;
};

__device__ float* carve(float*& p, int n) {
  float* r = p;
  p += n;
  return r;
}

__device__ SParams load_params(const float* __restrict__ g, int in, float*& sm) {
  const Offs o(in);
  SParams s;
  s.ld1 = in + 1;
  s.w1 = carve(sm, H * s.ld1);
  s.b1 = carve(sm, H);
  s.w2 = carve(sm, H * LDH);
  s.b2 = carve(sm, H);
  s.w3 = carve(sm, H * LDH);
  s.b3 = carve(sm, H);
  s.w4 = carve(sm, H);
  s.b4 = carve(sm, 4);
  for (int i = threadIdx.x; i < H * in; i += kThreads) s.w1[(i / in) * s.ld1 + i % in] = g[o.w1 + i];
  for (int i = threadIdx.x; i < H * H; i += kThreads) {
    s.w2[(i / H) * LDH + i % H] = g[o.w2 + i];
    s.w3[(i / H) * LDH + i % H] = g[o.w3 + i];
  }
  for (int i = threadIdx.x; i < H; i += kThreads) {
    s.b1[i] = g[o.b1 + i];
    s.b2[i] = g[o.b2 + i];
    s.b3[i] = g[o.b3 + i];
    s.w4[i] = g[o.w4 + i];
  }
  if (threadIdx.x == 0) s.b4[0] = g[o.b4];
  return s;
}

// out[s][j] = relu(sum_k W[j][k] in[s][k] + b[j]); thread: sample t/4,
// neurons (t%4) + 4i
__device__ __forceinline__ void dense_relu(const float* W, int ldw, const float* b, const float* in,
                                           int ldi, int K, float* out) {
  const int s = threadIdx.x >> 2, j0 = threadIdx.x & 3;
  float acc[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) acc[i] = b[j0 + 4 * i];
  for (int k = 0; k < K; ++k) {
    const float x = in[s * ldi + k];
#pragma unroll
    for (int i = 0; i < 16; ++i) acc[i] = fmaf(W[(j0 + 4 * i) * ldw + k], x, acc[i]);
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) out[s * LDH + j0 + 4 * i] = fmaxf(acc[i], 0.f);
}

// f[s] = w4 . h3[s] + b4 (4 threads per sample, fixed-order shuffle sum)
__device__ __forceinline__ float head(const SParams& P, const float* h3) {
  const int s = threadIdx.x >> 2, j0 = threadIdx.x & 3;
  float a = 0.f;
#pragma unroll
  for (int i = 0; i < 16; ++i) a = fmaf(P.w4[j0 + 4 * i], h3[s * LDH + j0 + 4 * i], a);
  a += __shfl_xor_sync(0xffffffffu, a, 1);
  a += __shfl_xor_sync(0xffffffffu, a, 2);
  return a + P.b4[0];
}

// rows [0, ns) of x (through idx) into sx[s][k], zero rows beyond
__device__ void load_x(const float* __restrict__ x, int in, const int32_t* __restrict__ idx,
                       int first, int ns, float* sx) {
  const int ldx = in + 1;
  for (int i = threadIdx.x; i < SB * in; i += kThreads) {
    const int s = i / in, k = i % in;
    float v = 0.f;
    if (s < ns) {
      const int64_t row = idx ? int64_t(idx[first + s]) : int64_t(first + s);
      v = x[row * in + k];
    }
    sx[s * ldx + k] = v;
  }
}

__global__ void __launch_bounds__(kThreads) k7_forward(const float* __restrict__ params, int in,
                                                       const float* __restrict__ x, int n,
                                                       float* __restrict__ out) {
  extern __shared__ __align__(16) float smem[];
  float* sm = smem;
  const SParams P = load_params(params, in, sm);
  float* sx = carve(sm, SB * (in + 1));
  float* h1 = carve(sm, SB * LDH);
  float* h2 = carve(sm, SB * LDH);
  for (int first = blockIdx.x * SB; first < n; first += gridDim.x * SB) {
    const int ns = min(SB, n - first);
    __syncthreads();
    load_x(x, in, nullptr, first, ns, sx);
    __syncthreads();
    dense_relu(P.w1, P.ld1, P.b1, sx, in + 1, in, h1);
    __syncthreads();
    dense_relu(P.w2, LDH, P.b2, h1, LDH, H, h2);
    __syncthreads();
    dense_relu(P.w3, LDH, P.b3, h2, LDH, H, h1);
    __syncthreads();
    const float f = head(P, h1);
    const int s = threadIdx.x >> 2;
    if ((threadIdx.x & 3) == 0 && s < ns) out[first + s] = f;
  }
}

// gW[j][k] += sum_s dz[s][j] in[s][k], gb[j] += sum_s dz[s][j]
// (thread: row j = t/4, columns (t%4) + 4i)
__device__ __forceinline__ void grad_weights(const float* dz, const float* in, int ldi, int K,
                                             float* gW, float* gb) {
  const int j = threadIdx.x >> 2, k0 = threadIdx.x & 3;
  float acc[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) acc[i] = 0.f;
  float ab = 0.f;
  for (int s = 0; s < SB; ++s) {
    const float d = dz[s * LDH + j];
    ab += d;
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (k0 + 4 * i < K) acc[i] = fmaf(d, in[s * ldi + k0 + 4 * i], acc[i]);
  }
#pragma unroll
  for (int i = 0; i < 16; ++i)
    if (k0 + 4 * i < K) gW[j * K + k0 + 4 * i] += acc[i];
  if (k0 == 0) gb[j] += ab;
}

// in place: h[s][k] <- (sum_j dz[s][j] W[j][k]) * (h[s][k] > 0)
__device__ __forceinline__ void back_relu(const float* dz, const float* W, float* h) {
  const int s = threadIdx.x >> 2, k0 = threadIdx.x & 3;
  float acc[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) acc[i] = 0.f;
  for (int j = 0; j < H; ++j) {
    const float d = dz[s * LDH + j];
#pragma unroll
    for (int i = 0; i < 16; ++i) acc[i] = fmaf(d, W[j * LDH + k0 + 4 * i], acc[i]);
  }
  __syncthreads();  // every thread has read dz before anyone overwrites h (dz may alias)
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    float* hp = &h[s * LDH + k0 + 4 * i];
    *hp = *hp > 0.f ? acc[i] : 0.f;
  }
}

__global__ void __launch_bounds__(kThreads)
    k7_backward(const float* __restrict__ params, int in, const float* __restrict__ x,
                const float* __restrict__ y, const int32_t* __restrict__ idx, int n, float scale,
                float* __restrict__ partial, float* __restrict__ loss_partial) {
  extern __shared__ __align__(16) float smem[];
  float* sm = smem;
  const SParams P = load_params(params, in, sm);
  const Offs o(in);
  float* sx = carve(sm, SB * (in + 1));
  float* h1 = carve(sm, SB * LDH);
  float* h2 = carve(sm, SB * LDH);
  float* h3 = carve(sm, SB * LDH);
  float* sg = carve(sm, (o.P + 3) & ~3);
  float* sl = carve(sm, kThreads / 32);
  for (int i = threadIdx.x; i < o.P; i += kThreads) sg[i] = 0.f;
  float loss = 0.f;
  for (int first = blockIdx.x * SB; first < n; first += gridDim.x * SB) {
    const int ns = min(SB, n - first);
    __syncthreads();
    load_x(x, in, idx, first, ns, sx);
    __syncthreads();
    dense_relu(P.w1, P.ld1, P.b1, sx, in + 1, in, h1);
    __syncthreads();
    dense_relu(P.w2, LDH, P.b2, h1, LDH, H, h2);
    __syncthreads();
    dense_relu(P.w3, LDH, P.b3, h2, LDH, H, h3);
    __syncthreads();
    const int s = threadIdx.x >> 2, k0 = threadIdx.x & 3;
    const float f = head(P, h3);
    float d = 0.f;
    if (s < ns) {
      const int64_t row = idx ? int64_t(idx[first + s]) : int64_t(first + s);
      const float r = f - y[row];
      d = scale * r;
      if (k0 == 0) loss += r * r;
    }
    // head gradients: gw4[k] = sum_s d_s h3[s][k], gb4 = sum_s d_s
    // dz3 = d_s w4[k] (h3 > 0), in place over h3 once h3 is consumed
    {
      // d of sample s lives in the 4 threads of s; stage it in h2's spare column
      if (k0 == 0) h2[s * LDH + H] = d;
    }
    __syncthreads();
    if (threadIdx.x < H) {
      float a = 0.f;
      for (int q = 0; q < SB; ++q) a = fmaf(h2[q * LDH + H], h3[q * LDH + threadIdx.x], a);
      sg[o.w4 + threadIdx.x] += a;
    } else if (threadIdx.x == H) {
      float a = 0.f;
      for (int q = 0; q < SB; ++q) a += h2[q * LDH + H];
      sg[o.b4] += a;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float* hp = &h3[s * LDH + k0 + 4 * i];
      *hp = *hp > 0.f ? d * P.w4[k0 + 4 * i] : 0.f;
    }
    __syncthreads();
    grad_weights(h3, h2, LDH, H, sg + o.w3, sg + o.b3);
    __syncthreads();
    back_relu(h3, P.w3, h2);  // dz2 over h2
    __syncthreads();
    grad_weights(h2, h1, LDH, H, sg + o.w2, sg + o.b2);
    __syncthreads();
    back_relu(h2, P.w2, h1);  // dz1 over h1
    __syncthreads();
    grad_weights(h1, sx, in + 1, in, sg + o.w1, sg + o.b1);
  }
  // block loss: fixed-order warp sums, then warps in order
  for (int off = 16; off > 0; off >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, off);
  if ((threadIdx.x & 31) == 0) sl[threadIdx.x >> 5] = loss;
  __syncthreads();
  for (int i = threadIdx.x; i < o.P; i += kThreads) partial[size_t(blockIdx.x) * o.P + i] = sg[i];
  if (threadIdx.x == 0) {
    float a = 0.f;
    for (int w = 0; w < kThreads / 32; ++w) a += sl[w];
    loss_partial[blockIdx.x] = a;
  }
}

// ---- small batches: kSmall samples per block -------------------------------------
// A training step has a few hundred samples.  In blocks of 64 it runs on four
// SMs and each waits on its own chain of dense layers (60 us for 256 samples);
// here a block takes four samples, so the step spreads over 64 blocks, and the
// time is that of loading the parameters (57 KB from the L2), eight short
// stages and one write of the block's gradients.  A block has one tile, so the
// gradients go to its partial without accumulators in shared memory.  Larger
// batches than one such wave keep k7_backward, which reads the parameters once
// per 64 samples.
constexpr int kSmall = 4;
constexpr int LDV = H + 4;  // row stride for 16-byte row reads: 17 units, distinct banks

struct SmallShared {  // (everything read as float4 sits on 16-byte boundaries)
  alignas(16) float w1[H * LDV];  // rows W[j][k], zero beyond the inputs
  alignas(16) float w2[H * LDV];
  alignas(16) float w3[H * LDV];
  alignas(16) float x[kSmall][LDV];
  alignas(16) float h1[kSmall][LDV];
  alignas(16) float h2[kSmall][LDV];
  alignas(16) float h3[kSmall][LDV];
  alignas(16) float dz[2][H][kSmall];  // deltas of a layer, by neuron then sample
  float part[4][kSmall][H];            // partial sums of a backward layer
  float b1[H], b2[H], b3[H], w4[H];
  float b4, d[kSmall];
};
static_assert(LDV % 4 == 0 && kSmall == 4 && kThreads == 4 * H, "float4 rows, one thread per (j, quarter)");

// out[s][j] = relu(sum_k W[j][k] in[s][k] + b[j]): thread (j, quarter of k) for
// every sample of the block, the quarters summed over neighbouring lanes
__device__ __forceinline__ void small_dense(const float* W, const float* b,
                                            const float (*in)[LDV], float (*out)[LDV]) {
  const int q = threadIdx.x & 3, j = threadIdx.x >> 2;
  float acc[kSmall] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 0; i < H / 16; ++i) {
    const int k = 4 * (q + 4 * i);
    const float4 w = *reinterpret_cast<const float4*>(W + j * LDV + k);
#pragma unroll
    for (int s = 0; s < kSmall; ++s) {
      const float4 x = *reinterpret_cast<const float4*>(&in[s][k]);
      acc[s] = fmaf(w.x, x.x, acc[s]);
      acc[s] = fmaf(w.y, x.y, acc[s]);
      acc[s] = fmaf(w.z, x.z, acc[s]);
      acc[s] = fmaf(w.w, x.w, acc[s]);
    }
  }
#pragma unroll
  for (int s = 0; s < kSmall; ++s) {
    acc[s] += __shfl_xor_sync(0xffffffffu, acc[s], 1);
    acc[s] += __shfl_xor_sync(0xffffffffu, acc[s], 2);
    if (q == s) out[s][j] = fmaxf(acc[s] + b[j], 0.f);
  }
}

// deltas one layer down: (sum_j dz[j][s] W[j][k]) where h[s][k] > 0
__device__ __forceinline__ void small_back(SmallShared& S, const float* W, const float (*dz)[kSmall],
                                           const float (*h)[LDV], float (*out)[kSmall]) {
  const int k = threadIdx.x & (H - 1), q = threadIdx.x / H;
  float acc[kSmall] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 0; i < H / 4; ++i) {
    const int j = q * (H / 4) + i;
    const float w = W[j * LDV + k];
    const float4 d = *reinterpret_cast<const float4*>(dz[j]);
    acc[0] = fmaf(d.x, w, acc[0]);
    acc[1] = fmaf(d.y, w, acc[1]);
    acc[2] = fmaf(d.z, w, acc[2]);
    acc[3] = fmaf(d.w, w, acc[3]);
  }
#pragma unroll
  for (int s = 0; s < kSmall; ++s) S.part[q][s][k] = acc[s];
  __syncthreads();
  const float a = (S.part[0][q][k] + S.part[1][q][k]) + (S.part[2][q][k] + S.part[3][q][k]);
  out[k][q] = h[q][k] > 0.f ? a : 0.f;  // (four quarters, four samples)
}

// gradients of a layer with K inputs straight to the block's partial
__device__ __forceinline__ void small_grad(const float (*dz)[kSmall], const float (*in)[LDV], int K,
                                           float* __restrict__ gw, float* __restrict__ gb) {
  // thread (k, quarter of the rows): its inputs stay in registers
  const int k = threadIdx.x & (H - 1), q = threadIdx.x / H;
  if (k < K) {
    float x[kSmall];
#pragma unroll
    for (int s = 0; s < kSmall; ++s) x[s] = in[s][k];
#pragma unroll
    for (int i = 0; i < H / 4; ++i) {
      const int j = q * (H / 4) + i;
      const float4 d = *reinterpret_cast<const float4*>(dz[j]);
      gw[j * K + k] = fmaf(d.w, x[3], fmaf(d.z, x[2], fmaf(d.y, x[1], d.x * x[0])));
    }
  }
  if (threadIdx.x < H) {
    const float4 d = *reinterpret_cast<const float4*>(dz[threadIdx.x]);
    gb[threadIdx.x] = (d.x + d.y) + (d.z + d.w);
  }
}

__global__ void __launch_bounds__(kThreads)
    k7_small(const float* __restrict__ params, int in, const float* __restrict__ x,
             const float* __restrict__ y, const int32_t* __restrict__ idx, int n, float scale,
             float* __restrict__ partial, float* __restrict__ loss_partial) {
  extern __shared__ __align__(16) float smem[];
  SmallShared& S = *reinterpret_cast<SmallShared*>(smem);
  const Offs o(in);
  const int t = threadIdx.x, first = blockIdx.x * kSmall, ns = min(kSmall, n - first);
  // every load of the parameters in flight at once (the block's longest wait);
  // the layers' offsets are multiples of 64 floats
  {
    float4 a[4], c[4];
    float e[H * H / kThreads];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      a[r] = *reinterpret_cast<const float4*>(params + o.w2 + 4 * (t + r * kThreads));
      c[r] = *reinterpret_cast<const float4*>(params + o.w3 + 4 * (t + r * kThreads));
    }
#pragma unroll
    for (int r = 0; r < H * H / kThreads; ++r) {
      const int i = t + r * kThreads, j = i / H, k = i % H;
      e[r] = k < in ? params[o.w1 + j * in + k] : 0.f;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = 4 * (t + r * kThreads), j = i / H, k = i % H;
      *reinterpret_cast<float4*>(&S.w2[j * LDV + k]) = a[r];
      *reinterpret_cast<float4*>(&S.w3[j * LDV + k]) = c[r];
    }
#pragma unroll
    for (int r = 0; r < H * H / kThreads; ++r) {
      const int i = t + r * kThreads;
      S.w1[(i / H) * LDV + i % H] = e[r];
    }
  }
  if (t < H) {
    S.b1[t] = params[o.b1 + t];
    S.b2[t] = params[o.b2 + t];
    S.b3[t] = params[o.b3 + t];
    S.w4[t] = params[o.w4 + t];
  }
  if (t == 0) S.b4 = params[o.b4];
  {
    const int s = t / H, k = t % H;  // one input per thread, zero beyond the samples
    float v = 0.f;
    if (s < ns && k < in) v = x[int64_t(idx ? idx[first + s] : first + s) * in + k];
    S.x[s][k] = v;
  }
  __syncthreads();
  small_dense(S.w1, S.b1, S.x, S.h1);
  __syncthreads();
  small_dense(S.w2, S.b2, S.h1, S.h2);
  __syncthreads();
  small_dense(S.w3, S.b3, S.h2, S.h3);
  __syncthreads();
  if (t < 32 * kSmall) {  // the head: a warp per sample
    const int s = t >> 5, l = t & 31;
    float a = fmaf(S.w4[l], S.h3[s][l], S.w4[l + 32] * S.h3[s][l + 32]);
    for (int off = 16; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
    if (l == 0) {
      float r = 0.f;
      if (s < ns) r = a + S.b4 - y[idx ? idx[first + s] : first + s];
      S.d[s] = scale * r;
      S.part[0][s][0] = r * r;
    }
  }
  __syncthreads();
  float* g = partial + size_t(blockIdx.x) * o.P;
  if (t == 0) {
    g[o.b4] = (S.d[0] + S.d[1]) + (S.d[2] + S.d[3]);
    loss_partial[blockIdx.x] = (S.part[0][0][0] + S.part[0][1][0]) + (S.part[0][2][0] + S.part[0][3][0]);
  }
  if (t < H) {
    float a = 0.f;
#pragma unroll
    for (int s = 0; s < kSmall; ++s) a = fmaf(S.d[s], S.h3[s][t], a);
    g[o.w4 + t] = a;
  }
  {
    const int s = t / H, k = t % H;
    S.dz[0][k][s] = S.h3[s][k] > 0.f ? S.d[s] * S.w4[k] : 0.f;
  }
  __syncthreads();
  small_grad(S.dz[0], S.h2, H, g + o.w3, g + o.b3);
  small_back(S, S.w3, S.dz[0], S.h2, S.dz[1]);
  __syncthreads();
  small_grad(S.dz[1], S.h1, H, g + o.w2, g + o.b2);
  small_back(S, S.w2, S.dz[1], S.h1, S.dz[0]);
  __syncthreads();
  small_grad(S.dz[0], S.x, in, g + o.w1, g + o.b1);
}

// the sum of the blocks' partials of parameter i, in order
__device__ __forceinline__ float sum_partials(const float* __restrict__ partial, int nblk, int P,
                                              int i) {
  float a = 0.f;
#pragma unroll 32
  for (int b = 0; b < nblk; ++b) a += partial[size_t(b) * P + i];
  return a;
}

__global__ void k7_reduce(const float* __restrict__ partial, const float* __restrict__ loss_partial,
                          int nblk, int P, float* __restrict__ grad, float* __restrict__ loss) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < P) grad[i] = sum_partials(partial, nblk, P, i);
  if (i == 0 && loss) {
    float a = 0.f;
    for (int b = 0; b < nblk; ++b) a += loss_partial[b];
    *loss = a;
  }
}

// one Adam step from the blocks' partials (the sum of k7_reduce in the same launch)
__global__ void k7_adam(float* __restrict__ params, const float* __restrict__ partial,
                        const float* __restrict__ loss_partial, int nblk, float* __restrict__ m,
                        float* __restrict__ v, int P, float lr, float b1, float b2, float eps,
                        float c1, float c2, float* __restrict__ loss) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    float a = 0.f;
    for (int b = 0; b < nblk; ++b) a += loss_partial[b];
    *loss = a;
  }
  if (i >= P) return;
  const float g = sum_partials(partial, nblk, P, i);
  const float mi = b1 * m[i] + (1.f - b1) * g;
  const float vi = b2 * v[i] + (1.f - b2) * g * g;
  m[i] = mi;
  v[i] = vi;
  params[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

size_t smem_forward(int in) {
  return sizeof(float) * size_t(H * (in + 1) + 3 * H + 2 * H * LDH + H + 4 + SB * (in + 1) +
                                 2 * SB * LDH);
}
size_t smem_backward(int in) {
  const Offs o(in);
  return smem_forward(in) + sizeof(float) * size_t(SB * LDH + ((o.P + 3) & ~3) + kThreads / 32);
}

}  // namespace

int launch_mlp_forward(const float* params, int in, const float* x, int n, float* out,
                       cudaStream_t s) {
  if (in < 1 || in > kMlpMaxIn) return set_error(HS_E_INVALID, "input width %d", in);
  if (n <= 0) return HS_OK;
  const size_t sm = smem_forward(in);
  HS_CUDA(cudaFuncSetAttribute(k7_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sm)));
  int dev = 0, sms = 148;
  HS_CUDA(cudaGetDevice(&dev));
  HS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int grid = std::min((n + SB - 1) / SB, sms);
  k7_forward<<<grid, kThreads, sm, s>>>(params, in, x, n, out);
  HS_CUDA(cudaGetLastError());
  return HS_OK;
}

int mlp_backward_blocks(int n, int sms) {
  const int small = (n + kSmall - 1) / kSmall;
  return small <= sms ? small : std::max(1, std::min((n + SB - 1) / SB, sms));
}

int launch_mlp_backward(const float* params, int in, const float* x, const float* y,
                        const int32_t* idx, int n, float scale, float* partial,
                        float* loss_partial, int nblk, cudaStream_t s) {
  if (in < 1 || in > kMlpMaxIn) return set_error(HS_E_INVALID, "input width %d", in);
  if (nblk == (n + kSmall - 1) / kSmall) {  // mlp_backward_blocks chose the small form
    HS_TRY(smem_optin(reinterpret_cast<const void*>(k7_small)));
    k7_small<<<nblk, kThreads, sizeof(SmallShared), s>>>(params, in, x, y, idx, n, scale, partial,
                                                         loss_partial);
    HS_CUDA(cudaGetLastError());
    return HS_OK;
  }
  const size_t sm = smem_backward(in);
  HS_CUDA(cudaFuncSetAttribute(k7_backward, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sm)));
  k7_backward<<<nblk, kThreads, sm, s>>>(params, in, x, y, idx, n, scale, partial, loss_partial);
  HS_CUDA(cudaGetLastError());
  return HS_OK;
}

int launch_mlp_reduce(const float* partial, const float* loss_partial, int nblk, int P,
                      float* grad, float* loss, cudaStream_t s) {
  k7_reduce<<<(P + 255) / 256, 256, 0, s>>>(partial, loss_partial, nblk, P, grad, loss);
  HS_CUDA(cudaGetLastError());
  return HS_OK;
}

int launch_mlp_adam(float* params, const float* partial, const float* loss_partial, int nblk,
                    float* m, float* v, int P, float lr, float beta1, float beta2, float eps,
                    int step, float* loss, cudaStream_t s) {
  const float c1 = 1.f - std::pow(beta1, float(step));
  const float c2 = 1.f - std::pow(beta2, float(step));
  k7_adam<<<(P + 127) / 128, 128, 0, s>>>(params, partial, loss_partial, nblk, m, v, P, lr, beta1,
                                          beta2, eps, c1, c2, loss);
  HS_CUDA(cudaGetLastError());
  return HS_OK;
}

}  // namespace hisv

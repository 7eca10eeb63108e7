// mlp.cu -- the path-guiding network on Blackwell tensor cores.
//
// No reference counterpart: Tracer has no path guiding. The network maps a
// path vertex (position normalised to the scene box, outgoing direction,
// roughness: 7 inputs) through four hidden layers of 64 ReLU units to the 40
// parameters of an 8-lobe von Mises-Fisher mixture. Weights and activations
// are fp16, accumulation fp32 (tcgen05.mma kind::f16 into tensor memory).
//
// Forward kernel: persistent CTAs of 128 threads, one 128-row tile at a
// time. All weights live in shared memory in the core-matrix layout of
// tc05.cuh; a layer is K/16 MMAs (M = 128, N = 64 or 48) issued by one
// thread into a 64-column TMEM accumulator; the four warps read their 32
// rows back (tcgen05.ld), add the bias, apply ReLU and write fp16 into the
// next layer's A operand.

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <utility>
#include <cstring>
#include <vector>

#include "context.h"
#include "mixture.cuh"
#include "mlp.h"
#include "tc05.cuh"

namespace trg {
namespace mlp {

// shared-memory image: W0..W4 (fp16, core layout), biases (fp32)
__host__ __device__ constexpr uint32_t w_off(int l) {
  return l == 0 ? 0u : (l == 1 ? 2048u : (l == 2 ? 10240u : (l == 3 ? 18432u : 26624u)));
}
constexpr uint32_t kBiasOff = 32768;                        // 4 x 64 + 48 floats
constexpr uint32_t kPackedBytes = kBiasOff + 304 * 4;        // 33984
constexpr uint32_t kAOff = 34048;                            // 128 x 64 fp16
constexpr uint32_t kMbarOff = kAOff + kTile * kHid * 2;      // 50432
constexpr uint32_t kSlotOff = kMbarOff + 8;
constexpr uint32_t kSmemBytes = kSlotOff + 8;
static_assert(kPackedBytes % 16 == 0, "packed image is copied in 16-byte units");
static_assert(w_off(4) + kOutPad * kHid * 2 == kBiasOff, "weight image layout");

__host__ __device__ constexpr int layer_k(int l) { return l == 0 ? kInPad : kHid; }
__host__ __device__ constexpr int layer_n(int l) { return l == 4 ? kOutPad : kHid; }
__host__ __device__ constexpr int layer_kin(int l) { return l == 0 ? kIn : kHid; }
__host__ __device__ constexpr int layer_nout(int l) { return l == 4 ? kOut : kHid; }

// Offsets of W_l (nout x kin, row-major) and b_l in the flat fp32 parameter vector.
__host__ __device__ constexpr int param_w(int l) {
  return l == 0 ? 0 : (l == 1 ? 512 : (l == 2 ? 4672 : (l == 3 ? 8832 : 12992)));
}
__host__ __device__ constexpr int param_b(int l) { return param_w(l) + layer_nout(l) * layer_kin(l); }
static_assert(param_b(4) + kOut == kParams, "parameter layout");

// Writes the shared-memory image (fp16 weights in core layout, fp32 biases)
// from the fp32 parameters; one thread per image element.
__global__ void k_pack(const float* __restrict__ p, uint8_t* __restrict__ img) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  // weights: element (n, k) of layer l
  int base = 0;
  for (int l = 0; l < kLayers; ++l) {
    const int N = layer_n(l), K = layer_k(l);
    if (i < base + N * K) {
      const int e = i - base, n = e / K, k = e % K;
      const float v = (n < layer_nout(l) && k < layer_kin(l)) ? p[param_w(l) + n * layer_kin(l) + k] : 0.0f;
      *reinterpret_cast<__half*>(img + w_off(l) + tc05::core_off(n, k, K)) = __float2half_rn(v);
      return;
    }
    base += N * K;
  }
  const int j = i - base;
  if (j < 304) {
    const int l = j < 256 ? j / 64 : 4, c = j < 256 ? j % 64 : j - 256;
    reinterpret_cast<float*>(img + kBiasOff)[j] = c < layer_nout(l) ? p[param_b(l) + c] : 0.0f;
  }
}
constexpr int kPackThreads = 64 * 16 + 3 * 64 * 64 + 48 * 64 + 304;  // W0, W1..W3, W4, biases

__device__ __forceinline__ uint32_t h2_bits(__half2 h) {
  uint32_t u;
  memcpy(&u, &h, 4);
  return u;
}
// max(x, 0) of two values as fp16; NaN gives 0 (as fmaxf does)
__device__ __forceinline__ uint32_t h2_relu(float a, float b) {
  return h2_bits(__hmax2(__floats2half2_rn(a, b), __float2half2_rn(0.0f)));
}

// A hidden layer's epilogue for 32 of a row's columns: c = fp32 sums, plus
// the bias, ReLU, fp16, into columns c0 .. c0 + 31 of the 64-column operand tile.
__device__ __forceinline__ void hidden_epilogue(const uint32_t (&c)[32], const float* bias, uint8_t* tile, int row, int c0) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float4 b0 = reinterpret_cast<const float4*>(bias + c0)[2 * q], b1 = reinterpret_cast<const float4*>(bias + c0)[2 * q + 1];
    const int k = 8 * q;
    int4 h;
    h.x = (int)h2_relu(__uint_as_float(c[k]) + b0.x, __uint_as_float(c[k + 1]) + b0.y);
    h.y = (int)h2_relu(__uint_as_float(c[k + 2]) + b0.z, __uint_as_float(c[k + 3]) + b0.w);
    h.z = (int)h2_relu(__uint_as_float(c[k + 4]) + b1.x, __uint_as_float(c[k + 5]) + b1.y);
    h.w = (int)h2_relu(__uint_as_float(c[k + 6]) + b1.z, __uint_as_float(c[k + 7]) + b1.w);
    *reinterpret_cast<int4*>(tile + tc05::core_off(row, c0 + k, kHid)) = h;
  }
}

// x: n x 7 fp32; out: n x 40 fp32 (decode: the 48 mixture floats per row).
__global__ void __launch_bounds__(128, 1)
    k_forward(const uint8_t* __restrict__ img, const float* __restrict__ x, int n, float* __restrict__ out, int* err,
              const unsigned int* __restrict__ n_dev, int decode) {
  extern __shared__ __align__(1024) uint8_t sm[];
  if (n_dev) n = (int)*n_dev;  // row count produced on the device (guided rendering)
  const int tid = threadIdx.x, warp = tid >> 5;
  for (int i = tid; i < (int)(kPackedBytes / 16); i += blockDim.x)
    reinterpret_cast<int4*>(sm)[i] = reinterpret_cast<const int4*>(img)[i];
  uint64_t* mbar = reinterpret_cast<uint64_t*>(sm + kMbarOff);
  uint32_t* slot = reinterpret_cast<uint32_t*>(sm + kSlotOff);
  if (tid == 0) tc05::mbar_init(mbar, 1);
  if (warp == 0) {
    tc05::tmem_alloc(slot, 64);
    tc05::tmem_relinquish();  // at once: the SM's other CTAs allocate their columns meanwhile
  }
  tc05::fence_before();
  __syncthreads();
  tc05::fence_after();
  const uint32_t tmem = *slot;
  const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
  const float* bias = reinterpret_cast<const float*>(sm + kBiasOff);
  uint8_t* A = sm + kAOff;
  const uint32_t a_addr = tc05::smem_u32(A);
  const uint32_t w_addr = tc05::smem_u32(sm);
  uint32_t phase = 0;
  bool ok = true;
  const int ntiles = (n + kTile - 1) / kTile;
  for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
    const int row = t * kTile + tid;
    {  // inputs, zero-padded to 16
      __align__(16) __half h[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) h[j] = __float2half_rn(j < kIn && row < n ? x[(size_t)row * kIn + j] : 0.0f);
      *reinterpret_cast<int4*>(A + tc05::core_off(tid, 0, kInPad)) = *reinterpret_cast<const int4*>(h);
      *reinterpret_cast<int4*>(A + tc05::core_off(tid, 8, kInPad)) = *reinterpret_cast<const int4*>(h + 8);
    }
    tc05::fence_proxy_async();
    __syncthreads();
#pragma unroll
    for (int l = 0; l < kLayers; ++l) {
      if (tid == 0) {
        tc05::fence_after();
        const uint32_t sbo = (uint32_t)(layer_k(l) / 8) * 128u;
        const tc05::Desc a = tc05::desc_of(a_addr, 128u, sbo), w = tc05::desc_of(w_addr + w_off(l), 128u, sbo);
#pragma unroll
        for (int kk = 0; kk < layer_k(l) / 16; ++kk)
          tc05::mma_f16(tmem, tc05::step(a, kk * 256u), tc05::step(w, kk * 256u),
                        tc05::idesc_f16_f32(128, (uint32_t)layer_n(l)), kk > 0 ? 1u : 0u);
        tc05::commit(mbar);
      }
      const bool got = tc05::mbar_wait(mbar, phase);
      ok = __syncthreads_and(got) != 0;
      if (!ok) break;
      phase ^= 1u;
      tc05::fence_after();
      if (l < kLayers - 1) {
        uint32_t c[32], d[32];
        tc05::tmem_ld32(tmem + lane_base, c);
        tc05::tmem_ld32(tmem + lane_base + 32u, d);
        tc05::tmem_wait(c);
        tc05::tmem_wait(d);
        hidden_epilogue(c, bias + 64 * l, A, tid, 0);
        hidden_epilogue(d, bias + 64 * l, A, tid, 32);
      } else {
        // the output row, whole in this thread: raw, or decoded into the
        // mixture's lobe parameters (guided rendering)
        float o[kOutPad];
#pragma unroll
        for (int c = 0; c < kOutPad / 16; ++c) {
          float v[16];
          tc05::tmem_ld16(tmem + lane_base + (uint32_t)(16 * c), v);
#pragma unroll
          for (int j = 0; j < 16; ++j) o[16 * c + j] = 16 * c + j < kOut ? v[j] + bias[256 + 16 * c + j] : 0.0f;
        }
        if (row < n) {
          if (decode) {
            float dd[kMixFloats];
            mixture_decode(o, dd);
            float4* dst = reinterpret_cast<float4*>(out + (size_t)row * kMixFloats);
#pragma unroll
            for (int q = 0; q < kMixFloats / 4; ++q)
              dst[q] = make_float4(dd[4 * q], dd[4 * q + 1], dd[4 * q + 2], dd[4 * q + 3]);
          } else if (((uintptr_t)out & 15u) == 0) {
            float4* dst = reinterpret_cast<float4*>(out + (size_t)row * kOut);
#pragma unroll
            for (int q = 0; q < kOut / 4; ++q) dst[q] = make_float4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
          } else {
#pragma unroll
            for (int j = 0; j < kOut; ++j) out[(size_t)row * kOut + j] = o[j];
          }
        }
      }
      tc05::fence_before();
      tc05::fence_proxy_async();
      __syncthreads();
    }
  }
  if (!ok) {
    if (tid == 0) atomicOr(err, 1);
    tc05::mbar_wait(mbar, phase);  // the same phase, bounded: let an MMA still in flight finish
  }
  __syncthreads();
  if (warp == 0) {
    tc05::tmem_dealloc(tmem, 64);
  }
}

// ------------------------------------------------------------ loss, Adam
//
// Negative log-likelihood of the directions under the 8-lobe vMF mixture,
// weighted per row: loss = -sum_i w_i log p(omega_i | x_i) / sum_i w_i.
// Lobe j of row i: out[5j] weight logit, out[5j+1] log kappa (clamped to
// [TR_GUIDE_LOG_KAPPA_MIN, TR_GUIDE_LOG_KAPPA_MAX]), out[5j+2..4]
// unnormalised mean direction;
// vMF(omega) = kappa / (2 pi (1 - exp(-2 kappa))) exp(kappa (mu.omega - 1)).

struct Lobe {
  float pi, kappa, mlen, c;
  float3 mu;
};

__device__ __forceinline__ float vmf_log_norm(float kappa) {
  // log(kappa / (2 pi (1 - exp(-2 kappa))))
  return logf(kappa) - 1.8378770664093453f - log1pf(-expf(-2.0f * kappa));
}

// log p(omega | z) of one row, and the gradient of -wi log p w.r.t. the row's
// network outputs z. The lobes may be split over several threads: this thread
// has LOBES of them (z, d: their 5 * LOBES outputs), and `row` gives a maximum
// (row.max) or the sum in lobe order (row.sum) over the row's threads.
template <int LOBES, class Row>
__device__ __forceinline__ float row_nll_grad(const float* z, float3 om, float wi, float* d, Row row) {
  float a_max = -INFINITY;
#pragma unroll
  for (int j = 0; j < LOBES; ++j) a_max = fmaxf(a_max, z[5 * j]);
  a_max = row.max(a_max);
  float lq[LOBES], pi[LOBES];
#pragma unroll
  for (int j = 0; j < LOBES; ++j) pi[j] = expf(z[5 * j] - a_max);
  const float esum = row.sum(pi);
  float lmax = -INFINITY;
  Lobe L[LOBES];
#pragma unroll
  for (int j = 0; j < LOBES; ++j) {
    pi[j] /= esum;
    const float s = fminf(fmaxf(z[5 * j + 1], TR_GUIDE_LOG_KAPPA_MIN), TR_GUIDE_LOG_KAPPA_MAX);
    const float kappa = expf(s);
    const float3 m = make_float3(z[5 * j + 2], z[5 * j + 3], z[5 * j + 4]);
    const float mlen = sqrtf(m.x * m.x + m.y * m.y + m.z * m.z) + 1e-6f;
    const float3 mu = make_float3(m.x / mlen, m.y / mlen, m.z / mlen);
    const float c = mu.x * om.x + mu.y * om.y + mu.z * om.z;
    L[j] = Lobe{pi[j], kappa, mlen, c, mu};
    lq[j] = logf(fmaxf(pi[j], 1e-30f)) + vmf_log_norm(kappa) + kappa * (c - 1.0f);
    lmax = fmaxf(lmax, lq[j]);
  }
  lmax = row.max(lmax);
  float qe[LOBES];
#pragma unroll
  for (int j = 0; j < LOBES; ++j) qe[j] = expf(lq[j] - lmax);
  const float logp = lmax + logf(row.sum(qe));
#pragma unroll
  for (int j = 0; j < LOBES; ++j) {
    const float q = expf(lq[j] - logp);  // responsibility
    const Lobe& b = L[j];
    d[5 * j] = -wi * (q - b.pi);
    const float s = z[5 * j + 1];
    const float e2 = expf(-2.0f * b.kappa);
    const float dlogk = 1.0f - 2.0f * b.kappa * e2 / fmaxf(-expm1f(-2.0f * b.kappa), 1e-30f) + b.kappa * (b.c - 1.0f);
    d[5 * j + 1] = (s > TR_GUIDE_LOG_KAPPA_MIN && s < TR_GUIDE_LOG_KAPPA_MAX) ? -wi * q * dlogk : 0.0f;
    const float f = -wi * q * b.kappa / b.mlen;
    d[5 * j + 2] = f * (om.x - b.c * b.mu.x);
    d[5 * j + 3] = f * (om.y - b.c * b.mu.y);
    d[5 * j + 4] = f * (om.z - b.c * b.mu.z);
  }
  return logp;
}

// A row whose eight lobes are all this thread's.
struct WholeRow {
  __device__ __forceinline__ float max(float v) const { return v; }
  __device__ __forceinline__ float sum(const float (&v)[kLobes]) const {
    float s = 0.0f;
#pragma unroll
    for (int j = 0; j < kLobes; ++j) s += v[j];
    return s;
  }
};

__global__ void k_loss(const float* __restrict__ out, const float* __restrict__ dir, const float* __restrict__ w,
                       int n, const float* __restrict__ wsum, float* __restrict__ dout, float* __restrict__ loss) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  float li = 0.0f;
  if (i < n) {
    const float3 om = make_float3(dir[3 * i], dir[3 * i + 1], dir[3 * i + 2]);
    const float wi = w[i] / fmaxf(*wsum, 1e-30f);
    li = -wi * row_nll_grad<kLobes>(out + (size_t)i * kOut, om, wi, dout + (size_t)i * kOut,
                                    WholeRow());
  }
  // block sum of the loss
  for (int o = 16; o > 0; o >>= 1) li += __shfl_xor_sync(0xffffffffu, li, o);
  if ((threadIdx.x & 31) == 0 && li != 0.0f) atomicAdd(loss, li);
}

__global__ void k_sum(const float* __restrict__ w, int n, float* __restrict__ out) {
  float s = 0.0f;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) s += w[i];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(out, s);
}

// ------------------------------------------------------------ fused training step
//
// One Adam step on a batch is two launches: k_train and k_update; a gradient
// for given output gradients is k_train<false> and k_grad_sum.
//
// k_train does a batch's forward pass, loss (or takes the outputs' gradient)
// and backward pass on the tensor cores. For a 128-row tile and layer l, with
// in_l the layer's input (x for l = 0, h_{l-1} otherwise):
//   Z_l    = in_l W_l^T          M = 128 rows, N = 64 or 48, K = 16 or 64
//   dW_l (+)= dZ_l^T in_l        M = 128 (64 outputs used), N = 16 or 64, K = 128 rows
//   db_l (+)= dZ_l^T 1           N = 16, a constant tile of ones (layer 0: a column of in_0)
//   dH     = dZ_l W_l            M = 128 rows, N = 64, K = 48 or 64
//   dZ_{l-1} = dH * (h_{l-1} > 0)
// A tile's in_l, its dZ and the weights lie in shared memory once, in the
// core-matrix layout; the products that need them transposed read the same
// bytes as MN-major operands (tc05.cuh). dW accumulates in tensor memory over
// the CTA's tiles and is written once per CTA as a partial sum (no atomics);
// k_update or k_grad_sum add the partials in a fixed order, so a step is
// deterministic.
//
// A tile is a chain of ten dependent MMAs and epilogues of a microsecond or
// two each, so a CTA (one per SM: the accumulators take 464 of the 512 TMEM
// columns) works on two tiles at once: two groups of four warps (a row per
// thread) run the epilogues and one thread of a ninth warp issues both
// groups' MMAs, each group's while the other's epilogue runs. The first
// version kept one tile per CTA with a __syncthreads per step and stored
// every activation and gradient a second time transposed (80 two-byte stores
// per row and layer): 93 us for 65,536 rows, 45 now; the gradient of 100,003
// rows 51 us instead of about 250 with stored activations. The MMA thread is
// busy 60% of that time: a product of 64 or 16 columns reads its 4 KB of A per
// 16 rows at shared-memory speed.
//
// Loss weighting: loss = sum_i -w_i log p_i / sum_i w_i. The rows carry
// s * w_i into the fp16 gradient chain, s = N / (64 W) for the weight sum W
// of N rows (the whole record set, or the batch), so the per-row values sit
// in fp16's normal range; k_update divides by s * sum_i w_i.

constexpr uint32_t kTOnes = 34048;                          // 128 x 16, column 0 one
constexpr uint32_t kTGroup = kTOnes + kTile * 16 * 2;       // per group: in_0, in_1..in_4, dZ
constexpr uint32_t kTileBytes = kTile * kHid * 2;           // 128 x 64 fp16
constexpr uint32_t kIn0Bytes = kTile * kInPad * 2;
constexpr uint32_t kGroupBytes = kIn0Bytes + 5 * kTileBytes;
__host__ __device__ constexpr uint32_t tin_off(int g, int l) {
  return kTGroup + (uint32_t)g * kGroupBytes + (l == 0 ? 0u : kIn0Bytes + (uint32_t)(l - 1) * kTileBytes);
}
__host__ __device__ constexpr uint32_t tdz_off(int g) { return tin_off(g, 5); }
// M = 128 reads 64 outputs beyond dZ's columns: the next row group, at the
// tile's end 1 KB past it (their products land in unused TMEM lanes)
constexpr uint32_t kTRed = kTGroup + 2 * kGroupBytes + 1024;  // per-warp sums
constexpr uint32_t kTXch = kTRed + 128;                     // per group: the two halves' partial values of a row
constexpr uint32_t kTMbar = kTXch + 2 * 2 * kTile * 4;      // ready[2], done[2], drain
constexpr uint32_t kTSlot = kTMbar + 5 * 8;
constexpr uint32_t kTSmemBytes = kTSlot + 16;
static_assert(kPackedBytes <= kTOnes && kTOnes % 128 == 0 && kTGroup % 128 == 0 && kTRed % 128 == 0, "k_train layout");
static_assert(kTSmemBytes <= 227 * 1024, "k_train shared memory");
// TMEM columns: a 64-column accumulator per group, then the weight gradients
__host__ __device__ constexpr uint32_t dw_col(int l) { return l == 0 ? 128u : 144u + 80u * (uint32_t)(l - 1); }
static_assert(dw_col(4) + 80 <= 512, "k_train tensor memory");
constexpr int kPartStride = kParams + 16;  // per-CTA partial: gradients, then weight sum and loss sum
constexpr int kWsumParts = 128;            // blocks of k_wsum
constexpr float kRowScale = 1.0f / 64.0f;
constexpr int kGroupThreads = 256;
constexpr int kTrainThreads = 2 * kGroupThreads + 32;  // two groups and the MMA warp

// The batch's row i: a record index drawn by a hash of (seed, i).
__device__ __forceinline__ unsigned int batch_record(unsigned long long seed, unsigned int i, unsigned int count) {
  unsigned long long h = seed * 0x9E3779B97F4A7C15ull + i * 0xBF58476D1CE4E5B9ull + 0x94D049BB133111EBull;
  h ^= h >> 31;
  h *= 0xD6E8FEB86659FD93ull;
  h ^= h >> 32;
  return (unsigned int)(h % count);
}

// Per-block sums of w[0..n) in a fixed order (kWsumParts blocks of 256).
__global__ void k_wsum(const float* __restrict__ w, unsigned int n, float* __restrict__ parts) {
  __shared__ float red[256];
  float s = 0.0f;
  for (unsigned int i = blockIdx.x * 256u + threadIdx.x; i < n; i += kWsumParts * 256u) s += w[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) parts[blockIdx.x] = red[0];
}

// The row scale s = nrows / (64 W) from k_wsum's partial sums, in a fixed
// order (every thread of a block of at least kWsumParts calls it).
__device__ __forceinline__ float row_scale(const float* __restrict__ parts, float nrows, int tid) {
  __shared__ float red[kWsumParts];
  if (tid < kWsumParts) red[tid] = parts[tid];
  __syncthreads();
  for (int o = kWsumParts / 2; o > 0; o >>= 1) {
    if (tid < o) red[tid] += red[tid + o];
    __syncthreads();
  }
  return nrows * kRowScale / fmaxf(red[0], 1e-30f);
}

// Two gradient values as fp16, clamped to the finite range with SAT (NaN to
// its lower end, as fminf(fmaxf()) does).
template <bool SAT>
__device__ __forceinline__ uint32_t h2_grad(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  if (SAT) h = __hmin2(__hmax2(h, __float2half2_rn(-65504.0f)), __float2half2_rn(65504.0f));
  return h2_bits(h);
}
// The halves of u where those of h are not zero (h: ReLU outputs).
__device__ __forceinline__ uint32_t h2_where(uint32_t u, uint32_t h) {
  return u & ((h & 0x7fffu ? 0xffffu : 0u) | (h & 0x7fff0000u ? 0xffff0000u : 0u));
}
// Meets the other threads of one group of k_train.
__device__ __forceinline__ void group_sync(int g) { tc05::bar_sync(g + 1, kGroupThreads); }

// A row whose lobes are split between two threads of a k_train group: the
// second half's sum goes on from the first half's, in lobe order.
struct HalfRow {
  float* x;  // two values per row of the group
  int g, half, r;
  __device__ __forceinline__ float max(float v) const {
    group_sync(g);
    x[kTile * half + r] = v;
    group_sync(g);
    return fmaxf(x[r], x[kTile + r]);
  }
  __device__ __forceinline__ float sum(const float (&v)[kLobes / 2]) const {
    float s = 0.0f;
    if (half == 0) {
#pragma unroll
      for (int j = 0; j < kLobes / 2; ++j) s += v[j];
    }
    group_sync(g);
    if (half == 0) x[r] = s;
    group_sync(g);
    if (half == 1) {
      s = x[r];
#pragma unroll
      for (int j = 0; j < kLobes / 2; ++j) s += v[j];
      x[kTile + r] = s;
    }
    group_sync(g);
    return x[kTile + r];
  }
};

// The MMAs of one step of a tile: forward layer L, and backward layer L.
template <int L>
__device__ __forceinline__ void train_forward_mma(uint32_t sm, uint32_t tmem, int g) {
  constexpr uint32_t sbo = (uint32_t)(layer_k(L) / 8) * 128u;
  const tc05::Desc in = tc05::desc_of(sm + tin_off(g, L), 128u, sbo), w = tc05::desc_of(sm + w_off(L), 128u, sbo);
#pragma unroll
  for (uint32_t kk = 0; kk < layer_k(L) / 16; ++kk)
    tc05::mma_f16(tmem + 64u * (uint32_t)g, tc05::step(in, kk * 256u), tc05::step(w, kk * 256u),
                  tc05::idesc_f16_f32(128, (uint32_t)layer_n(L)), kk > 0 ? 1u : 0u);
}
template <int L>
__device__ __forceinline__ void train_backward_mma(uint32_t sm, uint32_t tmem, int g, bool first) {
  constexpr uint32_t cols = L == 0 ? kInPad : kHid;
  const uint32_t dz = sm + tdz_off(g);
  const tc05::Desc a = tc05::desc_of(dz, 1024u, 128u), in = tc05::desc_of(sm + tin_off(g, L), cols * 16u, 128u),
                   one = tc05::desc_of(sm + kTOnes, 256u, 128u);
  if (L > 0) {  // first: the group's next epilogue waits for it
    const tc05::Desc ak = tc05::desc_of(dz, 128u, 1024u), w = tc05::desc_of(sm + w_off(L), 1024u, 128u);
#pragma unroll
    for (uint32_t kk = 0; kk < layer_n(L) / 16; ++kk)
      tc05::mma_f16(tmem + 64u * (uint32_t)g, tc05::step(ak, kk * 256u), tc05::step(w, kk * 2048u),
                    tc05::idesc_f16_f32(128, 64) | tc05::kTransB, kk > 0 ? 1u : 0u);
  }
#pragma unroll
  for (uint32_t kk = 0; kk < kTile / 16; ++kk) {
    const uint32_t acc = (!first || kk > 0) ? 1u : 0u;
    tc05::mma_f16(tmem + dw_col(L), tc05::step(a, kk * 2048u), tc05::step(in, kk * cols * 32u),
                  tc05::idesc_f16_f32(128, cols) | tc05::kTransA | tc05::kTransB, acc);
    if (L > 0)
      tc05::mma_f16(tmem + dw_col(L) + 64u, tc05::step(a, kk * 2048u), tc05::step(one, kk * 512u),
                    tc05::idesc_f16_f32(128, 16) | tc05::kTransA | tc05::kTransB, acc);
  }
}
// Step `step` of a tile: the forward layers 0 .. FWD - 1, then the backward
// layers 4 .. 0.
template <int FWD>
__device__ __forceinline__ void train_mma(int step, uint32_t sm, uint32_t tmem, int g, bool first) {
  switch (step) {
    case 0: train_forward_mma<0>(sm, tmem, g); return;
    case 1: train_forward_mma<1>(sm, tmem, g); return;
    case 2: train_forward_mma<2>(sm, tmem, g); return;
    case 3: train_forward_mma<3>(sm, tmem, g); return;
    case 4: if (FWD == 5) { train_forward_mma<4>(sm, tmem, g); return; }
  }
  switch (step - FWD) {
    case 0: train_backward_mma<4>(sm, tmem, g, first); return;
    case 1: train_backward_mma<3>(sm, tmem, g, first); return;
    case 2: train_backward_mma<2>(sm, tmem, g, first); return;
    case 3: train_backward_mma<1>(sm, tmem, g, first); return;
    default: train_backward_mma<0>(sm, tmem, g, first);
  }
}

// LOSS: rin: count x 7, rdir: count x 3, rw: count; gather != 0: row i of the
// batch is record batch_record(seed, i, count), else record i. Otherwise rin
// and rdir are the n inputs and the n x 40 gradients of the outputs.
// wparts: k_wsum's sums over the wrows weights. part: gridDim.x x kPartStride floats.
template <bool LOSS>
__global__ void __launch_bounds__(kTrainThreads, 1)
    k_train(const uint8_t* __restrict__ img, const float* __restrict__ rin, const float* __restrict__ rdir,
            const float* __restrict__ rw, unsigned int count, int n, unsigned long long seed, int gather,
            const float* __restrict__ wparts, float wrows, float* __restrict__ part, int* err) {
  extern __shared__ __align__(1024) uint8_t sm[];
  const int tid = threadIdx.x, warp = tid >> 5;
  const int grp = warp >> 3;        // 0, 1: epilogue groups; 2: the MMA warp
  const int half = (warp >> 2) & 1;  // which half of the row's columns is this thread's
  const int r = tid & (kTile - 1);   // this thread's tile row (TMEM lane)
  for (int i = tid; i < (int)(kPackedBytes / 16); i += kTrainThreads)
    reinterpret_cast<int4*>(sm)[i] = reinterpret_cast<const int4*>(img)[i];
  // the ones tile: column 0 (the other operands are written whole for every tile)
  if (tid < kTile) {
    uint8_t* one = sm + kTOnes;
    *reinterpret_cast<int4*>(one + tc05::core_off(tid, 0, 16)) = make_int4(0x3c00, 0, 0, 0);  // 1.0 in fp16
    *reinterpret_cast<int4*>(one + tc05::core_off(tid, 8, 16)) = make_int4(0, 0, 0, 0);
  }
  uint64_t* mbar = reinterpret_cast<uint64_t*>(sm + kTMbar);
  uint64_t *ready = mbar, *done = mbar + 2, *drain = mbar + 4;
  uint32_t* slot = reinterpret_cast<uint32_t*>(sm + kTSlot);
  int* failed = reinterpret_cast<int*>(sm + kTSlot + 4);
  if (tid == 0) {
    for (int g = 0; g < 2; ++g) {
      tc05::mbar_init(ready + g, kGroupThreads);
      tc05::mbar_init(done + g, 1);
    }
    tc05::mbar_init(drain, 1);
    *failed = 0;
  }
  if (warp == 16) {
    tc05::tmem_alloc(slot, 512);
    tc05::tmem_relinquish();
  }
  tc05::fence_before();
  tc05::fence_proxy_async();
  __syncthreads();
  tc05::fence_after();
  const uint32_t tmem = *slot;
  const uint32_t smem = tc05::smem_u32(sm);
  const int ntiles = (n + kTile - 1) / kTile, stride = 2 * (int)gridDim.x;
  constexpr int kFwd = LOSS ? 5 : 4;  // without a loss the outputs are not needed
  const float s = LOSS ? row_scale(wparts, wrows, tid) : 1.0f;
  float w_acc = 0.0f, l_acc = 0.0f;
  if (grp == 2) {
    if (tid == 2 * kGroupThreads) {
      uint32_t phase[2] = {0u, 0u};
      bool ok = true, first = true;
      for (int t = blockIdx.x; t < ntiles && ok; t += stride) {
        const int groups = t + (int)gridDim.x < ntiles ? 2 : 1;
        for (int step = 0; step < kFwd + 5 && ok; ++step)
          for (int g = 0; g < groups && ok; ++g) {
            ok = tc05::mbar_wait(ready + g, phase[g]);
            if (!ok) break;
            phase[g] ^= 1u;
            tc05::fence_after();
            train_mma<kFwd>(step, smem, tmem, g, first && g == 0);
            tc05::commit(done + g);
          }
        first = false;
      }
      if (!ok) *failed = 1;
    }
    __syncwarp();
  } else {
    const uint32_t acc = tmem + 64u * (uint32_t)grp + ((uint32_t)((warp & 3) * 32) << 16);
    const float* bias = reinterpret_cast<const float*>(sm + kBiasOff);
    uint8_t* dZ = sm + tdz_off(grp);
    uint32_t phase = 0;
    bool ok = true;
    for (int t = blockIdx.x + grp * (int)gridDim.x; t < ntiles && ok; t += stride) {
      const int i = t * kTile + r;
      const bool live = i < n;
      float x[kIn], om[3] = {0.0f, 0.0f, 0.0f}, w = 0.0f;
      const unsigned int j =
          live ? (LOSS && gather ? batch_record(seed, (unsigned int)i, count) : (unsigned int)i) : 0u;
#pragma unroll
      for (int k = 0; k < kIn; ++k) x[k] = live ? rin[(size_t)j * kIn + k] : 0.0f;
      if (LOSS && live) {
#pragma unroll
        for (int k = 0; k < 3; ++k) om[k] = rdir[(size_t)j * 3 + k];
        w = rw[j];
        // the weight sum, tile by tile in order: group 0 adds both groups' rows
        if (grp == 0 && half == 0) {
          w_acc += w;
          const long long i2 = (long long)i + (long long)gridDim.x * kTile;
          if (i2 < n) w_acc += rw[gather ? batch_record(seed, (unsigned int)i2, count) : (unsigned int)i2];
        }
      }
      {  // in_0: the inputs, a one for the bias gradient (its weights are zero), zeros; eight columns a thread
        __align__(16) __half h[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) h[k] = __float2half_rn(half ? 0.0f : (k < kIn ? x[k < kIn ? k : 0] : 1.0f));
        *reinterpret_cast<int4*>(sm + tin_off(grp, 0) + tc05::core_off(r, 8 * half, kInPad)) =
            *reinterpret_cast<const int4*>(h);
      }
      tc05::fence_proxy_async();
      tc05::mbar_arrive(ready + grp);
      const int c0 = 32 * half;
      // ---- forward
      for (int l = 0; l < 4; ++l) {
        ok = ok && tc05::mbar_wait(done + grp, phase);
        phase ^= 1u;
        tc05::fence_after();
        uint32_t c[32];
        tc05::tmem_ld32(acc + (uint32_t)c0, c);
        tc05::tmem_wait(c);
        hidden_epilogue(c, bias + 64 * l, sm + tin_off(grp, l + 1), r, c0);
        if (LOSS || l < 3) {
          tc05::fence_before();
          tc05::fence_proxy_async();
          tc05::mbar_arrive(ready + grp);
        }
      }
      {  // dZ_4: the loss and its gradient w.r.t. the outputs, or the given gradient (20 outputs a thread)
        constexpr int kMine = kOut / 2;
        float d[kMine];
#pragma unroll
        for (int k = 0; k < kMine; ++k) d[k] = 0.0f;
        if (LOSS) {
          ok = ok && tc05::mbar_wait(done + grp, phase);
          phase ^= 1u;
          tc05::fence_after();
          uint32_t c[32];
          tc05::tmem_ld32(acc + (uint32_t)(kMine * half), c);
          tc05::tmem_wait(c);
          float z[kMine];
#pragma unroll
          for (int k = 0; k < kMine; ++k) z[k] = __uint_as_float(c[k]) + bias[256 + kMine * half + k];
          float* xch = reinterpret_cast<float*>(sm + kTXch) + 2 * kTile * grp;
          const float logp = row_nll_grad<kLobes / 2>(z, make_float3(om[0], om[1], om[2]), w * s, d,
                                                      HalfRow{xch, grp, half, r});
          if (live && half == 0) l_acc -= w * logp;
        } else if (live) {
#pragma unroll
          for (int k = 0; k < kMine; ++k) d[k] = rdir[(size_t)i * kOut + kMine * half + k];
        }
        // columns 20 half .. + 19, in pairs (zeros from column 40 on stay)
#pragma unroll
        for (int k = 0; k < kMine; k += 2)
          *reinterpret_cast<uint32_t*>(dZ + tc05::core_off(r, kMine * half + k, kHid)) =
              live ? h2_grad<LOSS>(d[k], d[k + 1]) : 0u;
        if (half == 1) {
#pragma unroll
          for (int k = kOut; k < kHid; k += 8)
            *reinterpret_cast<int4*>(dZ + tc05::core_off(r, k, kHid)) = make_int4(0, 0, 0, 0);
        }
        tc05::fence_before();
        tc05::fence_proxy_async();
        tc05::mbar_arrive(ready + grp);
      }
      // ---- backward: dZ_{l-1} = dH * (h_{l-1} > 0); the step's MMAs have read dZ_l by now
      for (int l = kLayers - 1; l >= 0; --l) {
        ok = ok && tc05::mbar_wait(done + grp, phase);
        phase ^= 1u;
        if (l == 0) break;
        tc05::fence_after();
        uint32_t c[32];
        tc05::tmem_ld32(acc + (uint32_t)c0, c);
        tc05::tmem_wait(c);
        const uint8_t* in = sm + tin_off(grp, l);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t off = tc05::core_off(r, c0 + 8 * q, kHid);
          const int4 h = *reinterpret_cast<const int4*>(in + off);
          const int k = 8 * q;
          int4 u;
          u.x = (int)h2_where(h2_grad<LOSS>(__uint_as_float(c[k]), __uint_as_float(c[k + 1])), (uint32_t)h.x);
          u.y = (int)h2_where(h2_grad<LOSS>(__uint_as_float(c[k + 2]), __uint_as_float(c[k + 3])), (uint32_t)h.y);
          u.z = (int)h2_where(h2_grad<LOSS>(__uint_as_float(c[k + 4]), __uint_as_float(c[k + 5])), (uint32_t)h.z);
          u.w = (int)h2_where(h2_grad<LOSS>(__uint_as_float(c[k + 6]), __uint_as_float(c[k + 7])), (uint32_t)h.w);
          *reinterpret_cast<int4*>(dZ + off) = u;
        }
        tc05::fence_before();
        tc05::fence_proxy_async();
        tc05::mbar_arrive(ready + grp);
      }
      // A thread whose wait ran out has gone on without waiting, and arrived
      // like the others, to the end of the tile. The group leaves together: a
      // thread that left alone would be missing at the next tile's group_sync.
      ok = tc05::bar_all(grp + 1, kGroupThreads, ok);
    }
    if (!ok) *failed = 1;
  }
  tc05::fence_before();
  __syncthreads();
  tc05::fence_after();
  const bool ok = *failed == 0;
  if (!ok) {
    // whoever gave up did not see the MMAs issued so far end: wait for them
    // (bounded) before tensor memory is read and freed
    if (tid == 2 * kGroupThreads) {
      tc05::commit(drain);
      tc05::mbar_wait(drain, 0u);
    }
    if (tid == 0) atomicOr(err, 1);
    __syncthreads();
    tc05::fence_after();
  }
  // this CTA's partial: weight gradients from TMEM lanes 0..63 (one output
  // unit per lane), the layers split between the warps that read those lanes
  float* mine = part + (size_t)blockIdx.x * kPartStride;
  if (grp < 2 && (warp & 3) < 2) {
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    for (int l = 2 * grp + half; l < kLayers; l += 4) {
      const int kin = layer_kin(l), nout = layer_nout(l);
      for (int c0 = 0; c0 < (l == 0 ? kInPad : kHid + 16); c0 += 16) {
        float v[16];
        tc05::tmem_ld16(tmem + lanes + dw_col(l) + (uint32_t)c0, v);
        if (r >= nout) continue;
        if (l > 0 && c0 < kHid) {
          float4* dst = reinterpret_cast<float4*>(mine + param_w(l) + r * kHid + c0);
#pragma unroll
          for (int q = 0; q < 4; ++q)
            dst[q] = ok ? make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3])
                        : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        } else if (l > 0) {
          mine[param_b(l) + r] = ok ? v[0] : 0.0f;
        } else {
#pragma unroll
          for (int k = 0; k < kIn; ++k) mine[r * kin + k] = ok ? v[k] : 0.0f;
          mine[param_b(0) + r] = ok ? v[kIn] : 0.0f;
        }
      }
    }
  }
  for (int off = 16; off > 0; off >>= 1) {
    w_acc += __shfl_xor_sync(0xffffffffu, w_acc, off);
    l_acc += __shfl_xor_sync(0xffffffffu, l_acc, off);
  }
  float* red = reinterpret_cast<float*>(sm + kTRed);
  if ((tid & 31) == 0 && warp < 16) {
    red[2 * warp] = w_acc;
    red[2 * warp + 1] = l_acc;
  }
  tc05::fence_before();
  __syncthreads();
  if (tid == 0) {
    float ws = 0.0f, ls = 0.0f;
    for (int k = 0; k < 16; ++k) {
      ws += red[2 * k];
      ls += red[2 * k + 1];
    }
    mine[kParams] = ws;
    mine[kParams + 1] = ls;
  }
  if (warp == 16) tc05::tmem_dealloc(tmem, 512);
}

// Column i of the partials, summed over this thread's share of them (blocks of
// 32 columns x kSlices slices, ten loads in flight); the order is fixed.
constexpr int kSlices = 8;
__device__ __forceinline__ float part_slice(const float* __restrict__ part, int nparts, int i) {
  float g = 0.0f;
  for (int c0 = threadIdx.y; c0 < nparts; c0 += 10 * kSlices) {
    float v[10];
#pragma unroll
    for (int k = 0; k < 10; ++k)
      v[k] = c0 + k * kSlices < nparts ? part[(size_t)(c0 + k * kSlices) * kPartStride + i] : 0.0f;
#pragma unroll
    for (int k = 0; k < 10; ++k) g += v[k];
  }
  return g;
}

// The gradient itself: the sum of the partials.
__global__ void __launch_bounds__(32 * kSlices)
    k_grad_sum(const float* __restrict__ part, int nparts, float* __restrict__ grads) {
  __shared__ float red[kSlices][33];
  const int tx = threadIdx.x, ty = threadIdx.y, i = blockIdx.x * 32 + tx;
  red[ty][tx] = i < kParams ? part_slice(part, nparts, i) : 0.0f;
  __syncthreads();
  if (ty != 0 || i >= kParams) return;
  float g = 0.0f;
#pragma unroll
  for (int y = 0; y < kSlices; ++y) g += red[y][tx];
  grads[i] = g;
}

// Sums the nparts partials (32 parameters x kSlices partial slices per block),
// takes the Adam step, and writes the new weight (or bias) into the packed
// image. loss_out (optional) receives the batch loss.
__global__ void __launch_bounds__(32 * kSlices)
    k_update(const float* __restrict__ part, int nparts, const float* __restrict__ wparts, float wrows,
             float* __restrict__ p, float* __restrict__ m, float* __restrict__ v, float lr, float c1, float c2,
             uint8_t* __restrict__ img, float* __restrict__ loss_out) {
  __shared__ float red[kSlices][33];
  __shared__ float tot[kSlices][2];
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int i = blockIdx.x * 32 + tx;
  float g = i < kParams ? part_slice(part, nparts, i) : 0.0f, ws = 0.0f, ls = 0.0f;
  if (tx < 2) {
    const float t = part_slice(part, nparts, kParams + tx);
    tot[ty][tx] = t;
  }
  red[ty][tx] = g;
  const float scale = row_scale(wparts, wrows, 32 * ty + tx);  // (its barriers publish red and tot)
  if (ty != 0 || i >= kParams) return;
  g = 0.0f;
#pragma unroll
  for (int y = 0; y < kSlices; ++y) {
    g += red[y][tx];
    ws += tot[y][0];
    ls += tot[y][1];
  }
  if (loss_out && i == 0) *loss_out = ls / fmaxf(ws, 1e-30f);
  const float denom = scale * ws;
  g = denom > 1e-30f ? g / denom : 0.0f;
  const float mi = 0.9f * m[i] + 0.1f * g;
  const float vi = 0.999f * v[i] + 0.001f * g * g;
  m[i] = mi;
  v[i] = vi;
  const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + 1e-8f);
  p[i] = pi;
  int l = kLayers - 1;
  while (l > 0 && i < param_w(l)) --l;
  const int kin = layer_kin(l), e = i - param_w(l);
  if (e < layer_nout(l) * kin) {
    const int o = e / kin, k = e % kin;
    *reinterpret_cast<__half*>(img + w_off(l) + tc05::core_off(o, k, layer_k(l))) = __float2half_rn(pi);
  } else {
    const int o = e - layer_nout(l) * kin;
    reinterpret_cast<float*>(img + kBiasOff)[l < kLayers - 1 ? l * 64 + o : 256 + o] = pi;
  }
}

}  // namespace mlp

// ------------------------------------------------------------------ host

namespace {

uint32_t pcg_next(uint64_t& s) {
  const uint64_t old = s;
  s = old * 6364136223846793005ull + 1442695040888963407ull;
  const uint32_t xs = (uint32_t)(((old >> 18u) ^ old) >> 27u);
  const uint32_t rot = (uint32_t)(old >> 59u);
  return (xs >> rot) | (xs << ((32u - rot) & 31u));
}

}  // namespace

tr_status guide_reserve(tr_ctx* ctx) {
  if (!ctx->guide) ctx->guide = new GuideModel();
  GuideModel* g = ctx->guide;
  if (g->params.p) return TR_OK;
  cudaError_t e = cudaSuccess;
  for (auto pr : {std::make_pair(&g->params, (size_t)mlp::kParams * 4), std::make_pair(&g->img, (size_t)mlp::kPackedBytes),
                  
                  std::make_pair(&g->adam_m, (size_t)mlp::kParams * 4),
                  std::make_pair(&g->adam_v, (size_t)mlp::kParams * 4),
                  std::make_pair(&g->scal, (size_t)(16 + mlp::kWsumParts) * 4)})
    if ((e = pr.first->reserve(pr.second)) != cudaSuccess) return cuda_fail(ctx, e, "guide model allocation");
  if (!g->attr_set) {
    if ((e = cudaFuncSetAttribute(mlp::k_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, mlp::kSmemBytes)) !=
            cudaSuccess ||
        (e = cudaFuncSetAttribute(mlp::k_train<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  mlp::kTSmemBytes)) != cudaSuccess ||
        (e = cudaFuncSetAttribute(mlp::k_train<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  mlp::kTSmemBytes)) != cudaSuccess)
      return cuda_fail(ctx, e, "guide kernels' shared memory");
    g->attr_set = true;
  }
  return TR_OK;
}

// Resets the Adam state (new parameters start a new optimisation).
static tr_status guide_reset_adam(tr_ctx* ctx) {
  GuideModel* g = ctx->guide;
  TR_CUDA(ctx, cudaMemsetAsync(g->adam_m.p, 0, mlp::kParams * 4, ctx->stream));
  TR_CUDA(ctx, cudaMemsetAsync(g->adam_v.p, 0, mlp::kParams * 4, ctx->stream));
  g->step = 0;
  return TR_OK;
}

tr_status guide_pack(tr_ctx* ctx) {
  GuideModel* g = ctx->guide;
  mlp::k_pack<<<(mlp::kPackThreads + 255) / 256, 256, 0, ctx->stream>>>(g->params.as<float>(), g->img.as<uint8_t>());
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? TR_OK : cuda_fail(ctx, e, "guide weight packing");
}

// Forward: up to four CTAs per SM (50 KB of shared memory and 64 TMEM
// columns each), so that one CTA's MMAs overlap another's epilogue.
// Training and backward: one per SM (each holds 512 TMEM columns, the whole SM's).
static int guide_grid(tr_ctx* ctx, int n, int per_sm) {
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  const int tiles = (n + mlp::kTile - 1) / mlp::kTile;
  return std::max(1, std::min(tiles, sms * per_sm));
}

tr_status guide_forward(tr_ctx* ctx, const float* d_in, int n, float* d_out) {
  mlp::k_forward<<<guide_grid(ctx, n, 4), 128, mlp::kSmemBytes, ctx->stream>>>(
      ctx->guide->img.as<uint8_t>(), d_in, n, d_out, ctx->d_err.as<int>() + 2, nullptr, 0);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? TR_OK : cuda_fail(ctx, e, "k_forward");
}

tr_status guide_forward_rows_on_device(tr_ctx* ctx, const float* d_in, const unsigned int* d_n, float* d_out,
                                       cudaStream_t st) {
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  mlp::k_forward<<<std::max(sms, 1) * 4, 128, mlp::kSmemBytes, st>>>(
      ctx->guide->img.as<uint8_t>(), d_in, 0, d_out, ctx->d_err.as<int>() + 2, d_n, 1);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? TR_OK : cuda_fail(ctx, e, "k_forward");
}

// The partial sums (scal[16..]) of the weights w[0..n) of a training pass or
// step, from which its kernels take the row scale (row_scale).
static tr_status guide_scale(tr_ctx* ctx, const float* w, unsigned int n) {
  float* scal = ctx->guide->scal.as<float>();
  mlp::k_wsum<<<mlp::kWsumParts, 256, 0, ctx->stream>>>(w, n, scal + 16);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? TR_OK : cuda_fail(ctx, e, "guide weight sum");
}

// One Adam step on n rows (gather: drawn from `count` records by seed), two
// launches: k_train, k_update. The batch loss lands in *d_loss (device).
static tr_status guide_fused_step(tr_ctx* ctx, const float* in, const float* dir, const float* w, unsigned int count,
                                  int n, int gather, unsigned long long seed, float lr, float* d_loss) {
  GuideModel* g = ctx->guide;
  const int grid = guide_grid(ctx, n, 1);
  cudaError_t e;
  if ((e = g->part.reserve((size_t)grid * mlp::kPartStride * 4)) != cudaSuccess)
    return cuda_fail(ctx, e, "guide gradient partials");
  const float* wparts = g->scal.as<float>() + 16;  // guide_scale's sums over the `count` records
  mlp::k_train<true><<<grid, mlp::kTrainThreads, mlp::kTSmemBytes, ctx->stream>>>(
      g->img.as<uint8_t>(), in, dir, w, count, n, seed, gather, wparts, (float)count, g->part.as<float>(),
      ctx->d_err.as<int>() + 2);
  ++g->step;
  const float c1 = 1.0f - std::pow(0.9f, (float)g->step), c2 = 1.0f - std::pow(0.999f, (float)g->step);
  mlp::k_update<<<(mlp::kParams + 31) / 32, dim3(32, mlp::kSlices), 0, ctx->stream>>>(
      g->part.as<float>(), grid, wparts, (float)count, g->params.as<float>(), g->adam_m.as<float>(), g->adam_v.as<float>(), lr, c1,
      c2, g->img.as<uint8_t>(), d_loss);
  e = cudaGetLastError();
  return e == cudaSuccess ? TR_OK : cuda_fail(ctx, e, "guide training step");
}

tr_status guide_train_on(tr_ctx* ctx, const float* rec_in, const float* rec_dir, const float* rec_w, unsigned int count,
                         int steps, unsigned int batch, float lr, unsigned long long seed, float* mean_loss) {
  GuideModel* g = ctx->guide;
  cudaError_t e;
  if ((e = g->losses.reserve((size_t)std::max(steps, 1) * 4)) != cudaSuccess)
    return cuda_fail(ctx, e, "training losses");
  tr_status st = guide_scale(ctx, rec_w, count);
  if (st != TR_OK) return st;
  for (int s = 0; s < steps; ++s) {
    st = guide_fused_step(ctx, rec_in, rec_dir, rec_w, count, (int)batch, 1, seed * 1000003ull + (unsigned long long)s,
                          lr, g->losses.as<float>() + s);
    if (st != TR_OK) return st;
  }
  std::vector<float> l((size_t)steps);
  if (steps)
    TR_CUDA(ctx, cudaMemcpyAsync(l.data(), g->losses.p, (size_t)steps * 4, cudaMemcpyDeviceToHost, ctx->stream));
  TR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  double sum = 0.0;
  for (float v : l) sum += v;
  if (mean_loss) *mean_loss = steps ? (float)(sum / steps) : 0.0f;
  return TR_OK;
}

static tr_status guide_workspace(tr_ctx* ctx, int n) {
  GuideModel* g = ctx->guide;
  cudaError_t e;
  if ((e = g->out.reserve((size_t)n * mlp::kOut * 4)) != cudaSuccess ||
      (e = g->dout.reserve((size_t)n * mlp::kOut * 4)) != cudaSuccess)
    return cuda_fail(ctx, e, "guide training workspace");
  return TR_OK;
}

tr_status guide_backward(tr_ctx* ctx, const float* d_in, const float* d_dout, int n, float* d_grads) {
  GuideModel* g = ctx->guide;
  const int grid = guide_grid(ctx, n, 1);
  cudaError_t e = g->part.reserve((size_t)grid * mlp::kPartStride * 4);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "guide gradient partials");
  mlp::k_train<false><<<grid, mlp::kTrainThreads, mlp::kTSmemBytes, ctx->stream>>>(
      g->img.as<uint8_t>(), d_in, d_dout, nullptr, 0u, n, 0ull, 0, nullptr, 0.0f, g->part.as<float>(),
      ctx->d_err.as<int>() + 2);
  mlp::k_grad_sum<<<(mlp::kParams + 31) / 32, dim3(32, mlp::kSlices), 0, ctx->stream>>>(g->part.as<float>(), grid, d_grads);
  e = cudaGetLastError();
  return e == cudaSuccess ? TR_OK : cuda_fail(ctx, e, "guide backward pass");
}

// Loss and its gradient w.r.t. the network outputs (g->dout) for a batch;
// the loss lands in scal[1].
static tr_status guide_loss(tr_ctx* ctx, const float* d_in, const float* d_dir, const float* d_w, int n) {
  tr_status s = guide_workspace(ctx, n);
  if (s != TR_OK) return s;
  GuideModel* g = ctx->guide;
  s = guide_forward(ctx, d_in, n, g->out.as<float>());
  if (s != TR_OK) return s;
  float* scal = g->scal.as<float>();
  TR_CUDA(ctx, cudaMemsetAsync(scal, 0, 8, ctx->stream));
  mlp::k_sum<<<64, 256, 0, ctx->stream>>>(d_w, n, scal);
  mlp::k_loss<<<(n + 255) / 256, 256, 0, ctx->stream>>>(g->out.as<float>(), d_dir, d_w, n, scal,
                                                         g->dout.as<float>(), scal + 1);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? TR_OK : cuda_fail(ctx, e, "k_loss");
}

tr_status guide_train_step(tr_ctx* ctx, const float* d_in, const float* d_dir, const float* d_w, int n, float lr) {
  tr_status s = guide_scale(ctx, d_w, (unsigned int)n);
  if (s != TR_OK) return s;
  return guide_fused_step(ctx, d_in, d_dir, d_w, (unsigned int)n, n, 0, 0ull, lr, ctx->guide->scal.as<float>() + 1);
}

// Synchronises and turns a timed-out tensor-core wait into an error.
static tr_status guide_check(tr_ctx* ctx) {
  int e = 0;
  TR_CUDA(ctx, cudaMemcpyAsync(&e, ctx->d_err.as<int>() + 2, 4, cudaMemcpyDeviceToHost, ctx->stream));
  TR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (e) {
    cudaMemsetAsync(ctx->d_err.as<int>() + 2, 0, 4, ctx->stream);
    return set_err(ctx, TR_ERR_TIMEOUT, "tensor-core MMA wait timed out");
  }
  return TR_OK;
}

void release_guide(tr_ctx* ctx) {
  if (!ctx->guide) return;
  GuideModel* g = ctx->guide;
  for (DevBuf* b : {&g->params, &g->img, &g->adam_m, &g->adam_v, &g->out, &g->dout,
                    &g->scal, &g->part, &g->losses})
    b->release();
  delete g;
  ctx->guide = nullptr;
}

}  // namespace trg

using namespace trg;

extern "C" {

tr_status tr_guide_init(tr_ctx* ctx, uint64_t seed) {
  if (!ctx) return TR_ERR_ARG;
  TR_DEVICE_SCOPE(ctx);
  tr_status s = guide_reserve(ctx);
  if (s != TR_OK) return s;
  // uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) for weights and biases
  std::vector<float> p(mlp::kParams);
  uint64_t st = seed * 2 + 1;
  for (int l = 0; l < mlp::kLayers; ++l) {
    const float bound = 1.0f / std::sqrt((float)mlp::layer_kin(l));
    const int nw = mlp::layer_nout(l) * mlp::layer_kin(l);
    for (int i = 0; i < nw + mlp::layer_nout(l); ++i) {
      const float u = (float)(pcg_next(st) >> 8) * (1.0f / 16777216.0f);
      p[mlp::param_w(l) + i] = (2.0f * u - 1.0f) * bound;
    }
  }
  return tr_guide_set_params(ctx, p.data(), p.size());
}

tr_status tr_guide_set_params(tr_ctx* ctx, const float* params, size_t n) {
  if (!ctx || !params || n != (size_t)mlp::kParams) return TR_ERR_ARG;
  TR_DEVICE_SCOPE(ctx);
  tr_status s = guide_reserve(ctx);
  if (s != TR_OK) return s;
  TR_CUDA(ctx, cudaMemcpyAsync(ctx->guide->params.p, params, n * 4, cudaMemcpyHostToDevice, ctx->stream));
  s = guide_reset_adam(ctx);
  if (s != TR_OK) return s;
  s = guide_pack(ctx);
  if (s != TR_OK) return s;
  TR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return TR_OK;
}

tr_status tr_guide_get_params(tr_ctx* ctx, float* params, size_t n) {
  if (!ctx || !params || n != (size_t)mlp::kParams) return TR_ERR_ARG;
  if (!ctx->guide || !ctx->guide->params.p) return set_err(ctx, TR_ERR_STATE, "guide model not initialised");
  TR_DEVICE_SCOPE(ctx);
  TR_CUDA(ctx, cudaMemcpyAsync(params, ctx->guide->params.p, n * 4, cudaMemcpyDeviceToHost, ctx->stream));
  TR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return TR_OK;
}

tr_status tr_guide_forward_dev(tr_ctx* ctx, const float* d_in, size_t n, float* d_out) {
  if (!ctx || (n && (!d_in || !d_out))) return TR_ERR_ARG;
  if (!ctx->guide || !ctx->guide->params.p) return set_err(ctx, TR_ERR_STATE, "guide model not initialised");
  if (n > (1u << 30)) return set_err(ctx, TR_ERR_ARG, "too many rows");
  if (n == 0) return TR_OK;
  TR_DEVICE_SCOPE(ctx);
  tr_status s = guide_forward(ctx, d_in, (int)n, d_out);
  return s != TR_OK ? s : guide_check(ctx);
}

tr_status tr_guide_backward_dev(tr_ctx* ctx, const float* d_in, const float* d_dout, size_t n, float* d_grads) {
  if (!ctx || !d_grads || (n && (!d_in || !d_dout))) return TR_ERR_ARG;
  if (!ctx->guide || !ctx->guide->params.p) return set_err(ctx, TR_ERR_STATE, "guide model not initialised");
  if (n > (1u << 26)) return set_err(ctx, TR_ERR_ARG, "too many rows");
  TR_DEVICE_SCOPE(ctx);
  if (n == 0) {
    TR_CUDA(ctx, cudaMemsetAsync(d_grads, 0, mlp::kParams * 4, ctx->stream));
    return guide_check(ctx);
  }
  tr_status s = guide_backward(ctx, d_in, d_dout, (int)n, d_grads);
  return s != TR_OK ? s : guide_check(ctx);
}

tr_status tr_guide_loss_dev(tr_ctx* ctx, const float* d_in, const float* d_dir, const float* d_weight, size_t n,
                            float* d_dout, float* loss) {
  if (!ctx || !loss || !d_dout || n == 0 || !d_in || !d_dir || !d_weight) return TR_ERR_ARG;
  if (!ctx->guide || !ctx->guide->params.p) return set_err(ctx, TR_ERR_STATE, "guide model not initialised");
  if (n > (1u << 26)) return set_err(ctx, TR_ERR_ARG, "too many rows");
  TR_DEVICE_SCOPE(ctx);
  tr_status s = guide_loss(ctx, d_in, d_dir, d_weight, (int)n);
  if (s != TR_OK) return s;
  TR_CUDA(ctx, cudaMemcpyAsync(d_dout, ctx->guide->dout.p, n * mlp::kOut * 4, cudaMemcpyDeviceToDevice, ctx->stream));
  TR_CUDA(ctx, cudaMemcpyAsync(loss, ctx->guide->scal.as<float>() + 1, 4, cudaMemcpyDeviceToHost, ctx->stream));
  return guide_check(ctx);
}

tr_status tr_guide_train_step_dev(tr_ctx* ctx, const float* d_in, const float* d_dir, const float* d_weight,
                                  size_t n, float lr, float* loss) {
  if (!ctx || n == 0 || !d_in || !d_dir || !d_weight || !(lr > 0.0f)) return TR_ERR_ARG;
  if (!ctx->guide || !ctx->guide->params.p) return set_err(ctx, TR_ERR_STATE, "guide model not initialised");
  if (n > (1u << 26)) return set_err(ctx, TR_ERR_ARG, "too many rows");
  TR_DEVICE_SCOPE(ctx);
  tr_status s = guide_train_step(ctx, d_in, d_dir, d_weight, (int)n, lr);
  if (s != TR_OK) return s;
  float l = 0.0f;
  TR_CUDA(ctx, cudaMemcpyAsync(&l, ctx->guide->scal.as<float>() + 1, 4, cudaMemcpyDeviceToHost, ctx->stream));
  s = guide_check(ctx);
  if (loss) *loss = l;
  return s;
}

}  // extern "C"

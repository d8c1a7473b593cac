// phmm_mlp_train.cu -- training kernels of the band MLP (80-128-128-2, ReLU).
//
// Master weights are FP32; every step rounds them to BF16 (the precision the
// tensor-core inference kernel uses) and runs forward and backward in FP32 on
// those rounded values, so the gradient is that of the deployed network
// (straight-through rounding).  The products with 80 or 128 on every side run
// on the tensor cores (tcgen05.mma kind::f16: BF16 operands, FP32 accumulation
// in tensor memory) -- the two hidden layers' forward products (inputs, weights
// and hidden activations are BF16 values already), the hidden layers' weight
// gradients and the back-propagated hidden gradient (the FP32 gradient operands
// rounded to BF16, as mixed-precision training does); the products with the
// 2-wide output layer stay FP32.  The loss is an asymmetric squared error on
// the band's lower and upper edge (diagonals relative to the seed diagonal):
//   L = mean( w_lo (o_lo - t_lo)^2 + w_hi (o_hi - t_hi)^2 ),
//   w_lo = alpha if o_lo > t_lo (band too narrow below) else 1,
//   w_hi = alpha if o_hi < t_hi (band too narrow above) else 1,
// so under-covering the posterior spread costs alpha times more than
// over-covering it.  Optimiser: Adam.
//
// Two launches a step.  k_mlp_rows: a block per 128 rows of the minibatch runs
// the whole forward and backward pass of its rows with every operand in shared
// memory, and leaves the rows' hidden gradients and its partial products of the
// hidden weight gradients (K = its 128 rows).  k_mlp_update: sums the partial
// products block by block and the bias and output-layer gradients row by row,
// in a fixed order, so the weights are the same in every run, and applies Adam.
// (The reported loss is summed with atomics: its last bits may differ.)  The step
// is a chain of five small products and a 1,024-term sum, so latency is what
// counts: 1,024 rows take 47 us, where a launch per product, activation
// and sum (22 of them, operands through global memory) took 273.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "phmm_band.h"
#include "phmm_kernels.h"
#include "phmm_mlp.h"
#include "phmm_tc.cuh"

namespace bvphmm {
namespace {

using namespace tc;

constexpr int kRows = 128;          // minibatch rows per block (the MMA's M, and K of the weight gradients)
constexpr int kRowThreads = 256;    // warp w: rows 32 (w & 3) .., columns 64 (w >> 2) ..
constexpr int kW1 = kHid * kFeat, kW2 = kHid * kHid;
constexpr int kOffW1 = 0, kOffB1 = kW1, kOffW2 = kOffB1 + kHid, kOffB2 = kOffW2 + kW2, kOffW3 = kOffB2 + kHid,
              kOffB3 = kOffW3 + kOut * kHid;

struct RowsSmem {
  __nv_bfloat16 xa[kRows * kFeat];  // inputs [row][feature]
  __nv_bfloat16 w1[kHid * kFeat];   // W1 [out][feature]; after layer 1 the inputs transposed, [feature][row]
  __nv_bfloat16 w2[kHid * kHid];    // W2 [out][in]
  __nv_bfloat16 w2t[kHid * kHid];   // W2 transposed, [in][out]
  __nv_bfloat16 ra[kRows * kHid];   // H1, later dZ2, [row][unit]
  __nv_bfloat16 h1t[kHid * kRows];  // H1 transposed, [unit][row]
  __nv_bfloat16 dzt[kHid * kRows];  // dZ2, later dZ1, transposed, [unit][row]
  float b1[kHid], b2[kHid], w3[kOut][kHid], b3[kOut];
  float err[kRows][kOut], dout[kRows][kOut];
  uint64_t mbar;
  uint32_t tmem_base;
  int fail;
};

// eight consecutive values rounded to BF16 (nearest even)
__device__ __forceinline__ uint4 pack8(const float* v) {
  uint32_t w[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * t], v[2 * t + 1]);
    w[t] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
struct Eight {
  float v[8];
};
__device__ __forceinline__ Eight load8(const float* p) {  // 16-byte aligned
  const float4 a = __ldcg(reinterpret_cast<const float4*>(p)), b = __ldcg(reinterpret_cast<const float4*>(p) + 1);
  return Eight{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
}
__device__ __forceinline__ float as_bf16(float v) { return __bfloat162float(__float2bfloat16(v)); }

// D[tmem] = A . B^T over K, both operands in the canonical K-major layout.
template <int K, int N>
__device__ __forceinline__ void product(uint32_t d, const __nv_bfloat16* a, const __nv_bfloat16* b) {
  const unsigned char* pa = reinterpret_cast<const unsigned char*>(a);
  const unsigned char* pb = reinterpret_cast<const unsigned char*>(b);
#pragma unroll
  for (int k = 0; k < K / 16; ++k)
    mma_f16(d, mat_desc(pa + k * 2 * kLbo, kLbo, sbo_for(K)), mat_desc(pb + k * 2 * kLbo, kLbo, sbo_for(K)),
            instr_desc(kRows, N), k > 0);
}

__device__ __forceinline__ unsigned char* at(__nv_bfloat16* m, int row, int col, int k) {
  return reinterpret_cast<unsigned char*>(m) + core_offset(row, col, k);
}

// Forward (and backward) pass of rows [128 blockIdx.x, ..) of the minibatch of
// n rows.  The inputs are rows idx[r] of feat (training) or FP32 rows of X,
// rounded here (evaluation).
__global__ void __launch_bounds__(kRowThreads, 1)
    k_mlp_rows(MlpTrainBuffers b, const __nv_bfloat16* __restrict__ feat, const float* __restrict__ targets,
               const int32_t* __restrict__ idx, int n, float alpha, float inv_n, int backward) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  RowsSmem& s = *reinterpret_cast<RowsSmem*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, half = warp >> 2;
  const int row = (warp & 3) * 32 + (tid & 31);     // this thread's row (and TMEM lane)
  const int c0 = 64 * half;                         // and columns c0 .. c0 + 63
  const long long gr = (long long)blockIdx.x * kRows + row;
  const bool valid = gr < n;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmem_base)),
                 "r"(256)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&s.mbar)) : "memory");
    s.fail = 0;
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  // inputs: a row's ten 16-byte pieces, five a thread
  const long long src = !valid ? 0 : idx ? idx[gr] : gr;
#pragma unroll
  for (int q = 0; q < kFeat / 16; ++q) {
    const int c = 8 * (2 * q + half);
    uint4 v = make_uint4(0, 0, 0, 0);
    if (valid) {
      if (feat) {
        v = *reinterpret_cast<const uint4*>(feat + src * kFeat + c);
      } else {
        v = pack8(load8(b.X + src * kFeat + c).v);
      }
    }
    *reinterpret_cast<uint4*>(at(s.xa, row, c, kFeat)) = v;
  }
  // weights, rounded: 16-byte loads, several in flight a thread
  const float* gw1 = b.w + kOffW1;
  const float* gw2 = b.w + kOffW2;
#pragma unroll
  for (int x = tid; x < kW1 / 8; x += kRowThreads) {
    const int r = x / (kFeat / 8), c = 8 * (x % (kFeat / 8));
    *reinterpret_cast<uint4*>(at(s.w1, r, c, kFeat)) = pack8(load8(gw1 + r * kFeat + c).v);
  }
#pragma unroll 4
  for (int x = tid; x < kW2 / 8; x += kRowThreads) {
    const int r = x / (kHid / 8), c = 8 * (x % (kHid / 8));
    *reinterpret_cast<uint4*>(at(s.w2, r, c, kHid)) = pack8(load8(gw2 + r * kHid + c).v);
  }
  if (backward) {
#pragma unroll 4
    for (int x = tid; x < kW2 / 8; x += kRowThreads) {  // column r of W2, outputs c .. c + 7
      const int r = x % kHid, c = 8 * (x / kHid);
      float f[8];
#pragma unroll
      for (int t = 0; t < 8; ++t) f[t] = __ldcg(gw2 + (c + t) * kHid + r);
      *reinterpret_cast<uint4*>(at(s.w2t, r, c, kHid)) = pack8(f);
    }
  }
  if (tid < kHid) {
    s.b1[tid] = b.w[kOffB1 + tid];
    s.b2[tid] = b.w[kOffB2 + tid];
  }
  s.w3[half][tid & (kHid - 1)] = as_bf16(b.w[kOffW3 + tid]);
  if (tid < kOut) s.b3[tid] = b.w[kOffB3 + tid];
  unsigned phase = 0;
  // every thread's shared-memory writes towards the tensor cores, then one thread issues
  auto issue = [&](auto&& mmas) {
    fence_async_smem();
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    if (tid == 0) {
      mmas();
      mma_commit(&s.mbar);
    }
  };
  auto wait = [&]() -> bool {
    if (!mbar_wait_parity(&s.mbar, phase)) {
      s.fail = 1;
      mbar_wait_parity(&s.mbar, phase);  // again bounded: MMAs still reading shared memory
    }
    phase ^= 1u;
    fence_after_sync();
    __syncthreads();
    return !*reinterpret_cast<volatile int*>(&s.fail);
  };
  issue([&] { product<kFeat, kHid>(s.tmem_base, s.xa, s.w1); });
  const uint32_t d0 = s.tmem_base + ((uint32_t)((warp & 3) * 32) << 16), d1 = d0 + 128;
  bool ok = wait();
  uint32_t on1[2], on2[2];  // ReLU masks of this thread's columns
  if (ok) {
#pragma unroll 1
    for (int q = 0; q < 2; ++q) {
      float v[32];
      tmem_ld32(d0 + (uint32_t)(c0 + 32 * q), v);
      uint32_t m = 0;
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const float z = v[j] + s.b1[c0 + 32 * q + j];
        m |= (uint32_t)(z > 0.f) << j;
        v[j] = fmaxf(z, 0.f);
      }
      on1[q] = m;
#pragma unroll
      for (int j = 0; j < 32; j += 8) *reinterpret_cast<uint4*>(at(s.ra, row, c0 + 32 * q + j, kHid)) = pack8(v + j);
      if (backward) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          *reinterpret_cast<__nv_bfloat16*>(at(s.h1t, c0 + 32 * q + j, row, kRows)) = __float2bfloat16(v[j]);
      }
    }
    issue([&] { product<kHid, kHid>(s.tmem_base + 128, s.ra, s.w2); });
    if (backward) {  // the inputs transposed, where W1 was
#pragma unroll
      for (int q = 0; q < kFeat / 16; ++q) {
        const int c = 8 * (2 * q + half);
        const uint4 v = *reinterpret_cast<const uint4*>(at(s.xa, row, c, kFeat));
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int t = 0; t < 8; ++t)
          *reinterpret_cast<uint16_t*>(at(s.w1, c + t, row, kRows)) = (uint16_t)(w[t >> 1] >> (16 * (t & 1)));
      }
    }
    ok = wait();
  }
  if (ok) {
    // output layer: this thread sums output `half` of its row, hidden units in order
    float acc = 0.f;
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
      float v[32];
      tmem_ld32(d1 + (uint32_t)(32 * q), v);
      uint32_t m = 0;
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const float z = v[j] + s.b2[32 * q + j];
        m |= (uint32_t)(z > 0.f) << j;
        v[j] = as_bf16(fmaxf(z, 0.f));
        acc = fmaf(v[j], s.w3[half][32 * q + j], acc);
      }
      if ((q >> 1) == half) {
        if (q & 1) on2[1] = m;
        else on2[0] = m;
        if (backward && valid) {
#pragma unroll
          for (int j = 0; j < 32; j += 4)
            *reinterpret_cast<float4*>(b.H2 + gr * kHid + 32 * q + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        }
      }
    }
    const float o = acc + s.b3[half];
    const float t = valid ? (feat ? targets[2 * src + half] : b.T[2 * src + half]) : 0.f;
    const float e = o - t;
    const float w = (half == 0 ? e > 0.f : e < 0.f) ? alpha : 1.f;
    const float d = valid ? 2.f * w * e * inv_n : 0.f;
    s.err[row][half] = valid ? w * e * e : 0.f;
    s.dout[row][half] = d;
    if (valid) {
      b.O[2 * gr + half] = o;
      b.dO[2 * gr + half] = d;
    }
    __syncthreads();
    if (half == 0) {
      float l = s.err[row][0] + s.err[row][1];
      for (int k = 16; k > 0; k >>= 1) l += __shfl_xor_sync(0xffffffffu, l, k);
      if ((tid & 31) == 0) atomicAdd(b.loss, l * inv_n);
    }
  }
  if (ok && backward) {
    // dZ2 = (dO . W3) where Z2 > 0
    const float g0 = s.dout[row][0], g1 = s.dout[row][1];
#pragma unroll 1
    for (int q = 0; q < 2; ++q) {
      float v[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const int c = c0 + 32 * q + j;
        const float d = fmaf(g1, s.w3[1][c], fmaf(g0, s.w3[0][c], 0.f));
        v[j] = (on2[q] >> j & 1u) ? d : 0.f;
        *reinterpret_cast<__nv_bfloat16*>(at(s.dzt, c, row, kRows)) = __float2bfloat16(v[j]);
      }
#pragma unroll
      for (int j = 0; j < 32; j += 8) *reinterpret_cast<uint4*>(at(s.ra, row, c0 + 32 * q + j, kHid)) = pack8(v + j);
      if (valid) {
#pragma unroll
        for (int j = 0; j < 32; j += 4)
          *reinterpret_cast<float4*>(b.dH + gr * kHid + c0 + 32 * q + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
      }
    }
    issue([&] {
      product<kHid, kHid>(s.tmem_base, s.ra, s.w2t);         // dH1 = dZ2 W2
      product<kRows, kHid>(s.tmem_base + 128, s.dzt, s.h1t);  // this block's part of dW2 = dZ2^T H1
    });
    ok = wait();
    if (ok) {
      float* part2 = b.part2 + (size_t)blockIdx.x * kW2 + row * kHid + c0;
#pragma unroll 1
      for (int q = 0; q < 2; ++q) {
        float v[32];
        tmem_ld32(d1 + (uint32_t)(c0 + 32 * q), v);
#pragma unroll
        for (int j = 0; j < 32; j += 4)
          *reinterpret_cast<float4*>(part2 + 32 * q + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        tmem_ld32(d0 + (uint32_t)(c0 + 32 * q), v);
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          v[j] = (on1[q] >> j & 1u) ? v[j] : 0.f;  // dZ1
          *reinterpret_cast<__nv_bfloat16*>(at(s.dzt, c0 + 32 * q + j, row, kRows)) = __float2bfloat16(v[j]);
        }
        if (valid) {
#pragma unroll
          for (int j = 0; j < 32; j += 4)
            *reinterpret_cast<float4*>(b.dH2 + gr * kHid + c0 + 32 * q + j) =
                make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        }
      }
      issue([&] { product<kRows, kFeat>(s.tmem_base, s.dzt, s.w1); });  // part of dW1 = dZ1^T X
      ok = wait();
    }
    if (ok) {
      float* part1 = b.part1 + (size_t)blockIdx.x * kW1 + row * kFeat;
#pragma unroll 1
      for (int c = 32 * half; c < kFeat; c += 64) {  // columns 0-31 and 64-79, or 32-63
        float v[32];
        tmem_ld32(d0 + (uint32_t)c, v);
#pragma unroll
        for (int j = 0; j < 32; j += 4)
          if (c + j < kFeat) *reinterpret_cast<float4*>(part1 + c + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
      }
    }
  }
  if (!ok && tid == 0) atomicOr(b.tc_fail, 1u);
  fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s.tmem_base), "r"(256) : "memory");
  }
}

struct AdamArgs {
  int on;  // 0: the gradient goes to g (evaluation)
  float lr, b1, b2, eps, c1, c2;
};

// Gradient gg of parameter x: stored, or applied.
__device__ __forceinline__ void apply_grad(const MlpTrainBuffers& b, int x, float gg, const AdamArgs& a) {
  if (!a.on) {
    b.g[x] = gg;
    return;
  }
  const float mm = a.b1 * b.m[x] + (1.f - a.b1) * gg;
  const float vv = a.b2 * b.v[x] + (1.f - a.b2) * gg * gg;
  b.m[x] = mm;
  b.v[x] = vv;
  b.w[x] -= a.lr * (mm * a.c1) / (sqrtf(vv * a.c2) + a.eps);
}

// Blocks 0 .. kUpdElem - 1: the hidden weights, a parameter a thread, the partial
// products summed block by block.  Then a block per 32 columns of dZ1, dZ2 and
// H2: bias gradients (column sums) and the output layer's (sums of dO times H2),
// row by row: the rows are brought to shared memory kSumRows at a time, then
// one thread a sum adds them in order.
constexpr int kUpdThreads = 256;
constexpr int kUpdElem = (kW1 + kW2) / kUpdThreads;
constexpr int kSumRows = 1024;
constexpr int kSumCols = 32;
constexpr int kUpdSmem = kSumRows * (kSumCols + kOut) * (int)sizeof(float);
static_assert(kOffW2 % 4 == 0, "16-byte loads of W2");
static_assert((kW1 + kW2) % kUpdThreads == 0, "whole blocks of hidden weights");

__global__ void __launch_bounds__(kUpdThreads) k_mlp_update(MlpTrainBuffers b, int n, AdamArgs a) {
  extern __shared__ __align__(16) float tile[];
  const int tid = threadIdx.x;
  if (blockIdx.x < kUpdElem) {
    const int x = blockIdx.x * kUpdThreads + tid;
    const bool second = x >= kW1;
    const int e = second ? x - kW1 : x, size = second ? kW2 : kW1;
    const float* part = (second ? b.part2 : b.part1) + e;
    const int parts = (n + kRows - 1) / kRows;
    float acc = 0.f;
#pragma unroll 8
    for (int k = 0; k < parts; ++k) acc += part[(size_t)k * size];
    apply_grad(b, (second ? kOffW2 : kOffW1) + e, acc, a);
    return;
  }
  const int q = blockIdx.x - kUpdElem, what = q / (kHid / kSumCols), col = kSumCols * (q % (kHid / kSumCols));
  const float* rows = (what == 0 ? b.dH2 : what == 1 ? b.dH : b.H2) + col;
  float* dout = tile + kSumRows * kSumCols;
  // what 0, 1: thread c < 32 sums column c; 2: thread 32 o + c sums dO[o] H2[c], threads 64 + o sum dO[o]
  const int c = tid & 31, o = tid >> 5;
  const bool sums = what < 2 ? tid < 32 : tid < 64, sums_o = what == 2 && col == 0 && tid >= 64 && tid < 64 + kOut;
  float acc = 0.f;
  for (int r0 = 0; r0 < n; r0 += kSumRows) {
    const int nr = min(kSumRows, n - r0);
    __syncthreads();
#pragma unroll 16
    for (int x = tid; x < nr * (kSumCols / 4); x += kUpdThreads) {
      const int r = x / (kSumCols / 4), k = 4 * (x % (kSumCols / 4));
      *reinterpret_cast<float4*>(tile + r * kSumCols + k) =
          __ldcg(reinterpret_cast<const float4*>(rows + (size_t)(r0 + r) * kHid + k));
    }
    if (what == 2)
      for (int x = tid; x < nr * kOut; x += kUpdThreads) dout[x] = __ldcg(b.dO + (size_t)r0 * kOut + x);
    __syncthreads();
    if (sums) {
      if (what < 2) {
#pragma unroll 16
        for (int r = 0; r < nr; ++r) acc += tile[r * kSumCols + c];
      } else {
#pragma unroll 16
        for (int r = 0; r < nr; ++r) acc = fmaf(dout[r * kOut + o], tile[r * kSumCols + c], acc);
      }
    } else if (sums_o) {
#pragma unroll 16
      for (int r = 0; r < nr; ++r) acc += dout[r * kOut + tid - 64];
    }
  }
  if (sums) apply_grad(b, what == 0 ? kOffB1 + col + c : what == 1 ? kOffB2 + col + c : kOffW3 + o * kHid + col + c, acc, a);
  if (sums_o) apply_grad(b, kOffB3 + tid - 64, acc, a);
}

__global__ void k_export_params(const float* __restrict__ w, MlpParams* __restrict__ out) {
  const int n1 = kHid * kFeat, n2 = kHid * kHid, n3 = kOut * kHid;
  for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < kMlpParamCount; x += gridDim.x * blockDim.x) {
    const float v = w[x];
    if (x < n1) out->w1[x] = __float2bfloat16(v);
    else if (x < n1 + kHid) out->b1[x - n1] = v;
    else if (x < n1 + kHid + n2) out->w2[x - n1 - kHid] = __float2bfloat16(v);
    else if (x < n1 + 2 * kHid + n2) out->b2[x - n1 - kHid - n2] = v;
    else if (x < n1 + 2 * kHid + n2 + n3) out->w3[x - n1 - 2 * kHid - n2] = __float2bfloat16(v);
    else out->b3[x - n1 - 2 * kHid - n2 - n3] = v;
  }
}


cudaError_t launch_rows(const MlpTrainBuffers& b, const __nv_bfloat16* feat, const float* targets, const int32_t* idx, int n,
                        float alpha, bool backward, cudaStream_t st) {
  const cudaError_t e = raise_dynamic_smem(reinterpret_cast<const void*>(&k_mlp_rows), (int)sizeof(RowsSmem));
  if (e != cudaSuccess) return e;
  k_mlp_rows<<<(n + kRows - 1) / kRows, kRowThreads, sizeof(RowsSmem), st>>>(b, feat, targets, idx, n, alpha, 1.f / (float)n,
                                                                           backward);
  return cudaGetLastError();
}
cudaError_t launch_update(const MlpTrainBuffers& b, int n, const AdamArgs& a, cudaStream_t st) {
  const cudaError_t e = raise_dynamic_smem(reinterpret_cast<const void*>(&k_mlp_update), kUpdSmem);
  if (e != cudaSuccess) return e;
  k_mlp_update<<<kUpdElem + 3 * (kHid / kSumCols), kUpdThreads, kUpdSmem, st>>>(b, n, a);
  return cudaGetLastError();
}

}  // namespace

cudaError_t mlp_forward_backward(const MlpTrainBuffers& b, int n, float alpha, bool backward, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(b.loss, 0, sizeof(float), st);
  if (e == cudaSuccess) e = launch_rows(b, nullptr, nullptr, nullptr, n, alpha, backward, st);
  if (e == cudaSuccess && backward) e = launch_update(b, n, AdamArgs{}, st);
  return e;
}

cudaError_t mlp_train_step(const MlpTrainBuffers& b, const __nv_bfloat16* feat, const float* targets, const int32_t* idx,
                           int n, float alpha, int step, float lr, cudaStream_t st) {
  const float b1 = 0.9f, b2 = 0.999f;
  const AdamArgs a{1, lr, b1, b2, 1e-8f, 1.f / (1.f - powf(b1, (float)step)), 1.f / (1.f - powf(b2, (float)step))};
  const cudaError_t e = launch_rows(b, feat, targets, idx, n, alpha, true, st);
  return e == cudaSuccess ? launch_update(b, n, a, st) : e;
}

cudaError_t mlp_export(const float* w, MlpParams* out, cudaStream_t st) {
  k_export_params<<<64, 256, 0, st>>>(w, out);
  return cudaGetLastError();
}

}  // namespace bvphmm

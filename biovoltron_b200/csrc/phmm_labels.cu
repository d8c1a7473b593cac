// phmm_labels.cu -- training labels for the band MLP: the posterior spread of
// each pair's alignment over diagonals, from the full-DP forward-backward.
//
// For row r the posterior of cell (r, c) is p_r(c) ~ sum_s F_s(r,c) B_s(r,c)
// (s = M, X, Y), normalised to 1 over the row; pstar(d) = max_r p_r(d + r).
// The label is the lowest and highest diagonal d with pstar(d) >= tau.
// Recurrences are the reference's (avx-pairhmm-template.h:183-198) and their
// adjoint:
//   B_M(r,c) = mm(r+1) e(r+1,c+1) B_M(r+1,c+1) + mx(r+1) B_X(r+1,c) + my(r) B_Y(r,c+1) + [r==R]
//   B_X(r,c) = gp(r+1) e(r+1,c+1) B_M(r+1,c+1) + g(r+1) B_X(r+1,c) + [r==R]
//   B_Y(r,c) = gp(r+1) e(r+1,c+1) B_M(r+1,c+1) + g(r) B_Y(r,c+1)
//
// One warp per pair; lane l owns the C = ceil(H / 32) columns l C + 1 .. of a
// row and keeps their states in registers (template CM >= C: one launch per
// class of haplotype lengths; columns past the haplotype hold zeros).  M and X
// of a row depend only on the previous row (one shuffle brings the column left
// of the lane's first); the in-row Y recurrence is affine with a per-row
// constant (Y(c) = g Y(c-1) + t(c)), solved by a warp scan over the lanes'
// chunks.  Every row is renormalised by a power of two; the per-row
// normalisation of p_r makes the scales cancel.  Forward rows go to a per-warp
// global buffer, column-interleaved so that a warp's stores and loads are
// whole lines, and the backward reads them once.  pstar moves with the row: a
// lane's register for column c holds diagonal c - r, so going one row up
// shifts it by one column, and the diagonal that leaves column 1 is final.
//
// Bound by latency: a row's two affine chains, its warp scan and its three
// reductions follow one another, with 8 to 12 warps an SM to hide them (the
// forward rows' traffic, 24 bytes a cell, is a quarter of the time).  24 k pairs
// of 150 x 450: 10 ms.  States and pstar in shared memory (33 KB a warp, a lane
// stride of C words and its bank conflicts) took 80; classes of 256 and 128
// columns with a branch at every column 21; four columns a class leave the
// branch to the last three.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>
#include <utility>

#include "phmm_band.h"
#include "phmm_common.h"
#include "phmm_kernels.h"
#include "phmm_mlp.h"

namespace bvphmm {
namespace {

constexpr int kLabelMaxH = kBandMaxHap;   // columns per pair
constexpr int kLabelWarps = 4;

__device__ __forceinline__ uint32_t code_of(uint8_t b) {
  return b == 'C' ? 1u : b == 'T' ? 2u : b == 'G' ? 3u : b == 'N' ? 4u : 0u;
}

struct RowC {
  float mm, gp, mx, my, g, em, ex;
  uint32_t rc;
};

__device__ __forceinline__ RowC row_consts(const Tables* tb, const uchar4* quals, const uint8_t* bases, int r) {
  RowC k;
  const uchar4 q = quals[r - 1];
  const int qi = q.y & kQualMask, qd = q.z & kQualMask;
  const int mx = max(qi, qd), mn = min(qi, qd);
  k.mm = tb->mm_f[((mx * (mx + 1)) >> 1) + mn];
  k.g = tb->ph2pr_f[q.w & kQualMask];
  k.gp = 1.f - k.g;
  k.mx = tb->ph2pr_f[qi];
  k.my = tb->ph2pr_f[qd];
  const float eps = tb->ph2pr_f[q.x & kQualMask];
  k.em = 1.f - eps;
  k.ex = eps / 3.f;
  k.rc = code_of(bases[r - 1]);
  return k;
}

// Inclusive warp scan of affine maps y -> a*y + b (lane order = left to right
// when `forward`, right to left otherwise).  Returns the map composed over
// the lanes before this one applied to 0, i.e. the carry-in.
__device__ __forceinline__ float affine_carry(float a, float b, int lane, bool forward) {
  for (int o = 1; o < 32; o <<= 1) {
    const float ao = forward ? __shfl_up_sync(0xffffffffu, a, o) : __shfl_down_sync(0xffffffffu, a, o);
    const float bo = forward ? __shfl_up_sync(0xffffffffu, b, o) : __shfl_down_sync(0xffffffffu, b, o);
    const bool has = forward ? lane >= o : lane + o < 32;
    if (has) { b = a * bo + b; a = a * ao; }
  }
  const float prev = forward ? __shfl_up_sync(0xffffffffu, b, 1) : __shfl_down_sync(0xffffffffu, b, 1);
  return (forward ? lane == 0 : lane == 31) ? 0.f : prev;
}

__device__ __forceinline__ float warp_max(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Pairs whose C lies in (CL, CM]; `first`: this launch also marks the pairs
// that get no label.  Warps take `grab` pairs at a time from *next.
template <int CL, int CM>
__global__ void __launch_bounds__(kLabelWarps * 32, CM <= 20 ? 3 : 2)
    k_posterior_spread(DeviceBatch b, const Tables* tb, const int32_t* pair_read, const int32_t* pair_hap,
                       long long n_pairs, float tau, float* fbuf, long long fbuf_stride, long long max_area,
                       unsigned long long* next, int grab, bool first, int32_t* lo_out, int32_t* hi_out) {
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  float* F = fbuf + (blockIdx.x * (long long)kLabelWarps + wib) * fbuf_stride + lane;
  for (;;) {
    long long base = 0;
    if (lane == 0) base = (long long)atomicAdd(next, (unsigned long long)grab);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= n_pairs) break;
    for (long long pi = base; pi < min(base + grab, n_pairs); ++pi) {
      const int r_idx = pair_read[pi], h_idx = pair_hap[pi];
      const int64_t ro = b.read_off[r_idx], ho = b.hap_off[h_idx];
      const int R = (int)(b.read_off[r_idx + 1] - ro), H = (int)(b.hap_off[h_idx + 1] - ho);
      if (R < 1 || H < 1 || H > kLabelMaxH || R + H >= kBandMaxSpan || (long long)(R + 1) * 3 * (H + 2) > max_area) {
        if (first && lane == 0) { lo_out[pi] = INT32_MIN; hi_out[pi] = INT32_MIN; }
        continue;
      }
      const int C = (H + 31) / 32;
      if (C <= CL || C > CM) continue;
      const uchar4* quals = b.read_quals + ro;
      const uint8_t* bases = b.read_bases + ro;
      const int nc = max(0, min(C, H - lane * C));  // this lane's columns
      // bit j of match[h]: column j matches read code h
      uint32_t match[4] = {0, 0, 0, 0};
#pragma unroll
      for (int j = 0; j < CM; ++j)
        if (j < nc) {
          const uint32_t hc = code_of(b.hap_bases[ho + lane * C + j]);
#pragma unroll
          for (uint32_t h = 0; h < 4; ++h) match[h] |= (uint32_t)(hc == h || hc == 4u) << j;
        }
      auto row_match = [&](uint32_t rc) {
        return rc == 0 ? match[0] : rc == 1 ? match[1] : rc == 2 ? match[2] : rc == 3 ? match[3] : 0xffffffffu;
      };
      float M[CM], X[CM], Y[CM];
#pragma unroll
      for (int j = 0; j < CM; ++j) {
        M[j] = 0.f;
        X[j] = 0.f;
        Y[j] = j < nc ? 1.f : 0.f;
      }
      // ---- forward, rows 1..R; row r's states at F + r * 3 * 32 C: M, X, Y, column j of all lanes together
      const long long row_floats = 96ll * C;
      float tM = 0.f, tX = 0.f, tY = 1.f;  // the lane's last column
      RowC k = row_consts(tb, quals, bases, 1);
      for (int r = 1; r <= R; ++r) {
        const RowC kn = row_consts(tb, quals, bases, min(r + 1, R));
        const uint32_t mm = row_match(k.rc);
        float oM = __shfl_up_sync(0xffffffffu, tM, 1), oX = __shfl_up_sync(0xffffffffu, tX, 1);
        float oY = __shfl_up_sync(0xffffffffu, tY, 1);
        if (lane == 0) { oM = 0.f; oX = 0.f; oY = r == 1 ? 1.f : 0.f; }
        float lastM = 0.f;
#pragma unroll
        for (int j = 0; j < CM; ++j)
          if (j <= CL || j < C) {
            const float e = (mm >> j & 1u) ? k.em : k.ex;
            const float nM = e * (k.mm * oM + k.gp * (oX + oY));
            const float nX = k.mx * M[j] + k.g * X[j];
            oM = M[j]; oX = X[j]; oY = Y[j];
            M[j] = j < nc ? nM : 0.f;
            X[j] = nX;
            lastM = M[j];
          }
        // Y(c) = g Y(c-1) + my M(c-1): affine along the row
        float mleft = __shfl_up_sync(0xffffffffu, lastM, 1);
        if (lane == 0) mleft = 0.f;
        float a = 1.f, bb = 0.f;
        {
          float y = 0.f, m = mleft;
#pragma unroll
          for (int j = 0; j < CM; ++j)
            if (j <= CL || j < C) { y = k.g * y + k.my * m; m = M[j]; a *= k.g; }
          bb = y;
        }
        const float carry = affine_carry(a, bb, lane, true);
        float mx = 0.f;
        {
          float y = carry, m = mleft;
#pragma unroll
          for (int j = 0; j < CM; ++j)
            if (j <= CL || j < C) {
              y = k.g * y + k.my * m;
              Y[j] = j < nc ? y : 0.f;
              m = M[j];
              mx = fmaxf(mx, fmaxf(M[j], fmaxf(X[j], Y[j])));
            }
        }
        mx = warp_max(mx);
        const float sc = mx > 0.f ? ldexpf(1.f, -ilogbf(mx)) : 1.f;
        float* Fr = F + r * row_floats;
#pragma unroll
        for (int j = 0; j < CM; ++j)
          if (j <= CL || j < C) {
            M[j] *= sc;
            X[j] *= sc;
            Y[j] *= sc;
            Fr[j * 32] = M[j];
            Fr[(C + j) * 32] = X[j];
            Fr[(2 * C + j) * 32] = Y[j];
            tM = M[j]; tX = X[j]; tY = Y[j];
          }
        k = kn;
      }
      // ---- backward, rows R..1: M, X hold B of row r + 1, posterior per row
      float P[CM];  // pstar of diagonal c - r
#pragma unroll
      for (int j = 0; j < CM; ++j) { M[j] = 0.f; X[j] = 0.f; P[j] = 0.f; }
      int lo = INT32_MAX, hi = INT32_MIN;
      RowC k1{};  // constants of row r+1
      uint32_t mm1 = 0;
      RowC k0 = row_consts(tb, quals, bases, R);
      for (int r = R; r >= 1; --r) {
        const RowC kn = row_consts(tb, quals, bases, max(r - 1, 1));
        // the column right of the lane's last: B_M of row r + 1 and whether it matches
        float rM = __shfl_down_sync(0xffffffffu, M[0], 1);
        const bool rbit = __shfl_down_sync(0xffffffffu, mm1, 1) & 1u;
        if (lane == 31) rM = 0.f;
        // B_Y(c) = g(r) B_Y(c+1) + t(c), right to left, t(c) = gp(r+1) e(r+1,c+1) B_M(r+1,c+1)
        float a = 1.f, bb = 0.f;
        {
          float y = 0.f, nx = rM;
          bool bit = rbit;
#pragma unroll
          for (int j = CM - 1; j >= 0; --j)
            if (j <= CL || j < C) {
              const float t = __fmul_rn(__fmul_rn(k1.gp, bit ? k1.em : k1.ex), nx);
              y = __fmaf_rn(k0.g, y, t);
              if (j < nc) a *= k0.g;
              nx = M[j];
              bit = mm1 >> j & 1u;
            }
          bb = y;
        }
        const float carry = affine_carry(a, bb, lane, false);
        float mx = 0.f, tot = 0.f;
        {
          float y = carry, nx = rM;  // y: B_Y(r, c+1)
          bool bit = rbit;
#pragma unroll
          for (int j = CM - 1; j >= 0; --j)
            if (j <= CL || j < C) {
              const float byr = y, e = bit ? k1.em : k1.ex, nm = e * nx;
              const float t = __fmul_rn(__fmul_rn(k1.gp, e), nx);
              y = __fmaf_rn(k0.g, y, t);
              Y[j] = y;
              nx = M[j];
              bit = mm1 >> j & 1u;
              const float bm = k1.mm * nm + k1.mx * X[j] + k0.my * byr;
              const float bx = k1.gp * nm + k1.g * X[j];
              M[j] = r == R ? (j < nc ? 1.f : 0.f) : bm;
              X[j] = r == R ? (j < nc ? 1.f : 0.f) : bx;
              mx = fmaxf(mx, fmaxf(M[j], fmaxf(X[j], Y[j])));
            }
        }
        // posterior of row r
        const float* Fr = F + r * row_floats;
#pragma unroll
        for (int j = 0; j < CM; ++j)
          if (j <= CL || j < C) {
            // the sum's terms, kept for the row's normalised values
            Y[j] = Fr[j * 32] * M[j] + Fr[(C + j) * 32] * X[j] + Fr[(2 * C + j) * 32] * Y[j];
            tot += Y[j];
          }
        tot = warp_sum(tot);
        if (tot > 0.f) {
          const float inv = 1.f / tot;
#pragma unroll
          for (int j = 0; j < CM; ++j)
            if (j <= CL || j < C) P[j] = fmaxf(P[j], Y[j] * inv);
        }
        mx = warp_max(mx);
        const float sc = mx > 0.f ? ldexpf(1.f, -ilogbf(mx)) : 1.f;
#pragma unroll
        for (int j = 0; j < CM; ++j)
          if (j <= CL || j < C) { M[j] *= sc; X[j] *= sc; }
        if (r > 1) {  // one row up: diagonal 1 - r leaves column 1
          if (lane == 0 && P[0] >= tau) { lo = min(lo, 1 - r); hi = max(hi, 1 - r); }
          float in = __shfl_down_sync(0xffffffffu, P[0], 1);
          if (lane == 31) in = 0.f;
#pragma unroll
          for (int j = 0; j < CM; ++j)
            if (j <= CL || j < C) P[j] = j + 1 < CM && (j + 1 <= CL || j + 1 < C) ? P[j + 1 < CM ? j + 1 : j] : in;
        }
        k1 = k0;
        mm1 = row_match(k0.rc);
        k0 = kn;
      }
      // spread: lowest and highest diagonal with pstar >= tau (row 1: diagonal c - 1)
#pragma unroll
      for (int j = 0; j < CM; ++j)
        if (j < nc && P[j] >= tau) { lo = min(lo, lane * C + j); hi = max(hi, lane * C + j); }
      lo = __reduce_min_sync(0xffffffffu, lo);
      hi = __reduce_max_sync(0xffffffffu, hi);
      if (lane == 0) { lo_out[pi] = lo == INT32_MAX ? INT32_MIN : lo; hi_out[pi] = hi; }
    }
  }
}

template <int CL, int CM>
cudaError_t launch_class(const DeviceBatch& b, const Tables* tb, const int32_t* pair_read, const int32_t* pair_hap,
                         long long n_pairs, float tau, float* fbuf, const LabelRows& f, unsigned long long* next, bool first,
                         int32_t* lo, int32_t* hi, cudaStream_t st) {
  const int blocks = f.blocks;
  const int grab = (int)std::max<long long>(1, std::min<long long>(32, n_pairs / ((long long)blocks * kLabelWarps * 64)));
  k_posterior_spread<CL, CM><<<blocks, kLabelWarps * 32, 0, st>>>(b, tb, pair_read, pair_hap, n_pairs, tau, fbuf, f.stride,
                                                                  f.max_area, next, grab, first, lo, hi);
  return cudaGetLastError();
}

}  // namespace

// Rows of the longest read and haplotype the label kernel takes; a longer
// read may stand against a shorter haplotype as long as its rows fit that
// area (a row holds 32 C <= H + 31 columns, 29 more than the area counts).
LabelRows label_rows(int max_read, int longest, int max_hap, int sms, size_t max_bytes) {
  LabelRows f{};
  f.max_area = (long long)(max_read + 1) * 3 * (max_hap + 2);
  f.stride = (f.max_area + 3ll * 29 * (std::min(longest, kBandMaxSpan) + 1) + 31) / 32 * 32;
  const size_t per_block = (size_t)f.stride * sizeof(float) * kLabelWarps;
  f.blocks = (int)std::max<size_t>(1, std::min<size_t>((size_t)sms * 3, max_bytes / per_block));
  f.bytes = per_block * (size_t)f.blocks;
  return f;
}

cudaError_t launch_posterior_spread(const DeviceBatch& b, const Tables* tb, const int32_t* pair_read,
                                    const int32_t* pair_hap, long long n_pairs, float tau, float* fbuf,
                                    const LabelRows& f, int max_hap, unsigned long long* next, int32_t* lo, int32_t* hi,
                                    cudaStream_t st) {
  if (n_pairs <= 0) return cudaSuccess;
  const int c = (std::min(max_hap, kLabelMaxH) + 31) / 32;  // classes above the longest haplotype's are empty
  cudaError_t e = cudaSuccess;
  auto run = [&](auto cls) {
    constexpr int k = decltype(cls)::value;
    if (e == cudaSuccess && (k == 0 || c > 4 * k))
      e = launch_class<4 * k, 4 * k + 4>(b, tb, pair_read, pair_hap, n_pairs, tau, fbuf, f, next + k, k == 0, lo, hi, st);
  };
  [&]<int... K>(std::integer_sequence<int, K...>) {
    (run(std::integral_constant<int, K>{}), ...);
  }(std::make_integer_sequence<int, kLabelClasses>{});
  return e;
}

}  // namespace bvphmm

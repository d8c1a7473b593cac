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
// chunks.  Every row is renormalised by a power of two, folded into the next
// row's constants; the per-row normalisation of p_r makes the scales cancel.
// Forward rows go to a per-warp global buffer, M and X column-interleaved so
// that a warp's stores are whole lines, and of Y only what enters each lane's
// first column: the backward pass, which reads a row once, runs Y's chain again.
// It reads from two row buffers in shared memory, filled with cp.async two rows
// ahead.  pstar moves with the row: a lane's register for column c holds
// diagonal c - r, so going one row up shifts it by one column, and the diagonal
// that leaves column 1 is final.
//
// Bound by issue (70 %, 12 warps an SM at 168 registers; 16 warps at 128 give 1 %,
// classes of 20 columns lose by spilling) and by the forward rows' traffic, 16
// bytes a cell: 26 GB of 24 k uneven pairs (1.6 G cells), 3.9 of 6.5 ms.  Reading the
// rows where they are used took 9.5 ms (half the stalls waited for them), with
// the row buffers and one-instruction maxima 7.9, without Y's rows 6.9.
// Earlier forms: states and pstar in shared memory (33 KB a warp, a lane stride of
// C words and its bank conflicts) 80 ms; classes of 256 and 128 columns with a
// branch at every column 21; four columns a class leave the branch to the last
// three.
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
  float mm, gp, mx, my, g, gx, em, ex;
  uint32_t rc;
};

__device__ __forceinline__ RowC row_consts(const Tables* tb, const uchar4* quals, const uint8_t* bases, int r) {
  RowC k;
  const uchar4 q = quals[r - 1];
  const int qi = q.y & kQualMask, qd = q.z & kQualMask;
  const int mx = max(qi, qd), mn = min(qi, qd);
  k.mm = tb->mm_f[((mx * (mx + 1)) >> 1) + mn];
  k.g = tb->ph2pr_f[q.w & kQualMask];
  k.gx = k.g;
  k.gp = 1.f - k.g;
  k.mx = tb->ph2pr_f[qi];
  k.my = tb->ph2pr_f[qd];
  const float eps = tb->ph2pr_f[q.x & kQualMask];
  k.em = 1.f - eps;
  k.ex = eps / 3.f;
  k.rc = code_of(bases[r - 1]);
  return k;
}

// Inclusive warp scans of affine maps y -> a*y + b, `a` the same in every lane
// (a lane that takes a step has a full window of maps beside it: its factor is
// a power that all lanes know).  They return the map composed over the lanes
// before this one applied to 0, i.e. the carry-in.
__device__ __forceinline__ float carry_from_left(float a, float b, int lane) {
  for (int o = 1; o < 32; o <<= 1) {
    const float bo = __shfl_up_sync(0xffffffffu, b, o);
    if (lane >= o) b = a * bo + b;
    a = a * a;
  }
  const float prev = __shfl_up_sync(0xffffffffu, b, 1);
  return lane == 0 ? 0.f : prev;
}
// Right to left.  Lanes past the haplotype's end have b = 0, so that the one
// lane with fewer columns, and with it a smaller power, needs none of its own.
__device__ __forceinline__ float carry_from_right(float a, float b, int lane) {
  for (int o = 1; o < 32; o <<= 1) {
    const float bo = __shfl_down_sync(0xffffffffu, b, o);
    if (lane + o < 32) b = a * bo + b;
    a = a * a;
  }
  const float prev = __shfl_down_sync(0xffffffffu, b, 1);
  return lane == 31 ? 0.f : prev;
}
// The constants of a row that reads the states of a neighbouring row, those
// states to be multiplied by the power of two sc: exact, and cheaper than a
// product for every state.  (g also leads Y along its own row, which has no
// factor: gx is X's.)
__device__ __forceinline__ RowC scaled(RowC k, float sc) {
  k.mm *= sc;
  k.gp *= sc;
  k.mx *= sc;
  k.gx *= sc;
  return k;
}

// Of values >= 0: their bits are in the same order.
__device__ __forceinline__ float warp_max(float v) {
  return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v)));
}
__device__ __forceinline__ float warp_sum(float v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Until at most one group is in flight.
__device__ __forceinline__ void cp_async_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// A warp's two row buffers of the backward pass, floats.
template <int CM>
constexpr int kRowBufFloats = 2 * (64 * CM + 32);

// Pairs whose C lies in (CL, CM]; `first`: this launch also marks the pairs
// that get no label.  Warps take `grab` pairs at a time from *next.
template <int CL, int CM>
__global__ void __launch_bounds__(kLabelWarps * 32, CM <= 20 ? 3 : 2)
    k_posterior_spread(DeviceBatch b, const Tables* tb, const int32_t* pair_read, const int32_t* pair_hap,
                       long long n_pairs, float tau, float* fbuf, long long fbuf_stride, long long max_area,
                       unsigned long long* next, int grab, bool first, int32_t* lo_out, int32_t* hi_out) {
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  float* F = fbuf + (blockIdx.x * (long long)kLabelWarps + wib) * fbuf_stride + lane;
  extern __shared__ __align__(16) float row_bufs[];
  float* S = row_bufs + wib * kRowBufFloats<CM>;
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
      // ---- forward, rows 1..R; row r at F + r * row_floats: M, X (column j of all lanes together), Y's carries
      const long long row_floats = 64ll * C + 32;
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
            const float nX = k.mx * M[j] + k.gx * X[j];
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
          float m = mleft;
#pragma unroll
          for (int j = 0; j < CM; ++j)
            if (j <= CL || j < C) { bb = __fmaf_rn(k.g, bb, __fmul_rn(k.my, m)); m = M[j]; a *= k.g; }
        }
        const float carry = carry_from_left(a, bb, lane);
        float mx = 0.f;
        {
          float y = carry, m = mleft;
#pragma unroll
          for (int j = 0; j < CM; ++j)
            if (j <= CL || j < C) {
              y = __fmaf_rn(k.g, y, __fmul_rn(k.my, m));
              Y[j] = y;
              m = M[j];
              mx = fmaxf(mx, fmaxf(M[j], fmaxf(X[j], Y[j])));
            }
        }
        mx = warp_max(mx);
        const float sc = mx > 0.f ? ldexpf(1.f, -ilogbf(mx)) : 1.f;
        float* Fr = F + r * row_floats;
        Fr[64 * C] = carry;
#pragma unroll
        for (int j = 0; j < CM; ++j)
          if (j <= CL || j < C) {
            Fr[j * 32] = M[j];
            Fr[(C + j) * 32] = X[j];
            tM = M[j]; tX = X[j]; tY = Y[j];
          }
        k = scaled(kn, sc);
      }
      // ---- backward, rows R..1: M, X hold B of row r + 1, posterior per row
      // forward row r is copied to buffer r & 1 while row r + 2 and r + 1 are computed
      auto fetch = [&](int r) {
        if (r >= 1) {
          const float* src = F - lane + r * row_floats;
          float* dst = S + (r & 1) * (64 * CM + 32);
#pragma unroll
          for (int i = 0; i < (16 * CM + 8 + 31) / 32; ++i) {
            const int at = i * 32 + lane;
            if (at < 16 * C + 8) cp_async16(dst + 4 * at, src + 4 * at);
          }
        }
        cp_async_commit();  // a group a row, empty past the first
      };
      __syncwarp();
      fetch(R);
      fetch(R - 1);
      float P[CM];  // pstar of diagonal c - r
#pragma unroll
      for (int j = 0; j < CM; ++j) { M[j] = 0.f; X[j] = j < nc ? 1.f : 0.f; P[j] = 0.f; }
      int lo = INT32_MAX, hi = INT32_MIN;
      RowC k1{};  // constants of row r+1; above row R a row whose B_X = 1 gives B_M = B_X = 1 there
      k1.mx = 1.f;
      k1.gx = 1.f;
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
          float nx = rM;
          bool bit = rbit;
#pragma unroll
          for (int j = CM - 1; j >= 0; --j)
            if (j <= CL || j < C) {
              const float t = __fmul_rn(__fmul_rn(k1.gp, bit ? k1.em : k1.ex), nx);
              bb = __fmaf_rn(k0.g, bb, t);
              a *= k0.g;
              nx = M[j];
              bit = mm1 >> j & 1u;
            }
        }
        const float carry = carry_from_right(a, bb, lane);
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
              M[j] = k1.mm * nm + k1.mx * X[j] + k0.my * byr;
              X[j] = k1.gp * nm + k1.gx * X[j];
              mx = fmaxf(mx, fmaxf(M[j], fmaxf(X[j], Y[j])));
            }
        }
        // posterior of row r
        cp_async_wait1();
        __syncwarp();
        const float* Fr = S + (r & 1) * (64 * CM + 32) + lane;
        {
          float y = Fr[64 * C], m = lane == 0 ? 0.f : Fr[(C - 1) * 32 - 1];
#pragma unroll
          for (int j = 0; j < CM; ++j)
            if (j <= CL || j < C) {
              y = __fmaf_rn(k0.g, y, __fmul_rn(k0.my, m));
              m = Fr[j * 32];
              // the sum's terms, kept for the row's normalised values
              Y[j] = m * M[j] + Fr[(C + j) * 32] * X[j] + y * Y[j];
              tot += Y[j];
            }
        }
        __syncwarp();
        fetch(r - 2);
        tot = warp_sum(tot);
        // one row up: the diagonals move by one column (P: row r + 1's)
        {
          float in = __shfl_down_sync(0xffffffffu, P[0], 1);
          if (lane == 31) in = 0.f;
          const float inv = tot > 0.f ? 1.f / tot : 0.f;
#pragma unroll
          for (int j = 0; j < CM; ++j)
            if (j <= CL || j < C)
              P[j] = fmaxf(j + 1 < CM && (j + 1 <= CL || j + 1 < C) ? P[j + 1 < CM ? j + 1 : j] : in, Y[j] * inv);
        }
        if (r > 1 && lane == 0 && P[0] >= tau) { lo = min(lo, 1 - r); hi = max(hi, 1 - r); }  // leaves column 1
        mx = warp_max(mx);
        const float sc = mx > 0.f ? ldexpf(1.f, -ilogbf(mx)) : 1.f;
        k1 = scaled(k0, sc);
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
  const int smem = kLabelWarps * kRowBufFloats<CM> * (int)sizeof(float);
  if (cudaError_t e = raise_dynamic_smem(reinterpret_cast<const void*>(&k_posterior_spread<CL, CM>), smem); e != cudaSuccess)
    return e;
  k_posterior_spread<CL, CM><<<blocks, kLabelWarps * 32, smem, st>>>(b, tb, pair_read, pair_hap, n_pairs, tau, fbuf, f.stride,
                                                                  f.max_area, next, grab, first, lo, hi);
  return cudaGetLastError();
}

}  // namespace

// Rows of the longest read and haplotype the label kernel takes; a longer
// read may stand against a shorter haplotype as long as its rows fit that
// area.  (The buffer's rows hold M and X of 32 C <= H + 31 columns and 32
// carries: 2 (H + 2) + 90 floats at most, where the area counts 3 (H + 2).)
LabelRows label_rows(int max_read, int longest, int max_hap, int sms, size_t max_bytes) {
  LabelRows f{};
  f.max_area = (long long)(max_read + 1) * 3 * (max_hap + 2);
  f.stride = (f.max_area / 3 * 2 + 90ll * (std::min(longest, kBandMaxSpan) + 1) + 31) / 32 * 32;
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

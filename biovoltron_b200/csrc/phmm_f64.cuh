// phmm_f64.cuh -- the FP64 wavefront in the scaled, folded form, shared by the
// single-strip FP64 kernels (phmm_f64.cu) and the long-read kernel
// (phmm_long.cu).
//
// A warp's lane k owns RT consecutive rows and is at column s - k + 1 at step
// s, as in the FP32 kernels (phmm_device.cuh), with the same formulation: X
// and Y divided by their row's pMX / pMY and pMM folded into the emissions, so
// a cell takes five FP64 operations
//   M(r,c) = e'(r,c) (M(r-1,c-1) + cx' Xh(r-1,c-1) + cy' Yh(r-1,c-1))
//   Xh(r,c) = kap Xh(r-1,c) + M(r-1,c)        Yh(r,c) = g Yh(r,c-1) + M(r,c-1)
// instead of the eight of the unscaled recurrence (process_item<double>).  The
// lane above sends the two sums the top row consumes,
//   zx = kap(r) Xh(r-1,c) + M(r-1,c)
//   zm = M(r-1,c-1) + cx'(r) Xh(r-1,c-1) + cy'(r) Yh(r-1,c-1),
// so four shuffles a step.
//
// The single-strip kernels read the emissions from a table in shared memory
// (ETab, zero outside the haplotype except in the summing row).  The long-read
// kernel, 16 warps on an SM's shared memory, chooses them in registers: a byte
// per haplotype code holds the lane's match bits, one byte permute picks it,
// and every row selects between its two values.  A column outside the
// haplotype then has no zero emission; its cells stay zero because nothing
// above or left of column 1 is non-zero, and nothing is summed past the last
// column.
//
// The folded form needs pMM >= kF64FoldMin in every row and the scaled states
// need head-room, so callers start from 2^kF64Start / H (not 2^1020 / H) and
// hand a pair whose result is not safely inside the range to the unscaled,
// per-strip renormalised form (process_item_f64).
#pragma once
#include "phmm_device.cuh"

namespace bvphmm {

// Initial value's exponent in the single-strip kernels, and the smallest
// exponent of a result they keep: partial sums lost to underflow are then at
// least 2^400 below it.  X / pMX is at most 2^43 above X (qualities <= 127).
constexpr int kF64Start = 900;
constexpr int kF64InitExp = 1020;  // log2 of Tables::init_d
constexpr double kF64MinResult = 2.409919865102884e-181;  // 2^-600
// Rows whose pMM is smaller (indel qualities of 3 and less: pMM is zero, or 0.0061
// at least) do not fold.  FP64 holds coefficients of 1 / pMM, 2^8 at most, without
// loss; at FP32's limit of 0.5, 40 reads of up to 10 kb with some indel qualities
// of 5 and 6 were handed to the unscaled form and took 129 instead of 3.8 ms.
constexpr double kF64FoldMin = 0x1p-8;

template <int RT>
struct F64Rows {
  double cx[RT], cy[RT], kap[RT], g[RT], em[RT], ex[RT];
  double cxN, cyN, kapN;  // the row below the lane's last
  uint32_t ma, mb;        // match bits (bit j: row j) per haplotype code: bytes A C T G, N pad
  bool sums[RT];          // the summing row
};

struct F64Row {
  double cx, cy, kap, g, em, ex;
  uint32_t code;
  bool ok;  // the row can be folded
};

// Constants of padded row r (row 0 the initial row, negative padding, R + 1
// the summing row when SUM, rows past that padding).
template <bool SUM>
__device__ __forceinline__ F64Row f64_row(const Tables* __restrict__ tb, const uchar4* __restrict__ quals,
                                          const uint8_t* __restrict__ bases, int R, int r) {
  F64Row o;
  o.cx = 0.0; o.cy = 0.0; o.kap = 0.0; o.g = 1.0; o.em = 0.0; o.ex = 0.0; o.code = 6; o.ok = true;
  if (SUM && r == R + 1 && R >= 1) {
    o.cx = tb->const_mode ? tb->cd[1] : tb->ph2pr_d[quals[R - 1].y & kQualMask];
    o.em = 1.0;
    o.ex = 1.0;
  } else if (r >= 1 && r <= R) {
    const double* ph = tb->ph2pr_d;
    const uchar4 q = quals[r - 1];
    double mm, pmx, gpx, gx, gpy, gy, ap = 1.0, bp = 1.0;
    if (tb->const_mode) {
      const double* c = tb->cd;
      mm = c[0]; pmx = c[1]; gpx = c[3]; gx = c[4]; gpy = c[5]; gy = c[6];
      if (r >= 2) { ap = pmx; bp = c[2]; }
    } else {
      const int qi = q.y & kQualMask, qd = q.z & kQualMask;
      pmx = ph[qi];
      gx = ph[q.w & kQualMask];
      gy = gx;
      gpx = 1.0 - gx;
      gpy = gpx;
      mm = tb->mm_d[mm_index(qi, qd)];
      if (r >= 2) {
        const uchar4 pv = quals[r - 2];
        ap = ph[pv.y & kQualMask];
        bp = ph[pv.z & kQualMask];
      }
    }
    const double inv = 1.0 / mm;
    o.cx = gpx * ap * inv;
    o.cy = gpy * bp * inv;
    o.kap = gx * ap / pmx;
    o.g = gy;
    const double eps = ph[q.x & kQualMask];
    o.em = (1.0 - eps) * mm;
    o.ex = eps / 3.0 * mm;
    o.code = base_code(bases[r - 1]);
    o.ok = mm >= kF64FoldMin;
  }
  return o;
}

// The lane's rows [rbase, rbase + RT).  Returns whether all its rows fold.
template <int RT, bool SUM>
__device__ __forceinline__ bool f64_setup(const Tables* __restrict__ tb, const uchar4* __restrict__ quals,
                                          const uint8_t* __restrict__ bases, int R, int rbase, F64Rows<RT>& w) {
  static_assert(RT <= 8, "match bits of a code fit a byte");
  bool ok = true;
  w.ma = 0;
  w.mb = (1u << RT) - 1u;
#pragma unroll
  for (int j = 0; j < RT; ++j) {
    const F64Row o = f64_row<SUM>(tb, quals, bases, R, rbase + j);
    w.cx[j] = o.cx; w.cy[j] = o.cy; w.kap[j] = o.kap; w.g[j] = o.g; w.em[j] = o.em; w.ex[j] = o.ex;
    const uint32_t hit = o.code < 4 ? 1u << (8 * o.code) : o.code == 4 ? 0x01010101u : 0u;
    w.ma |= hit << j;
    w.sums[j] = SUM && rbase + j == R + 1;
    ok &= o.ok;
  }
  const F64Row n = f64_row<SUM>(tb, quals, bases, R, rbase + RT);
  w.cxN = n.cx; w.cyN = n.cy; w.kapN = n.kap;
  return ok;
}

template <int RT>
struct F64State {
  double M[RT], X[RT], Y[RT];
  double zx, zm;  // the sums the lane's top row consumes at the next step
};

// What the lane's last row gives the row below: (zx, zm) for its column c,
// from the row's values at c (M, X) and at c - 1 (dm, dx, dy).
template <int RT>
__device__ __forceinline__ double2 f64_sums(const F64Rows<RT>& w, const F64State<RT>& st, double dm, double dx,
                                            double dy) {
  return make_double2(fma_(w.kapN, st.X[RT - 1], st.M[RT - 1]), fma_(w.cyN, dy, fma_(w.cxN, dx, dm)));
}

// One column: the RT cells below the sums (st.zx, st.zm), e(j) the emission of
// the lane's row j.  Returns the last row's previous column in dm, dx, dy.
template <int RT, typename Emission>
__device__ __forceinline__ void f64_column(const F64Rows<RT>& w, F64State<RT>& st, Emission&& e, double& dm, double& dx,
                                           double& dy) {
  double um, ux;
  {
    const double mn = e(0) * st.zm;
    const double yn = fma_(w.g[0], st.Y[0], st.M[0]);
    dm = st.M[0]; dx = st.X[0]; dy = st.Y[0];
    um = mn; ux = st.zx;
    st.M[0] = mn; st.X[0] = ux; st.Y[0] = yn;
  }
#pragma unroll
  for (int j = 1; j < RT; ++j) {
    const double mn = e(j) * fma_(w.cy[j], dy, fma_(w.cx[j], dx, dm));
    const double xn = fma_(w.kap[j], ux, um);
    const double yn = fma_(w.g[j], st.Y[j], st.M[j]);
    dm = st.M[j]; dx = st.X[j]; dy = st.Y[j];
    um = mn; ux = xn;
    st.M[j] = mn; st.X[j] = xn; st.Y[j] = yn;
  }
}

// Emissions selected in registers by the code's match bits.
template <int RT>
__device__ __forceinline__ void f64_cells(const F64Rows<RT>& w, F64State<RT>& st, uint32_t code, double& dm, double& dx,
                                          double& dy) {
  const uint32_t hit = __byte_perm(w.ma, w.mb, code);
  f64_column(w, st, [&](int j) { return (hit & (1u << j)) ? w.em[j] : w.ex[j]; }, dm, dx, dy);
}

__device__ __forceinline__ double2 shfl_up_d2(double2 v) {
  return make_double2(__shfl_up_sync(0xffffffffu, v.x, 1), __shfl_up_sync(0xffffffffu, v.y, 1));
}

}  // namespace bvphmm

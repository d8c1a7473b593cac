// phmm_f64.cu -- FP64 forward pass of reads that fit one strip (up to
// kF64ShortMax bases), and the FP64 list.  The wavefront is phmm_f64.cuh's; a
// warp per read, one haplotype at a time.
//
// k_f64_units runs FP64 mode's work units, a bin of rows per lane at a time;
// k_f64_list drains the list of pairs the other kernels send to FP64 (the
// FP32 kernels' rescues, the pairs the unit and long-read kernels hand back).
// A pair that cannot take the folded form (a row with pMM < kF64FoldMin), whose
// result lies below 2^-600 (from a start of 2^900) or is not finite, and a
// read of several strips runs the unscaled recurrence strip after strip,
// renormalised between strips (process_item_f64: 128 rows a strip, 32 where those
// lose more than the range holds).
//
// Bound by issue: an FP64 instruction takes two slots, and a step of five rows a
// lane has 28 of them.  The emissions come from a table in shared memory, a
// load for two rows, where a select in registers costs two instructions a row
// (31 others a step); a column outside the haplotype then has emission zero,
// so nothing has to be injected on the way in.  75 k pairs of 50-250 bases
// take 3.05 ms (selects: 3.4; the unscaled two-strip kernel: 11.0); the rescue
// of 84 pairs of 46 k takes 0.1 instead of 0.28 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "phmm_f64.cuh"
#include "phmm_kernels.h"

namespace bvphmm {
namespace {

// The pair (rows set up in w, emissions in el's table) over its H columns.
// Lane 31 returns the summing row's total.
template <int RT>
__device__ __forceinline__ double f64_sweep(const F64Rows<RT>& w, const ELane el, const unsigned char* hc_lane, int H,
                                            int r0j, double y0) {
  F64State<RT> st;
#pragma unroll
  for (int j = 0; j < RT; ++j) {
    st.M[j] = 0.0;
    st.X[j] = 0.0;
    st.Y[j] = j == r0j ? y0 : 0.0;
  }
  double2 z = shfl_up_d2(f64_sums(w, st, 0.0, 0.0, st.Y[RT - 1]));
  st.zx = z.x;
  st.zm = z.y;
  // lane 31's last row (the summing row) takes column H + 1 at step H + 31
  const int nsteps = (H + kWarp + 3) / 4 * 4;
#pragma unroll 1
  for (int s = 0; s < nsteps; s += 4) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      double e[RT], dm, dx, dy;
      load_emissions<double, RT>(el, (unsigned)hc_lane[s + u] * ETab<double, RT>::kCodeStride, e);
      f64_column(w, st, [&](int j) { return e[j]; }, dm, dx, dy);
      z = shfl_up_d2(f64_sums(w, st, dm, dx, dy));
      st.zx = z.x;
      st.zm = z.y;
    }
  }
  return st.Y[RT - 1] + st.M[RT - 1];
}

// Scores a read (already set up) against one haplotype; false when the pair
// has to go to the unscaled kernel.
template <int RT>
__device__ __forceinline__ bool f64_pair(const KernelParams& p, const F64Rows<RT>& w, bool fold, int read, int R, int hap,
                                         long long out, unsigned char* hc, const ELane el, int lane) {
  const int64_t ho = p.batch.hap_off[hap];
  const int H = (int)(p.batch.hap_off[hap + 1] - ho);
  if (H == 0 || R == 0) {
    if (lane == kWarp - 1) p.out[out] = -INFINITY;
    return true;
  }
  if (!fold) return false;
  __syncwarp();
  stage_hap(p.batch.hap_bases + ho, H, hc, H + kWarp + 4 + kHapLead, lane);
  __syncwarp();
  const int pad = kWarp * RT - (R + 2);  // rows on top of row 0: >= 1 (the read fits RT rows a lane)
  const double y0 = ldexp(p.tables->init_d, kF64Start - kF64InitExp) / (double)H;
  const double res = f64_sweep<RT>(w, el, hc + kHapLead - lane, H, pad - lane * RT, y0);
  const bool ok = __shfl_sync(0xffffffffu, res >= kF64MinResult && isfinite(res), kWarp - 1);
  if (ok && lane == kWarp - 1) {
    write_result<double>(p, read, hap, out, res, kF64InitExp - kF64Start);
    if (p.cells_ctr) atomicAdd(p.cells_ctr, (unsigned long long)R * (unsigned long long)H);
  }
  return ok;
}

// Sets up a read's rows and their emission table (behind the haplotype codes).
template <int RT>
__device__ __forceinline__ bool f64_read(const KernelParams& p, int64_t ro, int R, int lane, unsigned char* etab,
                                         F64Rows<RT>& w) {
  __syncwarp();
  const bool fold = __all_sync(0xffffffffu, f64_setup<RT, true>(p.tables, p.batch.read_quals + ro,
                                                                p.batch.read_bases + ro, R,
                                                                lane * RT - (kWarp * RT - (R + 2)), w));
#pragma unroll
  for (int h = 0; h < kCodes; ++h) {
    const uint32_t hit = __byte_perm(w.ma, w.mb, h);
    double v[RT];
#pragma unroll
    for (int j = 0; j < RT; ++j) v[j] = h == kPadCode && !w.sums[j] ? 0.0 : (hit & (1u << j)) ? w.em[j] : w.ex[j];
    store_emissions<double, RT>(etab, lane, h, v);
  }
  return fold;
}

// Units of one bin (reads of the same rows per lane).
template <int RT>
__global__ void __launch_bounds__(kThreadsPerBlock, RT <= 5 ? 4 : 3) k_f64_units(KernelParams p) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & (kWarp - 1), wib = threadIdx.x >> 5;
  unsigned char* hc = smem + (size_t)wib * p.warp_smem_bytes;
  for (;;) {
    unsigned long long x = 0;
    if (lane == 0) x = atomicAdd(&p.ctr->unit_next[p.slot], 1ull);
    x = __shfl_sync(0xffffffffu, x, 0);
    if (x >= (unsigned long long)p.n_units) break;
    const Unit u = p.units[p.unit_base + x];
    const int64_t ro = p.batch.read_off[u.read];
    const int R = (int)(p.batch.read_off[u.read + 1] - ro);
    F64Rows<RT> w;
    unsigned char* etab = hc + p.hap_bytes;
    const bool fold = f64_read<RT>(p, ro, R, lane, etab, w);
    const ELane el = elane<double, RT>(etab, lane);
    for (int k = 0; k < u.nh; ++k) {
      if (f64_pair<RT>(p, w, fold, u.read, R, u.hap0 + k, u.out0 + k, hc, el, lane) || lane != 0) continue;
      // to the FP64 list, marked as seen (the read index complemented)
      const unsigned long long at = atomicAdd(&p.ctr->rescue_count, 1ull);
      if (at < (unsigned long long)p.rescue_cap) {
        p.rescue[at].read = ~u.read;
        p.rescue[at].hap = u.hap0 + k;
        p.rescue[at].out = u.out0 + k;
      } else {
        atomicOr(&p.ctr->status, 1ull);
      }
    }
  }
}

// The FP64 list: its front part (reads shorter than long_rows, and everything
// when there is no long-read kernel), then the long part's entries that the
// long-read kernel, which runs before, handed back.  A warp per pair: five
// rows a lane for the reads that fit them, eight for the other short ones,
// the unscaled strips for the rest.
__global__ void __launch_bounds__(kThreadsPerBlock, 3) k_f64_list(const __grid_constant__ KernelParams p) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & (kWarp - 1), wib = threadIdx.x >> 5;
  unsigned char* wsm = smem + (size_t)wib * p.warp_smem_bytes;
  double* bnd = reinterpret_cast<double*>(p.bnd) +
                (size_t)(blockIdx.x * (kThreadsPerBlock / kWarp) + wib) * p.bnd_cols * 4;
  const unsigned long long n_front = min(p.ctr->rescue_count, (unsigned long long)p.rescue_cap);
  const unsigned long long n_long =
      p.long_rows > 0 ? min(p.ctr->rescue_long_count, (unsigned long long)p.rescue_cap) : 0ull;
  for (;;) {
    unsigned long long x = 0;
    if (lane == 0) x = atomicAdd(&p.ctr->rescue_next, 1ull);
    x = __shfl_sync(0xffffffffu, x, 0);
    if (x >= n_front + n_long) break;
    const bool front = x < n_front;
    const long long at = front ? (long long)x : p.rescue_cap - 1 - (long long)(x - n_front);
    PairRef pr = p.rescue[at];
    const bool seen = pr.read < 0;  // handed back by a unit or the long-read kernel
    if (seen) pr.read = ~pr.read;
    else if (!front) continue;  // scored by the long-read kernel
    const int64_t ro = p.batch.read_off[pr.read];
    const int R = (int)(p.batch.read_off[pr.read + 1] - ro);
    bool done = false;
    if (!seen && R <= kF64ShortMax) {
      if (R + 3 <= 5 * kWarp) {
        F64Rows<5> w;
        const bool fold = f64_read<5>(p, ro, R, lane, wsm + p.hap_bytes, w);
        done = f64_pair<5>(p, w, fold, pr.read, R, pr.hap, pr.out, wsm, elane<double, 5>(wsm + p.hap_bytes, lane), lane);
      } else {
        F64Rows<8> w;
        const bool fold = f64_read<8>(p, ro, R, lane, wsm + p.hap_bytes, w);
        done = f64_pair<8>(p, w, fold, pr.read, R, pr.hap, pr.out, wsm, elane<double, 8>(wsm + p.hap_bytes, lane), lane);
      }
    }
    if (!done) process_item_f64(p, Item{pr.read, pr.hap, 1, pr.out}, wsm, lane, bnd);
    // the long part's mark is cleared: a replayed batch finds the list as it was staged
    if (!front && lane == 0) p.rescue[at].read = pr.read;
  }
}

const void* units_kernel(int rt) {
  switch (rt) {
    case 1: return reinterpret_cast<const void*>(&k_f64_units<1>);
    case 2: return reinterpret_cast<const void*>(&k_f64_units<2>);
    case 3: return reinterpret_cast<const void*>(&k_f64_units<3>);
    case 4: return reinterpret_cast<const void*>(&k_f64_units<4>);
    case 5: return reinterpret_cast<const void*>(&k_f64_units<5>);
    case 6: return reinterpret_cast<const void*>(&k_f64_units<6>);
    case 7: return reinterpret_cast<const void*>(&k_f64_units<7>);
    case 8: return reinterpret_cast<const void*>(&k_f64_units<8>);
  }
  return nullptr;
}
const void* kernel_of(int rt) { return rt == 0 ? reinterpret_cast<const void*>(&k_f64_list) : units_kernel(rt); }

}  // namespace

// Four warps fit a block for every haplotype length that is accepted (BV_PHMM_MAX_HAP_LEN: 172 KB).
int f64_warp_smem(int rt, int hap_bytes) {
  using S = WarpSmem<double, 4>;
  // the list's short reads need the table of eight rows a lane, its long ones that of four and the rings
  const int list = std::max(ETab<double, 8>::kBytes, S::kEtabBytes + S::kRingBytes);
  return hap_bytes + (rt == 0 ? list : kCodes * kWarp * rt * (int)sizeof(double));  // ETab<double, rt>::kBytes
}

int f64_blocks_per_sm(int rt, int smem_per_block) {
  int nb = 0;
  const void* k = kernel_of(rt);
  if (!k || raise_dynamic_smem(k, smem_per_block) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, kThreadsPerBlock, smem_per_block) != cudaSuccess) return 0;
  return nb;
}

cudaError_t launch_f64(int rt, const KernelParams& p, int grid, cudaStream_t st) {
  const void* k = kernel_of(rt);
  if (!k) return cudaErrorInvalidValue;
  KernelParams q = p;
  void* args[] = {&q};
  return cudaLaunchKernel(k, dim3(grid), dim3(kThreadsPerBlock), args, (size_t)p.warp_smem_bytes * (kThreadsPerBlock / kWarp),
                          st);
}

}  // namespace bvphmm

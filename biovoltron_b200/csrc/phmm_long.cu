// phmm_long.cu -- FP64 forward pass of long reads, several warps per pair.
//
// The FP64 pass (the rescue of pairs whose FP32 result falls below 1e-28, or
// every pair in FP64 mode) runs a long read strip after strip: strip s holds
// read rows [128 s, 128 s + 128) (4 rows per lane).  With one warp per pair
// the strips run one after the other and the longest pair sets the launch
// time; here a block of K warps takes one pair and warp w runs strips w,
// w + K, w + 2K, ... as a pipelined wavefront: strip s + 1 starts a 32-column
// chunk as soon as strip s has finished the next one.  The cells are the
// scaled, folded form of phmm_f64.cuh (five FP64 operations).
//
// Strip boundaries.  A strip hands the row below it, per column, the two sums
// that row's first cell consumes (zx, zm; phmm_f64.cuh): 16 bytes.  Inside a
// group of K consecutive strips (one per warp) they go to the next warp
// through a shared-memory channel of kLongSlots chunk slots; a slot's mbarriers
// say "full" (the producer's lane 31 arrives after writing the chunk) and
// "empty" (the consumer's lane 0 arrives once its warp has copied it).  From
// the group's last warp to the next group's first they go through the block's
// global boundary buffer, read back one chunk ahead of their use; a counter in
// shared memory says how many chunks are written, so the next group starts
// while the last one is still running.
//
// Scale.  Every strip keeps its own power of two E (true values are stored
// values * 2^E) and a chunk carries the E it was written with.  Before a
// chunk the warp looks at the largest exponent among its states and the
// incoming sums and, when that has left [2^560, 2^975], moves it to 2^965: all
// states are multiplied by exact powers of two.  E holds for all 128 rows of
// the strip, and the top rows are the largest: a path that loses a whole strip
// (a stretch of the read that does not align, insertion runs too dear to bridge
// it: 11 to 15 binary orders a row at base qualities 25 to 40) has to fit below
// them, and may still be the one that counts in the end.  So the largest state
// stands near the top of the range: some 1,980 binary orders a strip are kept,
// about as many as by the unscaled form (from 2^200, an exponent that leaves
// room for any growth, 922 to 1,422 are: a read of 300 bases whose bases 45-172
// do not align scored 10^-436 instead of 10^-384).  What lies further below is
// lost there as here.  Inside a chunk (32 columns) states grow by little: all of
// a row's mass comes from the row above it, and X / pMX by what the insertion
// quality falls from one row to the next, 2^43 at most.  A strip follows E
// wherever the incoming row leads: far from the alignment, where nothing is left
// in range, a chunk keeps the E of before, and the alignment may come back in a
// scale thousands of binary orders away.
//
// Up to a few hundred pairs: a cluster of up to eight blocks takes a pair, its warps numbered
// through, so that 16 x blocks strips run at once (long reads get more blocks
// than short ones: a launch for each cluster size, side by side, each picking
// its pairs from the list); the boundary rows between
// two blocks go through the producer's global buffer like a group's last row,
// with the chunk counter in global memory (release / acquire).  The cluster
// guarantees that its blocks run at the same time; a launch's pairs are dealt
// to its clusters in snake order, costliest first, and the blocks meet at the
// end of each.
//
// A pair with a row that cannot be folded, with a row between two strips whose
// largest sum lies below 2^-960 in the largest scale that the strip above wrote
// sums in (so that what it lost may count), or whose result lies below 2^-960 in
// the last strip's scale or is not finite, is handed back to k_f64_list (its
// list entry marked), which runs after this kernel.
//
// Bound by the issue slots of the FP64 instructions (two each): 40 reads of up to
// 10 kb take 3.7 ms with one to eight blocks of 16 warps a pair (6.8 with two
// each, 11 with one, 28 with four warps), 8 of them 2.8 ms with eight blocks, 2,000 of them 77 ms, where the unscaled form with four warps, emissions in shared memory and one scale
// a group of strips took 58 and 169.
//
// The haplotype codes are staged once per pair for all warps.  Every wait is
// bounded (status bit 8 when one gives up); after the first wait of a block
// that gives up the others are skipped, so a broken hand-over ends after one
// time-out.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "phmm_f64.cuh"
#include "phmm_kernels.h"

namespace bvphmm {
namespace {

constexpr int kLongRT = 4;                // rows per lane
constexpr int kStrip = kWarp * kLongRT;   // rows per strip
constexpr int kLongSlots = 4;             // chunk slots per channel
constexpr int kChunkB = 32 * 16;          // one 32-column chunk of (zx, zm)
constexpr int kTop = 965;                 // exponent the largest state is moved to
constexpr int kTopMax = 975, kTopMin = 560;
constexpr int kMinExp = -960;             // of a row's largest sum, and of the result
constexpr int kNoExp = -(1 << 24);        // "no value": below every exponent

// Dynamic shared memory of a block of K warps, after the staged haplotype
// codes (hap_bytes, a multiple of 16):
//   per warp: the 32 (zx, zm) its lane 0 consumes in the current chunk;
//   channels 0 .. K-2: kLongSlots chunks each, then their exponents;
//   barriers: full / empty per channel slot; the shared scalars.
template <int K>
struct LongLayout {
  static constexpr int kChan = K * kChunkB;
  static constexpr int kExp = kChan + (K - 1) * kLongSlots * kChunkB;
  static constexpr int kBars = kExp + ((K - 1) * kLongSlots * 4 + 15) / 16 * 16;
  static constexpr int kNumBars = 2 * (K - 1) * kLongSlots;
  static constexpr int kScalars = kBars + 8 * kNumBars;
  static constexpr int kBytes = kScalars + 64;
};

struct LongShared {  // at LongLayout::kScalars
  long long item;
  int done;  // chunks the block's last warp has written to the boundary buffer
  int fail;
};

struct LongIO {
  const double2* chin;  // input channel (warps 1 .. K-1)
  const int* chin_e;
  uint64_t* in_full;
  uint64_t* in_empty;
  double2* chout;       // output channel (warps 0 .. K-2)
  int* chout_e;
  uint64_t* out_full;
  uint64_t* out_empty;
  double2* bnd;         // the block's boundary buffer, its chunks' exponents and (clusters) how many are written
  int* bnd_e;
  int* bnd_done;
  const double2* src;   // the buffer warp 0 reads: the block's own, or the block's before it in the cluster
  const int* src_e;
  const int* src_done;
  double2* stage;       // the warp's staged chunk
};
enum LongMode { kZero = 0, kChan = 1, kGlobal = 2 };  // where a strip's input comes from (kZero: none), its output goes

__device__ __forceinline__ void mbar_arrive(uint64_t* mb) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(mb)) : "memory");
}
// Waits for the barrier's phase of parity ((bits >> i) & 1) and flips that
// bit.  Once any wait of the block has given up (*fail), waits are skipped.
__device__ __forceinline__ void wait_flip(uint64_t* mb, unsigned& bits, int i, volatile int* fail) {
  if (!*fail && !mbar_wait(mb, (bits >> i) & 1u)) *fail = 1;
  bits ^= 1u << i;
}
// Waits until `need` chunks of a boundary buffer have been written (CL: by a
// block of the cluster, the count in global memory).
template <bool CL>
__device__ __forceinline__ void wait_done(const int* done, int need, volatile int* fail) {
  for (unsigned it = 0; it < kBulkWaitLimit && !*fail; ++it) {
    int n;
    if (CL) asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(n) : "l"(done) : "memory");
    else n = *(const volatile int*)done;
    if (n >= need) {
      if (!CL) __threadfence_block();
      return;
    }
    __nanosleep(100);
  }
  *fail = 1;
}
template <bool CL>
__device__ __forceinline__ void post_done(int* done, int n) {
  if (CL) {
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(done), "r"(n) : "memory");
  } else {
    __threadfence_block();
    *(volatile int*)done = n;
  }
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Exponent of a non-negative value (kNoExp for zero and below 2^-1022).
__device__ __forceinline__ int exp_of(double v) {
  const int e = (__double2hiint(v) >> 20) & 0x7ff;
  return e == 0 ? kNoExp : e - 1023;
}
// 2^d, exact; zero below 2^-1022.  d <= 1000.
__device__ __forceinline__ double pow2(int d) { return d < -1022 ? 0.0 : __hiloint2double((d + 1023) << 20, 0); }
// v 2^d: a strip's scale may move by more than one power of two holds.
struct Pow2 {
  double a, b;
  __device__ __forceinline__ explicit Pow2(int d) {
    d = max(-2100, min(d, 2000));  // below: zero, as it should be; above: only zeros come
    a = pow2(d / 2);
    b = pow2(d - d / 2);
  }
  __device__ __forceinline__ double operator()(double v) const { return v * a * b; }
};

// The 32 steps of a chunk.  hc: the lane's first column code; stage: what lane
// 0 consumes; o: where lane 31's last row goes (kChan: shared, kGlobal: global
// memory).  RAMP: row 0 (lane l0, register j0) reaches column 0 at step l0 - 1.
// LAST: the last row is summed over the columns up to H (lane 31 is at column
// u + c31).  Specialised so that a step issues nothing but its cells, four
// shuffles, one load and one store: with these choices made inside the loop 40
// reads of up to 10 kb on a block of 16 warps each took 15.7 ms instead of 12.0.
template <LongMode OUT, bool RAMP, bool LAST>
__device__ __forceinline__ void run_chunk(const F64Rows<kLongRT>& w, F64State<kLongRT>& st, double2& z,
                                          const unsigned char* __restrict__ hc, const double2* __restrict__ stage,
                                          double2* __restrict__ o, int lane, int l0, int j0, double y0, int c31, int H,
                                          double& sumM, double& sumX) {
  const unsigned stage_at = smem_addr(stage);
  const unsigned o_at = OUT == kChan ? smem_addr(o) : 0u;
  const unsigned low = lane == 0, high = lane == kWarp - 1;
#pragma unroll(RAMP ? 1 : 4)
  for (int u = 0; u < 32; ++u) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p ld.shared.v2.f64 {%0, %1}, [%3];\n\t}"
                 : "+d"(z.x), "+d"(z.y) : "r"(low), "r"(stage_at + 16 * u) : "memory");
    st.zx = z.x;
    st.zm = z.y;
    double dm, dx, dy;
    f64_cells(w, st, hc[u], dm, dx, dy);
    if (RAMP && lane == l0 && u == l0 - 1) {
#pragma unroll
      for (int j = 0; j < kLongRT; ++j)
        if (j == j0) st.Y[j] = y0;
    }
    z = f64_sums(w, st, dm, dx, dy);
    if (OUT == kChan)
      asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.shared.v2.f64 [%3], {%0, %1};\n\t}"
                   ::"d"(z.x), "d"(z.y), "r"(high), "r"(o_at + 16 * u) : "memory");
    if (OUT == kGlobal && high) o[u] = z;
    if (LAST && u + c31 <= H) {
      sumM += st.M[kLongRT - 1];
      sumX += st.X[kLongRT - 1];
    }
    z = shfl_up_d2(z);
  }
}

// One strip of a long pair.  Entry x of a boundary row is its column x - 30:
// lane 31 is at that column at step x, and lane 0 consumes entry s + 31 at step
// s; chunk k holds the entries 32 k .. 32 k + 31.  fph (lane 0) and eph (lane
// 31) are the parities of the channel barriers' next phases.  Returns the
// strip's exponent; sumM, sumX: lane 31's last row summed over the haplotype's
// columns (last strip only).
template <bool CL>
__device__ __forceinline__ int run_strip_long(const F64Rows<kLongRT>& w, const unsigned char* __restrict__ hc_lane, int H,
                                              int nch, int lane, LongMode in, LongMode out, bool last, int in_done,
                                              int out_done, int l0, int j0, double y0, int y0_exp, const LongIO& io,
                                              LongShared& sh, unsigned& fph, unsigned& eph, double& sumM, double& sumX) {
  volatile int* fail = &sh.fail;
  F64State<kLongRT> st;
  const bool first = in == kZero;
#pragma unroll
  for (int j = 0; j < kLongRT; ++j) {
    st.M[j] = 0.0;
    st.X[j] = 0.0;
    st.Y[j] = (first && l0 == 0 && lane == 0 && j == j0) ? y0 : 0.0;
  }
  sumM = 0.0;
  sumX = 0.0;
  int E = y0_exp;
  // carry: lane 31 keeps the last entry of the chunk before the one being staged
  double2 carry = make_double2(0.0, 0.0);
  int carry_e = E;
  double2 ahead = make_double2(0.0, 0.0);  // global input: the chunk after the next, on its way
  int ahead_e = 0;
  if (in == kChan) {
    if (lane == 0) wait_flip(io.in_full, fph, 0, fail);
    __syncwarp();
    carry = io.chin[lane];
    carry_e = io.chin_e[0];
    __syncwarp();
    if (lane == 0) mbar_arrive(io.in_empty);
  } else if (in == kGlobal) {
    if (lane == 0) wait_done<CL>(io.src_done, in_done + min(2, nch), fail);
    __syncwarp();
    carry = __ldcg(io.src + lane);
    carry_e = __ldcg(io.src_e);
    if (nch > 1) {
      ahead = __ldcg(io.src + 32 + lane);
      ahead_e = __ldcg(io.src_e + 1);
    }
  }
  // the row above from column 2 on: its largest sum (this lane's share), the largest scale that sums came in
  int row_top = 2 * kNoExp, row_e = 2 * kNoExp;
  if (!first) E = carry_e;
  else io.stage[lane] = make_double2(0.0, 0.0);
  double2 z = make_double2(0.0, 0.0);  // nothing lies above column 0
  for (int k = 0; k < nch; ++k) {
    // the next chunk's entries, one a lane
    double2 nx = make_double2(0.0, 0.0);
    int nx_e = carry_e;
    if (in == kChan && k + 1 < nch) {
      const int sl = (k + 1) % kLongSlots;
      if (lane == 0) wait_flip(io.in_full + sl, fph, sl, fail);
      __syncwarp();
      nx = io.chin[sl * 32 + lane];
      nx_e = io.chin_e[sl];
      __syncwarp();
      if (lane == 0) mbar_arrive(io.in_empty + sl);
    } else if (in == kGlobal) {
      if (k + 1 < nch) {
        nx = ahead;
        nx_e = ahead_e;
      }
      if (k + 2 < nch) {
        if (lane == 0) wait_done<CL>(io.src_done, in_done + k + 3, fail);
        __syncwarp();
        ahead = __ldcg(io.src + 32 * (k + 2) + lane);
        ahead_e = __ldcg(io.src_e + k + 2);
      }
    }
    {
      // the scale of this chunk
      int top = max(max(exp_of(z.x), exp_of(z.y)), max(exp_of(sumM), exp_of(sumX)));
#pragma unroll
      for (int j = 0; j < kLongRT; ++j) top = max(top, max(exp_of(st.M[j]), max(exp_of(st.X[j]), exp_of(st.Y[j]))));
      top += E;
      top = max(top, max(exp_of(nx.x), exp_of(nx.y)) + nx_e);
      if (lane == kWarp - 1) top = max(top, max(exp_of(carry.x), exp_of(carry.y)) + carry_e);
      // (The broadcast says that the value is the warp's.  Without it the warp runs a strip's later chunks in parts:
      // the 40 pairs 8.4 instead of 3.7 ms.)
      top = __shfl_sync(0xffffffffu, __reduce_max_sync(0xffffffffu, top), 0);
      if (top > kNoExp / 2 && (top - E > kTopMax || top - E < kTopMin)) {
        const int d = E - (top - kTop);  // stored values times 2^d (beyond 2^2000 only when they are all zero)
        const Pow2 f(d);
#pragma unroll
        for (int j = 0; j < kLongRT; ++j) {
          st.M[j] = f(st.M[j]);
          st.X[j] = f(st.X[j]);
          st.Y[j] = f(st.Y[j]);
        }
        z.x = f(z.x);
        z.y = f(z.y);
        sumM = f(sumM);
        sumX = f(sumX);
        y0 = f(y0);
        E -= d;
      }
    }
    if (!first) {
      // lane 0's inputs of this chunk: the carried entry, then the next chunk's first 31
      const bool edge = lane == kWarp - 1;
      const Pow2 f((edge ? carry_e : nx_e) - E);
      io.stage[edge ? 0 : lane + 1] = make_double2(f(edge ? carry.x : nx.x), f(edge ? carry.y : nx.y));
      carry = nx;
      carry_e = nx_e;
      const int at = max(exp_of(nx.x), exp_of(nx.y)) + nx_e;
      row_top = max(row_top, at);
      row_e = max(row_e, __any_sync(0xffffffffu, at > kNoExp / 2) ? nx_e : 2 * kNoExp);  // (a branch here costs 2 %)
      if (k + 1 == nch && __reduce_max_sync(0xffffffffu, row_top) < row_e + kMinExp) {
        sumM = __longlong_as_double(0x7ff8000000000000ll);  // a NaN in the chunk's first column, or in the result
        st.M[kLongRT - 1] = sumM;
      }
    }
    const int slot = k % kLongSlots;
    if (lane == kWarp - 1 && out == kChan) {
      wait_flip(io.out_empty + slot, eph, slot, fail);
      io.chout_e[slot] = E;
    }
    double2* o = out == kChan ? io.chout + slot * 32 : io.bnd + 32 * k;
    __syncwarp();
    const unsigned char* hc = hc_lane + 32 * k;
    auto chunk = [&](auto mode, auto sum) {
      if (first && k == 0)
        run_chunk<decltype(mode)::value, true, decltype(sum)::value>(w, st, z, hc, io.stage, o, lane, l0, j0, y0,
                                                                     32 * k - 30, H, sumM, sumX);
      else
        run_chunk<decltype(mode)::value, false, decltype(sum)::value>(w, st, z, hc, io.stage, o, lane, l0, j0, y0,
                                                                      32 * k - 30, H, sumM, sumX);
    };
    using std::integral_constant;
    if (last) chunk(integral_constant<LongMode, kZero>{}, std::true_type{});
    else if (out == kChan) chunk(integral_constant<LongMode, kChan>{}, std::false_type{});
    else chunk(integral_constant<LongMode, kGlobal>{}, std::false_type{});
    if (lane == kWarp - 1) {
      if (out == kChan) {
        mbar_arrive(io.out_full + slot);
      } else if (out == kGlobal) {
        io.bnd_e[k] = E;
        post_done<CL>(io.bnd_done, out_done + k + 1);
      }
    }
    __syncwarp();  // lane 0 has read the staged entries
  }
  return E;
}

// A block of K warps (CL: a cluster of such blocks) per long pair: the FP64
// list's long part, read from the list's far end.
template <int K, bool CL>
__global__ void __launch_bounds__(K * kWarp, 16 / K) k_forward_long(KernelParams p) {
  using L = LongLayout<K>;
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & (kWarp - 1), w = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  unsigned char* hc = smem;
  unsigned char* base = smem + p.hap_bytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + L::kBars);
  uint64_t* full = bars;                          // [(K-1) * slots]
  uint64_t* empty = bars + (K - 1) * kLongSlots;  // [(K-1) * slots]
  LongShared& sh = *reinterpret_cast<LongShared*>(base + L::kScalars);
  if (threadIdx.x == 0) {
    for (int i = 0; i < L::kNumBars; ++i) mbar_init(bars + i, 1);
    sh.fail = 0;
  }
  __syncthreads();
  LongIO io{};
  if (w >= 1) {
    io.chin = reinterpret_cast<const double2*>(base + L::kChan) + (w - 1) * kLongSlots * 32;
    io.chin_e = reinterpret_cast<const int*>(base + L::kExp) + (w - 1) * kLongSlots;
    io.in_full = full + (w - 1) * kLongSlots;
    io.in_empty = empty + (w - 1) * kLongSlots;
  }
  if (w + 1 < K) {
    io.chout = reinterpret_cast<double2*>(base + L::kChan) + w * kLongSlots * 32;
    io.chout_e = reinterpret_cast<int*>(base + L::kExp) + w * kLongSlots;
    io.out_full = full + w * kLongSlots;
    io.out_empty = empty + w * kLongSlots;
  }
  // the blocks of a pair: rank in the cluster, their number, the cluster's and the clusters' number
  int rank = 0, blocks = 1;
  if (CL) {
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(blocks));
  }
  const int team = blockIdx.x / blocks, teams = gridDim.x / blocks;
  const int W = K * blocks, gw = rank * K + w;  // warps per pair, this warp's number
  // a buffer: bnd_cols rows of 32 bytes: 16 bytes an entry, the exponents behind them, the count at the end
  auto buffer = [&](int block) { return reinterpret_cast<double2*>(p.bnd) + (size_t)block * p.bnd_cols * 2; };
  auto count_of = [&](double2* buf) { return reinterpret_cast<int*>(buf + 2 * p.bnd_cols) - 4; };
  io.bnd = buffer(blockIdx.x);
  io.bnd_e = reinterpret_cast<int*>(io.bnd + p.bnd_cols);
  io.bnd_done = CL ? count_of(io.bnd) : &sh.done;
  const int before = (rank + blocks - 1) % blocks;  // whose last warp feeds this block's first
  double2* const src = buffer(team * blocks + before);
  io.src = src;
  io.src_e = reinterpret_cast<const int*>(src + p.bnd_cols);
  io.src_done = CL ? count_of(src) : &sh.done;
  if (threadIdx.x == 0) *io.bnd_done = 0;
  int in_base = 0, out_base = 0;  // chunks of earlier pairs (the counts run on over the pairs)
  io.stage = reinterpret_cast<double2*>(base) + w * 32;
  unsigned fph = 0;                        // lane 0: input channel slots' next full phases
  unsigned eph = (1u << kLongSlots) - 1u;  // lane 31: output slots; their first wait passes at once
  volatile int* fail = &sh.fail;
  const DeviceBatch& b = p.batch;
  const unsigned long long n_long = min(p.ctr->rescue_long_count, (unsigned long long)p.rescue_cap);
  __syncwarp();
  __shared__ long long member_cost[CL ? kLongMembers : 1];  // the listed pairs' costs, -1: other launches'
  __shared__ int members[CL ? kLongMembers : 1], n_members;
  if (CL) {
    // this launch's pairs, the costliest first (every block of every cluster finds the same order)
    const int n = (int)min(n_long, (unsigned long long)kLongMembers);
    long long cost = -1;
    if (threadIdx.x == 0) n_members = 0;
    if (threadIdx.x < n) {
      const PairRef pr = p.rescue[p.rescue_cap - 1 - threadIdx.x];
      const int read = pr.read < 0 ? ~pr.read : pr.read;  // handed back by another cluster already
      const long long R = b.read_off[read + 1] - b.read_off[read], H = b.hap_off[pr.hap + 1] - b.hap_off[pr.hap];
      if (long_blocks(R, H, p.long_cost) == blocks) cost = long_cost(R, H, blocks);
      member_cost[threadIdx.x] = cost;
    }
    __syncthreads();
    if (cost >= 0) {
      int at = 0;
      for (int t = 0; t < n; ++t) at += member_cost[t] > cost || (member_cost[t] == cost && t < threadIdx.x);
      members[at] = threadIdx.x;
      atomicAdd(&n_members, 1);
    }
    __syncthreads();
    cluster_sync();  // every count is zero
  }
  for (long long round = 0;; ++round) {
    long long wi;
    if (CL) {
      // dealt in snake order; every block of a cluster takes the same pairs, and leaves after the same one
      const long long m = round * teams + (round & 1 ? teams - 1 - team : team);
      if (round * teams >= n_members) break;
      if (m >= n_members) continue;
      wi = members[m];
    } else {
      if (threadIdx.x == 0) sh.item = (long long)atomicAdd(&p.ctr->rescue_long_next, 1ull);
      __syncthreads();
      wi = sh.item;
      if (wi >= (long long)n_long || *fail) break;
    }
    PairRef pr = p.rescue[p.rescue_cap - 1 - wi];
    if (CL && pr.read < 0) pr.read = ~pr.read;  // another block of the cluster is through and has handed it back
    const int64_t ro = b.read_off[pr.read], ho = b.hap_off[pr.hap];
    const int R = __shfl_sync(0xffffffffu, (int)(b.read_off[pr.read + 1] - ro), 0);
    const int H = __shfl_sync(0xffffffffu, (int)(b.hap_off[pr.hap + 1] - ho), 0);
    const uchar4* quals = b.read_quals + ro;
    const uint8_t* bases = b.read_bases + ro;
    if (H == 0 || R == 0) {
      if (threadIdx.x == 0) p.out[pr.out] = -INFINITY;
      if (!CL) __syncthreads();
      continue;
    }
    const int nch = (H + kWarp - 1 + 31) / 32;
    const int nstrips = (R + 1 + kStrip - 1) / kStrip;
    const int pad = nstrips * kStrip - (R + 1);  // padding rows on top of row 0
    // initial row: init / H, stored with exponent y0_exp, just below 2^(kTop + 9)
    const int y0_exp = kF64InitExp - kTop - 8 - (31 - __clz(H));
    const double y0 = ldexp(p.tables->init_d, -y0_exp) / (double)H;
    stage_hap_block(b.hap_bases + ho, H, hc, 32 * nch + kHapLead);
    __syncthreads();
    for (int s = gw; s < nstrips; s += W) {
      F64Rows<kLongRT> rw;
      // a row that cannot be folded makes the result NaN
      if (!f64_setup<kLongRT, false>(p.tables, quals, bases, R, s * kStrip + lane * kLongRT - pad, rw))
        rw.em[0] = rw.ex[0] = __longlong_as_double(0x7ff8000000000000ll);
      const LongMode in = s == 0 ? kZero : (w == 0 ? kGlobal : kChan);
      const bool last = s == nstrips - 1;
      const LongMode out = last ? kZero : (w == K - 1 ? kGlobal : kChan);
      double sumM, sumX;
      const int E = run_strip_long<CL>(rw, hc + kHapLead - lane, H, nch, lane, in, out, last,
                                       in_base + (s > 0 ? (s - 1) / W * nch : 0), out_base + s / W * nch,
                                       pad / kLongRT, pad % kLongRT, y0, y0_exp, io, sh, fph, eph, sumM, sumX);
      if (last && lane == kWarp - 1) {
        const double pmx = p.tables->const_mode ? p.tables->cd[1] : p.tables->ph2pr_d[quals[R - 1].y & kQualMask];
        const double res = sumM + pmx * sumX;
        if (res >= pow2(kMinExp) && isfinite(res)) {
          write_result<double>(p, pr.read, pr.hap, pr.out, res, E);
          if (p.cells_ctr) atomicAdd(p.cells_ctr, (unsigned long long)R * (unsigned long long)H);
        } else {
          // handed back: the entry is marked (read index complemented) for k_f64_list
          p.rescue[p.rescue_cap - 1 - wi].read = ~pr.read;
        }
      }
    }
    // strips but the last that end in a block's last warp: those numbers W i + (rank + 1) K - 1 < nstrips - 1
    auto ended = [&](int r) { return (max(0, nstrips - 1 - ((r + 1) * K - 1)) + W - 1) / W * nch; };
    in_base += ended(before);
    out_base += ended(rank);
    __syncwarp();
    if (CL) cluster_sync();  // the buffers are read
    else __syncthreads();
  }
  if (threadIdx.x == 0 && *fail) atomicOr(&p.ctr->status, 8ull);
}

template <int K, bool CL>
const void* kernel() { return reinterpret_cast<const void*>(&k_forward_long<K, CL>); }
const void* kernel_of(int warps, int blocks) {
  if (blocks > 0) return warps == 16 ? kernel<16, true>() : nullptr;
  return warps == 2 ? kernel<2, false>() : warps == 4 ? kernel<4, false>() : warps == 8 ? kernel<8, false>() : kernel<16, false>();
}
cudaLaunchConfig_t config_of(int grid, int smem, int warps, int blocks, cudaStream_t st, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(warps * kWarp);
  c.dynamicSmemBytes = (size_t)smem;
  c.stream = st;
  if (blocks > 0) {
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = (unsigned)blocks;
    attr->val.clusterDim.y = 1;
    attr->val.clusterDim.z = 1;
    c.attrs = attr;
    c.numAttrs = 1;
  }
  return c;
}
}  // namespace

int long_smem_bytes(int hap_bytes, int warps) {
  return hap_bytes + (warps == 2    ? LongLayout<2>::kBytes
                      : warps == 4  ? LongLayout<4>::kBytes
                      : warps == 8  ? LongLayout<8>::kBytes
                                    : LongLayout<16>::kBytes);
}

cudaError_t prepare_long(int smem, int warps, int blocks) { return raise_dynamic_smem(kernel_of(warps, blocks), smem); }

int long_blocks_per_sm(int smem, int warps) {
  int nb = 0;
  if (prepare_long(smem, warps, 0) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel_of(warps, 0), warps * kWarp, smem) != cudaSuccess) return 0;
  return nb;
}

cudaError_t launch_forward_long(const KernelParams& p, int grid, int smem, int warps, int blocks, cudaStream_t st) {
  cudaLaunchAttribute attr{};
  const cudaLaunchConfig_t c = config_of(grid, smem, warps, blocks, st, &attr);
  KernelParams q = p;
  void* args[] = {&q};
  return cudaLaunchKernelExC(&c, kernel_of(warps, blocks), args);
}

}  // namespace bvphmm

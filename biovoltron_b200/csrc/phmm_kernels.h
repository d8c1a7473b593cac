// phmm_kernels.h -- launch interface between the host engine and the kernels.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "phmm_common.h"

namespace bvphmm {

constexpr int kThreadsPerBlock = 128;

// Read-length bins of the full DP: 1 .. 8 rows a lane in one strip, then reads of several strips.
constexpr int kBins = 9;

// Makes a batch's units from its region arrays: bin rt's units start at
// start[column[rt]] (column -1: no units), region g's at base[column * n_regions
// + g] within them, read by read, per_unit haplotypes each.
struct MakeUnits {
  const int64_t* region_reads;  // [n_regions + 1]
  const int64_t* region_haps;   // [n_regions + 1]
  const int64_t* region_res;    // [n_regions] first result
  const uint32_t* base;         // [columns][n_regions]
  const int64_t* read_off;
  Unit* units;
  long long n_regions;
  long long start[kBins];
  int column[kBins + 1];
  int per_unit;
};
cudaError_t launch_make_units(const MakeUnits& m, int sms, cudaStream_t st);

struct KernelParams {
  DeviceBatch batch;
  const Tables* tables;
  const Unit* units;
  long long unit_base;
  long long n_units;
  const unsigned long long* n_units_dev;  // if set, the unit count is read from device memory
  int slot;               // work-queue head used by this launch
  Counters* ctr;
  double* out;            // log10 likelihoods, one per result slot
  PairRef* rescue;        // null: pairs below the FP32 threshold get NaN (audit runs)
  long long rescue_cap;
  int warps_per_block;    // block size of the launch / 32 (1..4)
  int hap_bytes;          // per-warp bytes for staged haplotype codes
  int code_row_bytes;     // entries of a staged code row (paired variants stage 4-byte entries)
  int warp_smem_bytes;    // per-warp dynamic shared memory
  void* bnd;              // per-warp strip-boundary buffers (multi-strip variants)
  long long bnd_cols;     // rows of 4 values per warp buffer
  int rescale;            // renormalise between strips (FP64, multi-strip)
  int rescale_target;     // binary exponent the boundary maximum is scaled to
  unsigned long long* cells_ctr;  // if set, FP64 launches add read x haplotype length per pair here
  long long long_cost;    // long-read kernel on clusters: the cost limit that gives each pair its blocks
  int long_rows;          // > 0: FP32 results of reads this long or longer go to the FP64 list's long part
};

// Reads of at most kF64ShortMax bases fit one strip of the FP64 wavefront
// (eight rows a lane, phmm_f64.cu).  rt = 1 .. 8: the unit kernel of that many
// rows a lane; rt = 0: the FP64 list.
constexpr int kF64ShortMax = 8 * kWarp - 3;
int f64_warp_smem(int rt, int hap_bytes);
int f64_blocks_per_sm(int rt, int smem_per_block);
cudaError_t launch_f64(int rt, const KernelParams& p, int grid, cudaStream_t st);

// Long reads in FP64: a block of `warps` warps per pair (phmm_long.cu; 2, 4,
// 8 or 16).  By default reads of more than kF64ShortMax bases take it, with as
// many warps as Engine::plan finds for the batch; a context whose warps per
// pair are set or tuned uses that many, for reads of at least 128 x warps
// bases.
constexpr int kLongWarps = 4;
int long_smem_bytes(int hap_bytes, int warps);
// `blocks` > 0 (16 warps each): clusters of that many blocks per pair, grid a multiple of it; the launch takes
// the listed pairs (kLongMembers at most) whose long_blocks is `blocks`.  0: a block per pair, all pairs.
constexpr int kLongMaxBlocks = 8;
constexpr int kLongMembers = 512;
// Wavefront steps of a pair on `blocks` blocks: strips of 128 rows on 16 x blocks
// warps, each strip some 96 columns behind the one above it.
__host__ __device__ inline long long long_cost(long long R, long long H, int blocks) {
  const long long strips = (R + 128) / 128, W = 16 * blocks, full = (strips - 1) / W;
  return full * (H > 96 * W ? H : 96 * W) + H + 96 * (strips - full * W);
}
// The fewest blocks (1, 2, 4, 8) that keep a pair's cost within the limit, or make it as small as it gets.
__host__ __device__ inline int long_blocks(long long R, long long H, long long limit) {
  int best = 1;
  for (int c = 2; c <= kLongMaxBlocks && long_cost(R, H, best) > limit; c *= 2)
    if (long_cost(R, H, c) < long_cost(R, H, best)) best = c;
  return best;
}
cudaError_t prepare_long(int smem, int warps, int blocks);
int long_blocks_per_sm(int smem, int warps);
cudaError_t launch_forward_long(const KernelParams& p, int grid, int smem, int warps, int blocks, cudaStream_t st);

// Variant table: (precision, rows per lane, multi-strip, two haplotypes per
// warp).  Paired variants exist for FP32 single strip only.
int variant_index(bool f64, int rows_per_lane, bool multi, bool paired = false);
bool variant_paired(int variant);
int warp_smem_bytes(int variant, int hap_bytes);
int blocks_per_sm(int variant, int smem_per_block, int threads = kThreadsPerBlock);
// Raises (never lowers) a kernel's dynamic shared-memory limit on the current
// device to at least `bytes`; safe to call from several host threads.
cudaError_t raise_dynamic_smem(const void* func, int bytes);
// Sets the variant's dynamic shared-memory limit; call before launching or capturing it.
cudaError_t prepare_variant(int variant, int smem_per_block);
cudaError_t launch_forward(int variant, const KernelParams& p, int grid, cudaStream_t st);
// Copies `bytes` (rounded up to 16; both sides 16-byte aligned) by a kernel.
cudaError_t launch_copy_small(const void* src, void* dst, size_t bytes, cudaStream_t st);
cudaError_t launch_pack_quals(const uint8_t* q, const uint8_t* i, const uint8_t* d, const uint8_t* c, uchar4* out,
                              long long n, int sms, cudaStream_t st);
// The same with the insertion, deletion and continuation qualities constant.
cudaError_t launch_pack_quals_uniform(const uint8_t* q, uint8_t gi, uint8_t gd, uint8_t gc, uchar4* out, long long n,
                                      int sms, cudaStream_t st);

#if defined(__CUDACC__)
// Appends a pair to the FP64 list: reads of at least long_rows bases to its
// long part, filled from the list's far end for the several-warps-per-pair
// kernel, the others to its front.
__device__ __forceinline__ void push_rescue(Counters* c, PairRef* list, long long cap, int long_rows, int R, int read,
                                            int hap, long long out) {
  const bool lng = long_rows > 0 && R >= long_rows;
  const unsigned long long slot = atomicAdd(lng ? &c->rescue_long_count : &c->rescue_count, 1ull);
  if (slot < (unsigned long long)cap) {
    PairRef& e = list[lng ? cap - 1 - (long long)slot : (long long)slot];
    e.read = read;
    e.hap = hap;
    e.out = out;
  } else {
    atomicOr(&c->status, 1ull);
  }
}
#endif

// Writes one 64-bit value on the device (graph-capturable).
cudaError_t launch_set_u64(unsigned long long* dst, unsigned long long v, cudaStream_t st);

// Host-side construction of the reference's probability tables (Context.h).
void build_tables(Tables* t);
// Constant transitions for every row (7 entries, PairHMM::TrasMatrx order), or
// back to the quality-derived ones (nullptr).
void set_constant_transitions(Tables* t, const double* trans);

}  // namespace bvphmm

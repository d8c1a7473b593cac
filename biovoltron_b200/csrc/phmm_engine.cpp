// phmm_engine.cpp -- host engine: validation, work planning, staging,
// launches, FP64 rescue, timing and graph replay.
//
// Work layout.  A result slot is one (read, haplotype) pair of one region,
// numbered region by region in read-major order, which is the layout of the
// [read][hap] matrix that AvxPairHMM::compute_likelihoods returns
// (include/biovoltron/algo/align/inexact_match/pairhmm_avx.hpp:160-171).
// A unit is one read scored against up to `haps_per_unit` consecutive
// haplotypes of its region, so the read's per-row constants and emission table
// are built once per unit.  Units are bucketed by kernel variant (rows per
// lane = ceil((read_len + 1) / 32), multi-strip above 256 rows); each bucket is
// one persistent launch whose warps pull units from a device work-queue head.
// The FP64 launch follows on the same stream and drains the list of pairs the
// FP32 launches flagged.
#include "phmm_engine.h"

#include "phmm_rows.h"

#include <emmintrin.h>

#include <algorithm>
#include <chrono>
#include <memory>
#include <cstring>
#include <numeric>
#include <string>

namespace bvphmm {

cudaError_t DevBuf::reserve(size_t bytes) {
  if (bytes <= cap_ && own_) {
    p_ = own_;
    return cudaSuccess;
  }
  release();
  size_t want = std::max<size_t>(bytes, 256);
  cudaError_t e = cudaMalloc(&own_, want);
  if (e != cudaSuccess) {
    own_ = nullptr;
    return e;
  }
  p_ = own_;
  cap_ = want;
  return cudaSuccess;
}

void DevBuf::release() {
  if (own_) cudaFree(own_);
  p_ = nullptr;
  own_ = nullptr;
  cap_ = 0;
}

namespace {
// Launch bins: the FP32 variants (variant_index), then FP64 mode's bins of 1 .. 8 rows a lane; reads of
// several strips go to the FP64 list.
constexpr int kF64Bin0 = 19;
constexpr int kF64List = 28;
constexpr int kMaxVariants = 28;
constexpr int kRescaleTarget = 1000;  // FP64 boundary rows are scaled to ~2^1000

// Small batches.  Eight copies from pageable memory, a packing kernel and two
// copies back cost more host time than the kernels of one window take; a batch
// whose inputs fit kStageBytes is laid out in page-locked memory instead
// (qualities packed there) and sent as one copy, and results that fit
// kSmallOutBytes come back with the counters in one.  Beyond that size the
// packing loop is slower than the copies it saves.
constexpr size_t kStageBytes = 512 << 10;
constexpr size_t kSmallOutBytes = 256 << 10;
constexpr size_t kCountersBytes = 512;
static_assert(sizeof(Counters) <= kCountersBytes, "results lie behind the counters");

int64_t round_up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

int hap_bytes_for(int max_hap, int chunk) {
  return (int)round_up((int64_t)max_hap + (kWarp - 1) + chunk + kHapLead + 16, 16);
}
long long bnd_cols_for(int max_hap) { return round_up((int64_t)max_hap + kWarp, 32) + 160; }
}  // namespace

Engine::Engine(const bv_phmm_options& opt) : opt_(opt) {
  // BV_MODE_BAND at creation: the band path with its default options (a fixed
  // band around the seed until MLP weights are trained or loaded).
  band_opt_.struct_size = (int32_t)sizeof(bv_band_options);
  band_opt_.enabled = opt.mode == BV_MODE_BAND;
  band_opt_.use_mlp = 0;
  band_opt_.fixed_half = 8;
  band_opt_.margin = 2;
  band_opt_.audit_period = 0;
  band_opt_.edge_threshold = 1e-3;
}

Engine::~Engine() {
  destroy_graph();
  if (stream_) {
    cudaStreamSynchronize(stream_);
    if (h_counters_) cudaFreeHost(h_counters_);
    if (h_chunk_off_) cudaFreeHost(h_chunk_off_);
    for (auto& e : ev_)
      if (e) cudaEventDestroy(e);
    for (auto& e : tune_ev_)
      if (e) cudaEventDestroy(e);
    for (auto& e : side_done_) cudaEventDestroy(e);
    if (fork_ev_) cudaEventDestroy(fork_ev_);
    for (auto& s : side_) cudaStreamDestroy(s);
    cudaStreamDestroy(stream_);
  }
}

bv_status Engine::fail(bv_status s, const std::string& msg) {
  err_ = msg;
  return s;
}

bv_status Engine::status_fail(unsigned long long status) {
  // Kernel status bits: 1 FP64 list overflow, 2 invalid pair, 4 band list
  // overflow, 8 a boundary-row copy or strip hand-over wait gave up, 16 a
  // tensor-core completion wait gave up.
  static const char* const kNames[] = {"FP64 list overflow", "invalid pair", "band list overflow",
                                       "boundary wait gave up", "tensor-core wait gave up"};
  std::string msg = "kernel reported an inconsistent state (";
  bool first = true;
  for (int b = 0; b < 5; ++b) {
    if (!(status >> b & 1ull)) continue;
    msg += first ? "" : ", ";
    msg += kNames[b];
    first = false;
  }
  if (status >> 5) msg += std::string(first ? "" : ", ") + "status " + std::to_string(status);
  return fail(BV_ERR_INTERNAL, msg + ")");
}

bv_status Engine::cuda_fail(cudaError_t e, const char* what) {
  err_ = std::string(what) + ": " + cudaGetErrorString(e);
  if (e == cudaErrorMemoryAllocation) return BV_ERR_OOM;
  if (e == cudaErrorNoDevice || e == cudaErrorInvalidDevice) return BV_ERR_NO_DEVICE;
  return BV_ERR_CUDA;
}

#define BV_CUDA(call, what)                         \
  do {                                              \
    cudaError_t e__ = (call);                       \
    if (e__ != cudaSuccess) return cuda_fail(e__, what); \
  } while (0)

bv_status Engine::set_transitions(const double* trans) {
  if (trans) {
    for (int k = 0; k < 7; ++k)
      if (!(trans[k] >= 0.0 && trans[k] <= 1.0)) return fail(BV_ERR_INVALID_ARG, "transition outside [0, 1]");
    if (band_enabled()) return fail(BV_ERR_UNSUPPORTED, "constant transitions run the full-DP path: disable the band");
  }
  BV_CUDA(cudaSetDevice(opt_.device), "cudaSetDevice");
  BV_CUDA(cudaStreamSynchronize(stream_), "sync before table update");
  set_constant_transitions(h_tables_.get(), trans);
  BV_CUDA(cudaMemcpy(d_tables_.get(), h_tables_.get(), sizeof(Tables), cudaMemcpyHostToDevice), "tables copy");
  ++config_version_;
  staged_ = false;
  destroy_graph();
  return BV_OK;
}

bool Engine::constant_transitions(double* trans) const {
  if (!h_tables_ || !h_tables_->const_mode) return false;
  if (trans)
    for (int k = 0; k < 7; ++k) trans[k] = h_tables_->cd[k];
  return true;
}

bv_status Engine::init() {
  int ndev = 0;
  cudaError_t e = cudaGetDeviceCount(&ndev);
  if (e != cudaSuccess || ndev == 0) return fail(BV_ERR_NO_DEVICE, "no CUDA device available");
  if (opt_.device < 0 || opt_.device >= ndev) return fail(BV_ERR_NO_DEVICE, "device ordinal out of range");
  BV_CUDA(cudaSetDevice(opt_.device), "cudaSetDevice");
  BV_CUDA(cudaDeviceGetAttribute(&sms_, cudaDevAttrMultiProcessorCount, opt_.device), "SM count");
  BV_CUDA(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking), "stream");
  for (auto& ev : ev_) BV_CUDA(cudaEventCreate(&ev), "event");
  h_tables_ = std::make_unique<Tables>();
  build_tables(h_tables_.get());
  BV_CUDA(d_tables_.reserve(sizeof(Tables)), "tables alloc");
  BV_CUDA(cudaMemcpyAsync(d_tables_.get(), h_tables_.get(), sizeof(Tables), cudaMemcpyHostToDevice, stream_),
          "tables copy");
  BV_CUDA(d_counters_.reserve(kCountersBytes + kSmallOutBytes), "counters alloc");
  BV_CUDA(cudaStreamSynchronize(stream_), "init sync");
  return BV_OK;
}

bv_status Engine::reserve_lanes(int n) {
  if (n > 1 && !fork_ev_) BV_CUDA(cudaEventCreateWithFlags(&fork_ev_, cudaEventDisableTiming), "event");
  while ((int)side_.size() < n - 1) {
    cudaStream_t s;
    BV_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "stream");
    side_.push_back(s);
  }
  while (side_done_.size() < side_.size()) {
    cudaEvent_t e;
    BV_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "event");
    side_done_.push_back(e);
  }
  return BV_OK;
}

bv_status Engine::fork(int n) {
  if (n < 2) return BV_OK;
  BV_CUDA(cudaEventRecord(fork_ev_, stream_), "event");
  for (int i = 1; i < n; ++i) BV_CUDA(cudaStreamWaitEvent(lane(i), fork_ev_, 0), "fork");
  return BV_OK;
}

bv_status Engine::join(int n) {
  for (int i = 1; i < n; ++i) {
    BV_CUDA(cudaEventRecord(side_done_[i - 1], lane(i)), "event");
    BV_CUDA(cudaStreamWaitEvent(stream_, side_done_[i - 1], 0), "join");
  }
  return BV_OK;
}

bv_status Engine::reserve_chunk_offsets(int64_t n) {
  if (n <= chunk_off_cap_) return BV_OK;
  if (h_chunk_off_) {
    BV_CUDA(cudaStreamSynchronize(stream_), "chunk offsets sync");
    cudaFreeHost(h_chunk_off_);
    h_chunk_off_ = nullptr;
    chunk_off_cap_ = 0;
  }
  BV_CUDA(cudaMallocHost(reinterpret_cast<void**>(&h_chunk_off_), sizeof(int64_t) * (size_t)n), "pinned chunk offsets");
  chunk_off_cap_ = n;
  return BV_OK;
}

bv_status Engine::validate(const bv_region_batch& b) { return validate_ranges(b, false); }
bv_status Engine::validate_outline(const bv_region_batch& b) { return validate_ranges(b, true); }

bv_status Engine::validate_ranges(const bv_region_batch& b, bool outline) {
  if (b.num_regions < 0 || b.num_reads < 0 || b.num_haps < 0) return fail(BV_ERR_INVALID_ARG, "negative count");
  if (b.num_regions > 0 && (!b.region_reads || !b.region_haps))
    return fail(BV_ERR_INVALID_ARG, "region offsets missing");
  if (b.num_reads > 0 && (!b.read_offsets)) return fail(BV_ERR_INVALID_ARG, "read offsets missing");
  if (b.num_haps > 0 && (!b.hap_offsets)) return fail(BV_ERR_INVALID_ARG, "hap offsets missing");
  if (b.num_reads >= INT32_MAX || b.num_haps >= INT32_MAX) return fail(BV_ERR_INVALID_ARG, "too many reads or haps");
  for (int64_t g = 0; g < b.num_regions; ++g) {
    if (b.region_reads[g] > b.region_reads[g + 1] || b.region_haps[g] > b.region_haps[g + 1])
      return fail(BV_ERR_INVALID_ARG, "region offsets decrease");
  }
  if (b.num_regions > 0) {
    if (b.region_reads[0] < 0 || b.region_haps[0] < 0 || b.region_reads[b.num_regions] > b.num_reads ||
        b.region_haps[b.num_regions] > b.num_haps)
      return fail(BV_ERR_INVALID_ARG, "region offsets out of range");
  }
  if (b.num_reads > 0) {
    if (b.read_offsets[0] < 0) return fail(BV_ERR_INVALID_ARG, "read offset negative");
    // outline: only the reads outside [region_reads[0], region_reads[num_regions])
    const int64_t skip0 = outline && b.num_regions > 0 ? b.region_reads[0] : b.num_reads;
    const int64_t skip1 = outline && b.num_regions > 0 ? b.region_reads[b.num_regions] : b.num_reads;
    for (int64_t r = 0; r < b.num_reads; ++r) {
      if (r == skip0 && skip1 > skip0) r = skip1;
      if (r >= b.num_reads) break;
      const int64_t l = b.read_offsets[r + 1] - b.read_offsets[r];
      if (l < 0) return fail(BV_ERR_INVALID_ARG, "read offsets decrease");
      if (l > BV_PHMM_MAX_READ_LEN) return fail(BV_ERR_INVALID_ARG, "read longer than BV_PHMM_MAX_READ_LEN");
    }
    const int n_gap_arrays = (b.read_i != nullptr) + (b.read_d != nullptr) + (b.read_c != nullptr);
    if (b.read_offsets[b.num_reads] > 0 && (!b.read_bases || !b.read_q || (n_gap_arrays != 0 && n_gap_arrays != 3)))
      return fail(BV_ERR_INVALID_ARG, "read arrays missing");
  }
  if (b.num_haps > 0) {
    if (b.hap_offsets[0] < 0) return fail(BV_ERR_INVALID_ARG, "hap offset negative");
    const int64_t skip0 = outline && b.num_regions > 0 ? b.region_haps[0] : b.num_haps;
    const int64_t skip1 = outline && b.num_regions > 0 ? b.region_haps[b.num_regions] : b.num_haps;
    for (int64_t h = 0; h < b.num_haps; ++h) {
      if (h == skip0 && skip1 > skip0) h = skip1;
      if (h >= b.num_haps) break;
      const int64_t l = b.hap_offsets[h + 1] - b.hap_offsets[h];
      if (l < 0) return fail(BV_ERR_INVALID_ARG, "hap offsets decrease");
      if (l > BV_PHMM_MAX_HAP_LEN) return fail(BV_ERR_INVALID_ARG, "haplotype longer than BV_PHMM_MAX_HAP_LEN");
    }
    if (b.hap_offsets[b.num_haps] > 0 && !b.hap_bases) return fail(BV_ERR_INVALID_ARG, "hap bases missing");
  }
  return BV_OK;
}

bv_status Engine::plan(const bv_region_batch& b) {
  units_.clear();
  f64_items_.clear();
  f64_long_items_.clear();
  plans_.clear();
  int64_t max_read = 0;
  n_results_ = 0;
  n_cells_ = 0;
  max_hap_ = 0;
  const int max_unit = std::max(1, opt_.haps_per_unit > 0 ? opt_.haps_per_unit : 8);
  const bool all_f64 = opt_.precision == BV_PRECISION_F64;
  const int v_multi = variant_index(false, 8, true);
  std::vector<int64_t> count(kMaxVariants, 0);
  std::vector<int> var_max_hap(kMaxVariants, 0);
  std::fill(bin_reads_, bin_reads_ + 9, 0);
  int64_t n_long = 0, long_rows_sum = 0;  // pairs the long-read kernel may get, and their reads' bases
  // pass 1: count units per variant
  std::vector<int> region_max_hap(std::max<int64_t>(b.num_regions, 1), 0);
  for (int64_t g = 0; g < b.num_regions; ++g) {
    int mh = 0;
    for (int64_t h = b.region_haps[g]; h < b.region_haps[g + 1]; ++h)
      mh = std::max<int>(mh, (int)(b.hap_offsets[h + 1] - b.hap_offsets[h]));
    region_max_hap[g] = mh;
    max_hap_ = std::max(max_hap_, mh);
  }
  // A read's bin: rows per lane of the single-strip kernels (row 0, the read, the summing row and one padding
  // row on top: phmm_device.cuh, rows_needed), kBins for reads of several strips.
  auto bin_of = [](int64_t rlen) { return (int)std::min<int64_t>((rlen + 3 + kWarp - 1) / kWarp, kBins); };
  // Haplotypes per unit: as many as the options allow when the batch still
  // gives every resident warp (about 16 an SM) eight units, so that the last
  // units of a launch do not leave the chip idle; fewer for smaller batches
  // (the row set-up a unit shares is ~1 % of one haplotype's sweep).  An even
  // count of at least two, for the paired kernels; one, with one haplotype per
  // warp, when the pairs do not even fill half the resident warps: a warp then
  // runs alone on its scheduler and only the length of its dependent chain
  // counts.  (FP32 kernels' time, ms, with 8 / 2 / 1 haplotypes a unit, the bins
  // one after the other: 64 reads x 8 haplotypes 0.108 / 0.035 / 0.027; 46 k
  // uneven pairs 2.07 / 1.26 / 1.28; 349 k 7.6 / 6.75 / 7.7, and with the bins
  // side by side 6.59 / 6.50 / 7.56.)
  int64_t n_pairs = 0;
  for (int64_t g = 0; g < b.num_regions; ++g)
    n_pairs += (b.region_reads[g + 1] - b.region_reads[g]) * (b.region_haps[g + 1] - b.region_haps[g]);
  const int64_t warps = (int64_t)sms_ * 16;
  // (FP64 mode: reads that fit a strip run in units too, one haplotype at a time)
  bool few = n_pairs * 2 <= warps && opt_.haps_per_warp != 2 && !band_runs() && !tuning_;
  // ... unless a read's bin was set or tuned to two haplotypes a warp, and they fit
  const bool two_fit = 4 * (4 * hap_bytes_for(max_hap_, 8) + warp_smem_bytes(variant_index(false, kTuneBins, false, true), 0)) <= 227 * 1024;
  for (int64_t g = 0; few && two_fit && g < b.num_regions; ++g)
    for (int64_t r = b.region_reads[g]; few && r < b.region_reads[g + 1]; ++r) {
      const int rt = bin_of(b.read_offsets[r + 1] - b.read_offsets[r]);
      few = !(rt <= kTuneBins && tune_[rt].set && tune_[rt].haps_per_warp == 2);
    }
  const int per_unit = band_runs() ? max_unit
                       : all_f64   ? (int)std::min<int64_t>(max_unit, std::max<int64_t>(1, n_pairs / (warps * 8)))
                       : few       ? 1
                                   : (int)std::min<int64_t>(max_unit, std::max<int64_t>(2, n_pairs / (warps * 8) / 2 * 2));
  // two haplotypes per warp (paired variants) unless the options or the bin's tuning ask for one
  auto pair_rows = [&](int64_t rt) {
    if (opt_.haps_per_warp == 1 || per_unit < 2 || rt < 1 || rt > kTuneBins) return false;
    return opt_.haps_per_warp == 2 || tune_[rt].haps_per_warp == 2;
  };
  int bin_variant[kBins + 1] = {};  // the launch a bin takes
  for (int rt = 1; rt <= kBins; ++rt)
    bin_variant[rt] = all_f64       ? (rt < kBins ? kF64Bin0 + rt : kF64List)
                      : rt == kBins ? v_multi
                                    : variant_index(false, rt, false, pair_rows(rt));
  // pass over the reads: units per bin and, per region, where its units of each bin start
  std::vector<uint32_t>* const base = region_base_;
  for (int rt = 1; rt <= kBins; ++rt) base[rt].clear();
  int64_t res = 0, bin_units[kBins + 1] = {};
  std::vector<int64_t>& res_off = region_res_;
  res_off.assign((size_t)std::max<int64_t>(b.num_regions, 1), 0);
  for (int64_t g = 0; g < b.num_regions; ++g) {
    const int64_t h0 = b.region_haps[g], nh = b.region_haps[g + 1] - h0;
    const int64_t r0 = b.region_reads[g], nr = b.region_reads[g + 1] - r0;
    res_off[g] = res;
    res += nr * nh;
    if (nh == 0 || nr == 0) continue;
    // reads and haplotypes are contiguous
    n_cells_ += (b.read_offsets[r0 + nr] - b.read_offsets[r0]) * (b.hap_offsets[h0 + nh] - b.hap_offsets[h0]);
    const int64_t chunks = (nh + per_unit - 1) / per_unit;
    int64_t cnt[kBins + 1] = {};
    for (int64_t r = r0; r < r0 + nr; ++r) {
      const int64_t rl = b.read_offsets[r + 1] - b.read_offsets[r];
      ++cnt[bin_of(rl)];
      max_read = std::max(max_read, rl);
      if (rl >= long_rows()) {
        n_long += nh;
        long_rows_sum += nh * rl;
      }
    }
    for (int rt = 1; rt <= kBins; ++rt) {
      if (cnt[rt] == 0) continue;
      bin_reads_[rt - 1] += cnt[rt];
      const int v = bin_variant[rt];
      if (v == kF64List) continue;
      if (base[rt].empty()) base[rt].assign((size_t)b.num_regions, 0);
      base[rt][g] = (uint32_t)bin_units[rt];
      bin_units[rt] += cnt[rt] * chunks;
      count[v] += cnt[rt] * chunks;
      var_max_hap[v] = std::max(var_max_hap[v], region_max_hap[g]);
    }
  }
  n_results_ = res;
  for (int rt = 1; rt <= kBins; ++rt)
    if (bin_units[rt] > UINT32_MAX) return fail(BV_ERR_INVALID_ARG, "too many pairs");
  std::vector<int64_t> start(kMaxVariants + 1, 0);
  for (int v = 0; v < kMaxVariants; ++v) start[v + 1] = start[v] + count[v];
  // the units, in result order within each bin: on the device (k_make_units, from the region arrays) or, for a
  // small batch, here; the FP64 list's pairs here
  n_units_ = start[kMaxVariants];
  unit_haps_ = per_unit;
  for (int rt = 1; rt <= kBins; ++rt) bin_start_[rt] = base[rt].empty() || n_units_ == 0 ? -1 : start[bin_variant[rt]];
  const bool lists = all_f64 && bin_reads_[kBins - 1] > 0;
  if (small_in_) units_.resize((size_t)n_units_);
  for (int64_t g = 0; (small_in_ || lists) && g < b.num_regions; ++g) {
    const int64_t h0 = b.region_haps[g], nh = b.region_haps[g + 1] - h0;
    int64_t out = res_off[g], fill[kBins + 1];
    for (int rt = 1; rt <= kBins; ++rt) fill[rt] = bin_start_[rt] < 0 ? 0 : bin_start_[rt] + base[rt][g];
    for (int64_t r = b.region_reads[g]; r < b.region_reads[g + 1]; ++r, out += nh) {
      const int64_t rl = b.read_offsets[r + 1] - b.read_offsets[r];
      const int rt = bin_of(rl);
      if (lists && rt == kBins) {
        auto& list = rl >= long_rows() ? f64_long_items_ : f64_items_;
        for (int64_t k = 0; k < nh; ++k) list.push_back(PairRef{(int32_t)r, (int32_t)(h0 + k), out + k});
        continue;
      }
      for (int64_t k = 0; small_in_ && k < nh; k += per_unit) {
        Unit u{};
        u.read = (int32_t)r;
        u.hap0 = (int32_t)(h0 + k);
        u.nh = (int32_t)std::min<int64_t>(per_unit, nh - k);
        u.out0 = out + k;
        units_[(size_t)fill[rt]++] = u;
      }
    }
  }
  unit_pairs_ = res - (int64_t)(f64_items_.size() + f64_long_items_.size());
  // launch plans
  int slot = 0;
  for (int v = 0; v < kMaxVariants; ++v) {
    if (count[v] == 0) continue;
    LaunchPlan lp;
    lp.variant = v;
    lp.slot = slot++;
    lp.unit_base = start[v];
    lp.n_units = count[v];
    lp.multi = (v == v_multi);
    lp.f64 = v > kF64Bin0;
    if (lp.f64) {
      lp.rows = v - kF64Bin0;
      lp.hap_bytes = hap_bytes_for(var_max_hap[v], 8);
      lp.warp_smem = f64_warp_smem(lp.rows, lp.hap_bytes);
      const int smem = lp.warp_smem * lp.warps_per_block;
      if (smem > 227 * 1024) return fail(BV_ERR_INVALID_ARG, "haplotype too long for shared-memory staging");
      const int64_t need = (count[v] + lp.warps_per_block - 1) / lp.warps_per_block;
      lp.grid = (int)std::min<int64_t>(need, (int64_t)sms_ * std::max(1, f64_blocks_per_sm(lp.rows, smem)));
      plans_.push_back(lp);
      continue;
    }
    lp.code_row_bytes = hap_bytes_for(var_max_hap[v], lp.multi ? 32 : 8);
    // a paired variant stages one 32-bit entry (both haplotypes' table offsets) per column
    lp.hap_bytes = variant_paired(v) ? 4 * lp.code_row_bytes : lp.code_row_bytes;
    lp.warp_smem = warp_smem_bytes(v, lp.hap_bytes);
    {
      // the bin's block size (rows per lane of a single-strip FP32 variant)
      int rt = 0;
      for (int t = 1; t <= kTuneBins; ++t)
        if (v == variant_index(false, t, false, false) || v == variant_index(false, t, false, true)) rt = t;
      lp.rows = rt;
      lp.warps_per_block = rt ? tune_[rt].warps_per_block : kThreadsPerBlock / kWarp;
    }
    const int smem_block = lp.warp_smem * lp.warps_per_block;
    if (lp.warp_smem * (kThreadsPerBlock / kWarp) > 227 * 1024)
      return fail(BV_ERR_INVALID_ARG, "haplotype too long for shared-memory staging");
    BV_CUDA(prepare_variant(v, lp.warp_smem * (kThreadsPerBlock / kWarp)), "kernel attribute");
    const int bps = std::max(1, blocks_per_sm(v, smem_block, lp.warps_per_block * kWarp));
    const int64_t need = (count[v] + lp.warps_per_block - 1) / lp.warps_per_block;
    lp.grid = (int)std::max<int64_t>(1, std::min<int64_t>(need, (int64_t)sms_ * bps));
    lp.bnd_cols = lp.multi ? bnd_cols_for(var_max_hap[v]) : 0;
    plans_.push_back(lp);
  }
  // The launches run beside each other (enqueue_kernels), the ones with the
  // longest units first: the shorter ones then fill their last waves.
  std::stable_sort(plans_.begin(), plans_.end(), [&](const LaunchPlan& x, const LaunchPlan& y) {
    return x.multi != y.multi ? x.multi : x.rows > y.rows;
  });
  if (bv_status ls = reserve_lanes(std::min((int)plans_.size(), kMaxLanes)); ls != BV_OK) return ls;
  // FP64 list: persistent over the whole device, whatever the other passes send there
  LaunchPlan rp;
  rp.multi = true;
  rp.f64 = true;
  rp.hap_bytes = hap_bytes_for(std::max(max_hap_, 1), 32);
  rp.warp_smem = f64_warp_smem(0, rp.hap_bytes);
  const int smem_block = rp.warp_smem * (kThreadsPerBlock / kWarp);
  if (smem_block > 227 * 1024) return fail(BV_ERR_INVALID_ARG, "haplotype too long for shared-memory staging");
  // (no more warps than pairs: an empty list after 60 pairs takes 4 instead of 8 us)
  rp.grid = (int)std::min<int64_t>((int64_t)sms_ * std::max(1, f64_blocks_per_sm(0, smem_block)),
                                   std::max<int64_t>(1, (n_results_ + kThreadsPerBlock / kWarp - 1) / (kThreadsPerBlock / kWarp)));
  rp.bnd_cols = bnd_cols_for(std::max(max_hap_, 1));
  rescue_plan_ = rp;
  // FP64 long reads: one block per pair, longest pairs first (the long list is
  // read from its far end, so the host list is in ascending order of cells).
  // The block's warps, unless they are set: twice as many while the pairs then
  // still fit the device's resident warps (16 an SM) at once and the longest
  // read has strips for them -- a pair then ends sooner -- and while the
  // average read gives every warp at least two strips.  FP64 pass, ms, with
  // 4 / 8 / 16 warps: 40 reads of up to 10 kb 28 / 17 / 12, 2000 of them 86 / 79 /
  // 77, 3000 of up to 1.5 kb 8.7 / 9.3 / 10.3, 400 of 400 bases 0.47 / 0.65 / 0.82.
  long_plan_ = LaunchPlan{};
  if (max_read >= long_rows() && n_long > 0) {
    const int64_t strips = (max_read + 1 + 127) / 128, strips_mean = long_rows_sum / n_long / 128 + 1;
    long_block_ = long_set_ ? long_warps_ : 2;
    while (!long_set_ && long_block_ < 16 &&
           ((2 * long_block_ * n_long <= warps && long_block_ < strips) || 4 * long_block_ <= strips_mean))
      long_block_ *= 2;
    long_smem_ = long_smem_bytes(rp.hap_bytes, long_block_);
    if (long_smem_ <= 227 * 1024) {
      // Up to a few hundred pairs: a cluster of blocks for each, the blocks dealt by the pairs' costs (long_cost):
      // the lowest limit for which all pairs' blocks together are at most the SMs (but eight: a cluster's have to be
      // neighbours, and one that finds no place waits for the others: 40 pairs 4.4-4.8 instead of 3.5-3.7 ms), or
      // 2/5 of them more than there are pairs.  FP64 pass of reads of up to 10 kb, one block a pair -> this, ms: 40 pairs 11.1 -> 3.7, 90 12.2 ->
      // 6.0, 148 11.9 -> 9.6, 256 15.9 -> 11.5, 512 25.7 -> 20.1 (one cluster size for all pairs: 40 pairs 6.8, 90
      // 12.2; totals of 112 to 400 blocks tried at 40 to 256 pairs).  Pairs of one length get a block each: then,
      // and beyond, the blocks take the next pair from the list.
      std::fill(long_grid_, long_grid_ + 4, 0);
      int64_t budget = 0;
      if (long_block_ == 16 && !long_set_ && n_long <= kLongMembers)
        budget = std::max<int64_t>(sms_ - 8, n_long + sms_ * 2 / 5);
      if (n_long <= budget) {
        std::vector<std::pair<int64_t, int64_t>> pairs;  // read and haplotype lengths
        std::vector<long long> limits;
        for (int64_t g = 0; g < b.num_regions; ++g)
          for (int64_t r = b.region_reads[g]; r < b.region_reads[g + 1]; ++r) {
            const int64_t rl = b.read_offsets[r + 1] - b.read_offsets[r];
            for (int64_t h = b.region_haps[g]; rl >= long_rows() && h < b.region_haps[g + 1]; ++h) {
              pairs.emplace_back(rl, b.hap_offsets[h + 1] - b.hap_offsets[h]);
              for (int c = 1; c <= kLongMaxBlocks; c *= 2) limits.push_back(long_cost(rl, pairs.back().second, c));
            }
          }
        std::sort(limits.begin(), limits.end());
        auto blocks = [&](long long limit) {
          int64_t n = 0;
          for (const auto& [rl, hl] : pairs) n += long_blocks(rl, hl, limit);
          return n;
        };
        long_limit_ = *std::partition_point(limits.begin(), limits.end() - 1, [&](long long t) { return blocks(t) > budget; });
        for (const auto& [rl, hl] : pairs) {
          const int c = long_blocks(rl, hl, long_limit_);
          long_grid_[c == 8 ? 0 : c == 4 ? 1 : c == 2 ? 2 : 3] += c;
        }
        if (long_grid_[3] == n_long) long_grid_[3] = 0;
      }
      long_plan_.grid = std::accumulate(long_grid_, long_grid_ + 4, 0);
      if (long_plan_.grid > 0) {
        BV_CUDA(prepare_long(long_smem_, long_block_, 1), "kernel attribute");
        if (bv_status ls = reserve_lanes(4); ls != BV_OK) return ls;
      } else {
        BV_CUDA(prepare_long(long_smem_, long_block_, 0), "kernel attribute");
        long_plan_.grid = (int)std::min<int64_t>(n_long, (int64_t)sms_ * std::max(1, long_blocks_per_sm(long_smem_, long_block_)));
      }
      long_plan_.hap_bytes = rp.hap_bytes;
      long_plan_.bnd_cols = rp.bnd_cols;
      long_plan_.f64 = true;
      long_plan_.multi = true;
    }
  }
  if (long_plan_.grid == 0) {  // no long kernel: the long reads stay on k_f64_list
    f64_items_.insert(f64_items_.end(), f64_long_items_.begin(), f64_long_items_.end());
    f64_long_items_.clear();
  }
  auto cells = [&](const PairRef& x) {
    return (b.read_offsets[x.read + 1] - b.read_offsets[x.read]) * (b.hap_offsets[x.hap + 1] - b.hap_offsets[x.hap]);
  };
  std::sort(f64_long_items_.begin(), f64_long_items_.end(),
            [&](const PairRef& x, const PairRef& y) { return cells(x) < cells(y); });
  return BV_OK;
}

bv_status Engine::reserve_host() {
  if (h_counters_) return BV_OK;
  unsigned char* p = nullptr;
  BV_CUDA(cudaMallocHost(reinterpret_cast<void**>(&p), kCountersBytes + kSmallOutBytes + kStageBytes), "pinned buffers");
  h_counters_ = reinterpret_cast<Counters*>(p);
  h_stage_ = p + kCountersBytes + kSmallOutBytes;
  return BV_OK;
}

// The next piece of the staged image: its host place, `dev` viewing its place
// on the device; nullptr when the image is full.
void* Engine::stage_piece(size_t bytes, DevBuf& dev) {
  const size_t at = stage_used_;
  const size_t end = (at + bytes + 255) / 256 * 256;
  if (end > kStageBytes) return nullptr;
  stage_used_ = end;
  dev.view(d_stage_.as<unsigned char>() + at);
  return h_stage_ + at;
}

// A small batch's inputs into the image (upload_plan sends it).
bv_status Engine::stage_inputs(const bv_region_batch& b) {
  if (bv_status s = reserve_host(); s != BV_OK) return s;
  BV_CUDA(d_stage_.reserve(kStageBytes), "alloc inputs");
  stage_used_ = 0;
  const size_t rb = (size_t)n_read_bytes_, hb = (size_t)n_hap_bytes_;
  auto put = [&](DevBuf& dev, const void* src, size_t bytes, size_t room) {
    void* p = stage_piece(room, dev);
    if (bytes) std::memcpy(p, src, bytes);
  };
  put(d_read_off_, b.read_offsets, n_reads_ > 0 ? sizeof(int64_t) * (n_reads_ + 1) : 0, sizeof(int64_t) * (n_reads_ + 1));
  put(d_hap_off_, b.hap_offsets, n_haps_ > 0 ? sizeof(int64_t) * (n_haps_ + 1) : 0, sizeof(int64_t) * (n_haps_ + 1));
  put(d_read_bases_, b.read_bases, rb, rb + 16);  // tail padding for the k-mer kernel's word loads
  put(d_hap_bases_, b.hap_bases, hb, hb + 16);
  uchar4* q = static_cast<uchar4*>(stage_piece(4 * rb + 16, d_quals4_));
  size_t x = 0;
  const __m128i gi = _mm_set1_epi8((char)gap_ins_), gd = _mm_set1_epi8((char)gap_del_), gc = _mm_set1_epi8((char)gap_gcp_);
  auto load = [&](const uint8_t* p) { return _mm_loadu_si128(reinterpret_cast<const __m128i*>(p + x)); };
  for (; x + 16 <= rb; x += 16) {  // 16 bases' four qualities interleaved
    const __m128i vq = load(b.read_q), vi = uniform_gaps_ ? gi : load(b.read_i);
    const __m128i vd = uniform_gaps_ ? gd : load(b.read_d), vc = uniform_gaps_ ? gc : load(b.read_c);
    const __m128i qi0 = _mm_unpacklo_epi8(vq, vi), qi1 = _mm_unpackhi_epi8(vq, vi);
    const __m128i dc0 = _mm_unpacklo_epi8(vd, vc), dc1 = _mm_unpackhi_epi8(vd, vc);
    __m128i* o = reinterpret_cast<__m128i*>(q + x);
    _mm_store_si128(o, _mm_unpacklo_epi16(qi0, dc0));
    _mm_store_si128(o + 1, _mm_unpackhi_epi16(qi0, dc0));
    _mm_store_si128(o + 2, _mm_unpacklo_epi16(qi1, dc1));
    _mm_store_si128(o + 3, _mm_unpackhi_epi16(qi1, dc1));
  }
  for (; x < rb; ++x)
    q[x] = uniform_gaps_ ? uchar4{b.read_q[x], gap_ins_, gap_del_, gap_gcp_}
                         : uchar4{b.read_q[x], b.read_i[x], b.read_d[x], b.read_c[x]};
  return BV_OK;
}

// Inputs: the byte arrays and offsets go to the device as soon as the batch
// is validated.  From page-locked arrays the copies run while the host plans the
// launches; from pageable ones a copy holds the host until it is staged (0.2 ms
// for 48 uneven regions, 1.1 for 256).
bv_status Engine::upload_inputs(const bv_region_batch& b) {
  n_reads_ = b.num_reads;
  n_haps_ = b.num_haps;
  n_read_bytes_ = b.num_reads > 0 ? b.read_offsets[b.num_reads] : 0;
  n_hap_bytes_ = b.num_haps > 0 ? b.hap_offsets[b.num_haps] : 0;
  const size_t rb = (size_t)std::max<int64_t>(n_read_bytes_, 1);
  // uniform gap penalties: no per-base i, d, c arrays to copy (see bv_region_batch)
  uniform_gaps_ = !b.read_i && !b.read_d && !b.read_c;
  gap_ins_ = b.gap_ins;
  gap_del_ = b.gap_del;
  gap_gcp_ = b.gap_gcp;
  small_in_ = 5 * rb + (size_t)n_hap_bytes_ + sizeof(int64_t) * (size_t)(n_reads_ + n_haps_ + 2) + 2048 <= kStageBytes;
  if (small_in_) return stage_inputs(b);
  // one allocation for all of them: a new context's first call, and one that grows its buffers, pays for
  // one instead of nine
  size_t total = 0;
  for (int pass = 0; pass < 2; ++pass) {
    if (pass == 1) BV_CUDA(d_inputs_.reserve(total), "alloc inputs");
    total = 0;
    auto piece = [&](DevBuf& dev, size_t bytes) {
      if (pass == 1) dev.view(d_inputs_.as<unsigned char>() + total);
      total += (bytes + 255) / 256 * 256;
    };
    piece(d_read_bases_, rb + 16);  // tail padding for the k-mer kernel's word loads
    piece(d_q_, rb);
    if (!uniform_gaps_) {
      piece(d_i_, rb);
      piece(d_d_, rb);
      piece(d_c_, rb);
    }
    piece(d_quals4_, rb * 4);
    piece(d_read_off_, sizeof(int64_t) * (n_reads_ + 1));
    piece(d_hap_bases_, (size_t)std::max<int64_t>(n_hap_bytes_, 1));
    piece(d_hap_off_, sizeof(int64_t) * (n_haps_ + 1));
  }
  BV_CUDA(cudaEventRecord(ev_[0], stream_), "event");
  // Offsets are copied verbatim; the byte arrays are copied from index 0 so
  // offsets index them directly.
  if (n_read_bytes_ > 0) {
    BV_CUDA(cudaMemcpyAsync(d_read_bases_.get(), b.read_bases, n_read_bytes_, cudaMemcpyHostToDevice, stream_), "H2D");
    BV_CUDA(cudaMemcpyAsync(d_q_.get(), b.read_q, n_read_bytes_, cudaMemcpyHostToDevice, stream_), "H2D");
    if (!uniform_gaps_) {
      BV_CUDA(cudaMemcpyAsync(d_i_.get(), b.read_i, n_read_bytes_, cudaMemcpyHostToDevice, stream_), "H2D");
      BV_CUDA(cudaMemcpyAsync(d_d_.get(), b.read_d, n_read_bytes_, cudaMemcpyHostToDevice, stream_), "H2D");
      BV_CUDA(cudaMemcpyAsync(d_c_.get(), b.read_c, n_read_bytes_, cudaMemcpyHostToDevice, stream_), "H2D");
    }
  }
  if (n_reads_ > 0)
    BV_CUDA(cudaMemcpyAsync(d_read_off_.get(), b.read_offsets, sizeof(int64_t) * (n_reads_ + 1), cudaMemcpyHostToDevice,
                            stream_), "H2D");
  if (n_hap_bytes_ > 0)
    BV_CUDA(cudaMemcpyAsync(d_hap_bases_.get(), b.hap_bases, n_hap_bytes_, cudaMemcpyHostToDevice, stream_), "H2D");
  if (n_haps_ > 0)
    BV_CUDA(cudaMemcpyAsync(d_hap_off_.get(), b.hap_offsets, sizeof(int64_t) * (n_haps_ + 1), cudaMemcpyHostToDevice,
                            stream_), "H2D");
  return BV_OK;
}

// The plan's device side: work units, result and list buffers, and the packed
// qualities.  Nothing here waits for the copies; run() reads the copy time
// once its own synchronisation has passed.
bv_status Engine::upload_plan(const bv_region_batch& b) {
  bool units_staged = false;
  stage_launches_ = small_in_ ? 0 : (n_units_ > 0) + (n_read_bytes_ > 0);  // units, packed qualities
  if (small_in_) {
    const size_t bytes = sizeof(Unit) * units_.size();
    if (void* p = stage_piece(std::max<size_t>(bytes, 1), d_units_)) {
      if (bytes) std::memcpy(p, units_.data(), bytes);
      units_staged = true;
    }
    BV_CUDA(cudaEventRecord(ev_[0], stream_), "event");
    BV_CUDA(cudaMemcpyAsync(d_stage_.get(), h_stage_, stage_used_, cudaMemcpyHostToDevice, stream_), "H2D");
  }
  if (!units_staged) BV_CUDA(d_units_.reserve(sizeof(Unit) * (size_t)std::max<int64_t>(n_units_, 1)), "alloc units");
  small_out_ = sizeof(double) * (size_t)n_results_ <= kSmallOutBytes;
  if (small_out_) d_out_.view(d_counters_.as<unsigned char>() + kCountersBytes);
  else BV_CUDA(d_out_.reserve(sizeof(double) * (size_t)std::max<int64_t>(n_results_, 1)), "alloc results");
  BV_CUDA(d_rescue_.reserve(sizeof(PairRef) * (size_t)std::max<int64_t>(n_results_, 1)), "alloc rescue list");
  // strip-boundary buffers for the multi-strip launches
  size_t need32 = 0;
  for (const auto& lp : plans_)
    if (lp.multi) need32 = std::max<size_t>(need32, (size_t)lp.grid * lp.warps_per_block * (size_t)lp.bnd_cols * 4 * sizeof(float));
  if (need32) BV_CUDA(d_bnd32_.reserve(need32), "alloc boundary buffers");
  const size_t need64 = std::max((size_t)rescue_plan_.grid * (kThreadsPerBlock / kWarp) * (size_t)rescue_plan_.bnd_cols,
                                 (size_t)long_plan_.grid * (size_t)long_plan_.bnd_cols) * 4 * sizeof(double);
  BV_CUDA(d_bnd64_.reserve(need64), "alloc FP64 boundary buffers");
  if (small_in_ && !units_staged && n_units_ > 0)
    BV_CUDA(cudaMemcpyAsync(d_units_.get(), units_.data(), sizeof(Unit) * units_.size(), cudaMemcpyHostToDevice,
                            stream_), "H2D");
  if (!small_in_ && n_units_ > 0) {
    // the region arrays in one copy: reads, haplotypes and results before each region, unit bases per bin
    const size_t ng = (size_t)b.num_regions;
    MakeUnits m{};
    m.n_regions = b.num_regions;
    m.per_unit = unit_haps_;
    int bins = 0;
    for (int rt = 1; rt <= kBins; ++rt) {
      m.column[rt] = bin_start_[rt] < 0 ? -1 : bins;
      if (bin_start_[rt] >= 0) m.start[bins++] = bin_start_[rt];
    }
    const size_t bytes = sizeof(int64_t) * (3 * ng + 2) + sizeof(uint32_t) * ng * (size_t)bins;
    region_img_.resize(bytes);
    unsigned char* p = region_img_.data();
    auto put = [&](const void* src, size_t n) {
      std::memcpy(p, src, n);
      p += n;
    };
    put(b.region_reads, sizeof(int64_t) * (ng + 1));
    put(b.region_haps, sizeof(int64_t) * (ng + 1));
    put(region_res_.data(), sizeof(int64_t) * ng);
    for (int rt = 1; rt <= kBins; ++rt)
      if (bin_start_[rt] >= 0) put(region_base_[rt].data(), sizeof(uint32_t) * ng);
    BV_CUDA(d_regions_.reserve(bytes), "alloc regions");
    BV_CUDA(cudaMemcpyAsync(d_regions_.get(), region_img_.data(), bytes, cudaMemcpyHostToDevice, stream_), "H2D");
    m.region_reads = d_regions_.as<int64_t>();
    m.region_haps = m.region_reads + ng + 1;
    m.region_res = m.region_haps + ng + 1;
    m.base = reinterpret_cast<const uint32_t*>(m.region_res + ng);
    m.read_off = d_read_off_.as<int64_t>();
    m.units = d_units_.as<Unit>();
    BV_CUDA(launch_make_units(m, sms_, stream_), "units");
  }
  if (!f64_items_.empty())
    BV_CUDA(cudaMemcpyAsync(d_rescue_.get(), f64_items_.data(), sizeof(PairRef) * f64_items_.size(),
                            cudaMemcpyHostToDevice, stream_), "H2D");
  if (!f64_long_items_.empty())  // at the list's far end
    BV_CUDA(cudaMemcpyAsync(d_rescue_.as<PairRef>() + (std::max<int64_t>(n_results_, 1) - (int64_t)f64_long_items_.size()),
                            f64_long_items_.data(), sizeof(PairRef) * f64_long_items_.size(), cudaMemcpyHostToDevice,
                            stream_), "H2D");
  if (small_in_) {  // packed in the image
  } else if (uniform_gaps_)
    BV_CUDA(launch_pack_quals_uniform(d_q_.as<uint8_t>(), gap_ins_, gap_del_, gap_gcp_, d_quals4_.as<uchar4>(),
                                      n_read_bytes_, sms_, stream_), "pack quals");
  else
    BV_CUDA(launch_pack_quals(d_q_.as<uint8_t>(), d_i_.as<uint8_t>(), d_d_.as<uint8_t>(), d_c_.as<uint8_t>(),
                              d_quals4_.as<uchar4>(), n_read_bytes_, sms_, stream_), "pack quals");
  BV_CUDA(cudaEventRecord(ev_[1], stream_), "event");
  h2d_time_pending_ = true;
  return BV_OK;
}

// The caller's host arrays are borrowed for the call: unless the caller runs
// the batch before returning (compute, whose run synchronises), stage waits
// for the copies, and every error path after the first copy waits for them too.
bv_status Engine::stage(const bv_region_batch& b, bool wait) {
  staged_ = false;
  destroy_graph();
  BV_CUDA(cudaSetDevice(opt_.device), "cudaSetDevice");
  bv_status s = validate(b);
  if (s != BV_OK) return s;
  s = upload_inputs(b);
  if (s == BV_OK) s = plan(b);
  if (s == BV_OK) s = upload_plan(b);
  if (s == BV_OK && band_runs()) s = band_prepare();
  if (s != BV_OK) {
    cudaStreamSynchronize(stream_);
    return s;
  }
  if (wait) BV_CUDA(cudaStreamSynchronize(stream_), "stage sync");
  staged_ = true;
  runs_since_stage_ = 0;
  return BV_OK;
}

// The staged bins' launches (of FP32 units, or of FP64 mode's).
bv_status Engine::enqueue_plans(bool capturing, bool f64, KernelParams& p) {
  if (band_runs() || plans_.empty() || plans_[0].f64 != f64) return BV_OK;
  if (tune_timing_ && !capturing) {
    while (tune_ev_.size() < 2 * plans_.size()) {
      cudaEvent_t e;
      BV_CUDA(cudaEventCreate(&e), "event");
      tune_ev_.push_back(e);
    }
  }
  // The bins side by side on the lanes' streams (one after the other while the
  // tuner times them): 48 uneven regions' eight bins, 46 k pairs, take 0.96
  // instead of 1.26 ms, since no bin waits for the last warps of another.
  const bool timed = tune_timing_ && !capturing;
  const int lanes = timed ? 1 : std::min((int)plans_.size(), kMaxLanes);
  if (bv_status fs = fork(lanes); fs != BV_OK) return fs;
  cudaError_t le = cudaSuccess;  // a failed launch still joins the lanes that started
  for (size_t pi = 0; pi < plans_.size(); ++pi) {
    const LaunchPlan& lp = plans_[pi];
    if (lp.f64 != f64) continue;
    if (timed) BV_CUDA(cudaEventRecord(tune_ev_[2 * pi], stream_), "event");
    p.unit_base = lp.unit_base;
    p.n_units = lp.n_units;
    p.slot = lp.slot;
    p.hap_bytes = lp.hap_bytes;
    p.code_row_bytes = lp.code_row_bytes;
    p.warps_per_block = lp.warps_per_block;
    p.warp_smem_bytes = lp.warp_smem;
    p.bnd = lp.multi ? d_bnd32_.get() : nullptr;
    p.bnd_cols = lp.bnd_cols;
    p.rescale = 0;
    p.rescale_target = 0;
    const cudaStream_t st = lane((int)pi % lanes);
    le = f64 ? launch_f64(lp.rows, p, lp.grid, st) : launch_forward(lp.variant, p, lp.grid, st);
    if (le != cudaSuccess) break;
    if (timed) BV_CUDA(cudaEventRecord(tune_ev_[2 * pi + 1], stream_), "event");
  }
  if (bv_status js = join(lanes); js != BV_OK) return js;
  BV_CUDA(le, "forward launch");
  return BV_OK;
}

bv_status Engine::enqueue_kernels(bool capturing) {
  // Inside stream capture, timing events become event-record nodes of the
  // graph only when recorded as external events.
  auto rec = [&](cudaEvent_t ev) {
    return capturing ? cudaEventRecordWithFlags(ev, stream_, cudaEventRecordExternal) : cudaEventRecord(ev, stream_);
  };
  BV_CUDA(cudaMemsetAsync(d_counters_.get(), 0, sizeof(Counters), stream_), "memset counters");
  if (!f64_items_.empty()) {
    BV_CUDA(launch_set_u64(&d_counters_.as<Counters>()->rescue_count, (unsigned long long)f64_items_.size(), stream_),
            "set FP64 count");
  }
  if (!f64_long_items_.empty()) {
    BV_CUDA(launch_set_u64(&d_counters_.as<Counters>()->rescue_long_count, (unsigned long long)f64_long_items_.size(),
                           stream_), "set FP64 count");
  }
  KernelParams p{};
  p.batch.read_bases = d_read_bases_.as<uint8_t>();
  p.batch.read_quals = d_quals4_.as<uchar4>();
  p.batch.read_off = d_read_off_.as<int64_t>();
  p.batch.hap_bases = d_hap_bases_.as<uint8_t>();
  p.batch.hap_off = d_hap_off_.as<int64_t>();
  p.tables = d_tables_.as<Tables>();
  p.units = d_units_.as<Unit>();
  p.ctr = d_counters_.as<Counters>();
  p.out = d_out_.as<double>();
  p.rescue = d_rescue_.as<PairRef>();
  p.rescue_cap = std::max<int64_t>(n_results_, 1);
  p.long_rows = long_plan_.grid > 0 ? long_rows() : 0;
  p.warps_per_block = kThreadsPerBlock / kWarp;  // band-path fallback and audit launches
  BV_CUDA(rec(ev_[2]), "event");
  if (band_runs()) {
    bv_status bs = enqueue_band(capturing, p);
    if (bs != BV_OK) return bs;
  }
  if (bv_status ps = enqueue_plans(capturing, false, p); ps != BV_OK) return ps;
  BV_CUDA(rec(ev_[3]), "event");
  if (bv_status ps = enqueue_plans(capturing, true, p); ps != BV_OK) return ps;
  {
    const LaunchPlan& lp = rescue_plan_;
    p.unit_base = 0;
    p.n_units = 0;
    p.hap_bytes = lp.hap_bytes;
    p.code_row_bytes = 0;
    p.warps_per_block = kThreadsPerBlock / kWarp;
    p.warp_smem_bytes = lp.warp_smem;
    p.bnd = d_bnd64_.get();
    p.bnd_cols = lp.bnd_cols;
    p.rescale = 1;
    p.rescale_target = kRescaleTarget;
    p.cells_ctr = &d_counters_.as<Counters>()->rescued_cells;
    if (long_plan_.grid > 0) {  // long reads first: a block per pair, longest first
      KernelParams q = p;
      q.hap_bytes = long_plan_.hap_bytes;
      q.bnd_cols = long_plan_.bnd_cols;
      if (long_grid_[0] + long_grid_[1] + long_grid_[2] + long_grid_[3] == 0) {
        BV_CUDA(launch_forward_long(q, long_plan_.grid, long_smem_, long_block_, 0, stream_), "FP64 long-read launch");
      } else {  // the largest clusters first, the smaller ones beside them
        q.long_cost = long_limit_;
        if (bv_status fs = fork(4); fs != BV_OK) return fs;
        cudaError_t le = cudaSuccess;  // a failed launch still joins the lanes that started
        for (int k = 0; k < 4 && le == cudaSuccess; ++k) {
          if (long_grid_[k] == 0) continue;
          le = launch_forward_long(q, long_grid_[k], long_smem_, long_block_, 8 >> k, lane(k));
          q.bnd = static_cast<unsigned char*>(q.bnd) + (size_t)long_grid_[k] * (size_t)q.bnd_cols * 4 * sizeof(double);
        }
        if (bv_status js = join(4); js != BV_OK) return js;
        BV_CUDA(le, "FP64 long-read launch");
      }
    }
    BV_CUDA(launch_f64(0, p, lp.grid, stream_), "FP64 forward launch");
    p.cells_ctr = nullptr;
  }
  BV_CUDA(rec(ev_[4]), "event");
  if (band_runs() && band_opt_.audit_period > 0) {
    BV_CUDA(launch_audit_compare(band_params(), d_audit_err_.as<double>(), stream_), "audit compare");
  }
  return BV_OK;
}

void Engine::destroy_graph() {
  if (graph_exec_) cudaGraphExecDestroy(graph_exec_);
  if (graph_) cudaGraphDestroy(graph_);
  graph_exec_ = nullptr;
  graph_ = nullptr;
}

bv_status Engine::run(bv_phmm_stats* stats) {
  bv_status s = launch();
  if (s != BV_OK) return s;
  return finish(stats);
}

bv_status Engine::launch(int64_t n_out) {
  if (!staged_) return fail(BV_ERR_INVALID_ARG, "no staged batch");
  BV_CUDA(cudaSetDevice(opt_.device), "cudaSetDevice");
  run_t0_ = std::chrono::steady_clock::now();
  if (bv_status hs = reserve_host(); hs != BV_OK) return hs;
  // The first run of a staged batch launches directly; later runs replay a
  // captured graph of the same launch sequence.
  if (runs_since_stage_ == 0 || !graph_exec_) {
    if (runs_since_stage_ >= 1 && !graph_exec_) {
      BV_CUDA(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal), "begin capture");
      bv_status s = enqueue_kernels(true);
      cudaGraph_t g = nullptr;
      cudaError_t ce = cudaStreamEndCapture(stream_, &g);
      if (s != BV_OK) {
        if (g) cudaGraphDestroy(g);
        return s;
      }
      BV_CUDA(ce, "end capture");
      graph_ = g;
      BV_CUDA(cudaGraphInstantiate(&graph_exec_, graph_, 0), "graph instantiate");
      BV_CUDA(cudaGraphLaunch(graph_exec_, stream_), "graph launch");
    } else {
      bv_status s = enqueue_kernels(false);
      if (s != BV_OK) return s;
    }
  } else {
    BV_CUDA(cudaGraphLaunch(graph_exec_, stream_), "graph launch");
  }
  ++runs_since_stage_;
  // page-locked destination: the copy is queued, the host goes on
  const size_t back = n_out > 0 ? kCountersBytes + sizeof(double) * (size_t)n_out : sizeof(Counters);
  // A small batch's come back by a kernel: a copy engine's start and end cost 8 us more.  Not beside large
  // batches, whose persistent blocks it would queue behind.
  if (small_in_) BV_CUDA(launch_copy_small(d_counters_.get(), h_counters_, back, stream_), "counters D2H");
  else BV_CUDA(cudaMemcpyAsync(h_counters_, d_counters_.get(), back, cudaMemcpyDeviceToHost, stream_), "counters D2H");
  return BV_OK;
}

bv_status Engine::finish(bv_phmm_stats* stats) {
  BV_CUDA(cudaStreamSynchronize(stream_), "run sync");
  if (h2d_time_pending_) {
    BV_CUDA(cudaEventElapsedTime(&ms_h2d_, ev_[0], ev_[1]), "event time");
    h2d_time_pending_ = false;
  }
  const Counters c = *h_counters_;
  if (c.status != 0) return status_fail(c.status);
  if (stats) *stats = bv_phmm_stats{};
  if (stats && band_runs()) {
    bv_status bs = band_stats(stats);
    if (bs != BV_OK) return bs;
  }
  if (stats) {
    float ms32 = 0, ms64 = 0;
    cudaEventElapsedTime(&ms32, ev_[2], ev_[3]);
    cudaEventElapsedTime(&ms64, ev_[3], ev_[4]);
    stats->pairs = n_results_;
    stats->cells = n_cells_;
    stats->rescued = (int64_t)(c.rescue_count + c.rescue_long_count);
    stats->rescued_cells = (int64_t)c.rescued_cells;
    if (opt_.precision == BV_PRECISION_F64) {  // every pair, on the list or in units
      stats->rescued = n_results_;
      stats->rescued_cells = n_cells_;
    }
    stats->fp32_skipped_cells = (int64_t)c.fp32_skipped_cells;
    stats->underflow = (int64_t)c.underflow_count;
    const int clusters = (int)(4 - std::count(long_grid_, long_grid_ + 4, 0));
    const int long_launches = long_plan_.grid == 0 ? 0 : clusters > 0 ? clusters : 1;
    // band mode: k-mer tables, nibble image, read k-mers, gap check, two featurisers, MLP, route,
    // scan, route; the banded kernels; the fallback's units and bins; the rescore's;
    // the audit's; the FP64 pass
    // (in both modes: the FP64 lists' counts, and a small batch's way back)
    const int small_launches = !f64_items_.empty() + !f64_long_items_.empty() + small_in_;
    stats->kernel_launches = band_runs()
                                 ? 9 + (band_opt_.use_mlp ? 1 : 0) + kBandWidths + 1 + full_bins_ +
                                       (band_opt_.cap_margin > 0 ? 1 + full_bins_ : 0) +
                                       (band_opt_.audit_period > 0 ? 2 + full_bins_ : 0) + 1 + long_launches + small_launches
                                 : (int64_t)plans_.size() + 1 + long_launches + small_launches;
    stats->ms_fp32 = ms32;
    stats->ms_fp64 = ms64;
    if (band_runs()) {
      float seed = 0, band = 0, full = 0;
      cudaEventElapsedTime(&seed, ev_[2], ev_[5]);
      cudaEventElapsedTime(&band, ev_[5], ev_[6]);
      cudaEventElapsedTime(&full, ev_[6], ev_[3]);
      stats->ms_seed = seed;
      stats->ms_band = band;
      stats->ms_full = full;
    } else {
      stats->ms_full = ms32;
    }
    stats->ms_h2d = ms_h2d_;
    stats->ms_total =
        std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - run_t0_).count();
  }
  return BV_OK;
}

bv_status Engine::fetch(double* out, int64_t n) {
  if (!staged_) return fail(BV_ERR_INVALID_ARG, "no staged batch");
  if (n < 0 || n > n_results_) return fail(BV_ERR_INVALID_ARG, "fetch size exceeds staged results");
  if (n == 0) return BV_OK;
  if (!out) return fail(BV_ERR_INVALID_ARG, "null output");
  BV_CUDA(cudaMemcpyAsync(out, d_out_.get(), sizeof(double) * n, cudaMemcpyDeviceToHost, stream_), "results D2H");
  BV_CUDA(cudaStreamSynchronize(stream_), "fetch sync");
  return BV_OK;
}

bv_status Engine::fetch_async(double* out, int64_t n) {
  if (!staged_) return fail(BV_ERR_INVALID_ARG, "no staged batch");
  if (n < 0 || n > n_results_) return fail(BV_ERR_INVALID_ARG, "fetch size exceeds staged results");
  if (n == 0) return BV_OK;
  if (!out) return fail(BV_ERR_INVALID_ARG, "null output");
  BV_CUDA(cudaMemcpyAsync(out, d_out_.get(), sizeof(double) * n, cudaMemcpyDeviceToHost, stream_), "results D2H");
  return BV_OK;
}

bv_status Engine::compute(const bv_region_batch& b, double* out, bv_phmm_stats* stats) {
  const auto t0 = std::chrono::steady_clock::now();
  if (!out && b.num_regions > 0) {
    // checked before any copy starts (a batch with results needs an output)
    bv_status v = validate(b);
    if (v != BV_OK) return v;
    int64_t res = 0;
    for (int64_t g = 0; g < b.num_regions; ++g)
      res += (b.region_reads[g + 1] - b.region_reads[g]) * (b.region_haps[g + 1] - b.region_haps[g]);
    if (res > 0) return fail(BV_ERR_INVALID_ARG, "null output");
  }
  bv_status s = stage(b, false);  // run() synchronises before this call returns
  if (s != BV_OK) return s;
  s = launch(small_out_ ? n_results_ : 0);
  if (s == BV_OK) s = finish(stats);
  if (s != BV_OK) {
    cudaStreamSynchronize(stream_);  // no copy from the caller's arrays outlives the call
    return s;
  }
  const auto t1 = std::chrono::steady_clock::now();
  if (small_out_) {
    if (n_results_ > 0)
      std::memcpy(out, reinterpret_cast<unsigned char*>(h_counters_) + kCountersBytes, sizeof(double) * (size_t)n_results_);
  } else {
    s = fetch(out, n_results_);
    if (s != BV_OK) return s;
  }
  if (stats) {
    stats->kernel_launches += stage_launches_;
    const auto t2 = std::chrono::steady_clock::now();
    stats->ms_d2h = std::chrono::duration<double, std::milli>(t2 - t1).count();
    stats->ms_total = std::chrono::duration<double, std::milli>(t2 - t0).count();
  }
  return BV_OK;
}

}  // namespace bvphmm

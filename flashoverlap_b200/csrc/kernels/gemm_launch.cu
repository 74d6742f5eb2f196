// Launcher of the fused sm_100a GEMM kernel: builds the TMA descriptors,
// picks the template instance for (tile width, dtype) and launches one CTA per
// SM.  Counterpart of the reference's per-tile-config launchers
// (reference: src/gemm/gemm.cu:29-113, src/overlap/gemm_signal.cu:28-110,
// src/overlap/gemm_scatter.cu:28-111), without a workspace allocation.
#include "gemm_launch.h"

#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <mutex>

#include <cstdlib>
#include <cstring>

#include "gemm_fused_sm100.cuh"

namespace fo {

#include "generated/algo_table.inc"

TileConfig algo_config(int algo) { return kAlgoTable[(algo < 0 || algo >= kNumAlgos) ? 0 : algo]; }

bool cooperative_launch_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("FLASHOVERLAP_COOPERATIVE");
    return e != nullptr && (std::strcmp(e, "1") == 0 || std::strcmp(e, "on") == 0);
  }();
  return on;
}

namespace {

PFN_cuTensorMapEncodeTiled_v12000 get_encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
    }
  });
  return fn;
}

// 2-D row-major [rows, cols] 16-bit matrix, box = 64 columns x box_rows rows,
// 128-byte swizzle.  Out-of-range parts of a box read as zero.
bool make_tensor_map(CUtensorMap* map, const void* base, int rows, int cols, int box_rows, DType dt) {
  auto encode = get_encode_fn();
  if (encode == nullptr) return false;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(cols) * 2};
  cuuint32_t box[2] = {64u, static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2] = {1u, 1u};
  CUresult r = encode(map, dt == DT_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                      const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                      CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

}  // namespace

int device_sm_count() {
  static int cached[kMaxDevices] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  const bool slot = dev >= 0 && dev < kMaxDevices;
  if (slot && cached[dev] > 0) return cached[dev];
  int n = 0;
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  if (slot) cached[dev] = n;
  return n;
}

cudaError_t prepare_fused(int algo, DType dtype) {
  if (algo < 0 || algo >= kNumAlgos) return cudaErrorInvalidValue;
  return kPrepareTable[algo][dtype == DT_BF16 ? 1 : 0]();
}

namespace {
int ceil_div(int a, int b) { return (a + b - 1) / b; }
int tile_columns(const GemmOperands& g, int bn) { return g.glu ? ceil_div(g.N / 2, bn / 2) : ceil_div(g.N, bn); }
bool can_run(const GemmOperands& g, const TileConfig& tc) { return !g.glu || (tc.ctas == 2 && tc.bn >= 128); }

// Estimated time in ns of a GEMM in one tile configuration: whole waves of tiles, each as long as K, plus what every wave
// costs and what the launch costs (start, pipeline fill, epilogue of the last tile).  Where the operands do not stay in L2
// the time is at least their way from HBM.
struct TileTime {
  double per_k, wave, fixed;
};
// From single waves (fp16, K from 2048 to 8192, all SMs busy).  A CTA takes in 110 to 125 GB/s of operands, which is what
// the tiles of up to 128 columns wait for; only the 256-wide ones wait for the tensor cores.  A stage of 64 K-values costs
// 290 ns at least, one of 128 K-values 430 ns.  Like the table below taken while four warps stored every tile; what rests on
// the two is the configuration that plan_plain and find_plan start from and weigh other forms against.
constexpr TileTime kSingleWave[] = {{6.7, 300, 7000}, {4.6, 300, 7000},  {4.5, 300, 6000}, {6.1, 300, 9500},
                                    {4.7, 300, 8700}, {4.5, 300, 7700},  {4.1, 300, 6300}, {3.4, 300, 5500},
                                    {6.0, 300, 9000}, {3.75, 300, 8300}, {3.4, 300, 7300}};
// Fitted to whole calls: 1500 shapes (M 128 to 8192, N 512 to 14336, K 256 to 16384, both types, with RMSNorm and without)
// in every configuration that divides them; least squares of the logarithm, 10 % rms.  Several waves share L2 and power,
// so that a value of K costs more, and the epilogue of a large tile shows in every wave.
constexpr TileTime kWholeCalls[] = {{7.49, 1500, 5900}, {5.48, 900, 5000},  {4.75, 500, 4300}, {5.65, 2400, 5900},
                                    {4.92, 1200, 5600}, {4.81, 600, 5500},  {5.30, 900, 5000}, {4.04, 600, 4700},
                                    {5.85, 2300, 6200}, {4.09, 1600, 5600}, {3.71, 900, 5500}};
static_assert(sizeof(kSingleWave) / sizeof(kSingleWave[0]) == kNumAlgos, "one entry per tile configuration");
static_assert(sizeof(kWholeCalls) / sizeof(kWholeCalls[0]) == kNumAlgos, "one entry per tile configuration");

double estimate_ns(const TileTime (&times)[kNumAlgos], const GemmOperands& g, int algo, int ctas) {
  const TileConfig& tc = kAlgoTable[algo];
  const int waves = ceil_div(ceil_div(g.M, tc.bm) * tile_columns(g, tc.bn), std::max(1, ctas / tc.ctas));
  const double operands = 2.0 * (static_cast<double>(g.M) + g.N) * g.K / 6000;  // bytes at 6 TB/s
  return std::max(waves * static_cast<double>(g.K) * times[algo].per_k, operands) + times[algo].fixed +
         times[algo].wave * waves;
}
}  // namespace

// Another tile than the named one runs when it is the fastest by the single waves, clearly, and no slower by the whole
// calls.  On 700 shapes other than the fitted ones, the tile that runs is more than 3 % slower than the named one in 0.3 %
// of the calls that name the first of gather_algo_candidates (5.1 % without the second condition) and in 1.4 % (4.1 %) of
// those that name any other; it is 1.25 times as fast on average over all (shares and average with the epilogue of that
// time, four warps).
static int plan_algo(const GemmOperands& g, int ctas) {
  if (!g.any_tile) return g.algo;
  int best = g.algo;
  double best_ns = 0.97 * estimate_ns(kSingleWave, g, g.algo, ctas);
  for (int algo = 0; algo < kNumAlgos; ++algo) {
    const double ns = estimate_ns(kSingleWave, g, algo, ctas);
    if (ns < best_ns && ctas >= kAlgoTable[algo].ctas && can_run(g, kAlgoTable[algo])) {
      best_ns = ns;
      best = algo;
    }
  }
  return estimate_ns(kWholeCalls, g, best, ctas) <= estimate_ns(kWholeCalls, g, g.algo, ctas) ? best : g.algo;
}

namespace {
// Clusters of so many CTAs that fit the chip together (148 SMs in groups of unequal size); the plan asks for no more.  Counted
// on one B200: where fewer fit, the others run in a second round.
constexpr int kMaxSplit = 8;
constexpr int kClusters[kMaxSplit + 1] = {0, 148, 73, 44, 32, 25, 21, 14, 14};

// A plain GEMM in a tile of any width, its K split over `split` CTAs, in ns: least squares of the logarithm (8 % rms) over
// 11000 timings, the dozen most promising forms of 1300 random shapes (M 128 to 16384, N 1024 to 14336, K 256 to 28672, both
// types).  A value of K costs what the tensor cores take (more as the chip warms up), what a CTA takes in (see NormFit), or
// its part of the least time of a stage; a split adds the way of the sums through distributed shared memory.
double plain_ns(const GemmOperands& g, int algo, int bn, int split, int ctas) {
  const TileConfig& tc = kAlgoTable[algo];
  const int tiles = ceil_div(g.M, tc.bm) * tile_columns(g, bn);
  const int waves = split > 1 ? 1 : ceil_div(tiles, std::max(1, ctas / tc.ctas));
  const double k = static_cast<double>(ceil_div(ceil_div(g.K, tc.bk), split)) * tc.bk;
  const double mma = 0.0203 * bn * (1 + 0.096 * std::min(1.0, waves * static_cast<double>(g.K) * 0.0203 * bn / 200e3));
  const double intake = 2.0 * (128 + bn / tc.ctas) / (tc.ctas == 1 ? 120.0 : 100.1) *
                        (g.K % 16 != 0 ? (tc.ctas == 1 ? 1.52 : 1.37) : g.K % 64 != 0 ? 1.10 : 1.0);
  const double per_k = std::max(std::max(mma, intake) * (tc.bk == 64 ? 0.985 : 1.0), 324.0 / tc.bk);
  const double main = waves * (k * per_k + 117.0 + 5.84 * bn);
  const double operands = 2.0 * (static_cast<double>(g.M) + g.N) * g.K / std::min(7833.0, 150.0 * std::min(ctas, tiles * split * tc.ctas));
  return std::sqrt(main * main + operands * operands) + 4425.0 + 0.52 * bn + (tc.ctas == 2 ? 1231.0 : 0) +
         (split > 1 ? 1777.0 + 21.2 * bn * (split - 1) / split : 0);
}

// The plan of a plain GEMM: the configuration that plan_algo finds, in the width that suits the wave, or another one where
// that is clearly better.  Short K gives little to go by (rounds of the epilogue and of HBM writes), and a split pays where
// the tiles leave SMs without work.  Over the fitted shapes 1.11 times as fast as plan_algo's tile alone (1.15 with the best
// choice each time), slower by more than 3 % in 0.2 %.  Against plan_algo's tile with the epilogue of four warps, two
// libraries in turn: 1152 x 5120 x 1720 bf16 38.4 -> 26.5 us (256 x 192), 128 x 10240 x 8192 bf16 42.2 -> 37.6 (two CTAs per
// 128 x 160 tile), 128 x 1024 x 28672 bf16 98 -> 27 (eight per 128 x 96), 2048 x 8192 x 1024 fp16 31.9 -> 30.7 (256 x 224).
LaunchPlan plan_plain(const GemmOperands& g, int base, int ctas) {
  LaunchPlan plan{base, kAlgoTable[base].bn, 0, 1, 0};
  const TileConfig& named = kAlgoTable[base];
  const double base_ns = plain_ns(g, base, named.bn, 1, ctas);
  const bool idle = ceil_div(g.M, named.bm) * tile_columns(g, named.bn) * named.ctas <= 0.6 * ctas;
  double best = base_ns;
  for (int algo = 0; algo < kNumAlgos; ++algo) {
    const TileConfig& tc = kAlgoTable[algo];
    if (ctas < tc.ctas || !can_run(g, tc)) continue;
    const int step = g.glu ? 64 : 32;  // of the gated form every CTA of a pair stages whole chunks
    for (int bn = tc.bn; bn >= 64 && (bn == tc.bn || bn > tc.bn / 2); bn -= step) {
      const int tiles = ceil_div(g.M, tc.bm) * tile_columns(g, bn);
      for (int split = 1; split <= (tc.ctas == 1 ? kMaxSplit : 1); ++split) {
        if (split > 1 && (split == 7 || tiles > kClusters[split] || tiles * split > ctas || ceil_div(g.K, tc.bk) < 3 * split)) continue;
        const bool same = algo == base && split == 1;
        const double ns = plain_ns(g, algo, bn, split, ctas);
        const double limit = same ? 0.95 : split > 1 ? (idle ? 0.9 : 0.79) : g.K >= 1024 ? 0.92 : 0.78;
        if (ns >= limit * base_ns) continue;
        const double rank = same ? 0.97 * ns : ns;  // among equals the configuration stays
        if (rank < best) {
          best = rank;
          plan = LaunchPlan{algo, bn, 0, split, 0};
        }
      }
    }
  }
  return plan;
}

// GEMM + RMSNorm of one rank, staged and resident, in ns.  Both are least-squares fits (of the logarithm; 8 % rms) to 900
// random shapes (M 128 to 16384, N 1024 to 14336, K 256 to 28672, both types), timed call after call in every form.  A value
// of K costs what the tensor cores take for bn columns (more as the chip warms up), or what a CTA takes in: 107 to 119 GB/s
// from L2, less where the rows of 128 bytes that the copy engine reads straddle two lines, or two sectors.
struct NormFit {
  double mma, droop, rate_one, rate_pair, odd_line, odd_sector;
};
double per_k_ns(const NormFit& f, int K, int ctas, int bn, int waves) {
  const double mma = f.mma * bn * (1 + f.droop * std::min(1.0, waves * static_cast<double>(K) * f.mma * bn / 200e3));
  const double intake = 2.0 * (128 + bn / ctas) / (ctas == 1 ? f.rate_one : f.rate_pair) *
                        (K % 16 != 0 ? f.odd_sector : K % 64 != 0 ? f.odd_line : 1.0);
  return std::max(mma, intake);
}
double staged_ns(const GemmOperands& g, int algo, int ctas) {
  constexpr NormFit kFit = {0.0210, 0.09, 117.2, 108.9, 1.04, 1.39};
  const TileConfig& tc = kAlgoTable[algo];
  const int waves = ceil_div(ceil_div(g.M, tc.bm) * tile_columns(g, tc.bn), std::max(1, ctas / tc.ctas));
  const double main = waves * static_cast<double>(g.K) * per_k_ns(kFit, g.K, tc.ctas, tc.bn, waves);
  return std::max(main, 2.0 * (static_cast<double>(g.M) + g.N) * g.K / 4230) + 10700 + 0.5 * tc.bn +
         0.96e-3 * g.M * static_cast<double>(g.N) + (tc.ctas == 2 ? 780 : 0);
}
double resident_ns(const GemmOperands& g, const TileConfig& tc, int bn, int tn, int rows, int waves) {
  constexpr NormFit kFit = {0.0211, 0.05, 118.9, 107.0, 1.10, 1.37};
  const double main = g.K * per_k_ns(kFit, g.K, tc.ctas, bn, waves) + 1760;
  // collecting a row's statistics, and the whole epilogue of a tile from its last MMA to its last store
  const double collect = 19 * tn + 805 * ceil_div(tn, 40), epilogue = 380 + 16.8 * bn + collect;
  const double hbm = std::min(3960.0, 64.0 * rows * tn * tc.ctas);  // few CTAs do not fill it
  return std::max((waves - 1) * std::max(main, epilogue) + main, 2.0 * (static_cast<double>(g.M) + g.N) * g.K / hbm) + 4480 +
         4.8 * bn + collect + (tc.ctas == 2 ? 1480 : 0);
}
}  // namespace

// A resident RMSNorm (see resident_norm) takes as many tile rows per wave as have all their tiles in it.  It runs where it
// is expected to save 5 %: in 89 % of the fitted shapes, slower than the staged form by more than 3 % in 1.6 % of all, 1.17
// times as fast over all (1.19 with the best choice each time).  Against the best tile of the staged form, fp16, in turn on a
// warm chip: 4096 x 8192 x 1024 83.5 -> 76.8 us, 2048 x 4096 x 2048 40.6 -> 34.2, 4096 x 4096 x 512 35.2 -> 29.1, 128 x 8192
// x 1024 15.6 -> 12.2.  From 1.5e11
// multiply-adds on (some 220 us) every form runs at the power cap, and the staged one, whose tiles have the full width, comes
// out the same or better: 4096 x 8192 x 8192 464 against 474, 8192 x 8192 x 28672 bf16 2950 against 3098.
// Among forms within the fit's error the configuration of a call without RMSNorm is kept.
static LaunchPlan find_plan(const GemmOperands& g, int ctas, bool whole_chip) {
  LaunchPlan plan{plan_algo(g, ctas), 0, 0, 1, 0};
  plan.bn = kAlgoTable[plan.algo].bn;
  if (!g.any_tile) return plan;
  if (!g.normed) return plan_plain(g, plan.algo, ctas);
  if (!g.may_keep) return plan;
  const int plain = plan.algo;
  double expected = staged_ns(g, plain, ctas);
  if (static_cast<double>(g.M) * g.N * g.K < 1.5e11) {
    const double limit = 0.95 * expected;
    double best = limit;
    for (int algo : {8, 9, 0, 6, 7}) {
      const TileConfig& tc = kAlgoTable[algo];
      const int slots = ctas / tc.ctas, tm = ceil_div(g.M, tc.bm);
      for (int bn = tc.bn; bn >= 32 && (tc.bn == 64 || bn > tc.bn / 2); bn -= 32) {
        const int tn = ceil_div(g.N, bn), rows = std::min(tm, slots / tn);
        if (rows == 0) continue;
        const double ns = resident_ns(g, tc, bn, tn, rows, ceil_div(tm, rows));
        if (ns >= limit) continue;
        const double rank = algo == plain ? 0.92 * ns : ns;
        if (rank < best) {
          best = rank;
          expected = ns;
          plan = LaunchPlan{algo, bn, rows, 1, 0};
        }
      }
    }
  }
  // A plain GEMM, in a tile of any width and with its K split, and an RMSNorm kernel that reads the product from L2: 2.3 us
  // and 0.76 ns per 1000 values more than the GEMM.  Over 800 shapes 1.09 times as fast as the better of the other forms
  // where it is expected to save 3 % (27 % of them; 1.56 times where K is split), nowhere slower by more than 3 %.  Against
  // the better of the other forms (the plan on 147 SMs), in turn: 256 x 1664 x 11904 bf16 47.6 -> 24.5 us, 384 x 1280 x 22256
  // fp16 82 -> 35.5, 128 x 1024 x 28672 bf16 100 -> 27; without a split 2176 x 4096 x 4096 fp16 65 to 81 -> 61 to 65.  Not
  // for calls of less than 14 us, which is what the host takes for two launches and the way to them.
  // Not for calls that leave SMs to other streams either: the RMSNorm kernel takes every SM.
  if (!whole_chip) return plan;
  const LaunchPlan two = plan_plain(g, plain, ctas);
  const double two_ns = plain_ns(g, two.algo, two.bn, two.split, ctas) + 2280 + 0.76e-3 * g.M * static_cast<double>(g.N);
  if (two_ns < 0.97 * expected && two_ns >= 14000) {
    plan = two;
    plan.norm_after = 1;
  }
  return plan;
}

// Comparing the forms takes some 3 us of host time, as long as a launch: each thread remembers the plans of its last shapes.
LaunchPlan plan_launch(const GemmOperands& g, int ctas, bool whole_chip) {
  struct Entry {
    int key[6];
    LaunchPlan plan;
  };
  static thread_local Entry seen[64] = {};
  if (!g.any_tile) return find_plan(g, ctas, whole_chip);
  const int key[6] = {g.M, g.N, g.K, g.algo, ctas, g.glu | g.normed << 1 | g.may_keep << 2 | (whole_chip ? 8 : 0)};
  const uint32_t slot = (static_cast<uint32_t>(g.M / 32) * 31u + static_cast<uint32_t>(g.N / 32)) * 31u + static_cast<uint32_t>(g.K / 8) * 7u + key[5];
  Entry& e = seen[slot % 64];
  if (!std::equal(key, key + 6, e.key)) {  // (no shape has M = 0)
    e.plan = find_plan(g, ctas, whole_chip);
    std::copy(key, key + 6, e.key);
  }
  return e.plan;
}

cudaError_t launch_fused(const GemmOperands& g, FusedParams& p, cudaStream_t stream, const char** why) {
  const char* dummy;
  if (why == nullptr) why = &dummy;
  *why = "";
  TileConfig tc = algo_config(g.algo);
  if (g.algo < 0 || g.algo >= kNumAlgos) {
    *why = "Algo index out of range";
    return cudaErrorInvalidValue;
  }
  if (g.M <= 0 || g.N <= 0 || g.K <= 0 || g.M % tc.bm != 0 || g.N % tc.bn != 0 || g.K % 8 != 0) {
    *why = "shape not supported: need M % tile_m == 0, N % tile_n == 0, K % 8 == 0";
    return cudaErrorInvalidValue;
  }
  if ((reinterpret_cast<uintptr_t>(g.A) & 15u) || (reinterpret_cast<uintptr_t>(g.B) & 15u)) {
    *why = "A and B must be 16-byte aligned";
    return cudaErrorInvalidValue;
  }
  // every store of the epilogue and of the reduce phase, and every load of the weights, is 16 bytes wide
  if ((reinterpret_cast<uintptr_t>(p.epi_base[0]) & 15u) ||
      (p.reduce && (reinterpret_cast<uintptr_t>(p.out[p.me]) & 15u)) ||
      (p.reduce && p.norm && (reinterpret_cast<uintptr_t>(p.gamma) & 15u))) {
    *why = "the result and the RMSNorm weights must be 16-byte aligned";
    return cudaErrorInvalidValue;
  }
  if (!can_run(g, tc)) {
    *why = "the gated form needs a CTA-pair tile of at least 128 columns";
    return cudaErrorInvalidValue;
  }
  int grid = g.sm_count > 0 ? g.sm_count : device_sm_count();
  const int sms = device_sm_count();
  if (grid > sms) grid = sms;  // every CTA must be resident: CTAs wait on one another's output
  const LaunchPlan plan = plan_launch(g, grid, grid == sms);
  const int algo = plan.algo;
  p.algo = algo;
  p.bn = plan.bn;
  p.split = plan.split;
  p.trace_cols = tc.bn;
  tc = kAlgoTable[algo];
  // every CTA stages 128 rows of A and (for a CTA pair) half of the B tile, 64 K-values per box
  const int a_rows = g.a_rows > 0 && g.a_rows < g.M ? g.a_rows : g.M;  // the copy engine fills the rows after them with zero
  if (!make_tensor_map(&p.tmA, g.A, a_rows, g.K, 128, g.dtype) ||
      !make_tensor_map(&p.tmB, g.B, g.N, g.K, p.bn / tc.ctas, g.dtype)) {
    *why = "cuTensorMapEncodeTiled failed";
    return cudaErrorInvalidValue;
  }
  p.a_own_begin = p.a_own_end = 0;
  if (g.A_own != nullptr && g.own_rows > 0) {
    if ((reinterpret_cast<uintptr_t>(g.A_own) & 15u) || g.own_begin < 0 || g.own_begin % 128 != 0 ||
        g.own_rows % 128 != 0 || g.own_begin + g.own_rows > g.M) {
      *why = "own rows of A must be 16-byte aligned whole blocks of 128 rows inside the matrix";
      return cudaErrorInvalidValue;
    }
    if (!make_tensor_map(&p.tmA_own, g.A_own, g.own_rows, g.K, 128, g.dtype)) {
      *why = "cuTensorMapEncodeTiled failed";
      return cudaErrorInvalidValue;
    }
    p.a_own_begin = g.own_begin;
    p.a_own_end = g.own_begin + g.own_rows;
  }
  p.glu = g.glu ? g.N / 2 : 0;
  p.M = g.M;
  p.N = g.N;
  p.K = g.K;
  p.TM = ceil_div(g.M, tc.bm);
  p.TN = tile_columns(g, p.bn);
  if (g.any_tile && p.reduce) p.flag_target = static_cast<uint32_t>(p.TN);
  p.norm_after = plan.norm_after;
  if (p.norm_after) {
    p.reduce = 0;
    p.flag[0] = nullptr;
    p.ssq = nullptr;
    p.raster_taper = 0;
  }
  p.resident = plan.rows > 0 ? 1 : 0;
  if (p.resident) {
    p.reduce = 0;
    p.epi_base[0] = p.out[p.me];
    p.raster_group = plan.rows;
    p.raster_taper = 0;
    grid = tc.ctas * plan.rows * p.TN;
  }
  const OutLayout& L = p.epi_layout;
  p.epi_direct = (p.own_mode == OWN_SINGLE || p.nvls) && (!L.tiled || (L.row_map == nullptr && L.bm % 32 == 0 && L.bn % 64 == 0));
  p.epi_wide = reinterpret_cast<uintptr_t>(p.epi_base[0]) % 32 == 0 && (L.tiled || L.ld % 16 == 0);
  // 3584 x 9472 x 256 fp16: 35.4 us with four epilogue warps and the transpose, 26.7 with eight and without; 4096 x 8192 x
  // 1024 74.5 -> 60.9; one wave of 512 x 9472 x 256 10.3 -> 8.6.
  p.epi_halves = p.epi_direct && !p.reduce && !p.ag_push ? 2 : 1;
  if (p.split > 1 && p.epi_halves != 2) {
    *why = "a split K needs the epilogue of eight warps";
    return cudaErrorInvalidValue;
  }
  if (p.raster_group <= 0) p.raster_group = 1;
  if (p.raster_group > p.TM) p.raster_group = p.TM;
  if (p.rot < 0 || p.rot >= p.TM) p.rot = 0;
  if (p.reduce && p.job_counter == nullptr) {
    *why = "the reduce phase needs a row-job counter";
    return cudaErrorInvalidValue;
  }
  if (!p.reduce && !p.force_full_grid && grid > p.TM * p.TN * tc.ctas) grid = p.TM * p.TN * tc.ctas;
  if (p.split > 1) grid = p.TM * p.TN * p.split;  // one tile per cluster
  if (tc.ctas == 2 && grid < 2) grid = 2;
  if (tc.ctas == 2) grid &= ~1;
  return kLaunchTable[algo][g.dtype == DT_BF16 ? 1 : 0](p, grid, stream);
}

}  // namespace fo

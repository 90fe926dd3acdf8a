// FP64 GEMM engine for sm_100a: picks the CTA tile and the split of every
// launch (the kernels are dgemm_tile.cuh's), reduces split-K partials, and holds
// the profiler and the split-K autotuner.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "dgemm_tile.cuh"
#include "gemm_f64.cuh"
#include "ozaki.cuh"

namespace uw12b {

namespace {

constexpr int BK = kDgemmBK;
constexpr long long kSMs = 148;

// C = alpha * sum_s work[s] + beta * C (fixed summation order).  Bound by the
// latency of the partials' loads at the small outputs that split: eight are in
// flight per thread.  I: index type (32-bit divisions where the output allows).
template <typename I>
__global__ void splitk_reduce(const double* work, int split, I m, I mn, I total,
                              I nbo1, double alpha, double beta, double* C, long long ldc,
                              long long sCo1, long long sCo2) {
  chain_wait();
  const I step = static_cast<I>(gridDim.x) * blockDim.x;
  for (I idx = static_cast<I>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total; idx += step) {
    const I bo = idx / mn;
    const I e = idx - bo * mn;
    const I c = e / m;
    const I r = e - c * m;
    const double* w = work + idx;
    double s = 0.0;
#pragma unroll 8
    for (int q = 0; q < split; ++q) s += w[static_cast<long long>(q) * total];
    double* dst = C + (bo % nbo1) * sCo1 + (bo / nbo1) * sCo2 + r + ldc * c;
    const double v = alpha * s;
    *dst = (beta == 0.0) ? v : v + beta * (*dst);
  }
}

// C = beta * C for an empty contraction.
__global__ void scale_only(long long m, long long n, long long nbo, long long nbo1, double beta,
                           double* C, long long ldc, long long sCo1, long long sCo2) {
  chain_wait();
  const long long total = m * n * nbo;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long mn = m * n;
    const long long bo = idx / mn;
    const long long e = idx - bo * mn;
    double* dst = C + (bo % nbo1) * sCo1 + (bo / nbo1) * sCo2 + (e % m) + ldc * (e / m);
    *dst = (beta == 0.0) ? 0.0 : beta * (*dst);
  }
}

// The tile and the split of a launch come from a cost model of the kernel,
// fitted to a sweep of every tile and split over 41 shapes (outputs from 24 x 24
// to 160000 x 600, contractions from 24 to 1.08 million terms, all layouts): its
// pick is within 4 % of the measured best on all of them.
// In cycles, for a CTA on one SM:
//   mma   its k tile at the tensor pipe's 64 multiply-adds per cycle, over the
//         share of that rate which the tile reaches with all its CTAs resident
//         (what is lost is operand traffic: 33.6, 31.5 and 30.1 TFLOP/s of 37.2
//         for 64 x 64, 64 x 32 and 32 x 32 at 45000 x 9000 x 900);
//   lone  its k tile when it has the SM to itself (fragment and barrier latency);
//   lsu   its k tile's 8-byte copies where an operand does not allow 16-byte ones.
// A split adds the partials' round trip and one launch.  The old rule, one
// 128 x 128 tile, left 95 % of the tensor pipe idle at 360 x 360 x 360 and
// computed 64 % padding at 300 x 300.
struct TileCost {
  const DgemmTile* tile;
  double eff, lone;
};
const TileCost kTiles[] = {{&kTile64x64, 0.905, 1500.0},
                           {&kTile64x32, 0.86, 900.0},
                           {&kTile32x32, 0.82, 600.0},
                           {&kTile128x16, 0.78, 1180.0},
                           {&kTile128x8, 0.62, 940.0}};
constexpr int kSplits[] = {1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64};
constexpr double kCtaStart = 2500.0;    // prologue, epilogue and launch of a wave
constexpr double kSplitLaunch = 5500.0; // the reduction's launch
constexpr double kSplitBytes = 1600.0;  // partial bytes per cycle through L2 / HBM
// Partial tiles of an automatic split: at most 256 MiB.
constexpr double kMaxPartials = double(1LL << 25);

struct Plan {
  const DgemmTile* tile = nullptr;
  int split = 1;
};

// Fewest predicted cycles over the tiles and, when `split` is 0, over the
// splits whose partials stay within max_partials doubles and leave every CTA
// two k tiles.
Plan choose_plan(const GemmDesc& d, bool va, bool vb, int split, double max_partials) {
  const long long nbo = d.nbo1 * d.nbo2;
  const long long kt = (d.k + BK - 1) / BK * d.nbr1 * d.nbr2;
  const double out = double(d.m) * double(d.n) * double(nbo);
  Plan best;
  double best_cost = 1e300;
  for (const TileCost& t : kTiles) {
    const DgemmTile& g = *t.tile;
    const long long tiles = ((d.m + g.bm - 1) / g.bm) * ((d.n + g.bn - 1) / g.bn) * nbo;
    double mma = g.bm * g.bn * BK / 64.0 / t.eff;
    const double lsu = (va ? 0.0 : g.bm * (d.a_kcontig ? 6.5 : 5.0)) +
                       (vb ? 0.0 : g.bn * (d.b_ncontig ? 5.0 : 6.5));
    mma = std::max(mma, lsu);
    const double occ = g.ctas_per_sm;
    for (const int s : kSplits) {
      if (split > 0 ? s != kSplits[0] : (s > 1 && (kt / s < 2 || out * s > max_partials))) break;
      const int sp = split > 0 ? split : s;
      const long long ctas = tiles * sp;
      if (ctas > 0x7fffffffLL) break;
      const double ktl = double((kt + sp - 1) / sp);
      const long long per_sm = (ctas + kSMs - 1) / kSMs;
      const long long full = per_sm / g.ctas_per_sm, rem = per_sm % g.ctas_per_sm;
      double cost;
      if (full >= 2)  // several waves: the CTAs of an SM drift apart and its last ones overlap
        cost = ktl * (double(ctas) / kSMs + 1.0) * std::max(mma, t.lone / occ) + kCtaStart;
      else  // 5 %: fewer CTAs than fill every SM alike
        cost = ktl * (double(full) * std::max(occ * mma, t.lone) * 1.05 +
                      (rem ? std::max(double(rem) * mma * 1.05, t.lone) : 0.0)) +
               kCtaStart * double(full + (rem ? 1 : 0));
      if (sp > 1) cost += kSplitLaunch + (sp + 1) * out * 8.0 / kSplitBytes;
      if (cost < best_cost) {
        best_cost = cost;
        best = Plan{t.tile, sp};
      }
    }
  }
  if (!best.tile) throw Error(kErrInvalid, "gemm: too many output tiles for one launch");
  return best;
}

// A 16-byte copy needs the operand base, leading dimension and every batch
// stride to be even (in doubles); tile origins are multiples of 8.
bool vec_ok(const double* base, long long ld, long long s1, long long s2, long long s3,
            long long s4) {
  return (reinterpret_cast<std::uintptr_t>(base) % 16 == 0) && (ld % 2 == 0) && (s1 % 2 == 0) &&
         (s2 % 2 == 0) && (s3 % 2 == 0) && (s4 % 2 == 0);
}

// Fills the kernel parameters up to the tile and the split.  Returns false for
// an empty output; *empty_k is set when the contraction is empty (C = beta C).
bool prepare(const GemmDesc& d, KParams& p, bool* empty_k) {
  const long long nbo = d.nbo1 * d.nbo2;
  const long long nbr = d.nbr1 * d.nbr2;
  *empty_k = false;
  if (d.m <= 0 || d.n <= 0 || nbo <= 0) return false;
  if (d.k <= 0 || nbr <= 0) {
    *empty_k = true;
    return true;
  }
  if (!d.A || !d.B || !d.C) throw Error(kErrInvalid, "gemm: null operand");
  p = KParams{};
  p.A = d.A; p.B = d.B; p.C = d.C;
  p.lda = d.lda; p.ldb = d.ldb; p.ldc = d.ldc;
  p.m = d.m; p.n = d.n; p.k = d.k;
  p.alpha = d.alpha; p.beta = d.beta;
  p.nbo1 = d.nbo1; p.nbo = nbo;
  p.sAo1 = d.sAo1; p.sAo2 = d.sAo2; p.sBo1 = d.sBo1; p.sBo2 = d.sBo2;
  p.sCo1 = d.sCo1; p.sCo2 = d.sCo2;
  p.nbr1 = d.nbr1;
  p.sAr1 = d.sAr1; p.sAr2 = d.sAr2; p.sBr1 = d.sBr1; p.sBr2 = d.sBr2;
  p.ktiles_pb = (d.k + BK - 1) / BK;
  p.ktiles_total = p.ktiles_pb * nbr;
  return true;
}

bool a_vec(const GemmDesc& d) { return vec_ok(d.A, d.lda, d.sAo1, d.sAo2, d.sAr1, d.sAr2); }
bool b_vec(const GemmDesc& d) { return vec_ok(d.B, d.ldb, d.sBo1, d.sBo2, d.sBr1, d.sBr2); }

// The plan for a given split (at most one per k tile), or for the rule's own
// choice (split 0).
Plan make_plan(const GemmDesc& d, const KParams& p, long long split,
               double max_partials = kMaxPartials) {
  return choose_plan(d, a_vec(d), b_vec(d),
                     static_cast<int>(std::min<long long>(split, p.ktiles_total)), max_partials);
}

void launch_scale_only(const GemmDesc& d, cudaStream_t s) {
  if (d.beta == 1.0) return;
  const long long nbo = d.nbo1 * d.nbo2;
  const long long total = d.m * d.n * nbo;
  const int blocks = static_cast<int>(std::min<long long>((total + 255) / 256, kSMs * 16));
  launch_chained(scale_only, blocks, 256, 0, s, d.m, d.n, nbo, d.nbo1, d.beta, d.C, d.ldc, d.sCo1,
                 d.sCo2);
  UW12_LAUNCHED();
}

// Makes the layout's kernels of every tile resident on the current device at
// the layout's first use there, so that no later size of it loads a kernel.
void load_layout(int layout) {
  static bool loaded[64][16] = {};
  static std::mutex mu;
  int dev = 0;
  UW12_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  if (dev < 64 && loaded[dev][layout]) return;
  for (const TileCost& t : kTiles) t.tile->load(layout);
  if (dev < 64) loaded[dev][layout] = true;
}

// Launches the GEMM (and the split-K reduction when the plan splits, with
// partial tiles in p.work).
void launch(const GemmDesc& d, KParams p, const Plan& plan, cudaStream_t s) {
  const DgemmTile& t = *plan.tile;
  p.tiles_m = (d.m + t.bm - 1) / t.bm;
  p.tiles_n = (d.n + t.bn - 1) / t.bn;
  p.tiles_mn = p.tiles_m * p.tiles_n;
  p.split = plan.split;
  const int layout = int(d.a_kcontig) | int(d.b_ncontig) << 1 | int(a_vec(d)) << 2 |
                     int(b_vec(d)) << 3;
  load_layout(layout);
  t.launch(p, layout, p.tiles_mn * p.nbo * p.split, s);
  if (p.split > 1) {
    const long long total = d.m * d.n * p.nbo;
    const int blocks = static_cast<int>(std::min<long long>((total + 255) / 256, kSMs * 16));
    if (total < (1LL << 31))
      launch_chained(splitk_reduce<unsigned>, blocks, 256, 0, s, p.work, p.split,
                     static_cast<unsigned>(d.m), static_cast<unsigned>(d.m * d.n),
                     static_cast<unsigned>(total), static_cast<unsigned>(d.nbo1), d.alpha, d.beta,
                     d.C, d.ldc, d.sCo1, d.sCo2);
    else
      launch_chained(splitk_reduce<long long>, blocks, 256, 0, s, p.work, p.split, d.m, d.m * d.n,
                     total, d.nbo1, d.alpha, d.beta, d.C, d.ldc, d.sCo1, d.sCo2);
    UW12_LAUNCHED();
  }
}

// ---- profiling -------------------------------------------------------------
struct ProfRec {
  cudaEvent_t a, b;
  double flops;
  std::string shape;  // "m n k nbo nbr split layout vec" for the per-launch log
  int kind;
};
std::mutex g_prof_mu;
bool g_prof_on = false;
std::vector<ProfRec> g_prof_recs;
KernelStats g_prof_acc[kProfKinds];

void prof_collect_locked() {
  for (auto& r : g_prof_recs) {
    UW12_CUDA(cudaEventSynchronize(r.b));
    float ms = 0.f;
    UW12_CUDA(cudaEventElapsedTime(&ms, r.a, r.b));
    KernelStats& acc = g_prof_acc[r.kind];
    acc.launches += 1;
    acc.ms += ms;
    acc.flops += r.flops;
    if (const char* path = std::getenv("UW12_PROFILE_LOG")) {
      if (FILE* f = std::fopen(path, "a")) {
        std::fprintf(f, "%.4f %s\n", ms, r.shape.c_str());
        std::fclose(f);
      }
    }
    cudaEventDestroy(r.a);
    cudaEventDestroy(r.b);
  }
  g_prof_recs.clear();
}

}  // namespace

void profile_enable(bool on) {
  std::lock_guard<std::mutex> lk(g_prof_mu);
  g_prof_on = on;
}

bool profile_enabled() {
  std::lock_guard<std::mutex> lk(g_prof_mu);
  return g_prof_on;
}

void profile_reset() {
  std::lock_guard<std::mutex> lk(g_prof_mu);
  prof_collect_locked();
  for (auto& a : g_prof_acc) a = KernelStats{};
}

KernelStats profile_read_gemm() { return profile_read_kind(kProfDgemm); }

KernelStats profile_read_kind(int kind) {
  std::lock_guard<std::mutex> lk(g_prof_mu);
  prof_collect_locked();
  return g_prof_acc[kind];
}

void profile_record(int kind, cudaEvent_t a, cudaEvent_t b, double work, std::string shape) {
  std::lock_guard<std::mutex> lk(g_prof_mu);
  g_prof_recs.push_back({a, b, work, std::move(shape), kind});
}

// ---- split-K autotuner ------------------------------------------------------
//
// choose_plan predicts the split-K factor of a launch.  The autotuner replaces
// it by measurement: a shape class is (output CTAs = 128 x 128 output tiles x
// output batches, power-of-two bucket of the k tiles over all reduction
// batches, power-of-two bucket of the 32 x 8 blocks that cover the output: launches
// use tiles from 64 x 64 down to 32 x 32 and 128 x 8, so 24 x 24 and 128 x 128, one
// CTA of 128 x 128 both, want different splits); in tuning mode the first
// automatic-split GEMM of a class not yet in
// the table is launched once with every candidate split (1, 2, 3, 4, 6, 8, 12,
// 16, 24, 32, 48, 64 while each CTA keeps >= 4 k tiles and the partial tiles stay
// within 256 MiB or the rule's), each with the tile the cost model picks for it
// and timed with CUDA events on the current stream, and the fastest is recorded
// and launched last, so C holds its result.  Only GEMMs with beta = 0 are tuned
// (their repeated launches overwrite C); the others, and every GEMM in "use"
// mode, take the table's split for their class when it has one and the rule's
// otherwise.  Outputs of at least 8 waves of 128 x 128 tiles are not tuned.
// A file's line without the last bucket (tables of one-tile kernels) stands for every
// output of its CTA count that has no entry of its own, and does not keep tuning mode
// from measuring one.
namespace {
struct TuneKey {
  long long ctas;
  int kbucket;
  int blocks;  // bucket of the output's 32 x 8 blocks, -1: any
  bool operator<(const TuneKey& o) const {
    return std::tie(ctas, kbucket, blocks) < std::tie(o.ctas, o.kbucket, o.blocks);
  }
};
struct TuneEntry {
  int split;
  double ms;
};
std::mutex g_tune_mu;
int g_tune_mode = 0;  // 0 off, 1 tune, 2 use
std::map<TuneKey, TuneEntry> g_tune;

int kbucket_of(long long ktiles_total) {
  int b = 0;
  while ((1LL << (b + 1)) <= ktiles_total) ++b;
  return b;
}

TuneKey tune_key(long long m, long long n, long long k, long long nbo, long long nbr) {
  const long long tiles = ((m + 127) / 128) * ((n + 127) / 128);
  const long long blocks = ((m + 31) / 32) * ((n + 7) / 8);
  return TuneKey{tiles * nbo, kbucket_of(((k + BK - 1) / BK) * nbr), kbucket_of(blocks * nbo)};
}
TuneKey tune_key(const GemmDesc& d) {
  return tune_key(d.m, d.n, d.k, d.nbo1 * d.nbo2, d.nbr1 * d.nbr2);
}

// the table's split for a class, or 0 (the caller holds g_tune_mu)
int table_split(TuneKey key) {
  auto it = g_tune.find(key);
  if (it == g_tune.end()) {
    key.blocks = -1;
    it = g_tune.find(key);
  }
  return it == g_tune.end() ? 0 : it->second.split;
}

// the table's split for d's class, or 0
int tuned_split(const GemmDesc& d) {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  return g_tune_mode == 0 ? 0 : table_split(tune_key(d));
}

bool tuning_wanted(const GemmDesc& d) {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  if (g_tune_mode != 1 || d.split > 0 || d.beta != 0.0) return false;
  const TuneKey key = tune_key(d);
  if (key.ctas >= 8 * kSMs) return false;
  return g_tune.find(key) == g_tune.end();
}

// Times every candidate split of d (beta = 0) on stream s, records the fastest
// for the class and leaves C with the result of a launch with it.
void tune_and_launch(const GemmDesc& d, KParams p, cudaStream_t s) {
  const int heuristic = make_plan(d, p, 0).split;
  // a candidate's partial tiles stay within 2^25 doubles (256 MiB) or the
  // rule's own, so tuning needs no more memory than the evaluation around it
  const double per_split = double(p.nbo) * double(d.m) * double(d.n);
  const double cap = std::max(double(1LL << 25), per_split * heuristic);
  std::vector<int> cands;
  for (int c : kSplits)
    if (c == 1 || (p.ktiles_total / c >= 4 && per_split * c <= cap)) cands.push_back(c);
  if (std::find(cands.begin(), cands.end(), heuristic) == cands.end()) cands.push_back(heuristic);
  struct Events {  // destroyed on every exit, a failed launch included
    cudaEvent_t a = nullptr, b = nullptr;
    ~Events() {
      if (a) cudaEventDestroy(a);
      if (b) cudaEventDestroy(b);
    }
  } ev;
  UW12_CUDA(cudaEventCreate(&ev.a));
  UW12_CUDA(cudaEventCreate(&ev.b));
  cudaEvent_t e0 = ev.a, e1 = ev.b;
  int best = heuristic;
  double best_ms = 1e300;
  for (int c : cands) {
    const Plan plan = make_plan(d, p, c);
    DevBuf work;
    if (c > 1) {
      work.alloc(static_cast<size_t>(c) * p.nbo * d.m * d.n, s);
      p.work = work.get();
    }
    launch(d, p, plan, s);  // warm-up (caches, first-launch set-up)
    UW12_CUDA(cudaEventRecord(e0, s));
    launch(d, p, plan, s);
    launch(d, p, plan, s);
    UW12_CUDA(cudaEventRecord(e1, s));
    UW12_CUDA(cudaEventSynchronize(e1));
    float ms = 0.f;
    UW12_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    if (ms / 2.0 < best_ms) {
      best_ms = ms / 2.0;
      best = c;
    }
  }
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tune[tune_key(d)] = TuneEntry{best, best_ms};
  }
  DevBuf work;
  if (best > 1) {
    work.alloc(static_cast<size_t>(best) * p.nbo * d.m * d.n, s);
    p.work = work.get();
  }
  launch(d, p, make_plan(d, p, best), s);
}
}  // namespace

void autotune_set(int mode, const char* path) {
  if (mode < 0 || mode > 2) throw Error(kErrInvalid, "autotune: mode must be 0, 1 or 2");
  std::map<TuneKey, TuneEntry> loaded;
  if (path && *path) {
    if (FILE* f = std::fopen(path, "r")) {
      char line[256];
      int lineno = 0;
      while (std::fgets(line, sizeof(line), f)) {
        ++lineno;
        if (line[0] == '#' || line[0] == '\n') continue;
        long long ctas = 0;
        int kb = 0, split = 0, blocks = -1;
        double ms = 0.0;
        if (std::sscanf(line, "%lld %d %d %lf %d", &ctas, &kb, &split, &ms, &blocks) < 4 ||
            ctas <= 0 || kb < 0 || kb > 62 || split < 1 || split > 64 || blocks < -1 ||
            blocks > 62) {
          std::fclose(f);
          throw Error(kErrInvalid, std::string("autotune: malformed line ") +
                                       std::to_string(lineno) + " in " + path);
        }
        loaded[TuneKey{ctas, kb, blocks}] = TuneEntry{split, ms};
      }
      std::fclose(f);
    }
  }
  std::lock_guard<std::mutex> lk(g_tune_mu);
  for (const auto& kv : loaded) g_tune[kv.first] = kv.second;
  g_tune_mode = mode;
}

void autotune_save(const char* path) {
  if (!path || !*path) throw Error(kErrInvalid, "autotune: no path");
  std::lock_guard<std::mutex> lk(g_tune_mu);
  FILE* f = std::fopen(path, "w");
  if (!f) throw Error(kErrInvalid, std::string("autotune: cannot write ") + path);
  std::fprintf(f, "# output_ctas k_tile_bucket split ms output_block_bucket\n");
  for (const auto& kv : g_tune) {
    std::fprintf(f, "%lld %d %d %.6f", kv.first.ctas, kv.first.kbucket, kv.second.split,
                 kv.second.ms);
    if (kv.first.blocks >= 0) std::fprintf(f, " %d", kv.first.blocks);
    std::fprintf(f, "\n");
  }
  std::fclose(f);
}

void autotune_clear() {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  g_tune.clear();
}

long long autotune_size() {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  return static_cast<long long>(g_tune.size());
}

int autotune_lookup(long long m, long long n, long long k, long long nbo, long long nbr) {
  if (m <= 0 || n <= 0 || k <= 0 || nbo <= 0 || nbr <= 0) return 0;
  std::lock_guard<std::mutex> lk(g_tune_mu);
  return table_split(tune_key(m, n, k, nbo, nbr));
}

void gemm(const GemmDesc& d) {
  const int L = split_moduli();
  if (L > 0) {
    const double flops = 2.0 * double(d.m) * double(d.n) * double(d.k) * double(d.nbo1) *
                         double(d.nbo2) * double(d.nbr1) * double(d.nbr2);
    const double min_flops = split_min_flops();
    if (flops >= min_flops && (min_flops == 0.0 || ozaki_profitable(d, L)) && ozaki_supported(d)) {
      gemm_ozaki(d, L);
      return;
    }
  }
  gemm_dmma(d);
}

void gemm_dmma(const GemmDesc& d) {
  KParams p;
  bool empty_k = false;
  if (!prepare(d, p, &empty_k)) return;
  cudaStream_t s = current_stream();
  if (empty_k) {
    launch_scale_only(d, s);
    return;
  }
  const bool prof = profile_enabled();
  if (d.split <= 0 && !prof && tuning_wanted(d)) {
    tune_and_launch(d, p, s);
    return;
  }
  const Plan plan = make_plan(d, p, d.split > 0 ? d.split : tuned_split(d));
  DevBuf work;
  if (plan.split > 1) {
    work.alloc(static_cast<size_t>(plan.split) * p.nbo * d.m * d.n, s);
    p.work = work.get();
  }
  cudaEvent_t ev_a = nullptr, ev_b = nullptr;
  if (prof) {
    UW12_CUDA(cudaEventCreate(&ev_a));
    UW12_CUDA(cudaEventCreate(&ev_b));
    UW12_CUDA(cudaEventRecord(ev_a, s));
  }
  launch(d, p, plan, s);
  if (prof) {
    UW12_CUDA(cudaEventRecord(ev_b, s));
    std::lock_guard<std::mutex> lk(g_prof_mu);
    char shape[256];
    std::snprintf(shape, sizeof(shape), "%lld %lld %lld %lld %lld %d %d%d %d%d %dx%d", d.m, d.n,
                  d.k, p.nbo, d.nbr1 * d.nbr2, plan.split, int(d.a_kcontig), int(d.b_ncontig),
                  int(a_vec(d)), int(b_vec(d)), plan.tile->bm, plan.tile->bn);
    g_prof_recs.push_back({ev_a, ev_b, 2.0 * double(d.m) * double(d.n) * double(d.k) *
                                           double(p.nbo) * double(d.nbr1 * d.nbr2),
                           shape, kProfDgemm});
  }
}

// ---- allocation-free variant -------------------------------------------------
//
// Split-K partial tiles normally live in a stream-ordered allocation.  For
// callers that must not allocate, they go into this fixed device array
// instead: every device that loads the library keeps it (16 MiB) until the
// process exits.  Host code cannot use the symbol itself as a pointer (it is a
// host-side shadow), so the device address is looked up once per device.
namespace {
static __device__ __align__(256) double g_noalloc_scratch[kNoAllocScratchDoubles];

std::mutex g_scratch_mu;
double* g_scratch_ptr[64] = {};

double* noalloc_scratch_for_current_device() {
  int dev = 0;
  UW12_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) throw Error(kErrInvalid, "gemm_noalloc: device index out of range");
  std::lock_guard<std::mutex> lk(g_scratch_mu);
  if (!g_scratch_ptr[dev]) {
    void* ptr = nullptr;
    UW12_CUDA(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
    g_scratch_ptr[dev] = static_cast<double*>(ptr);
  }
  return g_scratch_ptr[dev];
}

// At a device's first call: the fixed array and every kernel that a later call may launch
// (all layouts of all tiles, the split reduction, the empty contraction), so that no later
// one loads device code, which takes device memory.
void load_all_for_current_device() {
  static bool loaded[64] = {};
  static std::mutex mu;
  int dev = 0;
  UW12_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  if (dev < 0 || dev >= 64 || loaded[dev]) return;
  noalloc_scratch_for_current_device();
  for (int layout = 0; layout < 16; ++layout) load_layout(layout);
  cudaFuncAttributes fa{};
  UW12_CUDA(cudaFuncGetAttributes(&fa, splitk_reduce<unsigned>));
  UW12_CUDA(cudaFuncGetAttributes(&fa, splitk_reduce<long long>));
  UW12_CUDA(cudaFuncGetAttributes(&fa, scale_only));
  loaded[dev] = true;
}
}  // namespace

void gemm_noalloc(const GemmDesc& d) {
  load_all_for_current_device();
  KParams p;
  bool empty_k = false;
  if (!prepare(d, p, &empty_k)) return;
  cudaStream_t s = current_stream();
  if (empty_k) {
    launch_scale_only(d, s);
    return;
  }
  const double per_split = double(p.nbo) * double(d.m) * double(d.n);
  // an automatic split keeps its partial tiles within the array (split 1 needs none)
  const Plan plan = make_plan(d, p, std::max(0, d.split), double(kNoAllocScratchDoubles));
  if (d.split > 1 && per_split * plan.split > double(kNoAllocScratchDoubles))
    throw Error(kErrInvalid,
                "gemm_noalloc: split * batches * m * n = " +
                    std::to_string(static_cast<long long>(per_split * plan.split)) +
                    " doubles exceeds the fixed scratch of " +
                    std::to_string(kNoAllocScratchDoubles) + " doubles (16 MiB)");
  if (plan.split > 1) p.work = noalloc_scratch_for_current_device();
  launch(d, p, plan, s);
}

}  // namespace uw12b

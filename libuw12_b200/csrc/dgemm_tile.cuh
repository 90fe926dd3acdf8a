// The FP64 tensor-core GEMM kernel (mma.sync m16n8k4 .f64), one template for
// every CTA tile shape; each tile shape is instantiated in a file of its own
// (dgemm_tile_*.cu) for the four operand layouts and the two copy widths of
// each operand, and gemm_f64.cu picks the tile and the split of a launch.
//
// What bounds it.  A wide product is bound by the double-precision tensor
// pipe (64 multiply-adds per SM and cycle; one m16n8k4 occupies a quarter of
// the SM for 32 cycles), thin ones by the operand stream, small ones by the
// latency of one k tile.  So:
//  * fragments are double buffered in registers: those of the next four k are
//    read from shared memory while the tensor pipe works on the current four,
//    across k tiles too (the wait and the barrier for the next tile come
//    before the last MMA group of the current one), so the pipe does not drain
//    at a tile's end;
//  * the tiles are small enough for three to five CTAs per SM, whose
//    prologues, barriers and epilogues overlap each other's MMAs.  An FP64 MMA
//    is slow enough that a 64 x 64 tile needs only 16 bytes per cycle from L2;
//  * tiles from 64 x 64 down to 32 x 32, and two thin ones (128 x 16, 128 x 8),
//    keep the padding of ragged, thin and small outputs low, which is computed
//    like the rest.
// Measured (one B200, kernel alone), against the same pipeline depth at one
// 128 x 128 CTA per SM without fragment double buffering (30.3 TFLOP/s at
// 45000 x 9000 x 900): 64 x 64 33.0 TFLOP/s there, 64 x 32 31.0, 32 x 32 30.0
// (2 % more on other devices); 360 x 360 x 360 64 -> 10 us (32 x 32);
// 480 x 12 x 120, 360 batches, 242 -> 44 us (128 x 16); 125250 x 2 x 1500
// 1.62 -> 0.24 ms (128 x 8, 6.4 TB/s of operand).
#pragma once

#include <cstdint>
#include <mutex>

#include "common.cuh"

namespace uw12b {

constexpr int kDgemmBK = 16;  // k extent of one pipeline stage

struct KParams {
  const double* A;
  const double* B;
  double* C;
  double* work;  // split > 1: partial tiles [split][nbo][m*n]
  long long lda, ldb, ldc;
  long long m, n, k;
  double alpha, beta;
  long long nbo1, nbo;
  long long sAo1, sAo2, sBo1, sBo2, sCo1, sCo2;
  long long nbr1;
  long long sAr1, sAr2, sBr1, sBr2;
  long long tiles_m, tiles_n, tiles_mn;
  long long ktiles_pb, ktiles_total;
  int split;
};

// One tile shape: extents, resident CTAs per SM, and its launcher.  `layout`
// is a_kcontig | b_ncontig << 1 | va << 2 | vb << 3 (va, vb: 16-byte copies of
// A and B are possible).  `load` makes the layout's kernel resident on the
// current device (its shared-memory size is raised).
struct DgemmTile {
  int bm, bn, ctas_per_sm;
  void (*launch)(const KParams& p, int layout, long long grid, cudaStream_t s);
  void (*load)(int layout);
};

extern const DgemmTile kTile64x64, kTile64x32, kTile32x32, kTile128x16, kTile128x8;

namespace dgemm_detail {

__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

// 8- or 16-byte asynchronous global -> shared copy; bytes beyond src_bytes
// are zero-filled (src_bytes = 0 reads nothing).
template <int BYTES>
__device__ __forceinline__ void cp_async(double* dst, const double* src, int src_bytes) {
  if (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(src_bytes));
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__device__ __forceinline__ void dmma(double (&c)[4], double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

// Loader of one operand tile (kDgemmBK deep, W wide) into shared memory.
//   KC  : the operand is contiguous along k in global memory ([w][k] tile,
//         row LDK) -- otherwise along the wide dimension ([k][w], row LDW);
//   VEC : copies of two consecutive doubles (16 bytes) along the contiguous
//         dimension; requires even leading dimension / offsets.
// The contiguous index is the fastest-varying across threads.  Row lengths are
// 4 mod 16 doubles: the eight-by-four fragment reads then touch every 8-byte
// bank once per half warp.
template <bool KC, bool VEC, int W, int THREADS>
struct TileLoader {
  static constexpr int BK = kDgemmBK;
  static constexpr int LDW = (W + 15) / 16 * 16 + 4;
  static constexpr int LDK = BK + 4;
  static constexpr int ELEMS = KC ? W * LDK : BK * LDW;  // doubles per stage
  static constexpr int E = VEC ? 2 : 1;                  // doubles per copy
  static constexpr int TPC = (KC ? BK : W) / E;          // threads along the contiguous dimension
  static constexpr int STEP = THREADS / TPC;             // other-dimension stride
  static constexpr int OTHER = KC ? W : BK;
  static constexpr int COPIES = (OTHER + STEP - 1) / STEP;
  static constexpr bool EXACT = OTHER % STEP == 0;
  static_assert(THREADS % TPC == 0, "threads cover whole rows of copies");

  int c0;  // contiguous index of this thread's first element
  int o0;  // other index of this thread's first copy

  __device__ __forceinline__ explicit TileLoader(int tid) : c0((tid % TPC) * E), o0(tid / TPC) {}

  // Element (w, kk) of the tile lives at global offset w + ld*kk (not KC) or
  // kk + ld*w (KC).
  __device__ __forceinline__ long long base(long long w0, long long ld) const {
    return KC ? (c0 + ld * (w0 + o0)) : (w0 + c0 + ld * o0);
  }
  __device__ __forceinline__ long long kstep(long long ld) const { return KC ? BK : BK * ld; }
  static __device__ __forceinline__ int at(int w, int kk) {
    return KC ? w * LDK + kk : kk * LDW + w;
  }

  // Copies this thread's share of a tile.  wlim = extent left along the wide
  // dimension from the tile start, klim = extent left along k (both clamped).
  __device__ __forceinline__ void load(double* s, const double* g, const double* dummy, int wlim,
                                       int klim, long long ld) const {
    const int left = (KC ? klim : wlim) - c0;
    const int full = left >= E ? 8 * E : (left > 0 ? 8 * left : 0);
    const int lim_o = KC ? wlim : klim;
    double* dst = s + (KC ? o0 * LDK + c0 : o0 * LDW + c0);
#pragma unroll
    for (int r = 0; r < COPIES; ++r) {
      const int o = o0 + r * STEP;
      if (!EXACT && o >= OTHER) break;
      const int bytes = o < lim_o ? full : 0;
      const double* src = bytes ? g + r * STEP * ld : dummy;
      cp_async<8 * E>(dst + r * STEP * (KC ? LDK : LDW), src, bytes);
    }
  }
};

// WM x WN warps, each MI x NI MMA tiles of 16 x 8; STAGES pipeline stages.
template <int WM, int WN, int MI, int NI, int STAGES, int CTAS, bool AK, bool BNC, bool VA,
          bool VB>
__global__ void __launch_bounds__(32 * WM * WN, CTAS) dgemm_dmma(const KParams p) {
  constexpr int BK = kDgemmBK;
  constexpr int THREADS = 32 * WM * WN;
  constexpr int BM = WM * MI * 16, BN = WN * NI * 8;
  // CTAs that run together share A panels across about 1024 columns of B
  constexpr int GROUP_N = 1024 / BN;
  using LA = TileLoader<AK, VA, BM, THREADS>;
  using LB = TileLoader<!BNC, VB, BN, THREADS>;
  extern __shared__ __align__(16) double smem[];
  double* As = smem;
  double* Bs = smem + STAGES * LA::ELEMS;

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int g = lane >> 2;  // groupID
  const int t = lane & 3;   // thread in group
  const int wm = (warp % WM) * (MI * 16);
  const int wn = (warp / WM) * (NI * 8);

  // Block -> (tile, output batch, split).  Tiles are visited in groups of
  // GROUP_N n-tiles, m-tile outermost inside a group, so the CTAs that run at
  // once touch a few A panels and GROUP_N B panels.
  long long bid = blockIdx.x;
  const long long tile = bid % p.tiles_mn;
  bid /= p.tiles_mn;
  const long long bo = bid % p.nbo;
  const int sp = static_cast<int>(bid / p.nbo);
  const long long per_group = p.tiles_m * GROUP_N;
  const long long grp = tile / per_group;
  const long long gn0 = grp * GROUP_N;
  const long long gsize = (p.tiles_n - gn0) < GROUP_N ? (p.tiles_n - gn0) : GROUP_N;
  const long long local = tile - grp * per_group;
  const long long tn = gn0 + local % gsize;
  const long long tm = local / gsize;
  const long long m0 = tm * BM;
  const long long n0 = tn * BN;
  const long long bo1 = bo % p.nbo1;
  const long long bo2 = bo / p.nbo1;

  const long long kt_begin = p.ktiles_total * sp / p.split;
  const long long kt_end = p.ktiles_total * (sp + 1) / p.split;

  const LA la(tid);
  const LB lb(tid);
  const long long a_kstep = la.kstep(p.lda);
  const long long b_kstep = lb.kstep(p.ldb);
  const int a_wlim = static_cast<int>(min(p.m - m0, static_cast<long long>(BM)));
  const int b_wlim = static_cast<int>(min(p.n - n0, static_cast<long long>(BN)));

  // Incremental (reduction batch, k offset) iterator of the next stage to
  // load: no integer division inside the main loop.
  long long it_kin, it_br1;
  const double* itA;
  const double* itB;
  {
    const long long br = kt_begin / p.ktiles_pb;
    const long long kt_in = kt_begin - br * p.ktiles_pb;
    it_kin = kt_in * BK;
    it_br1 = br % p.nbr1;
    const long long br2 = br / p.nbr1;
    itA = p.A + bo1 * p.sAo1 + bo2 * p.sAo2 + it_br1 * p.sAr1 + br2 * p.sAr2 + kt_in * a_kstep +
          la.base(m0, p.lda);
    itB = p.B + bo1 * p.sBo1 + bo2 * p.sBo2 + it_br1 * p.sBr1 + br2 * p.sBr2 + kt_in * b_kstep +
          lb.base(n0, p.ldb);
  }
  const long long k_pad = p.ktiles_pb * BK;

  auto load_stage = [&](int slot) {
    const int klim = static_cast<int>(min(p.k - it_kin, static_cast<long long>(BK)));
    la.load(As + slot * LA::ELEMS, itA, p.A, a_wlim, klim, p.lda);
    lb.load(Bs + slot * LB::ELEMS, itB, p.B, b_wlim, klim, p.ldb);
    it_kin += BK;
    itA += a_kstep;
    itB += b_kstep;
    if (it_kin >= k_pad) {
      it_kin = 0;
      itA += p.sAr1 - p.ktiles_pb * a_kstep;
      itB += p.sBr1 - p.ktiles_pb * b_kstep;
      if (++it_br1 == p.nbr1) {
        it_br1 = 0;
        itA += p.sAr2 - p.nbr1 * p.sAr1;
        itB += p.sBr2 - p.nbr1 * p.sBr1;
      }
    }
  };

  double acc[MI][NI][4];
#pragma unroll
  for (int a = 0; a < MI; ++a)
#pragma unroll
    for (int b = 0; b < NI; ++b)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[a][b][c] = 0.0;

  double af[2][MI][2], bf[2][NI];
  auto load_frags = [&](int buf, int slot, int kq) {
    const double* as = As + slot * LA::ELEMS;
    const double* bs = Bs + slot * LB::ELEMS;
    const int kk = kq * 4 + t;
#pragma unroll
    for (int mi = 0; mi < MI; ++mi) {
      af[buf][mi][0] = as[LA::at(wm + mi * 16 + g, kk)];
      af[buf][mi][1] = as[LA::at(wm + mi * 16 + g + 8, kk)];
    }
#pragma unroll
    for (int ni = 0; ni < NI; ++ni) bf[buf][ni] = bs[LB::at(wn + ni * 8 + g, kk)];
  };

  chain_wait();
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (kt_begin + s < kt_end) load_stage(s);
    cp_async_commit();
  }
  cp_async_wait<STAGES - 2>();
  __syncthreads();
  load_frags(0, 0, 0);

  int slot = 0;
  int load_slot = STAGES - 1;
  for (long long kt = kt_begin; kt < kt_end; ++kt) {
#pragma unroll
    for (int kq = 0; kq < BK / 4; ++kq) {
      if (kq == BK / 4 - 1) {
        // the next tile has landed for every thread, and every warp has read
        // its last fragments of this one
        cp_async_wait<STAGES - 2>();
        __syncthreads();
        slot = (slot + 1 == STAGES) ? 0 : slot + 1;
      }
      load_frags((kq + 1) & 1, slot, (kq + 1) % (BK / 4));
      if (kq == 0) {
        // refills the slot of the previous tile, whose last reads precede the
        // barrier above
        if (kt + STAGES - 1 < kt_end) load_stage(load_slot);
        cp_async_commit();
        load_slot = (load_slot + 1 == STAGES) ? 0 : load_slot + 1;
      }
#pragma unroll
      for (int mi = 0; mi < MI; ++mi)
#pragma unroll
        for (int ni = 0; ni < NI; ++ni)
          dmma(acc[mi][ni], af[kq & 1][mi][0], af[kq & 1][mi][1], bf[kq & 1][ni]);
    }
  }
  chain_release();  // the epilogue is left
  cp_async_wait<0>();

  // Epilogue: C = alpha acc + beta C, or the raw partial tile for split-K.
  double* Cb = p.split == 1 ? p.C + bo1 * p.sCo1 + bo2 * p.sCo2
                            : p.work + (static_cast<long long>(sp) * p.nbo + bo) * (p.m * p.n);
  const long long ldc = p.split == 1 ? p.ldc : p.m;
#pragma unroll
  for (int mi = 0; mi < MI; ++mi)
#pragma unroll
    for (int ni = 0; ni < NI; ++ni)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const long long r = m0 + wm + mi * 16 + g + 8 * h;
        if (r >= p.m) continue;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const long long c = n0 + wn + ni * 8 + 2 * t + q;
          if (c >= p.n) continue;
          double* dst = Cb + r + ldc * c;
          if (p.split == 1) {
            const double v = p.alpha * acc[mi][ni][2 * h + q];
            *dst = (p.beta == 0.0) ? v : v + p.beta * (*dst);
          } else {
            *dst = acc[mi][ni][2 * h + q];
          }
        }
      }
}

template <int WM, int WN, int MI, int NI, int STAGES, int CTAS>
struct Ops {
  static constexpr int THREADS = 32 * WM * WN;
  static constexpr int BM = WM * MI * 16, BN = WN * NI * 8;

  template <bool AK, bool BNC, bool VA, bool VB>
  static constexpr size_t smem_bytes() {
    return size_t(STAGES) * sizeof(double) *
           (TileLoader<AK, VA, BM, THREADS>::ELEMS + TileLoader<!BNC, VB, BN, THREADS>::ELEMS);
  }
  // f(kernel, shared memory) for the layout
  template <int L, typename F>
  static void visit(F&& f) {
    constexpr bool AK = L & 1, BNC = L & 2, VA = L & 4, VB = L & 8;
    static_assert(CTAS * (smem_bytes<AK, BNC, VA, VB>() + 1024) <= 228 * 1024,
                  "resident CTAs exceed an SM's shared memory");
    f(dgemm_dmma<WM, WN, MI, NI, STAGES, CTAS, AK, BNC, VA, VB>, smem_bytes<AK, BNC, VA, VB>());
  }
  template <typename F>
  static void dispatch(int layout, F&& f) {
    switch (layout) {
      case 0: visit<0>(f); break;
      case 1: visit<1>(f); break;
      case 2: visit<2>(f); break;
      case 3: visit<3>(f); break;
      case 4: visit<4>(f); break;
      case 5: visit<5>(f); break;
      case 6: visit<6>(f); break;
      case 7: visit<7>(f); break;
      case 8: visit<8>(f); break;
      case 9: visit<9>(f); break;
      case 10: visit<10>(f); break;
      case 11: visit<11>(f); break;
      case 12: visit<12>(f); break;
      case 13: visit<13>(f); break;
      case 14: visit<14>(f); break;
      default: visit<15>(f); break;
    }
  }
  static void launch(const KParams& p, int layout, long long grid, cudaStream_t s) {
    dispatch(layout, [&](auto kernel, size_t smem) {
      launch_chained(kernel, dim3(static_cast<unsigned>(grid)), THREADS, smem, s, p);
    });
    UW12_LAUNCHED();
  }
  static void load(int layout) {
    dispatch(layout, [&](auto kernel, size_t smem) {
      UW12_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(smem)));
    });
  }
  static constexpr DgemmTile tile() { return DgemmTile{BM, BN, CTAS, &launch, &load}; }
};

}  // namespace dgemm_detail
}  // namespace uw12b

// Split-precision FP64 GEMM: int8 residue products on the tcgen05 tensor
// cores, recombined by the Chinese remainder theorem (see ozaki.cuh).
//
// Kernels per GEMM (slab):
//   k_row_exponent per row of A / column of B: the binary exponent of its
//                 largest element; rows are scaled by 2^(beta - exponent) so
//                 that every element is below 2^beta in magnitude;
//   k_residues    FP64 -> rint(x 2^shift) -> L int8 residue planes, K-major
//                 (row r of plane (l, p) is K_pad contiguous bytes);
//   k_i8_mma      persistent, one CTA pair (or CTA) per SM pair (SM); work item =
//                 one 256 x 256 (128 x 256) output tile of one modulus and one K
//                 chunk: TMA (128-byte swizzled boxes, ring of stages) -> shared
//                 memory -> tcgen05.mma.cta_group::2 (::1) kind::i8 with the int32
//                 accumulator in TMEM (two 256-column buffers) -> tcgen05.ld ->
//                 residue mod p -> uint8 rows in HBM.  Warp roles: 0 TMA producer,
//                 1 TMEM owner + MMA issuer, 2..5 epilogue (TMEM lane quarter =
//                 warp % 4);
//   k_crt         per output element: sum the K-chunk residues mod p, CRT on
//                 <= 41-bit chunks in FP64 (exact integer arithmetic), join the
//                 chunks error-free (TwoSum), scale by 2^-(sa+sb), apply
//                 alpha / beta, store FP64.
// The MMA's M side (TMEM lanes) runs over the output column j (B's n index)
// and its N side over the output row i (A's m index), so that one thread of
// the epilogue owns 256 consecutive i of one column j and the residue planes
// and C are both i-contiguous.
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <mutex>
#include <string>

#include "ozaki.cuh"

namespace uw12b {

namespace {

// Pairwise-coprime moduli <= 256 (residues fit int8: [-128, 127]).
constexpr uint32_t kModuli[kOzakiMaxModuli] = {256, 255, 253, 251, 247, 241, 239, 233,
                                               229, 227, 223, 217, 211, 199, 197, 193};
// CRT weights are split into nch chunks of cw <= 41 bits: r_l * chunk < 2^49
// and the sum over <= 16 moduli < 2^53, so every chunk sum is exact in FP64.
constexpr int kMaxChunkBits = 41;
constexpr int kMaxChunks = 4;  // 4 x 41 bits >= log2(M) for 16 moduli (~125.3)
constexpr long long kMaxKChunk = 65536;  // |acc| <= 65536 * 128^2 = 2^30 per split

struct Consts {
  int L = 0, nch = 0, cw = 0, beta = 0;
  uint32_t p[kOzakiMaxModuli];
  uint32_t barrett[kOzakiMaxModuli];  // floor(2^32 / p)
  double inv_p[kOzakiMaxModuli];
  double w[kOzakiMaxModuli][kMaxChunks];  // chunks of (M/p_l) * ((M/p_l)^-1 mod p_l) mod M
  double mc[kMaxChunks];                  // chunks of M
  double inv_m;
  double log2_m;
  // the same weights for k_crt_pipe: byte b of w_l for the moduli 4t .. 4t + 3 as
  // the bytes of w8[b][t]; 32-bit digits m of M; 2^(32 m) / M; and 2^52 plus what
  // the 128 added to every residue adds to digit m
  uint32_t w8[16][4];
  double m32[4], per_m[4], bias[4];
};

using u128 = unsigned __int128;

long long inv_mod(long long a, long long p) {
  long long t = 0, nt = 1, r = p, nr = a % p;
  while (nr) {
    const long long q = r / nr;
    std::swap(t, nt); nt -= q * t;
    std::swap(r, nr); nr -= q * r;
  }
  if (r != 1) throw Error(kErrInvalid, "split-precision moduli are not coprime");
  return t < 0 ? t + p : t;
}

Consts make_consts(int L) {
  Consts c;
  c.L = L;
  u128 M = 1;
  c.log2_m = 0.0;
  for (int l = 0; l < L; ++l) {
    const uint32_t p = kModuli[l];
    M *= p;
    c.log2_m += std::log2(double(p));
    c.p[l] = p;
    c.barrett[l] = static_cast<uint32_t>((1ULL << 32) / p);
    c.inv_p[l] = 1.0 / double(p);
  }
  int bits = 0;
  for (u128 t = M; t; t >>= 1) ++bits;
  c.nch = (bits + kMaxChunkBits - 1) / kMaxChunkBits;
  c.cw = (bits + c.nch - 1) / c.nch;
  const int kChunkBits = c.cw;
  const u128 mask = (u128(1) << kChunkBits) - 1;
  for (int l = 0; l < L; ++l) {
    const u128 Ml = M / kModuli[l];
    const long long y = inv_mod(static_cast<long long>(Ml % kModuli[l]), kModuli[l]);
    const u128 w = Ml * u128(y);  // < M: Ml * y < Ml * p_l
    for (int ch = 0; ch < kMaxChunks; ++ch)
      c.w[l][ch] = ch < c.nch ? double(static_cast<uint64_t>((w >> (kChunkBits * ch)) & mask))
                              : 0.0;
  }
  for (int ch = 0; ch < kMaxChunks; ++ch)
    c.mc[ch] = ch < c.nch ? double(static_cast<uint64_t>((M >> (kChunkBits * ch)) & mask)) : 0.0;
  c.inv_m = 1.0 / static_cast<double>(M);
  for (auto& row : c.w8)
    for (uint32_t& v : row) v = 0;
  for (int m = 0; m < 4; ++m) {
    c.m32[m] = double(static_cast<uint32_t>(M >> (32 * m)));
    c.per_m[m] = std::ldexp(1.0, 32 * m) / static_cast<double>(M);
    c.bias[m] = 0x1p52;
  }
  for (int l = 0; l < L; ++l) {
    const u128 Ml = M / kModuli[l];
    const u128 w = Ml * u128(inv_mod(static_cast<long long>(Ml % kModuli[l]), kModuli[l]));
    for (int b = 0; b < 16; ++b) c.w8[b][l / 4] |= static_cast<uint32_t>((w >> (8 * b)) & 255) << (8 * (l % 4));
    for (int m = 0; m < 4; ++m) c.bias[m] += 128.0 * double(static_cast<uint32_t>(w >> (32 * m)));
  }
  return c;
}

const Consts& consts_for(int L) {
  static std::once_flag once[kOzakiMaxModuli + 1];
  static Consts table[kOzakiMaxModuli + 1];
  std::call_once(once[L], [&] { table[L] = make_consts(L); });
  return table[L];
}

thread_local int g_split_moduli = 0;
thread_local double g_split_min_flops = kOzakiMinFlops;

// device error flags (a pipeline wait timed out): kOzakiErrorSlots ints per
// device; a host thread uses the slot set by set_error_slot (0 by default), so
// that concurrent evaluations on different threads (uw12c_fock_batched's
// workers) read and clear only their own flag
constexpr int kMaxDevices = 64;
std::mutex g_err_mu;
int* g_err_ptr[kMaxDevices] = {};
thread_local int t_err_slot = 0;

int* err_flag() {
  int dev = 0;
  UW12_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices)
    throw Error(kErrInvalid, "split-precision GEMM: device index beyond 63");
  std::lock_guard<std::mutex> lk(g_err_mu);
  if (!g_err_ptr[dev]) {
    UW12_CUDA(cudaMalloc(reinterpret_cast<void**>(&g_err_ptr[dev]),
                         kOzakiErrorSlots * sizeof(int)));
    UW12_CUDA(cudaMemset(g_err_ptr[dev], 0, kOzakiErrorSlots * sizeof(int)));
  }
  return g_err_ptr[dev] + t_err_slot;
}

// ---------------------------------------------------------------------------
// operand preparation
// ---------------------------------------------------------------------------
// Operand rows: element (row, kt) of plane (p1, p2), kt = kk + k * (r1 + nbr1 r2),
// lives at base + p1*po1 + p2*po2 + row*rs + kk*ks + r1*sr1 + r2*sr2.
struct OperandView {
  const double* base;
  long long rows, k, k_total;
  long long rs, ks, sr1, sr2, nbr1;
  long long po1, po2;
  int np1, np2;
};

// Offsets (kk*ks + r1*sr1 + r2*sr2) of the 128 k of the tile starting at k0
// (-1 beyond k_total), one division per k.
__device__ __forceinline__ void tile_k_offsets(const OperandView& v, long long k0,
                                               long long* koff) {
  if (threadIdx.x < 128) {
    const long long kt = k0 + threadIdx.x;
    long long off = -1;
    if (kt < v.k_total) {
      const long long r = kt / v.k, kk = kt - r * v.k;
      off = kk * v.ks + (r % v.nbr1) * v.sr1 + (r / v.nbr1) * v.sr2;
    }
    koff[threadIdx.x] = off;
  }
}

// Shared-memory tile of 32 rows x 128 k, unpadded, element (r, c) at
// r * 128 + (c ^ ((c >> 4) & 7) ^ (r & 15)).  The swizzle stays inside each
// 16-element group and is a bijection per row; every warp access of the
// kernels below touches all 16 8-byte bank pairs exactly twice (two
// wavefronts for 256 bytes, the minimum): the column fill of 32 rows at one k,
// the row fill of 32 consecutive k, and the compute reads (16 lanes per row,
// lane t at k = 8 t + q for one q).
__device__ __forceinline__ int tile_at(int r, int c) {
  return r * 128 + (c ^ ((c >> 4) & 7) ^ (r & 15));
}

// Loads the 32 x 128 tile (rows row0.., k k0..) of one plane, zeros outside,
// reading along whichever of rows / k is contiguous in memory: 16 asynchronous
// 8-byte copies per thread, all in flight at once (a copy of 0 source bytes
// writes a zero), then waits for them.
template <bool KCONTIG>
__device__ __forceinline__ void load_tile(const OperandView& v, int plane, long long row0,
                                          const long long* koff, double* tile) {
  const double* pb = v.base + (plane % v.np1) * v.po1 + (plane / v.np1) * v.po2;
#pragma unroll
  for (int it = 0; it < 16; ++it) {
    const int e = threadIdx.x + 256 * it;
    const int r = KCONTIG ? (e >> 7) : (e & 31);
    const int c = KCONTIG ? (e & 127) : (e >> 5);
    const long long row = row0 + r;
    const long long ko = koff[c];
    const bool in = row < v.rows && ko >= 0;
    const double* src = in ? pb + row * v.rs + ko : pb;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(
                     static_cast<unsigned>(__cvta_generic_to_shared(&tile[tile_at(r, c)]))),
                 "l"(src), "r"(in ? 8 : 0)
                 : "memory");
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// Per row: exponent e of its largest element (2^(e-1) <= max|x| < 2^e),
// stored as e + 2048 through atomicMax (0 = all zeros).  Bound by HBM (8 bytes per
// element, once).  One block covers 32 rows x kExpTileK k of one plane (grid: row
// tiles, k tiles, planes) and reads straight into registers, eight or more loads in
// flight per thread: KCONTIG (rows contiguous along k) lets each warp sweep 4 rows
// along k, a pair of elements per load where the view allows it (PAIRS, as in
// k_residues: 2 % of the preparation), otherwise each warp takes every 8th k of all
// 32 rows (consecutive rows per warp load; pairs of rows by half warps were slower).
constexpr int kExpTileK = 512;

__device__ __forceinline__ void note_exponent(unsigned* eplus, double mx) {
  if (mx > 0.0) {
    int e = 0;
    frexp(mx, &e);
    atomicMax(eplus, static_cast<unsigned>(e + 2048));
  }
}

template <bool KCONTIG, bool PAIRS>
__global__ void __launch_bounds__(256) k_row_exponent(OperandView v,
                                                      unsigned* __restrict__ eplus) {
  __shared__ long long koff[kExpTileK];
  __shared__ double part[8][33];
  const int plane = blockIdx.z;
  const long long row0 = static_cast<long long>(blockIdx.x) * 32;
  const long long k0 = static_cast<long long>(blockIdx.y) * kExpTileK;
  for (int c = threadIdx.x; c < kExpTileK; c += 256) {
    const long long kt = k0 + c;
    long long off = -1;
    if (kt < v.k_total) {
      const long long r = kt / v.k, kk = kt - r * v.k;
      off = kk * v.ks + (r % v.nbr1) * v.sr1 + (r / v.nbr1) * v.sr2;
    }
    koff[c] = off;
  }
  __syncthreads();
  const double* pb = v.base + (plane % v.np1) * v.po1 + (plane / v.np1) * v.po2;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  if (KCONTIG) {
#pragma unroll
    for (int rr = 0; rr < 4; ++rr) {
      const long long row = row0 + warp * 4 + rr;
      double mx = 0.0;
      if (row < v.rows) {
        const double* rp = pb + row * v.rs;
        if (PAIRS) {
#pragma unroll
          for (int t = 0; t < kExpTileK / 64; ++t) {
            const long long ko = koff[2 * lane + 64 * t];
            if (ko >= 0) {
              const double2 d = __ldg(reinterpret_cast<const double2*>(rp + ko));
              mx = fmax(mx, fmax(fabs(d.x), fabs(d.y)));
            }
          }
        } else {
#pragma unroll
          for (int t = 0; t < kExpTileK / 32; ++t) {
            const long long ko = koff[lane + 32 * t];
            if (ko >= 0) mx = fmax(mx, fabs(rp[ko]));
          }
        }
      }
      for (int o = 16; o; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      if (lane == 0 && row < v.rows) note_exponent(&eplus[plane * v.rows + row], mx);
    }
  } else {
    const long long row = row0 + lane;
    double mx = 0.0;
    if (row < v.rows) {
      const double* rp = pb + row * v.rs;
#pragma unroll 16
      for (int t = 0; t < kExpTileK / 8; ++t) {
        const long long ko = koff[warp + 8 * t];
        if (ko >= 0) mx = fmax(mx, fabs(rp[ko]));
      }
    }
    part[warp][lane] = mx;
    __syncthreads();
    if (warp == 0) {
      for (int w = 1; w < 8; ++w) mx = fmax(mx, part[w][lane]);
      if (row < v.rows) note_exponent(&eplus[plane * v.rows + row], mx);
    }
  }
}

// shift = beta - e (0 for an all-zero row).
__global__ void k_exponent_to_shift(const unsigned* __restrict__ eplus, long long n, int beta,
                                    int* __restrict__ shift) {
  const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t < n) shift[t] = eplus[t] ? beta - (static_cast<int>(eplus[t]) - 2048) : 0;
}

// x 2^e for exponents outside the normal range, out of line: kept off the
// per-element paths (inlined, its branches would run predicated on every
// element).
__device__ __noinline__ double ldexp_slow(double x, int e) { return ldexp(x, e); }

// 2^e as a double for -1022 <= e <= 1023 (exponent bits only).
__device__ __forceinline__ double pow2(int e) {
  return __longlong_as_double(static_cast<long long>(e + 1023) << 52);
}

struct ResidueMods {
  int L;
  int pi[kOzakiMaxModuli];
  double inv_p[kOzakiMaxModuli];
};

// FP64 integer tricks that keep the conversion unit out of the inner loops:
// (x + 1.5 2^52) - 1.5 2^52 rounds |x| < 2^51 to the nearest integer, and
// the low word of r + 1.5 2^52 is the integer r as a two's-complement int32.
constexpr double kRound = 6755399441055744.0;  // 1.5 * 2^52
__device__ __forceinline__ double round_int(double x) {
  return __dadd_rn(__dadd_rn(x, kRound), -kRound);
}
__device__ __forceinline__ int int_of(double r) { return __double2loint(__dadd_rn(r, kRound)); }

// Residues of the integer v (|v| <= 2^50) modulo p as int8 bytes.  With
// q = rint(v / p) the remainder r = v - q p lies in [-(p-1)/2, (p-1)/2] for odd
// p <= 255 and in [-128, 128] for p = 256; its low byte is r as int8 (128 as
// -128, congruent mod 256).  fma(v, 1/p, 1.5 2^52) rounds v / p exactly (for
// odd p, v / p is at least 1/(2p) >= 2^-9 away from a half-integer while the
// product's error is below |v / p| 2^-53 < 2^-10.6; p = 256 is exact) and its
// low word is q as an int32; with vl = v mod 2^32, r mod 2^32 = vl - q p.  One
// DFMA and one integer multiply-add per residue.
__device__ __forceinline__ uint32_t residue_low(int vl, double v, double inv_p, int p) {
  const int q = __double2loint(fma(v, inv_p, kRound));
  return static_cast<uint32_t>(vl - q * p);  // low byte = residue
}

// How k_residues reads its operand (residue_load picks it): 16 bytes at a time along
// k straight into registers, 16 bytes at a time along the rows through shared
// memory, or 8 bytes at a time through shared memory where alignment, an odd k or
// strides forbid pairs.
enum ResidueLoad { kPairsK = 0, kPairsRows = 1, kSingleK = 2, kSingleRows = 3 };

// Shared tile of kPairsRows, element (r, c) at c * 32 + 2 * ((r / 2) ^ (c / 8)) + r % 2:
// a copy's pair of rows stays together, and the compute reads (16 lanes per row,
// lane t at k = 8 t + q, two rows of a pair per warp) touch every bank once.
__device__ __forceinline__ int pair_at(int r, int c) {
  return c * 32 + 2 * ((r >> 1) ^ ((c >> 3) & 15)) + (r & 1);
}

// Tile of 32 rows x 128 k of one plane -> L residue rows per row: row r of
// modulus l of a plane is out row ((plane * tiles + r / T) * L + l) * T + r % T
// (T = tile_rows, the MMA tile height of this operand; tiles = rows_pad / T),
// each k_pad bytes; zeros in padding.  The L residue rows of a tile are
// T * k_pad bytes apart.  Thread (row pair rr, rr + 16; lane t of 16) converts
// the 8 consecutive k 8t .. 8t+7 of each of its rows and stores 8 residue bytes
// per modulus (16 lanes: 128 contiguous bytes per row and modulus).  The
// moduli loop is unrolled to kOzakiMaxModuli, so that p and 1/p are
// immediate constant-bank operands.  Grid: (row tiles, k tiles, planes).
//
// Bound by instruction issue, 75 % busy at 41 % of DRAM with 125 instructions per
// element, of which the 14 residues need 40 (a DFMA, a multiply-add and packing
// each): so a pair of elements is loaded at once, addresses advance by constants,
// one FMA scales an element, rounds it and leaves its low word (the scaling is
// by a power of two, so x 2^sh + 1.5 2^52 rounds once, to the same integer), and
// modulus 256, always the first, is the low byte itself.  Preparation of both operands
// (with the exponent pass): 500 x 500 x 2000 in 300 reduction batches 3.65 -> 3.13
// ms (5.8 TB/s of 16 + L bytes per element), 1200 x 900 x 900 in 64 batches 0.50 ->
// 0.45, 20000 x 6000 x 1500 0.305 -> 0.275.
template <int LOAD, int LM>
__global__ void __launch_bounds__(256, 4) k_residues(OperandView v, const int* __restrict__ shift,
                                                  ResidueMods mods, int tile_rows,
                                                  long long tiles, long long k_pad,
                                                  uint8_t* __restrict__ out) {
  __shared__ __align__(16) double tile[LOAD == kPairsK ? 2 : 32 * 128];
  __shared__ long long koff[128];
  const int plane = blockIdx.z;
  const long long row0 = static_cast<long long>(blockIdx.x) * 32;
  const long long k0 = static_cast<long long>(blockIdx.y) * 128;
  const double* pb = v.base + (plane % v.np1) * v.po1 + (plane / v.np1) * v.po2;
  tile_k_offsets(v, k0, koff);
  __syncthreads();
  const int t = threadIdx.x & 15;
  double x[2][8];
  if (LOAD == kPairsK) {
#pragma unroll
    for (int it = 0; it < 2; ++it) {
      const long long row = row0 + (threadIdx.x >> 4) + 16 * it;
      const double* rp = pb + row * v.rs;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const long long ko = koff[8 * t + 2 * q];
        double2 d = make_double2(0.0, 0.0);
        if (row < v.rows && ko >= 0) d = __ldg(reinterpret_cast<const double2*>(rp + ko));
        x[it][2 * q] = d.x;
        x[it][2 * q + 1] = d.y;
      }
    }
  } else if (LOAD == kPairsRows) {
    const long long row = row0 + 2 * t;
    const long long left = v.rows - row;
    const int full = left >= 2 ? 16 : left == 1 ? 8 : 0;
    const double* rp = pb + (full ? row : 0);
#pragma unroll
    for (int it = 0; it < 8; ++it) {
      const int c = (threadIdx.x >> 4) + 16 * it;
      const long long ko = koff[c];
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                       static_cast<unsigned>(__cvta_generic_to_shared(&tile[pair_at(2 * t, c)]))),
                   "l"(ko >= 0 ? rp + ko : pb), "r"(ko >= 0 ? full : 0)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
  } else {
    load_tile<LOAD == kSingleK>(v, plane, row0, koff, tile);
    __syncthreads();
  }
  const long long lstep = k_pad * tile_rows;  // next modulus of the same row
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const int r = (threadIdx.x >> 4) + 16 * it;
    const long long row = row0 + r;
    const int sh = row < v.rows ? shift[plane * v.rows + row] : 0;
    double xr[8];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      xr[q] = LOAD == kPairsK      ? x[it][q]
              : LOAD == kPairsRows ? tile[pair_at(r, 8 * t + q)]
                                   : tile[tile_at(r, 8 * t + q)];
    int vl[8];
    if (sh > -1000 && sh < 1000) {  // 2^sh is a normal double: scale and round in one FMA
      const double sc = pow2(sh);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const double y = fma(xr[q], sc, kRound);
        vl[q] = __double2loint(y);
        xr[q] = __dadd_rn(y, -kRound);
      }
    } else {
      for (int q = 0; q < 8; ++q) {
        xr[q] = round_int(ldexp_slow(xr[q], sh));
        vl[q] = int_of(xr[q]);
      }
    }
    // row of modulus 0 in the residue layout
    const unsigned ti = static_cast<unsigned>(row) / static_cast<unsigned>(tile_rows);
    const long long base_row =
        ((plane * tiles + ti) * mods.L) * tile_rows + (static_cast<unsigned>(row) - ti * tile_rows);
    uint8_t* dst = out + base_row * k_pad + k0 + 8 * t;
#pragma unroll
    for (int l = 0; l < (LM ? LM : kOzakiMaxModuli); ++l) {
      if (LM || l < mods.L) {
        const double ip = mods.inv_p[l];
        const int p = mods.pi[l];
        uint32_t low[8];
#pragma unroll
        for (int q = 0; q < 8; ++q)
          low[q] = l == 0 ? static_cast<uint32_t>(vl[q]) : residue_low(vl[q], xr[q], ip, p);
        *reinterpret_cast<uint2*>(dst) =
            make_uint2(__byte_perm(__byte_perm(low[0], low[1], 0x0040),
                                   __byte_perm(low[2], low[3], 0x0040), 0x5410),
                       __byte_perm(__byte_perm(low[4], low[5], 0x0040),
                                   __byte_perm(low[6], low[7], 0x0040), 0x5410));
        dst += lstep;
      }
    }
  }
}

// Pairs need 16-byte aligned addresses: even strides and base (in doubles), and along
// k an even k, so that no pair spans two reduction batches.
ResidueLoad residue_load(const OperandView& v) {
  const bool even = reinterpret_cast<std::uintptr_t>(v.base) % 16 == 0 && v.sr1 % 2 == 0 &&
                    v.sr2 % 2 == 0 && (v.np1 == 1 || v.po1 % 2 == 0) &&
                    (v.np2 == 1 || v.po2 % 2 == 0);
  if (v.ks == 1) return even && v.rs % 2 == 0 && v.k % 2 == 0 ? kPairsK : kSingleK;
  return even && v.ks % 2 == 0 ? kPairsRows : kSingleRows;
}

template <int LM>
void launch_residues(const OperandView& v, const int* shift, const ResidueMods& mods,
                     int tile_rows, long long tiles, long long k_pad, uint8_t* out, dim3 g,
                     cudaStream_t s) {
  switch (residue_load(v)) {
    case kPairsK: k_residues<kPairsK, LM><<<g, 256, 0, s>>>(v, shift, mods, tile_rows, tiles, k_pad, out); break;
    case kPairsRows: k_residues<kPairsRows, LM><<<g, 256, 0, s>>>(v, shift, mods, tile_rows, tiles, k_pad, out); break;
    case kSingleK: k_residues<kSingleK, LM><<<g, 256, 0, s>>>(v, shift, mods, tile_rows, tiles, k_pad, out); break;
    default: k_residues<kSingleRows, LM><<<g, 256, 0, s>>>(v, shift, mods, tile_rows, tiles, k_pad, out); break;
  }
}

// ---------------------------------------------------------------------------
// tcgen05 int8 product kernel
// ---------------------------------------------------------------------------
// Work item: TJ = 128 (one CTA) or 256 (a CTA pair) output columns j by tile_i
// <= 256 output rows i of one modulus and one K chunk.  A CTA holds 128 columns j
// in its 128 TMEM lanes; the two 256-column TMEM accumulators are double-buffered
// across items.
//
// What bounds it: at K = 1500 the int8 tensor pipe under the power cap (1.59 ms for
// 20000 x 6000 x 1500 and 14 moduli with no epilogue at all, 3.16 POPS) and, below
// about K = 1000, the epilogue's arithmetic and stores.  The single critical thread
// of each role must stay off that path: items advance without divisions, and the
// epilogue reduces with one conversion, FMA and multiply-add per accumulator and
// stores whole sectors.  A CTA pair (cta_group::2) shares both operands of its
// 256 x 256 tile: each CTA loads its own 128 columns j and half of the rows i, 32
// instead of 48 KiB from L2 per 512 tensor cycles.  Measured (one CTA, decoding
// every item, remainders in [0, p), 16-byte stores -> now): 20000 x 6000 x 1500 2.05
// -> 1.78 ms, 2500 x 200000 x 2000 11.7 -> 9.9, 2500 x 200000 x 500 5.0 -> 4.2,
// 1200 x 900 x 900 in 64 batches 1.06 -> 0.88.  Eight epilogue warps instead of four
// gain 3 % at K = 500 and lose 2 % at K = 1500.
constexpr int kLanes = 128;     // TMEM lanes: output columns j per CTA
constexpr int kMaxTileI = 256;  // MMA N (TMEM columns): output rows i
constexpr int kTileK = 128;     // bytes of K per pipeline stage (one 128-byte swizzle row)
constexpr int kBytesJ = kLanes * kTileK;  // 16 KiB
constexpr int kMmaK = 32;                 // K of one kind::i8 MMA
constexpr int kEpiWarps = 4;              // one per TMEM lane quarter
constexpr int kThreads = 64 + 32 * kEpiWarps;
// stages of 48 (one CTA) or 32 KiB (pair)
constexpr int stages_of(bool pair) { return pair ? 6 : 4; }
constexpr int bytes_i_of(bool pair) { return (pair ? kMaxTileI / 2 : kMaxTileI) * kTileK; }
constexpr unsigned long long kWaitLimitNs = 4000000000ULL;  // 4 s

struct MmaArgs {
  int tiles_j, tiles_i, tile_j, tile_i, L, splits, nbatch, nbo1;
  unsigned n_items;
  int step[6];  // mixed-radix digits (tj, ti, l, split, b1, b2) of the number of groups
  int a_var1, a_var2, b_var1, b_var2;  // operand planes vary with bo1 / bo2
  int planes_a, planes_b;
  long long m_pad, n_pad;
  int kb_per_split, kb_total;
  int p[kOzakiMaxModuli], c16[kOzakiMaxModuli], mode[kOzakiMaxModuli];
  float inv_p[kOzakiMaxModuli];
  uint8_t* R;
  int* err;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait for the phase of the given parity to complete.  Gives up
// (returns false, sets the CTA's abort flag and the device error flag) after
// kWaitLimitNs, or when another role of the CTA has aborted.
__device__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* err,
                          int code) {
  if (mbar_test(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  for (unsigned it = 1;; ++it) {
    if (mbar_test(bar, parity)) return true;
    if ((it & 255u) == 0) {
      if (*abort_flag) return false;
      if (global_ns() - t0 > kWaitLimitNs) {
        *abort_flag = 1;
        atomicExch(err, code);
        return false;
      }
    }
  }
}
// 2-D box load into this CTA's shared memory; bytes are counted on the barrier
// at the shared::cluster address bar (the pair's leader's when PAIR).
template <bool PAIR>
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y,
                                            uint32_t bar) {
  if (PAIR)
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        ".cta_group::2 [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
  else
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
// shared::cluster address of this CTA's shared address `a` in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_rank(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row core
// groups 1024 bytes apart (stride byte offset), version 1.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr) {
  return static_cast<uint64_t>((addr >> 4) & 0x3fffu) | (1ull << 16) |
         (static_cast<uint64_t>(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// Instruction descriptor of kind::i8: s32 accumulator, signed int8 A and B,
// both K-major, N = tile_i, M = 128 (one CTA) or 256 (pair).
__device__ __forceinline__ uint32_t i8_idesc(int tile_i, int m) {
  return (2u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(tile_i >> 3) << 17) |
         (static_cast<uint32_t>(m >> 4) << 24);
}

template <bool PAIR>
__device__ __forceinline__ void mma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                       uint32_t idesc, uint32_t accumulate) {
  if (PAIR)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, "
        "p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}" ::"r"(
            tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}
// Arrives on the barrier (of both CTAs of a pair) when the MMAs issued so far
// have completed.
template <bool PAIR>
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  if (PAIR)
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 "
        "[%0], %1;" ::"r"(bar),
        "h"(static_cast<uint16_t>(3))
        : "memory");
  else
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
        : "memory");
}

#define UW12_TMEM_LD32(taddr, v)                                                               \
  asm volatile(                                                                                \
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "  \
      "%11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, "  \
      "%28, %29, %30, %31}, [%32];"                                                            \
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),    \
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),             \
        "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),          \
        "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),          \
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]),          \
        "=r"(v[31])                                                                            \
      : "r"(taddr))

// Product residues: byte (split, batch b, column j, modulus l, row i) at
// (((split * nbatch + b) * n_pad + j) * L + l) * m_pad + i, so that the L
// residues of one column lie within L * m_pad bytes of each other.
__device__ __forceinline__ long long residue_offset(const MmaArgs& a, int split, int b,
                                                    long long j, int l) {
  return (((static_cast<long long>(split) * a.nbatch + b) * a.n_pad + j) * a.L + l) * a.m_pad;
}

// Residue bytes of an accumulator v (|v| <= 2^30) modulo p: r = v - q p with
// q = rint(float(v) / p) taken from the low bits of fma(float(v), 1/p, 1.5 2^23), as
// a signed byte stored with 128 added.  float(v) and 1/p are each off by 2^-24, so
// |r| <= p / 2 + |v| 2^-23: below 128 for short enough K chunks (kFast).  Where it
// may not be, v is first replaced by (v mod 2^16) + floor(v / 2^16) (2^16 mod p), at
// most 2^21.04, congruent modulo p (kFold).  p = 256: the low byte (kMask).  A
// conversion, an FMA and a multiply-add per accumulator, against seven integer
// instructions at half rate for a remainder in [0, p).
enum ResidueMode { kMask = 0, kFast = 1, kFold = 2 };

template <int MODE>
__device__ __forceinline__ uint32_t residue_of(uint32_t acc, int p, int c16, float inv_p) {
  int v = static_cast<int>(acc);
  if (MODE == kMask) return acc;
  if (MODE == kFold) v = (v & 0xffff) + (v >> 16) * c16;
  const int q = __float_as_int(fmaf(__int2float_rn(v), inv_p, 12582912.0f));
  return static_cast<uint32_t>(v - q * p);  // low byte: the offset 1.5 2^23 has none
}

// Four residues to one word of bytes, 128 added to each.
template <int MODE>
__device__ __forceinline__ uint32_t residue_word(const uint32_t* v, int p, int c16, float inv_p) {
  const uint32_t b01 = __byte_perm(residue_of<MODE>(v[0], p, c16, inv_p),
                                   residue_of<MODE>(v[1], p, c16, inv_p), 0x0040);
  const uint32_t b23 = __byte_perm(residue_of<MODE>(v[2], p, c16, inv_p),
                                   residue_of<MODE>(v[3], p, c16, inv_p), 0x0040);
  return __byte_perm(b01, b23, 0x5410) ^ 0x80808080u;
}

__device__ __forceinline__ uint32_t mod_u32(uint32_t u, uint32_t p, uint32_t barrett) {
  uint32_t r = u - __umulhi(u, barrett) * p;
  return r >= p ? r - p : r;
}

// One work item = one tile_j x tile_i output tile of one modulus, one K chunk and
// one batch; items are numbered tile fastest (j, then i), then modulus, K chunk,
// batch: the digits of a mixed-radix number.  A role decodes its first item and
// then adds the digits of the step (the number of groups) with carries: decoding
// every item took five 64-bit divisions, about 3000 cycles of each role's single
// critical thread per item of 2048 (K = 512) to 6144 (K = 1536) tensor cycles.
struct WorkItem {
  int tj, ti, l, split, b1, b2;

  __device__ __forceinline__ WorkItem(const MmaArgs& a, unsigned w) {
    tj = static_cast<int>(w % a.tiles_j);
    w /= a.tiles_j;
    ti = static_cast<int>(w % a.tiles_i);
    w /= a.tiles_i;
    l = static_cast<int>(w % a.L);
    w /= a.L;
    split = static_cast<int>(w % a.splits);
    w /= a.splits;
    b1 = static_cast<int>(w % a.nbo1);
    b2 = static_cast<int>(w / a.nbo1);
  }
  __device__ __forceinline__ void advance(const MmaArgs& a) {
    int carry = 0;
    auto add = [&](int& digit, int step, int radix) {
      digit += step + carry;
      carry = digit >= radix;
      digit -= carry ? radix : 0;
    };
    add(tj, a.step[0], a.tiles_j);
    add(ti, a.step[1], a.tiles_i);
    add(l, a.step[2], a.L);
    add(split, a.step[3], a.splits);
    add(b1, a.step[4], a.nbo1);
    b2 += a.step[5] + carry;
  }
  __device__ __forceinline__ int kb0(const MmaArgs& a) const { return split * a.kb_per_split; }
  __device__ __forceinline__ int nkb(const MmaArgs& a) const {
    return min(a.kb_per_split, a.kb_total - kb0(a));
  }
  // first residue row of the tile: ((plane * tiles + tile) * L + l) * tile rows
  __device__ __forceinline__ int row_j(const MmaArgs& a) const {
    const int pb = (a.b_var1 ? b1 : 0) + (a.b_var1 ? a.nbo1 : 1) * (a.b_var2 ? b2 : 0);
    return ((pb * a.tiles_j + tj) * a.L + l) * a.tile_j;
  }
  __device__ __forceinline__ int row_i(const MmaArgs& a) const {
    const int pa = (a.a_var1 ? b1 : 0) + (a.a_var1 ? a.nbo1 : 1) * (a.a_var2 ? b2 : 0);
    return ((pa * a.tiles_i + ti) * a.L + l) * a.tile_i;
  }
};

// Arrive on the barrier at a shared::cluster address.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar)
               : "memory");
}

// Persistent: one CTA (or CTA pair) per SM (pair) walks the work items group id,
// + number of groups, ... through a ring of TMA stages.  Warp roles in every
// CTA: 0 TMA producer, 1 TMEM owner and, in the pair's leader (cluster rank 0),
// MMA issuer, 2.. epilogue.  Barriers: full (the leader's; bytes of both CTAs),
// empty and acc_full (each CTA's, arrived by the commits), acc_empty (the
// leader's, arrived by the epilogue warps of both).
template <bool PAIR>
__global__ void __launch_bounds__(kThreads, 1)
    k_i8_mma(const __grid_constant__ CUtensorMap tm_j, const __grid_constant__ CUtensorMap tm_i,
             const MmaArgs a) {
  constexpr int STAGES = stages_of(PAIR);
  constexpr int BYTES_I = bytes_i_of(PAIR);
  constexpr int CTAS = PAIR ? 2 : 1;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sj = base;                            // STAGES x 16 KiB
  uint8_t* si = base + STAGES * kBytesJ;         // STAGES x BYTES_I
  uint64_t* bars = reinterpret_cast<uint64_t*>(si + STAGES * BYTES_I);
  uint64_t* full = bars;
  uint64_t* empty = bars + STAGES;
  uint64_t* acc_full = bars + 2 * STAGES;       // [2]
  uint64_t* acc_empty = bars + 2 * STAGES + 2;  // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const uint32_t rank = PAIR ? cluster_rank() : 0u;
  const unsigned group = blockIdx.x / CTAS, groups = gridDim.x / CTAS;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&full[s]), 1);
      mbar_init(smem_u32(&empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&acc_full[b]), 1);
      mbar_init(smem_u32(&acc_empty[b]), CTAS * kEpiWarps);  // one arrival per epilogue warp
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                       smem_u32(tmem_slot)),
                   "r"(static_cast<uint32_t>(2 * kMaxTileI))
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                       smem_u32(tmem_slot)),
                   "r"(static_cast<uint32_t>(2 * kMaxTileI))
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync();  // the peer's barriers are initialised
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0 && lane == 0) {
    // ---- TMA producer: this CTA's 128 columns j and its share of the rows i
    const int rows_i = a.tile_i / CTAS;
    const uint32_t bytes = static_cast<uint32_t>(CTAS * (kBytesJ + rows_i * kTileK));
    int s = 0;        // ring slot and its phase, continued across items
    uint32_t ph = 0;
    bool ok = true;
    WorkItem it(a, group);
    for (unsigned w = group; ok && w < a.n_items; w += groups, it.advance(a)) {
      const int yj = it.row_j(a) + static_cast<int>(rank) * kLanes;
      const int yi = it.row_i(a) + static_cast<int>(rank) * rows_i;
      const int kb0 = it.kb0(a), nkb = it.nkb(a);
      for (int kb = 0; kb < nkb; ++kb) {
        if (!mbar_wait(smem_u32(&empty[s]), ph ^ 1, abort_flag, a.err, 1)) {
          ok = false;
          break;
        }
        uint32_t fb = smem_u32(&full[s]);
        if (rank == 0) mbar_expect_tx(fb, bytes);
        if (PAIR) fb = map_rank(fb, 0);
        const int x = (kb0 + kb) * kTileK;
        tma_load_2d<PAIR>(smem_u32(sj + s * kBytesJ), &tm_j, x, yj, fb);
        tma_load_2d<PAIR>(smem_u32(si + s * BYTES_I), &tm_i, x, yi, fb);
        if (++s == STAGES) {
          s = 0;
          ph ^= 1;
        }
      }
    }
    if (!ok) {
      // the copies already issued land before the CTA exits: they count on barriers
      // whose phase may never complete now, so give them a millisecond
      for (const unsigned long long t0 = global_ns(); global_ns() - t0 < 1000000ULL;) {
      }
    }
  } else if (warp == 1 && lane == 0 && rank == 0) {
    // ---- MMA issuer
    const uint32_t idesc = i8_idesc(a.tile_i, CTAS * kLanes);
    int s = 0, t = 0, last_buf = -1;
    uint32_t ph = 0, last_use = 0;
    WorkItem it(a, group);
    for (unsigned w = group; w < a.n_items; w += groups, it.advance(a), ++t) {
      const int buf = t & 1;
      const uint32_t use = static_cast<uint32_t>(t >> 1);
      if (!mbar_wait(smem_u32(&acc_empty[buf]), (use & 1) ^ 1, abort_flag, a.err, 2)) break;
      tc_fence_after();
      const uint32_t d = tmem + static_cast<uint32_t>(buf * kMaxTileI);
      bool ok = true;
      const int nkb = it.nkb(a);
      for (int kb = 0; kb < nkb; ++kb) {
        if (!mbar_wait(smem_u32(&full[s]), ph, abort_flag, a.err, 2)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint64_t dj = sw128_desc(smem_u32(sj + s * kBytesJ));
        const uint64_t di = sw128_desc(smem_u32(si + s * BYTES_I));
#pragma unroll
        for (int kk = 0; kk < kTileK / kMmaK; ++kk) {
          // advance along K inside the swizzle row: +32 bytes = +2 in the
          // 16-byte address field
          mma_i8<PAIR>(d, dj + 2 * kk, di + 2 * kk, idesc, (kb | kk) != 0);
        }
        mma_commit<PAIR>(smem_u32(&empty[s]));
        if (++s == STAGES) {
          s = 0;
          ph ^= 1;
        }
      }
      mma_commit<PAIR>(smem_u32(&acc_full[buf]));  // also on failure, so the epilogue wakes
      last_buf = buf;
      last_use = use;
      if (!ok) break;
    }
    if (last_buf >= 0)  // every MMA of this CTA (pair) has completed before TMEM is released
      (void)mbar_wait(smem_u32(&acc_full[last_buf]), last_use & 1, abort_flag, a.err, 4);
  } else if (warp >= 2) {
    // ---- epilogue: TMEM -> residues mod p -> uint8 rows
    const int q = warp & 3;               // TMEM lane quarter this warp may access
    int t = 0;
    WorkItem it(a, group);
    for (unsigned w = group; w < a.n_items; w += groups, it.advance(a), ++t) {
      const int buf = t & 1;
      const uint32_t use = static_cast<uint32_t>(t >> 1);
      // warp-uniform, so that the .sync.aligned TMEM loads below are convergent
      const bool ok =
          __all_sync(0xffffffffu, mbar_wait(smem_u32(&acc_full[buf]), use & 1, abort_flag, a.err, 3));
      tc_fence_after();
      if (!ok) break;
      const int p = a.p[it.l], c16 = a.c16[it.l], mode = a.mode[it.l];
      const float inv_p = a.inv_p[it.l];
      const long long j = static_cast<long long>(it.tj) * a.tile_j + rank * kLanes + q * 32 + lane;
      uint8_t* rowp = a.R + residue_offset(a, it.split, it.b1 + a.nbo1 * it.b2, j, it.l) +
                      static_cast<long long>(it.ti) * a.tile_i;
      const uint32_t tq = tmem + static_cast<uint32_t>(buf * kMaxTileI) +
                          (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < a.tile_i / 32; ++c) {
        uint32_t v[32];
        UW12_TMEM_LD32(tq + c * 32, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        uint32_t wd[8];
        if (mode == kFast) {
#pragma unroll
          for (int e = 0; e < 8; ++e) wd[e] = residue_word<kFast>(v + 4 * e, p, c16, inv_p);
        } else if (mode == kFold) {
#pragma unroll
          for (int e = 0; e < 8; ++e) wd[e] = residue_word<kFold>(v + 4 * e, p, c16, inv_p);
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) wd[e] = residue_word<kMask>(v + 4 * e, p, c16, inv_p);
        }
        // one whole 32-byte sector per lane
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(rowp + c * 32),
                     "r"(wd[0]), "r"(wd[1]), "r"(wd[2]), "r"(wd[3]), "r"(wd[4]), "r"(wd[5]),
                     "r"(wd[6]), "r"(wd[7])
                     : "memory");
      }
      // this warp's TMEM reads are done: release the accumulator
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        const uint32_t bar = smem_u32(&acc_empty[buf]);
        mbar_arrive_cluster(PAIR ? map_rank(bar, 0) : bar);
      }
    }
  }

  tc_fence_before();
  __syncwarp();
  __syncthreads();
  if (PAIR) cluster_sync();  // no MMA, copy or arrival of the pair is outstanding
  if (warp == 1) {
    tc_fence_after();
    __syncwarp();
    if (PAIR)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                   "r"(static_cast<uint32_t>(2 * kMaxTileI))
                   : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                   "r"(static_cast<uint32_t>(2 * kMaxTileI))
                   : "memory");
  }
}

// ---------------------------------------------------------------------------
// CRT reconstruction
// ---------------------------------------------------------------------------
struct CrtArgs {
  const uint8_t* R;
  long long m, n, m_pad, n_pad;
  int splits, L, nch, nbatch, nbo1;
  const int* shift_a;
  const int* shift_b;
  int a_var1, a_var2, b_var1, b_var2;
  long long rows_a, rows_b;  // rows per shift plane (m, n)
  double* C;
  long long ldc, sCo1, sCo2;
  double alpha, beta;
  uint32_t p[kOzakiMaxModuli], barrett[kOzakiMaxModuli];
  uint32_t red_off[kOzakiMaxModuli];  // REDUCE: undoes the 128 added to each K chunk's residue
  double w[kOzakiMaxModuli][kMaxChunks];
  double mc[kMaxChunks];
  double inv_m;
  int cw;          // CRT chunk width in bits
  uint32_t w8[16][4];                  // k_crt_pipe (Consts)
  double m32[4], per_m[4], bias[4];
  int c_aligned;   // C, ldc and the batch strides allow 16-byte accesses
};

// Several K chunks (small outputs): one thread = four consecutive rows i of a
// column j of one batch; grid (row blocks of 1024, columns strided by gridDim.y,
// batches).  The L residue words of a column (and the elements of C when beta != 0)
// are loaded before any is used, the K-chunk sums of the four bytes are kept as
// pairs of 16-bit lanes, the CRT runs on NCH chunks of cw bits, and C is read and
// written 16 bytes at a time when aligned.
// x 2^e: one multiply by an exactly representable power of two when 2^e is a
// normal double, ldexp otherwise.
__device__ __forceinline__ double scale_pow2(double x, int e) {
  if (e >= -1022 && e <= 1023) return x * pow2(e);
  return ldexp_slow(x, e);
}

// s + e = a + b exactly (Knuth's TwoSum, six FP64 operations).
__device__ __forceinline__ double two_sum(double a, double b, double& e) {
  const double s = __dadd_rn(a, b);
  const double bb = __dsub_rn(s, a);
  e = __dadd_rn(__dsub_rn(a, __dsub_rn(s, bb)), __dsub_rn(b, bb));
  return s;
}

// sum_c d[c] 2^(cw c) for integer-valued doubles |d[c]| < 2^53: every term
// d[c] 2^(cw c) is exact, the running sum is carried error-free (TwoSum) and
// the integer errors are added at the end, so the result equals the exact sum
// whenever that is a double and is within one unit in the last place
// otherwise.
template <int NCH>
__device__ __forceinline__ double join_chunks(const double (&d)[NCH], double chunk) {
  double pw = 1.0;
  double terms[NCH];
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    terms[c] = d[c] * pw;  // exact: a power-of-two scaling
    pw *= chunk;
  }
  double sum = terms[NCH - 1], err = 0.0;
#pragma unroll
  for (int c = NCH - 2; c >= 0; --c) {
    double e;
    sum = two_sum(sum, terms[c], e);
    err += e;
  }
  return sum + err;
}

// Residue (< 2^16) to double without the conversion unit.
__device__ __forceinline__ double small_to_double(uint32_t r) {
  return __dsub_rn(__hiloint2double(0x43300000, static_cast<int>(r)), 4503599627370496.0);
}

// Stored residues are bytes in [0, 255], 128 more than a residue in [-128, 127]; the
// sums of the (at most 256) K chunks' bytes are reduced mod p, red_off undoing the
// 128 of each.
template <int NCH>
__global__ void __launch_bounds__(256, 2) k_crt(const CrtArgs a) {
  constexpr int E = 4;
  const long long i0 = (static_cast<long long>(blockIdx.x) * 256 + threadIdx.x) * E;
  if (i0 >= a.m) return;
  const int b = blockIdx.z;
  const int b1 = b % a.nbo1, b2 = b / a.nbo1;
  const int pa = (a.a_var1 ? b1 : 0) + (a.a_var1 ? a.nbo1 : 1) * (a.a_var2 ? b2 : 0);
  const int pb = (a.b_var1 ? b1 : 0) + (a.b_var1 ? a.nbo1 : 1) * (a.b_var2 ? b2 : 0);
  // residue layout of k_i8_mma: (((split * nbatch + b) * n_pad + j) * L + l) * m_pad + i
  const long long lstride = a.m_pad;                                             // next modulus
  const long long sstride = static_cast<long long>(a.nbatch) * a.n_pad * a.L * a.m_pad;  // K chunk
  int sa[E];
#pragma unroll
  for (int e = 0; e < E; ++e)
    sa[e] = i0 + e < a.m ? a.shift_a[pa * a.rows_a + i0 + e] : 0;
  const double chunk = __longlong_as_double(static_cast<long long>(a.cw + 1023) << 52);  // 2^cw

  const bool vec = i0 + E - 1 < a.m && a.c_aligned;
  for (long long j = blockIdx.y; j < a.n; j += gridDim.y) {
    const uint8_t* base = a.R + (static_cast<long long>(b) * a.n_pad + j) * a.L * a.m_pad + i0;
    double* Cb = a.C + b1 * a.sCo1 + b2 * a.sCo2 + j * a.ldc;
    uint32_t w0[kOzakiMaxModuli];
#pragma unroll
    for (int l = 0; l < kOzakiMaxModuli; ++l)
      if (l < a.L) w0[l] = __ldg(reinterpret_cast<const uint32_t*>(base + l * lstride));
    double cold[E];
#pragma unroll
    for (int e = 0; e < E; ++e) cold[e] = 0.0;
    if (a.beta != 0.0) {
      if (vec) {
#pragma unroll
        for (int e = 0; e < E; e += 2) {
          const double2 c2 = *reinterpret_cast<const double2*>(Cb + i0 + e);
          cold[e] = c2.x;
          cold[e + 1] = c2.y;
        }
      } else {
#pragma unroll
        for (int e = 0; e < E; ++e)
          if (i0 + e < a.m) cold[e] = Cb[i0 + e];
      }
    }
    double S[E][NCH];
#pragma unroll
    for (int e = 0; e < E; ++e)
#pragma unroll
      for (int c = 0; c < NCH; ++c) S[e][c] = 0.0;
    // byte sums in 16-bit lanes (bytes 0, 2 and 1, 3), reduced mod p
    uint32_t s02[kOzakiMaxModuli], s13[kOzakiMaxModuli];
#pragma unroll
    for (int l = 0; l < kOzakiMaxModuli; ++l) {
      if (l < a.L) {
        s02[l] = w0[l] & 0x00ff00ffu;
        s13[l] = (w0[l] >> 8) & 0x00ff00ffu;
      }
    }
    for (int sp = 1; sp < a.splits; ++sp) {
#pragma unroll
      for (int l = 0; l < kOzakiMaxModuli; ++l) {
        if (l < a.L) {
          const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(base + sp * sstride + l * lstride));
          s02[l] += w & 0x00ff00ffu;
          s13[l] += (w >> 8) & 0x00ff00ffu;
        }
      }
    }
#pragma unroll
    for (int l = 0; l < kOzakiMaxModuli; ++l) {
      if (l < a.L) {
        const uint32_t p = a.p[l], bm = a.barrett[l];
        const uint32_t u[4] = {s02[l] & 0xffffu, s13[l] & 0xffffu, s02[l] >> 16, s13[l] >> 16};
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const double r = small_to_double(mod_u32(u[e] + a.red_off[l], p, bm));
#pragma unroll
          for (int c = 0; c < NCH; ++c) S[e][c] = fma(r, a.w[l][c], S[e][c]);
        }
      }
    }
    const int sb = a.shift_b[pb * a.rows_b + j];
    double out[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      double approx = 0.0;
#pragma unroll
      for (int c = NCH - 1; c >= 0; --c) approx = fma(approx, chunk, S[e][c]);
      const double q = round_int(approx * a.inv_m);  // |q| < 2^13
      double dig[NCH];
#pragma unroll
      for (int c = 0; c < NCH; ++c) dig[c] = fma(-q, a.mc[c], S[e][c]);  // exact
      out[e] = a.alpha * scale_pow2(join_chunks<NCH>(dig, chunk), -(sa[e] + sb));
      if (a.beta != 0.0) out[e] = fma(a.beta, cold[e], out[e]);
    }
    if (vec) {
#pragma unroll
      for (int e = 0; e < E; e += 2)
        *reinterpret_cast<double2*>(Cb + i0 + e) = make_double2(out[e], out[e + 1]);
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e)
        if (i0 + e < a.m) Cb[i0 + e] = out[e];
    }
  }
}

// One K chunk, pipelined: a block owns 512 rows i of a batch and walks its
// columns j = blockIdx.y, + gridDim.y, ...; the L residue rows of the next
// kCrtStages - 1 columns are copied into shared memory (16-byte cp.async.cg) while
// the current one is reconstructed.
//
// The weighted sum sum_l r_l w_l of an element is a small matrix product of bytes:
// 16 residues by the 16 bytes of every weight.  On the FP64 pipe it took 42 FMAs
// and 14 conversions per element, the larger part of the 224 instructions that
// bounded this kernel; mma.sync m16n8k32 (u8) forms it instead.  The A operand's row
// holds four elements 16 apart (four groups of 16 moduli along K, two k steps),
// read by ldmatrix.trans out of the modulus-major rows; column n of B carries one
// byte of the weights in the K group n / 2 only, so that the two columns a thread
// holds of every product are bytes 2 j and 2 j + 1 of one element: each thread ends
// up with all 16 byte sums (exact, below 2^20) of two elements, with no exchange
// between lanes.  Half of the products are with zeros: 16 MMAs per 64 elements, 68
// cycles of the tensor pipe per 32, beside 64 of the FP64 pipe.
//
// Byte sums join to four digits of 32 bits (below 2^44) in integers, become doubles
// (minus the bias of the 128 in every stored residue), lose q M, q the rounded
// quotient by M (|C'| <= M / 4), and join error-free: exactly when the product is a
// double, within one unit in the last place otherwise.  20000 x 6000 at 14 moduli 0.95
// -> 0.77 ms; now 60 % of the pipe that FP64 and these MMAs share, half each.
constexpr int kCrtStages = 3;
constexpr int kCrtRows = 512;             // rows i per block, 128 per warp
constexpr int kCrtThreads = 128;
constexpr int kCrtPitch = kCrtRows + 16;  // bytes of a modulus row: ldmatrix rows in distinct banks

__device__ __forceinline__ void mma_u8(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int LM>
__global__ void __launch_bounds__(kCrtThreads, 4) k_crt_pipe(const CrtArgs a) {
  extern __shared__ __align__(16) uint8_t crt_smem[];  // kCrtStages x L x kCrtPitch bytes
  const int L = LM ? LM : a.L;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const long long iblk = static_cast<long long>(blockIdx.x) * kCrtRows;
  const long long iw = iblk + warp * 128;  // first row of this warp
  const int b = blockIdx.z;
  const int b1 = b % a.nbo1, b2 = b / a.nbo1;
  const int pa = (a.a_var1 ? b1 : 0) + (a.a_var1 ? a.nbo1 : 1) * (a.a_var2 ? b2 : 0);
  const int pb = (a.b_var1 ? b1 : 0) + (a.b_var1 ? a.nbo1 : 1) * (a.b_var2 ? b2 : 0);
  // bytes of this block's rows inside one residue row (a multiple of 32)
  const int row_bytes = static_cast<int>(min(static_cast<long long>(kCrtRows), a.m_pad - iblk));
  const long long nj = (a.n - blockIdx.y + gridDim.y - 1) / gridDim.y;
  const bool active = iw < a.m;
  // this thread's elements: rows iw + 64 z + 16 t + g + 8 h
  int sa[2][2];
#pragma unroll
  for (int z = 0; z < 2; ++z)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long long i = iw + 64 * z + 16 * t + g + 8 * h;
      sa[z][h] = i < a.m ? a.shift_a[pa * a.rows_a + i] : 0;
    }
  uint32_t w[8], in_group[4];
#pragma unroll
  for (int q = 0; q < 8; ++q) w[q] = a.w8[2 * q + (g & 1)][t];
#pragma unroll
  for (int u = 0; u < 4; ++u) in_group[u] = (g >> 1) == u ? 0xffffffffu : 0u;
  // ldmatrix row of this lane: modulus lane % 16 of the first or second matrix
  const unsigned ld_row = static_cast<unsigned>(__cvta_generic_to_shared(crt_smem)) +
                          min(lane & 15, L - 1) * kCrtPitch + warp * 128 + 16 * (lane >> 4);

  // copy lane: 16 bytes at (threadIdx.x % 32) of every fourth modulus row
  const int cp_off = (threadIdx.x & 31) * 16;
  const bool cp_in = cp_off < row_bytes;
  auto issue = [&](long long q, int slot) {
    const long long j = blockIdx.y + q * gridDim.y;
    const uint8_t* src = a.R + ((static_cast<long long>(b) * a.n_pad + j) * L + warp) * a.m_pad +
                         iblk + (cp_in ? cp_off : 0);
    unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(crt_smem)) +
                   (slot * L + warp) * kCrtPitch + cp_off;
#pragma unroll
    for (int l0 = 0; l0 < (LM ? LM : kOzakiMaxModuli); l0 += 4) {
      if (l0 + warp < L)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src),
                     "r"(cp_in ? 16 : 0)
                     : "memory");
      src += 4 * a.m_pad;
      dst += 4 * kCrtPitch;
    }
  };

#pragma unroll
  for (int q = 0; q < kCrtStages - 1; ++q) {
    if (q < nj) issue(q, q);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  int slot = 0;
  for (long long q = 0; q < nj; ++q) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kCrtStages - 2) : "memory");
    __syncthreads();  // column q landed; the slot refilled below is no longer read
    {
      const long long qn = q + kCrtStages - 1;
      const int to = slot == 0 ? kCrtStages - 1 : slot - 1;  // (slot + kCrtStages - 1) % kCrtStages
      if (qn < nj) issue(qn, to);
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    const unsigned ld = ld_row + slot * L * kCrtPitch;
    slot = slot + 1 == kCrtStages ? 0 : slot + 1;
    if (!active) continue;
    const long long j = blockIdx.y + q * gridDim.y;
    double* Cb = a.C + b1 * a.sCo1 + b2 * a.sCo2 + j * a.ldc + iw + 16 * t + g;
    const int sb = a.shift_b[pb * a.rows_b + j];
#pragma unroll
    for (int z = 0; z < 2; ++z) {
      double* dst = Cb + 64 * z;
      bool in[2];
      double cold[2];  // read ahead of the products
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        in[h] = iw + 64 * z + 16 * t + g + 8 * h < a.m;
        cold[h] = a.beta != 0.0 && in[h] ? dst[8 * h] : 0.0;
      }
      int acc[8][4];
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[n][c] = 0;
#pragma unroll
      for (int ks = 0; ks < 2; ++ks) {
        uint32_t r[4];
        asm volatile("ldmatrix.sync.aligned.m16n16.x2.trans.shared.b8 {%0, %1, %2, %3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(ld + 64 * z + 32 * ks)
                     : "memory");
#pragma unroll
        for (int n = 0; n < 8; ++n)
          mma_u8(acc[n], r, w[n] & in_group[2 * ks], w[n] & in_group[2 * ks + 1]);
      }
      double x[2][4], v[2];
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t lo = static_cast<uint32_t>(acc[2 * m][2 * h] + (acc[2 * m][2 * h + 1] << 8));
          const uint32_t hi =
              static_cast<uint32_t>(acc[2 * m + 1][2 * h] + (acc[2 * m + 1][2 * h + 1] << 8));
          const unsigned long long d = lo + (static_cast<unsigned long long>(hi) << 16);
          x[h][m] = __dsub_rn(__longlong_as_double(static_cast<long long>(d | 0x4330000000000000ULL)),
                              a.bias[m]);
        }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        // the low digits are below 2^-31 of M at the default modulus count
        double approx = fma(x[h][3], a.per_m[3], x[h][2] * a.per_m[2]);
        if (!LM) approx = fma(x[h][1], a.per_m[1], fma(x[h][0], a.per_m[0], approx));
        const double quo = round_int(approx);  // |q| < 2^13
#pragma unroll
        for (int m = 0; m < 4; ++m) x[h][m] = fma(-quo, a.m32[m], x[h][m]);  // exact
        if (LM) {
          const double d[3] = {x[h][0], x[h][1], fma(x[h][3], 4294967296.0, x[h][2])};  // exact: < 2^47
          v[h] = join_chunks<3>(d, 4294967296.0);
        } else {
          v[h] = join_chunks<4>(x[h], 4294967296.0);
        }
      }
      const int e0 = -(sa[z][0] + sb), e1 = -(sa[z][1] + sb);
      if (min(e0, e1) >= -1022 && max(e0, e1) <= 1023) {
        v[0] *= pow2(e0);
        v[1] *= pow2(e1);
      } else {
        v[0] = scale_pow2(v[0], e0);
        v[1] = scale_pow2(v[1], e1);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (in[h]) dst[8 * h] = a.beta != 0.0 ? fma(a.beta, cold[h], a.alpha * v[h]) : a.alpha * v[h];
    }
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                 const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                 const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_fn() {
  static std::once_flag once;
  static EncodeTiled fn = nullptr;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiled>(p);
  });
  if (!fn) throw Error(kErrCuda, "cuTensorMapEncodeTiled is not available");
  return fn;
}

// 2-D uint8 map over rows x k_pad bytes, box = box_rows x 128 bytes, 128-byte swizzle.
CUtensorMap make_map(const uint8_t* base, long long rows, long long k_pad, int box_rows) {
  CUtensorMap m;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(k_pad), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(k_pad)};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(kTileK), static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(base),
                                 dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                 CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    throw Error(kErrCuda, "cuTensorMapEncodeTiled failed (" + std::to_string(int(r)) + ")");
  return m;
}

constexpr size_t mma_smem(bool pair) {
  return size_t(stages_of(pair)) * (kBytesJ + bytes_i_of(pair)) + 1024 /*alignment*/ +
         256 /*barriers*/;
}

long long round_up(long long x, long long m) { return (x + m - 1) / m * m; }

int num_sms() {
  static int n[kMaxDevices] = {};
  static std::mutex mu;
  int dev = 0;
  UW12_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) throw Error(kErrInvalid, "device index out of range");
  std::lock_guard<std::mutex> lk(mu);
  if (!n[dev]) UW12_CUDA(cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev));
  return n[dev];
}

struct Timer {
  int kind;
  double work;
  std::string shape;
  cudaEvent_t a = nullptr, b = nullptr;
  cudaStream_t s;
  Timer(int kind_, double work_, std::string shape_, cudaStream_t s_)
      : kind(kind_), work(work_), shape(std::move(shape_)), s(s_) {
    if (!profile_enabled()) return;
    UW12_CUDA(cudaEventCreate(&a));
    UW12_CUDA(cudaEventCreate(&b));
    UW12_CUDA(cudaEventRecord(a, s));
  }
  void stop() {
    if (!a) return;
    UW12_CUDA(cudaEventRecord(b, s));
    profile_record(kind, a, b, work, shape);
    a = b = nullptr;
  }
};

// Output tile of the int8 products: the pair's 256 columns j unless they would be
// mostly padding (one CTA is 1.2 to 1.4 times slower per padded column), and the
// rows i per tile, a multiple of 32, that pad m least (the wider one of two
// that differ by less than a sixteenth).
struct ProductTile {
  bool pair;
  int tile_j, tile_i;
};
ProductTile product_tile(long long m, long long n) {
  ProductTile t;
  t.pair = 4 * round_up(n, 2 * kLanes) <= 5 * round_up(n, kLanes);
  t.tile_j = t.pair ? 2 * kLanes : kLanes;
  t.tile_i = kMaxTileI;
  for (int ti = kMaxTileI; ti >= 128; ti -= 32)
    if (16 * round_up(m, ti) < 15 * round_up(m, t.tile_i)) t.tile_i = ti;
  return t;
}

// Runs one GEMM whose temporaries fit.  d.nbo2 == 1 or both batch dims are
// handled through the plane maps.
void run_core(const GemmDesc& d, const Consts& cs, int beta, cudaStream_t s) {
  const int L = cs.L;
  const long long nbo1 = d.nbo1, nbo2 = d.nbo2, nbatch = nbo1 * nbo2;
  const long long k_total = d.k * d.nbr1 * d.nbr2;
  const long long k_pad = round_up(k_total, kTileK);
  const ProductTile pt = product_tile(d.m, d.n);
  const long long m_pad = round_up(d.m, pt.tile_i), n_pad = round_up(d.n, pt.tile_j);
  const int a_var1 = d.sAo1 != 0 && nbo1 > 1, a_var2 = d.sAo2 != 0 && nbo2 > 1;
  const int b_var1 = d.sBo1 != 0 && nbo1 > 1, b_var2 = d.sBo2 != 0 && nbo2 > 1;
  const int pa1 = a_var1 ? int(nbo1) : 1, pa2 = a_var2 ? int(nbo2) : 1;
  const int pb1 = b_var1 ? int(nbo1) : 1, pb2 = b_var2 ? int(nbo2) : 1;
  const long long planes_a = pa1 * pa2, planes_b = pb1 * pb2;

  // K chunks: <= kMaxKChunk bytes each; more chunks when the tile grid alone
  // would leave SMs idle.
  const long long kb_total = k_pad / kTileK;
  const long long tiles_j = n_pad / pt.tile_j, tiles_i = m_pad / pt.tile_i;
  const long long items = tiles_j * tiles_i * L * nbatch;
  const long long groups = num_sms() / (pt.pair ? 2 : 1);
  long long splits = (k_pad + kMaxKChunk - 1) / kMaxKChunk;
  const long long want = (2 * groups + items - 1) / items;
  splits = std::max(splits, std::min(want, std::max<long long>(1, kb_total / 8)));
  splits = std::min(splits, std::max<long long>(1, 65535 / nbatch));
  splits = std::min<long long>(splits, 256);  // byte sums of the chunks fit 16 bits
  long long kb_per = (kb_total + splits - 1) / splits;
  kb_per = std::min<long long>(kb_per, kMaxKChunk / kTileK);
  splits = (kb_total + kb_per - 1) / kb_per;
  if (splits * nbatch > 65535) throw Error(kErrInvalid, "split-precision GEMM: too many batches");

  DevBuf resA((L * planes_a * m_pad * k_pad + 7) / 8, s);
  DevBuf resB((L * planes_b * n_pad * k_pad + 7) / 8, s);
  DevBuf shA((planes_a * d.m + 1) / 2, s), shB((planes_b * d.n + 1) / 2, s);
  DevBuf exA((planes_a * d.m + 1) / 2, s), exB((planes_b * d.n + 1) / 2, s);
  unsigned* ea = reinterpret_cast<unsigned*>(exA.get());
  unsigned* eb = reinterpret_cast<unsigned*>(exB.get());
  DevBuf R((splits * L * nbatch * n_pad * m_pad + 7) / 8, s);
  uint8_t* ra = reinterpret_cast<uint8_t*>(resA.get());
  uint8_t* rb = reinterpret_cast<uint8_t*>(resB.get());
  int* sa = reinterpret_cast<int*>(shA.get());
  int* sb = reinterpret_cast<int*>(shB.get());

  // ---- operand views: A rows = i (m), B rows = j (n)
  OperandView va{d.A, d.m, d.k, k_total,
                 d.a_kcontig ? d.lda : 1, d.a_kcontig ? 1 : d.lda, d.sAr1, d.sAr2, d.nbr1,
                 d.sAo1, d.sAo2, pa1, pa2};
  OperandView vb{d.B, d.n, d.k, k_total,
                 d.b_ncontig ? 1 : d.ldb, d.b_ncontig ? d.ldb : 1, d.sBr1, d.sBr2, d.nbr1,
                 d.sBo1, d.sBo2, pb1, pb2};
  ResidueMods mods;
  mods.L = L;
  for (int l = 0; l < L; ++l) {
    mods.pi[l] = static_cast<int>(cs.p[l]);
    mods.inv_p[l] = cs.inv_p[l];
  }
  {
    const double bytes = 8.0 * double(planes_a * d.m + planes_b * d.n) * double(k_total) * 2.0 +
                         double(L) * double(planes_a * m_pad + planes_b * n_pad) * double(k_pad);
    Timer tm(kProfSplitPrep, bytes, "prep", s);
    auto prep = [&](const OperandView& v, long long planes, long long rows_pad, int tile_rows,
                    int* sh, unsigned* ep, uint8_t* out) {
      UW12_CUDA(cudaMemsetAsync(ep, 0, planes * v.rows * sizeof(unsigned), s));
      dim3 ge(static_cast<unsigned>(rows_pad / 32),
              static_cast<unsigned>((k_pad + kExpTileK - 1) / kExpTileK),
              static_cast<unsigned>(planes));
      switch (residue_load(v)) {
        case kPairsK: k_row_exponent<true, true><<<ge, 256, 0, s>>>(v, ep); break;
        case kSingleK: k_row_exponent<true, false><<<ge, 256, 0, s>>>(v, ep); break;
        default: k_row_exponent<false, false><<<ge, 256, 0, s>>>(v, ep); break;
      }
      dim3 g(static_cast<unsigned>(rows_pad / 32), static_cast<unsigned>(k_pad / 128),
             static_cast<unsigned>(planes));
      UW12_LAUNCHED();
      const long long nsh = planes * v.rows;
      k_exponent_to_shift<<<static_cast<unsigned>((nsh + 255) / 256), 256, 0, s>>>(ep, nsh, beta,
                                                                                  sh);
      UW12_LAUNCHED();
      const long long tiles = rows_pad / tile_rows;
      // the default modulus count runs a fully unrolled, unguarded moduli loop
      if (L == kOzakiDefaultModuli)
        launch_residues<kOzakiDefaultModuli>(v, sh, mods, tile_rows, tiles, k_pad, out, g, s);
      else
        launch_residues<0>(v, sh, mods, tile_rows, tiles, k_pad, out, g, s);
      UW12_LAUNCHED();
    };
    prep(va, planes_a, m_pad, pt.tile_i, sa, ea, ra);
    prep(vb, planes_b, n_pad, pt.tile_j, sb, eb, rb);
    tm.stop();
  }

  // ---- int8 products
  {
    static std::mutex attr_mu;
    static bool attr_set[64] = {};
    {
      int dev = 0;
      UW12_CUDA(cudaGetDevice(&dev));
      std::lock_guard<std::mutex> lk(attr_mu);
      if (!attr_set[dev]) {
        UW12_CUDA(cudaFuncSetAttribute(k_i8_mma<false>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(mma_smem(false))));
        UW12_CUDA(cudaFuncSetAttribute(k_i8_mma<true>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(mma_smem(true))));
        attr_set[dev] = true;
      }
    }
    const CUtensorMap tmj = make_map(rb, L * planes_b * n_pad, k_pad, kLanes);
    const CUtensorMap tmi = make_map(ra, L * planes_a * m_pad, k_pad,
                                     pt.tile_i / (pt.pair ? 2 : 1));
    MmaArgs ma{};
    ma.tiles_j = static_cast<int>(tiles_j);
    ma.tiles_i = static_cast<int>(tiles_i);
    ma.tile_j = pt.tile_j;
    ma.tile_i = pt.tile_i;
    const long long n_items = tiles_j * tiles_i * L * splits * nbatch;
    if (n_items >= (1LL << 31) || L * planes_a * m_pad >= (1LL << 31) ||
        L * planes_b * n_pad >= (1LL << 31))
      throw Error(kErrInvalid, "split-precision GEMM: too many output tiles");
    ma.n_items = static_cast<unsigned>(n_items);
    ma.L = L;
    ma.splits = static_cast<int>(splits);
    ma.nbatch = static_cast<int>(nbatch);
    ma.nbo1 = static_cast<int>(nbo1);
    ma.a_var1 = a_var1; ma.a_var2 = a_var2; ma.b_var1 = b_var1; ma.b_var2 = b_var2;
    ma.planes_a = static_cast<int>(planes_a);
    ma.planes_b = static_cast<int>(planes_b);
    ma.m_pad = m_pad;
    ma.n_pad = n_pad;
    ma.kb_per_split = static_cast<int>(kb_per);
    ma.kb_total = static_cast<int>(kb_total);
    for (int l = 0; l < L; ++l) {
      const int p = static_cast<int>(cs.p[l]);
      const double vmax = double(std::min(k_total, kb_per * kTileK)) * double(p / 2) * (p / 2);
      ma.p[l] = p;
      ma.inv_p[l] = 1.0f / float(p);
      ma.c16[l] = 65536 % p > p / 2 ? 65536 % p - p : 65536 % p;
      ma.mode[l] = p == 256 ? kMask : 0.5 * p + vmax * 0x1p-23 < 127.99 ? kFast : kFold;
    }
    ma.R = reinterpret_cast<uint8_t*>(R.get());
    ma.err = err_flag();
    const double ops = 2.0 * double(d.m) * double(d.n) * double(k_total) * double(L) * nbatch;
    char shape[160];
    std::snprintf(shape, sizeof(shape), "i8 %lld %lld %lld %lld L%d s%lld", d.m, d.n, k_total,
                  nbatch, L, splits);
    Timer tm(kProfI8Mma, ops, shape, s);
    const unsigned n_groups = static_cast<unsigned>(std::min<long long>(n_items, groups));
    {
      const int radix[5] = {ma.tiles_j, ma.tiles_i, ma.L, ma.splits, ma.nbo1};
      unsigned rest = n_groups;
      for (int q = 0; q < 5; ++q) {
        ma.step[q] = static_cast<int>(rest % radix[q]);
        rest /= radix[q];
      }
      ma.step[5] = static_cast<int>(rest);
    }
    if (pt.pair) {
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3(2 * n_groups);
      cfg.blockDim = dim3(kThreads);
      cfg.dynamicSmemBytes = mma_smem(true);
      cfg.stream = s;
      cudaLaunchAttribute attr{};
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = 2;
      attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
      cfg.attrs = &attr;
      cfg.numAttrs = 1;
      UW12_CUDA(cudaLaunchKernelEx(&cfg, k_i8_mma<true>, tmj, tmi, ma));
    } else {
      k_i8_mma<false><<<n_groups, kThreads, mma_smem(false), s>>>(tmj, tmi, ma);
    }
    UW12_LAUNCHED();
    tm.stop();
  }

  // ---- CRT reconstruction
  {
    CrtArgs ca{};
    ca.R = reinterpret_cast<const uint8_t*>(R.get());
    ca.m = d.m; ca.n = d.n; ca.m_pad = m_pad; ca.n_pad = n_pad;
    ca.splits = static_cast<int>(splits);
    ca.L = L;
    ca.nch = cs.nch;
    ca.nbatch = static_cast<int>(nbatch);
    ca.nbo1 = static_cast<int>(nbo1);
    ca.shift_a = sa; ca.shift_b = sb;
    ca.a_var1 = a_var1; ca.a_var2 = a_var2; ca.b_var1 = b_var1; ca.b_var2 = b_var2;
    ca.rows_a = d.m; ca.rows_b = d.n;
    ca.C = d.C; ca.ldc = d.ldc; ca.sCo1 = d.sCo1; ca.sCo2 = d.sCo2;
    ca.alpha = d.alpha; ca.beta = d.beta;
    for (int l = 0; l < L; ++l) {
      ca.p[l] = cs.p[l];
      ca.barrett[l] = cs.barrett[l];
      ca.red_off[l] = cs.p[l] - static_cast<uint32_t>(128 * splits % cs.p[l]);
      for (int c = 0; c < kMaxChunks; ++c) ca.w[l][c] = cs.w[l][c];
    }
    for (int q = 0; q < 16; ++q)
      for (int t = 0; t < 4; ++t) ca.w8[q][t] = cs.w8[q][t];
    for (int m = 0; m < 4; ++m) {
      ca.m32[m] = cs.m32[m];
      ca.per_m[m] = cs.per_m[m];
      ca.bias[m] = cs.bias[m];
    }
    for (int c = 0; c < kMaxChunks; ++c) ca.mc[c] = cs.mc[c];
    ca.inv_m = cs.inv_m;
    ca.cw = cs.cw;
    ca.c_aligned = (reinterpret_cast<std::uintptr_t>(d.C) % 16 == 0) && d.ldc % 2 == 0 &&
                   d.sCo1 % 2 == 0 && d.sCo2 % 2 == 0;
    const double bytes = double(splits * L) * double(d.m * d.n * nbatch) +
                         8.0 * double(d.m * d.n * nbatch) * (d.beta != 0.0 ? 2.0 : 1.0);
    Timer tm(kProfSplitCrt, bytes, "crt", s);
    if (splits == 1) {
      // about eight waves of 4 blocks per SM (a short tail), each block walking its
      // share of the columns
      const long long gx = (d.m + kCrtRows - 1) / kCrtRows;
      const long long per_col = gx * nbatch;
      const long long gy = std::min<long long>(
          std::min<long long>(d.n, 65535),
          std::max<long long>(1, (32LL * num_sms() + per_col - 1) / per_col));
      const dim3 g(static_cast<unsigned>(gx), static_cast<unsigned>(gy),
                   static_cast<unsigned>(nbatch));
      const size_t smem = size_t(kCrtStages) * L * kCrtPitch;
      if (L == kOzakiDefaultModuli)
        k_crt_pipe<kOzakiDefaultModuli><<<g, kCrtThreads, smem, s>>>(ca);
      else
        k_crt_pipe<0><<<g, kCrtThreads, smem, s>>>(ca);
    } else {
      const dim3 g(static_cast<unsigned>((d.m + 1023) / 1024),
                   static_cast<unsigned>(std::min<long long>(d.n, 65535)),
                   static_cast<unsigned>(nbatch));
      switch (cs.nch) {
        case 1: k_crt<1><<<g, 256, 0, s>>>(ca); break;
        case 2: k_crt<2><<<g, 256, 0, s>>>(ca); break;
        case 3: k_crt<3><<<g, 256, 0, s>>>(ca); break;
        default: k_crt<4><<<g, 256, 0, s>>>(ca); break;
      }
    }
    UW12_LAUNCHED();
    tm.stop();
  }
}

long long slab_bytes(long long L, long long m, long long n, long long k_total, long long nbatch,
                     long long planes_a, long long planes_b) {
  const long long k_pad = round_up(k_total, kTileK);
  const ProductTile pt = product_tile(m, n);
  const long long m_pad = round_up(m, pt.tile_i), n_pad = round_up(n, pt.tile_j);
  const long long splits = std::max<long long>(1, (k_pad + kMaxKChunk - 1) / kMaxKChunk);
  return L * (planes_a * m_pad + planes_b * n_pad) * k_pad +
         std::max<long long>(splits, 4) * L * nbatch * m_pad * n_pad;
}

constexpr long long kSlabBudget = 8LL << 30;  // temporaries of one slab

// Splits the GEMM into slabs (batches, then rows i / columns j) whose
// temporaries stay within kSlabBudget, and runs each.
void run_slabs(const GemmDesc& d, const Consts& cs, int beta, cudaStream_t s) {
  const long long L = cs.L;
  const long long k_total = d.k * d.nbr1 * d.nbr2;
  auto planes = [](long long var1n, long long var2n) { return var1n * var2n; };
  // 1. batches: one bo2 at a time, then ranges of bo1
  if (d.nbo2 > 1 &&
      slab_bytes(L, d.m, d.n, k_total, d.nbo1 * d.nbo2,
                 planes(d.sAo1 ? d.nbo1 : 1, d.sAo2 ? d.nbo2 : 1),
                 planes(d.sBo1 ? d.nbo1 : 1, d.sBo2 ? d.nbo2 : 1)) > kSlabBudget) {
    for (long long b2 = 0; b2 < d.nbo2; ++b2) {
      GemmDesc e = d;
      e.nbo2 = 1;
      e.A += b2 * d.sAo2; e.B += b2 * d.sBo2; e.C += b2 * d.sCo2;
      e.sAo2 = e.sBo2 = e.sCo2 = 0;
      run_slabs(e, cs, beta, s);
    }
    return;
  }
  if (d.nbo1 > 1) {
    long long nb = d.nbo1;
    while (nb > 1 && slab_bytes(L, d.m, d.n, k_total, nb * d.nbo2, d.sAo1 ? nb : 1,
                                d.sBo1 ? nb : 1) > kSlabBudget)
      nb = (nb + 1) / 2;
    if (nb < d.nbo1) {
      for (long long b0 = 0; b0 < d.nbo1; b0 += nb) {
        GemmDesc e = d;
        e.nbo1 = std::min(nb, d.nbo1 - b0);
        e.A += b0 * d.sAo1; e.B += b0 * d.sBo1; e.C += b0 * d.sCo1;
        run_slabs(e, cs, beta, s);
      }
      return;
    }
  }
  const long long nbatch = d.nbo1 * d.nbo2;
  const long long pa = (d.sAo1 && d.nbo1 > 1 ? d.nbo1 : 1) * (d.sAo2 && d.nbo2 > 1 ? d.nbo2 : 1);
  const long long pb = (d.sBo1 && d.nbo1 > 1 ? d.nbo1 : 1) * (d.sBo2 && d.nbo2 > 1 ? d.nbo2 : 1);
  // 2. long contractions into a small output: when the operands' residues
  // exceed half the budget but the output's fit in the other half, K is cut
  // into consecutive ranges (reduction batches, else k) whose products are
  // reconstructed one after another and accumulated in C (beta = 1 after the
  // first); row / column slabs would prepare each operand once per slab of
  // the other.  A large output is cut into row / column slabs instead (each
  // K range would reconstruct all of it).
  const ProductTile pt = product_tile(d.m, d.n);
  const long long m_pad = round_up(d.m, pt.tile_i), n_pad = round_up(d.n, pt.tile_j);
  const long long op_bytes = L * (pa * m_pad + pb * n_pad) * round_up(k_total, kTileK);
  const long long out_bytes = 4 * L * nbatch * m_pad * n_pad;
  if (op_bytes > kSlabBudget / 2 && out_bytes <= kSlabBudget / 2 && k_total > kTileK) {
    const long long pieces = (2 * op_bytes + kSlabBudget - 1) / kSlabBudget;
    const long long nred = d.nbr1 * d.nbr2;
    if (nred > 1) {
      // ranges of reduction batches (r1 fastest); one r2 at a time when nbr2 > 1
      if (d.nbr2 > 1) {
        for (long long r2 = 0; r2 < d.nbr2; ++r2) {
          GemmDesc e = d;
          e.nbr2 = 1;
          e.A += r2 * d.sAr2; e.B += r2 * d.sBr2;
          e.sAr2 = e.sBr2 = 0;
          if (r2 > 0) e.beta = 1.0;
          run_slabs(e, cs, beta, s);
        }
        return;
      }
      const long long per = std::max<long long>(1, (d.nbr1 + pieces - 1) / pieces);
      for (long long r0 = 0; r0 < d.nbr1; r0 += per) {
        GemmDesc e = d;
        e.nbr1 = std::min(per, d.nbr1 - r0);
        e.A += r0 * d.sAr1; e.B += r0 * d.sBr1;
        if (r0 > 0) e.beta = 1.0;
        run_slabs(e, cs, beta, s);
      }
      return;
    }
    const long long kc = round_up((d.k + pieces - 1) / pieces, kTileK);
    if (kc < d.k) {
      for (long long k0 = 0; k0 < d.k; k0 += kc) {
        GemmDesc e = d;
        e.k = std::min(kc, d.k - k0);
        e.A += k0 * (d.a_kcontig ? 1 : d.lda);
        e.B += k0 * (d.b_ncontig ? d.ldb : 1);
        if (k0 > 0) e.beta = 1.0;
        run_slabs(e, cs, beta, s);
      }
      return;
    }
  }
  // 3. rows i / columns j
  long long ms = m_pad, ns = n_pad;
  while (slab_bytes(L, ms, ns, k_total, nbatch, pa, pb) > kSlabBudget) {
    if (ms >= ns && ms > kMaxTileI)
      ms = round_up(ms / 2, kMaxTileI);
    else if (ns > 2 * kLanes)
      ns = round_up(ns / 2, 2 * kLanes);
    else
      break;
  }
  for (long long i0 = 0; i0 < d.m; i0 += ms)
    for (long long j0 = 0; j0 < d.n; j0 += ns) {
      GemmDesc e = d;
      e.m = std::min(ms, d.m - i0);
      e.n = std::min(ns, d.n - j0);
      e.A += i0 * (d.a_kcontig ? d.lda : 1);
      e.B += j0 * (d.b_ncontig ? 1 : d.ldb);
      e.C += i0 + j0 * d.ldc;
      run_core(e, cs, beta, s);
    }
}

}  // namespace

void set_split_moduli(int n_moduli) {
  if (n_moduli < 0 || n_moduli > kOzakiMaxModuli)
    throw Error(kErrInvalid, "number of split-precision moduli must be 0..16");
  g_split_moduli = n_moduli;
}

int split_moduli() { return g_split_moduli; }

void set_split_min_flops(double flops) {
  if (!(flops >= 0.0)) throw Error(kErrInvalid, "split-precision threshold must be >= 0");
  g_split_min_flops = flops;
}

double split_min_flops() { return g_split_min_flops; }

int ozaki_bits(int n_moduli, long long k_total) {
  const Consts& cs = consts_for(n_moduli);
  const double kb = std::ceil(std::log2(double(std::max<long long>(k_total, 1))));
  const int beta = static_cast<int>(std::floor((cs.log2_m - 2.0 - kb) / 2.0));
  return std::min(beta, 50);  // |A'| <= 2^50: the FP64 rounding tricks stay exact
}

#ifndef UW12_COST_FP64_TFS
#define UW12_COST_FP64_TFS 26.0
#endif
#ifndef UW12_COST_PREP_TBS
#define UW12_COST_PREP_TBS 3.2
#endif
#ifndef UW12_COST_CRT_TBS
#define UW12_COST_CRT_TBS 2.0
#endif
#ifndef UW12_COST_I8_POPS
#define UW12_COST_I8_POPS 2.2
#endif

bool ozaki_profitable(const GemmDesc& d, int n_moduli) {
  // Estimated times on a B200: operand preparation streams each operand
  // element twice in FP64 and writes L residue bytes (UW12_COST_PREP_TBS
  // TB/s); the CRT reads L residue bytes (and C when beta != 0) and writes C
  // (UW12_COST_CRT_TBS); the int8 products run at UW12_COST_I8_POPS; the FP64
  // DMMA GEMM at UW12_COST_FP64_TFS TFLOP/s.  Split when it is clearly faster.
  // The rates are those of earlier kernels (today 5.8 and 3.4 TB/s, 2.9 POPS,
  // 32 TFLOP/s), kept because they decide which products keep FP64's bits:
  // today's would send sums of K = 7e5 to the split path, where 14 moduli hold
  // 44 bits of an operand (48 at K = 1500).
  const double L = double(n_moduli);
  const double k_total = double(d.k) * double(d.nbr1) * double(d.nbr2);
  const double nbatch = double(d.nbo1) * double(d.nbo2);
  const double pa = double(d.sAo1 && d.nbo1 > 1 ? d.nbo1 : 1) *
                    double(d.sAo2 && d.nbo2 > 1 ? d.nbo2 : 1);
  const double pb = double(d.sBo1 && d.nbo1 > 1 ? d.nbo1 : 1) *
                    double(d.sBo2 && d.nbo2 > 1 ? d.nbo2 : 1);
  const double m = double(d.m), n = double(d.n);
  const double flops = 2.0 * m * n * k_total * nbatch;
  const double t_fp64 = flops / (UW12_COST_FP64_TFS * 1e12);
  const double t_prep = (pa * m + pb * n) * k_total * (16.0 + L) / (UW12_COST_PREP_TBS * 1e12);
  const double t_crt = nbatch * m * n * (L + 8.0 + (d.beta != 0.0 ? 8.0 : 0.0)) /
                       (UW12_COST_CRT_TBS * 1e12);
  const double t_i8 = flops * L / (UW12_COST_I8_POPS * 1e15);
  return t_prep + t_crt + t_i8 + 30e-6 < 0.9 * t_fp64;
}

bool ozaki_supported(const GemmDesc& d) {
  const long long k_total = d.k * d.nbr1 * d.nbr2;
  return d.m <= (1LL << 30) && d.n <= (1LL << 30) && k_total <= 65535LL * kTileK &&
         d.nbo1 * d.nbo2 <= 65535;
}

void gemm_ozaki(const GemmDesc& d, int n_moduli) {
  if (n_moduli < 1 || n_moduli > kOzakiMaxModuli)
    throw Error(kErrInvalid, "number of split-precision moduli must be 1..16");
  if (d.m <= 0 || d.n <= 0 || d.nbo1 <= 0 || d.nbo2 <= 0) return;
  if (d.k <= 0 || d.nbr1 <= 0 || d.nbr2 <= 0) {
    gemm_dmma(d);  // C = beta C
    return;
  }
  if (!ozaki_supported(d)) throw Error(kErrInvalid, "split-precision GEMM: shape too large");
  const long long k_total = d.k * d.nbr1 * d.nbr2;
  const int beta = ozaki_bits(n_moduli, k_total);
  if (beta < 4)
    throw Error(kErrInvalid, "split-precision GEMM: too few moduli for a contraction of " +
                                 std::to_string(k_total) + " terms");
  cudaStream_t s = current_stream();
  const Consts& cs = consts_for(n_moduli);
  char shape[160];
  std::snprintf(shape, sizeof(shape), "split %lld %lld %lld %lld %lld L%d", d.m, d.n, d.k,
                d.nbo1 * d.nbo2, d.nbr1 * d.nbr2, n_moduli);
  Timer tm(kProfSplitGemm,
           2.0 * double(d.m) * double(d.n) * double(k_total) * double(d.nbo1 * d.nbo2), shape,
           s);
  run_slabs(d, cs, beta, s);
  tm.stop();
}

int set_error_slot(int slot) {
  const int prev = t_err_slot;
  t_err_slot = ((slot % kOzakiErrorSlots) + kOzakiErrorSlots) % kOzakiErrorSlots;
  return prev;
}

int ozaki_error_read_and_clear() {
  int* f = err_flag();
  cudaStream_t s = current_stream();
  int h = 0;
  UW12_CUDA(cudaMemcpyAsync(&h, f, sizeof(int), cudaMemcpyDeviceToHost, s));
  UW12_CUDA(cudaStreamSynchronize(s));
  if (h) UW12_CUDA(cudaMemsetAsync(f, 0, sizeof(int), s));
  return h;
}

}  // namespace uw12b

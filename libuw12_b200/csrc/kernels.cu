#include <algorithm>

#include "kernels.cuh"

namespace uw12b {

namespace {

constexpr int kT = 256;

inline int grid_for(long long total, int per_sm = 16) {
  const long long want = (total + kT - 1) / kT;
  return static_cast<int>(std::max<long long>(1, std::min<long long>(want, 148LL * per_sm)));
}

__device__ __forceinline__ long long tri(long long i) { return i * (i + 1) / 2; }

// Tile t of the lower triangle of a matrix of 32 x 32 tiles -> tile row and
// column (tj <= ti), t = ti (ti + 1) / 2 + tj.
__device__ __forceinline__ void lower_tile(int t, int& ti, int& tj) {
  ti = static_cast<int>((sqrtf(8.0f * t + 1.0f) - 1.0f) * 0.5f);
  while (ti * (ti + 1) / 2 > t) --ti;
  while ((ti + 1) * (ti + 2) / 2 <= t) ++ti;
  tj = t - ti * (ti + 1) / 2;
}

// Bound by HBM: every packed element is read once and written to both halves.
// A block takes one 32 x 32 tile of the lower triangle of one column: its rows
// are contiguous in the packed storage and in the upper half of the output, and
// go to the lower half through shared memory, so all three streams are
// coalesced (an element per thread instead reads the packed rows of half of the
// output at a stride, and divides twice in 64 bits per element: 300 x 300 x 900
// 0.34 -> 0.19 ms, 5.1 TB/s).
__global__ void __launch_bounds__(256) k_unpack_sym(const double* P, long long ldp,
                                                    int n, long long ncols, double* out,
                                                    long long ldo, long long so, double alpha,
                                                    double beta) {
  chain_wait();
  __shared__ double tile[32][33];
  int ti, tj;
  lower_tile(blockIdx.x, ti, tj);
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int i0 = ti * 32, j0 = tj * 32;
  for (long long c = blockIdx.y; c < ncols; c += gridDim.y) {
    const double* p = P + ldp * c;
    double* o = out + so * c;
    double v[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = i0 + ty + 8 * r, j = j0 + tx;
      v[r] = (i < n && j <= i) ? alpha * p[tri(i) + j] : 0.0;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = i0 + ty + 8 * r, j = j0 + tx;
      tile[ty + 8 * r][tx] = v[r];
      if (i < n && j <= i) {
        double* d = o + j + ldo * i;
        *d = beta == 0.0 ? v[r] : v[r] + beta * *d;
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = i0 + tx, j = j0 + ty + 8 * r;
      if (i < n && j < i) {
        const double w = tile[tx][ty + 8 * r];
        double* d = o + i + ldo * j;
        *d = beta == 0.0 ? w : w + beta * *d;
      }
    }
    __syncthreads();
  }
}

__global__ void k_pack_density(const double* C, long long ldc, long long n,
                               long long nc, double scale, double* d) {
  chain_wait();
  const long long total = tri(n);
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    // invert idx = i(i+1)/2 + j
    long long i = static_cast<long long>((sqrt(8.0 * double(idx) + 1.0) - 1.0) * 0.5);
    while (tri(i) > idx) --i;
    while (tri(i + 1) <= idx) ++i;
    const long long j = idx - tri(i);
    double s = 0.0;
    for (long long k = 0; k < nc; ++k) s += C[i + ldc * k] * C[j + ldc * k];
    d[idx] = scale * (i != j ? 2.0 : 1.0) * s;
  }
}

template <typename I>
__global__ void k_scale_rc(const double* X, long long ldx, long long rows,
                           long long cols, const double* r,
                           const double* c, double alpha, double* Y, long long ldy) {
  chain_wait();
  const I nr = static_cast<I>(rows), total = nr * static_cast<I>(cols);
  for (I idx = blockIdx.x * static_cast<I>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<I>(gridDim.x) * blockDim.x) {
    const I j = idx / nr, i = idx - j * nr;
    double v = alpha * X[i + ldx * j];
    if (r) v *= r[i];
    if (c) v *= c[j];
    Y[i + ldy * j] = v;
  }
}

template <typename I>
__global__ void k_copy3d(const double* src, long long s1, long long s2, double* dst,
                         long long d1, long long d2, long long n0, long long n1, long long n2,
                         double alpha, double beta) {
  chain_wait();
  const I m0 = static_cast<I>(n0), m1 = static_cast<I>(n1);
  const I total = m0 * m1 * static_cast<I>(n2);
  for (I idx = blockIdx.x * static_cast<I>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<I>(gridDim.x) * blockDim.x) {
    const I rest = idx / m0, i = idx - rest * m0;
    const I l = rest / m1, j = rest - l * m1;
    double* d = dst + i + d1 * j + d2 * l;
    const double v = alpha * src[i + s1 * j + s2 * l];
    *d = beta != 0.0 ? v + beta * *d : v;
  }
}

// Block partial sums -> partials[blockIdx.x]; fixed tree order.
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double sh[kT / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0) {
    for (int q = 0; q < kT / 32; ++q) s += sh[q];
  }
  __syncthreads();
  return s;
}

// acc[slot] += coef * (sum of every block's s): the block that takes the last
// ticket adds the partial sums in a fixed order and hands the ticket back.  One
// launch instead of a second single-thread kernel whose serial sum of up to 592
// partials took longer (7.6 us) than the products (4.1 us at 500 x 500).
__device__ __forceinline__ void finish_reduction(double s, double* partials, double coef,
                                                 double* acc, int slot) {
  __shared__ bool last;
  unsigned* ticket = reinterpret_cast<unsigned*>(acc + kAccSlots);
  s = block_sum(s);
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = s;
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double v = 0.0;
  for (unsigned q = threadIdx.x; q < gridDim.x; q += kT) v += __ldcg(partials + q);
  v = block_sum(v);
  if (threadIdx.x == 0) {
    acc[slot] += coef * v;
    *ticket = 0u;
  }
}

template <typename I>
__global__ void k_wdot(const double* x, long long ldx, const double* y,
                       long long ldy, long long rows, long long cols, const double* rw,
                       const double* cw, double* partials, double coef, double* acc,
                       int slot) {
  chain_wait();
  const I nr = static_cast<I>(rows), total = nr * static_cast<I>(cols);
  double s = 0.0;
  for (I idx = blockIdx.x * static_cast<I>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<I>(gridDim.x) * blockDim.x) {
    const I j = idx / nr, i = idx - j * nr;
    double v = x[i + ldx * j] * y[i + ldy * j];
    if (rw) v *= rw[i];
    if (cw) v *= cw[j];
    s += v;
  }
  finish_reduction(s, partials, coef, acc, slot);
}

struct SpinDots {
  const double* X[2];
  const double* t[2];
  const double* T[2];
  double cx[4], ct[4];
};

// The direct energies' products of all spin pairs: each matrix is read once, in one launch
// instead of one per spin pair and term (bound by launches when small: open-shell
// energy at N=61 231 -> 221 us).  The last block finishes both sums as in finish_reduction.
template <int NS>
__global__ void __launch_bounds__(kT) k_spin_dots(SpinDots a, long long n, double* partials,
                                                  double* acc, int slot_x, int slot_t) {
  chain_wait();
  double sx = 0.0, st = 0.0;
  for (long long e = blockIdx.x * (long long)kT + threadIdx.x; e < n;
       e += (long long)gridDim.x * kT) {
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      const double T = a.T[q][e];
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        if (a.cx[s + 2 * q] != 0.0) sx += a.cx[s + 2 * q] * (a.X[s][e] * T);
        if (a.ct[s + 2 * q] != 0.0) st += a.ct[s + 2 * q] * (T * a.t[s][e]);
      }
    }
  }
  __shared__ bool last;
  unsigned* ticket = reinterpret_cast<unsigned*>(acc + kAccSlots);
  sx = block_sum(sx);
  st = block_sum(st);
  if (threadIdx.x == 0) {
    partials[2 * blockIdx.x] = sx;
    partials[2 * blockIdx.x + 1] = st;
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  sx = st = 0.0;
  for (unsigned q = threadIdx.x; q < gridDim.x; q += kT) {
    sx += __ldcg(partials + 2 * q);
    st += __ldcg(partials + 2 * q + 1);
  }
  sx = block_sum(sx);
  st = block_sum(st);
  if (threadIdx.x == 0) {
    acc[slot_x] += sx;
    acc[slot_t] += st;
    *ticket = 0u;
  }
}

template <typename I>
__global__ void k_permdot_4el(const double* X, const double* Y,
                              long long a, long long o, double* partials, double coef,
                              double* acc, int slot) {
  chain_wait();
  const I na = static_cast<I>(a), nao = na * static_cast<I>(o);
  const I total = nao * nao;  // (i, l, j, k)
  const long long ao = a * o;
  double s = 0.0;
  for (I idx = blockIdx.x * static_cast<I>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<I>(gridDim.x) * blockDim.x) {
    const I col = idx / nao, row = idx - col * nao;  // row = i + a*l, col = j + a*k
    const I l = row / na, i = row - l * na, k = col / na, j = col - k * na;
    s += X[row + ao * col] * Y[(i + a * k) + ao * (j + a * l)];
  }
  finish_reduction(s, partials, coef, acc, slot);
}

// One warp per (i, j, k) triple, summing the contiguous p index.
__global__ void k_permdot_3el(const double* Yw, const double* Zv, long long rp, PairColumns q,
                              double* partials, double coef, double* acc, int slot) {
  chain_wait();
  const long long triples = q.a * q.a * q.nk;
  const int lane = threadIdx.x & 31;
  const long long warp_global = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  const long long ra = rp * q.a;
  double s = 0.0;
  for (long long tix = warp_global; tix < triples; tix += nwarps) {
    const long long i = tix % q.a;
    const long long rest = tix / q.a;
    const long long j = rest % q.a, k = q.k0 + rest / q.a;
    const double* y = Yw + rp * i + ra * q.column(j, k);
    const double* z = Zv + rp * j + ra * q.column(i, k);
    for (long long p = lane; p < rp; p += 32) s += y[p] * z[p];
  }
  finish_reduction(s, partials, coef, acc, slot);
}

__global__ void k_symmetrise(const double* G, long long ldg, long long n, double* F,
                             long long ldf) {
  chain_wait();
  const long long total = n * n;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long i = idx % n, j = idx / n;
    F[i + ldf * j] = 0.5 * (G[i + ldg * j] + G[j + ldg * i]);
  }
}

__global__ void k_symmetry_stats(const double* A, long long lda, long long n,
                                 double* partials) {
  chain_wait();
  const long long total = n * n;
  double dmax = 0.0, amax = 0.0;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long i = idx % n, j = idx / n;
    const double v = A[i + lda * j];
    dmax = fmax(dmax, fabs(v - A[j + lda * i]));
    amax = fmax(amax, fabs(v));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    dmax = fmax(dmax, __shfl_down_sync(0xffffffffu, dmax, o));
    amax = fmax(amax, __shfl_down_sync(0xffffffffu, amax, o));
  }
  __shared__ double sd[kT / 32], sa[kT / 32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) { sd[w] = dmax; sa[w] = amax; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double d = 0.0, a = 0.0;
    for (int q = 0; q < kT / 32; ++q) { d = fmax(d, sd[q]); a = fmax(a, sa[q]); }
    partials[2 * blockIdx.x] = d;
    partials[2 * blockIdx.x + 1] = a;
  }
}

__global__ void k_max_pairs(const double* partials, int n, double* out) {
  chain_wait();
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double d = 0.0, a = 0.0;
    for (int q = 0; q < n; ++q) { d = fmax(d, partials[2 * q]); a = fmax(a, partials[2 * q + 1]); }
    out[0] = d;
    out[1] = a;
  }
}

struct CombineArgs {
  const double* T[2];
  const double* X[2];
  double cT[2];
  double cX[2];
};

template <typename I>
__global__ void k_combine_y(double* Y, long long m, CombineArgs a, int nq,
                            const double* r, const double* c) {
  chain_wait();
  const I nr = static_cast<I>(m), total = nr * nr;
  for (I idx = blockIdx.x * static_cast<I>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<I>(gridDim.x) * blockDim.x) {
    const I j = idx / nr, i = idx - j * nr;
    double t = 0.0, x = 0.0;
    for (int q = 0; q < nq; ++q) {
      if (a.cT[q] != 0.0) t += a.cT[q] * a.T[q][idx];
      if (a.cX[q] != 0.0) x += a.cX[q] * a.X[q][idx];
    }
    Y[idx] = t - r[i] * c[j] * x;
  }
}

struct VecArgs {
  double coef[4];
};

__global__ void k_combine_vecs(const double* U, long long m, int ns, VecArgs a,
                               const double* w, double* V) {
  chain_wait();
  const long long total = m * ns;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long i = idx % m;
    const int s = static_cast<int>(idx / m);
    double v = 0.0;
    for (int q = 0; q < ns; ++q) v += a.coef[s * ns + q] * U[i + m * q];
    V[idx] = w[i] * v;
  }
}

struct LincombArgs {
  const double* M[kMaxLincomb];
  double coef[kMaxLincomb];
  int scaled[kMaxLincomb];
};

template <typename I>
__global__ void k_lincomb(double* Y, long long m, long long n, int nt, LincombArgs a,
                          const double* r, const double* c) {
  chain_wait();
  const I nr = static_cast<I>(m), total = nr * static_cast<I>(n);
  for (I idx = blockIdx.x * static_cast<I>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<I>(gridDim.x) * blockDim.x) {
    const I j = idx / nr, i = idx - j * nr;
    const double rc = (r ? r[i] : 1.0) * (c ? c[j] : 1.0);
    double plain = 0.0, sc = 0.0;
    for (int q = 0; q < nt; ++q) {
      if (a.coef[q] == 0.0) continue;
      if (a.scaled[q])
        sc += a.coef[q] * a.M[q][idx];
      else
        plain += a.coef[q] * a.M[q][idx];
    }
    Y[idx] = plain + rc * sc;
  }
}

// Row i and column j <= i of element q of a packed lower triangle.
__device__ __forceinline__ void triangle_index(long long q, long long& i, long long& j) {
  i = static_cast<long long>((sqrt(8.0 * static_cast<double>(q) + 1.0) - 1.0) * 0.5);
  while (i * (i + 1) / 2 > q) --i;
  while ((i + 1) * (i + 2) / 2 <= q) ++i;
  j = q - i * (i + 1) / 2;
}

// x^ of orbital pairs before the metric: a few MB at most, one block per pair so
// that the pair is found once; its strided reads of B2 are shared in L2 by the
// neighbouring pairs' blocks.
__global__ void k_pack_pairs(const double* B2, PairColumns q, long long o, long long m,
                             const double* r, double h, double* out) {
  chain_wait();
  const long long k = q.k0 + blockIdx.x / q.a, j = blockIdx.x % q.a, ao = q.a * o;
  const bool both = q.mirrored(j, k);
  if (both && j > k - q.c) return;  // the pair's other block writes it
  const long long p = q.column(j, k), n = q.count();
  const long long mirror = both ? k - q.c + q.a * (q.c + j) : 0;
  for (long long A = threadIdx.x; A < m; A += blockDim.x) {
    double v = B2[j + q.a * k + ao * A];
    if (both) v = h * (v + B2[mirror + ao * A]);
    out[p + n * A] = r ? r[A] * v : v;
  }
}

__global__ void k_unpack_pairs(const double* X, PairColumns q, long long o, long long m,
                               const double* r, double h, double* out) {
  chain_wait();
  const long long k = q.k0 + blockIdx.x / q.a, j = blockIdx.x % q.a, ao = q.a * o;
  const double f = q.mirrored(j, k) ? h : 1.0;
  const long long p = q.column(j, k), n = q.count();
  for (long long A = threadIdx.x; A < m; A += blockDim.x)
    out[j + q.a * k + ao * A] = f * (r ? r[A] : 1.0) * X[p + n * A];
}

struct PairRange {
  long long a, c, k0, nk, i0, core_pairs, size;  // core_pairs: those of the range's core orbitals
};

// Bound by HBM: two or three matrices read and one written per pair.  A block
// finds its pair once and takes a run of its elements, 16 bytes per load where
// every matrix starts on 16 bytes (VEC 2): 6.5 TB/s at 136 pairs of 1000 x 200.
template <int VEC>
__global__ void __launch_bounds__(kT) k_sum_pairs(const double* Y, const double* Y2, PairRange g,
                                                  long long run, long long runs, double coef,
                                                  double h, const double* S, double coef_s,
                                                  double* out) {
  chain_wait();
  const long long p = blockIdx.x / runs, part = blockIdx.x - p * runs;
  long long j, k;
  const double* mirror = nullptr;
  if (p < g.core_pairs) {
    k = g.k0 + p / g.a;
    j = p % g.a;
  } else {
    long long i;
    triangle_index(p - g.core_pairs + g.i0 * (g.i0 + 1) / 2, i, j);
    k = g.c + i;
    if (j < g.i0)
      mirror = Y2 + g.size * (j + g.i0 * (i - g.i0));
    else if (j < i)
      mirror = Y + g.size * ((g.c + j - g.k0) + g.nk * i);
  }
  const double* y = Y + g.size * ((k - g.k0) + g.nk * j);
  const double f = mirror ? coef * h : coef;
  const long long end = (part + 1) * run < g.size ? (part + 1) * run : g.size;
  const double* s = S ? S + g.size * p : nullptr;
  double* d = out + g.size * p;
  for (long long e = part * run + VEC * threadIdx.x; e < end; e += VEC * kT) {
    if constexpr (VEC == 2) {
      double2 v = *reinterpret_cast<const double2*>(y + e);
      if (mirror) {
        const double2 w = *reinterpret_cast<const double2*>(mirror + e);
        v.x += w.x;
        v.y += w.y;
      }
      v.x *= f;
      v.y *= f;
      if (s) {
        const double2 w = *reinterpret_cast<const double2*>(s + e);
        v.x += coef_s * w.x;
        v.y += coef_s * w.y;
      }
      *reinterpret_cast<double2*>(d + e) = v;
    } else {
      double v = y[e];
      if (mirror) v += mirror[e];
      v *= f;
      if (s) v += coef_s * s[e];
      d[e] = v;
    }
  }
}

// out[i(i+1)/2 + j, a] = G[i, j, a] + G[j, i, a] (j < i), G[i, i, a] (j = i):
// the gradient of a function of sq(x) with respect to the packed x.  Bound by
// HBM and L2 (G[i, j] is read at a stride; its lines serve the neighbouring rows
// from L2).  One packed element per thread with 32-bit indices (0.34 -> 0.26 ms
// over the four launches of an open-shell gradient at N = 200, M = 600); tiles
// through shared memory as in k_unpack_sym took 0.36 ms, two dependent phases
// for no fewer bytes.
template <typename I>
__global__ void k_pack_sym_sum(const double* G, I n, I np, I total, double* out,
                               long long ldo, double beta) {
  chain_wait();
  for (I idx = blockIdx.x * static_cast<I>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<I>(gridDim.x) * blockDim.x) {
    const I a = idx / np, p = idx - a * np;
    // row i of the packed index: i(i+1)/2 <= p < (i+1)(i+2)/2
    I i = static_cast<I>((sqrtf(8.0f * static_cast<float>(p) + 1.0f) - 1.0f) * 0.5f);
    while (i * (i + 1) / 2 > p) --i;
    while ((i + 1) * (i + 2) / 2 <= p) ++i;
    const I j = p - i * (i + 1) / 2;
    const double* g = G + static_cast<long long>(n) * n * a;
    const double v = (i == j) ? g[i + n * i] : g[i + n * j] + g[j + n * i];
    double* o = out + p + ldo * a;
    *o = beta != 0.0 ? beta * *o + v : v;
  }
}

// Pairs and active orbitals i by block, so that no element divides; bound by HBM.
__global__ void __launch_bounds__(kT) k_perm_3el(const double* Z, double* out, long long rp,
                                                 PairColumns q, double alpha) {
  chain_wait();
  const long long i = blockIdx.x % q.a, t = blockIdx.x / q.a;
  const long long k = q.k0 + t / q.a, j = t % q.a, ra = rp * q.a;
  const bool both = q.mirrored(j, k);
  if (both && j > k - q.c) return;  // the pair's other blocks write it
  const double* z = Z + rp * j + ra * q.column(i, k);
  const double* w = both ? Z + rp * (k - q.c) + ra * q.column(i, q.c + j) : nullptr;
  double* d = out + rp * i + ra * q.column(j, k);
  for (long long p = threadIdx.x; p < rp; p += kT) d[p] = alpha * (w ? z[p] + w[p] : z[p]);
}

// out[i + a*l + ao*(j + a*k)] = alpha * V[i + a*k + ao*(j + a*l)], ao = a*o:
// the occupied indices of rows and columns of (ik|jl) exchanged.
template <typename I>
__global__ void k_perm_4el(const double* V, double* out,
                           long long a, long long o, double alpha) {
  chain_wait();
  const I na = static_cast<I>(a), no = static_cast<I>(o), total = na * no * na * no;
  const long long ao = a * o;
  for (I idx = blockIdx.x * static_cast<I>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<I>(gridDim.x) * blockDim.x) {
    const I t0 = idx / na, i = idx - t0 * na;
    const I t1 = t0 / no, l = t0 - t1 * no;
    const I k = t1 / na, j = t1 - k * na;
    out[idx] = alpha * V[i + a * k + ao * (j + a * l)];
  }
}

__global__ void k_scale_pinv_cols(double* Q, long long n, const double* lam,
                                  double tol) {
  chain_wait();
  const long long total = n * n;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long j = idx / n;
    const double l = lam[j];
    Q[idx] = (fabs(l) > tol) ? Q[idx] / l : 0.0;
  }
}

__global__ void k_set_identity(double* A, long long n) {
  chain_wait();
  const long long total = n * n;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x)
    A[idx] = (idx % n == idx / n) ? 1.0 : 0.0;
}

__global__ void k_gather_scale_cols(const double* src, long long rows,
                                    const int* idxv, const double* s,
                                    long long nq, double* dst) {
  chain_wait();
  const long long total = rows * nq;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long i = idx % rows, q = idx / rows;
    dst[idx] = src[i + rows * idxv[q]] * s[q];
  }
}

// Grid of k_unpack_sym: lower-triangle tiles x columns.
inline dim3 tile_grid(long long n, long long ncols) {
  const long long t = (n + 31) / 32;
  return dim3(static_cast<unsigned>(t * (t + 1) / 2),
              static_cast<unsigned>(std::min<long long>(ncols, 65535)));
}

// Index arithmetic in 32 bits where the element count allows it: the divisions
// that turn an element's number into its indices otherwise take longer than
// the element's traffic.
inline bool small_index(long long total) { return total < (1LL << 31); }

}  // namespace

void unpack_sym(const double* P, long long ldp, long long n, long long ncols, double* out,
                long long ldo, long long so, double alpha, double beta) {
  const long long total = n * n * ncols;
  if (total <= 0) return;
  launch_chained(k_unpack_sym, tile_grid(n, ncols), kT, 0, current_stream(), P, ldp,
                 static_cast<int>(n), ncols, out, ldo, so, alpha, beta);
  UW12_LAUNCHED();
}

void pack_density(const double* C, long long ldc, long long n, long long nc, double scale,
                  double* d) {
  const long long total = n * (n + 1) / 2;
  if (total <= 0) return;
  launch_chained(k_pack_density, grid_for(total), kT, 0, current_stream(), C, ldc, n, nc, scale, d);
  UW12_LAUNCHED();
}

void scale_rc(const double* X, long long ldx, long long rows, long long cols, const double* r,
              const double* c, double alpha, double* Y, long long ldy) {
  const long long total = rows * cols;
  if (total <= 0) return;
  if (small_index(total))
    launch_chained(k_scale_rc<unsigned>, grid_for(total), kT, 0, current_stream(), X, ldx, rows,
                   cols, r, c, alpha, Y, ldy);
  else
    launch_chained(k_scale_rc<long long>, grid_for(total), kT, 0, current_stream(), X, ldx, rows,
                   cols, r, c, alpha, Y, ldy);
  UW12_LAUNCHED();
}

void copy3d(const double* src, long long s1, long long s2, double* dst, long long d1,
            long long d2, long long n0, long long n1, long long n2, double alpha, double beta) {
  const long long total = n0 * n1 * n2;
  if (total <= 0) return;
  if (small_index(total))
    launch_chained(k_copy3d<unsigned>, grid_for(total), kT, 0, current_stream(), src, s1, s2, dst,
                   d1, d2, n0, n1, n2, alpha, beta);
  else
    launch_chained(k_copy3d<long long>, grid_for(total), kT, 0, current_stream(), src, s1, s2, dst,
                   d1, d2, n0, n1, n2, alpha, beta);
  UW12_LAUNCHED();
}

void wdot(const double* x, long long ldx, const double* y, long long ldy, long long rows,
          long long cols, const double* rw, const double* cw, double coef, double* acc,
          int slot) {
  const long long total = rows * cols;
  if (total <= 0 || coef == 0.0) return;
  cudaStream_t s = current_stream();
  const int blocks = grid_for(total, 4);
  DevBuf part(blocks, s);
  if (small_index(total))
    launch_chained(k_wdot<unsigned>, blocks, kT, 0, s, x, ldx, y, ldy, rows, cols, rw, cw,
                   part.get(), coef, acc, slot);
  else
    launch_chained(k_wdot<long long>, blocks, kT, 0, s, x, ldx, y, ldy, rows, cols, rw, cw,
                   part.get(), coef, acc, slot);
  UW12_LAUNCHED();
}

void spin_dots(const double* const* X, const double* const* t, const double* const* T, int ns,
               long long n, const double* cx, const double* ct, double* acc, int slot_x,
               int slot_t) {
  if (n <= 0) return;
  SpinDots a{};
  for (int s = 0; s < ns; ++s) {
    a.X[s] = X[s];
    a.t[s] = t[s];
    a.T[s] = T[s];
  }
  for (int i = 0; i < 4; ++i) {
    a.cx[i] = cx[i];
    a.ct[i] = ct[i];
  }
  cudaStream_t s = current_stream();
  const int blocks = grid_for(n, 4);
  DevBuf part(2 * blocks, s);
  if (ns == 1)
    launch_chained(k_spin_dots<1>, blocks, kT, 0, s, a, n, part.get(), acc, slot_x, slot_t);
  else
    launch_chained(k_spin_dots<2>, blocks, kT, 0, s, a, n, part.get(), acc, slot_x, slot_t);
  UW12_LAUNCHED();
}

void permdot_4el(const double* X, const double* Y, long long a, long long o, double coef,
                 double* acc, int slot) {
  const long long total = a * o * a * o;
  if (total <= 0 || coef == 0.0) return;
  cudaStream_t s = current_stream();
  const int blocks = grid_for(total, 4);
  DevBuf part(blocks, s);
  if (small_index(total))
    launch_chained(k_permdot_4el<unsigned>, blocks, kT, 0, s, X, Y, a, o, part.get(), coef, acc,
                   slot);
  else
    launch_chained(k_permdot_4el<long long>, blocks, kT, 0, s, X, Y, a, o, part.get(), coef, acc,
                   slot);
  UW12_LAUNCHED();
}

void permdot_3el(const double* Y, const double* Z, long long rp, const PairColumns& q,
                 double coef, double* acc, int slot) {
  const long long triples = q.a * q.a * q.nk;
  if (triples <= 0 || rp <= 0 || coef == 0.0) return;
  cudaStream_t s = current_stream();
  const int blocks = grid_for(triples * 32, 8);
  DevBuf part(blocks, s);
  launch_chained(k_permdot_3el, blocks, kT, 0, s, Y, Z, rp, q, part.get(), coef, acc, slot);
  UW12_LAUNCHED();
}

void symmetrise(const double* G, long long ldg, long long n, double* F, long long ldf) {
  const long long total = n * n;
  if (total <= 0) return;
  launch_chained(k_symmetrise, grid_for(total), kT, 0, current_stream(), G, ldg, n, F, ldf);
  UW12_LAUNCHED();
}

void symmetry_stats(const double* A, long long lda, long long n, double* out) {
  cudaStream_t s = current_stream();
  const long long total = n * n;
  const int blocks = grid_for(std::max<long long>(total, 1), 4);
  DevBuf part(2 * blocks, s);
  launch_chained(k_symmetry_stats, blocks, kT, 0, s, A, lda, n, part.get());
  UW12_LAUNCHED();
  launch_chained(k_max_pairs, 1, 32, 0, s, part.get(), blocks, out);
  UW12_LAUNCHED();
}

void combine_y(double* Y, long long m, const double* const* T, const double* coefT,
               const double* const* X, const double* coefX, int nq, const double* r,
               const double* c) {
  const long long total = m * m;
  if (total <= 0) return;
  CombineArgs a{};
  for (int q = 0; q < nq; ++q) {
    a.T[q] = T[q]; a.X[q] = X[q]; a.cT[q] = coefT[q]; a.cX[q] = coefX[q];
  }
  if (small_index(total))
    launch_chained(k_combine_y<unsigned>, grid_for(total), kT, 0, current_stream(), Y, m, a, nq, r,
                   c);
  else
    launch_chained(k_combine_y<long long>, grid_for(total), kT, 0, current_stream(), Y, m, a, nq, r,
                   c);
  UW12_LAUNCHED();
}

void combine_vecs(const double* U, long long m, int ns, const double* coef, const double* w,
                  double* V) {
  if (m <= 0) return;
  VecArgs a{};
  for (int q = 0; q < ns * ns; ++q) a.coef[q] = coef[q];
  launch_chained(k_combine_vecs, grid_for(m * ns), kT, 0, current_stream(), U, m, ns, a, w, V);
  UW12_LAUNCHED();
}

void lincomb(double* Y, long long m, long long n, int nt, const double* const* mats,
             const double* coefs, const int* scaled, const double* r, const double* c) {
  const long long total = m * n;
  if (total <= 0) return;
  if (nt > kMaxLincomb) throw Error(kErrInvalid, "lincomb: too many terms");
  LincombArgs a{};
  for (int q = 0; q < nt; ++q) {
    a.M[q] = mats[q];
    a.coef[q] = coefs[q];
    a.scaled[q] = scaled ? scaled[q] : 0;
  }
  if (small_index(total))
    launch_chained(k_lincomb<unsigned>, grid_for(total), kT, 0, current_stream(), Y, m, n, nt, a, r,
                   c);
  else
    launch_chained(k_lincomb<long long>, grid_for(total), kT, 0, current_stream(), Y, m, n, nt, a,
                   r, c);
  UW12_LAUNCHED();
}

// blocks of a kernel with one per (j, k) of the range, times `each`
static unsigned pair_blocks(const PairColumns& q, long long each) {
  const long long n = q.a * q.nk * each;
  if (n >= (1LL << 31)) throw Error(kErrInvalid, "too many orbital pairs for one launch");
  return static_cast<unsigned>(n);
}

void pack_pairs(const double* B2, const PairColumns& q, long long o, long long m, const double* r,
                double h, double* out) {
  if (q.a * q.nk <= 0 || m <= 0) return;
  launch_chained(k_pack_pairs, pair_blocks(q, 1), kT, 0, current_stream(), B2, q, o, m, r, h, out);
  UW12_LAUNCHED();
}

void unpack_pairs(const double* X, const PairColumns& q, long long o, long long m, const double* r,
                  double h, double* out) {
  if (q.a * q.nk <= 0 || m <= 0) return;
  launch_chained(k_unpack_pairs, pair_blocks(q, 1), kT, 0, current_stream(), X, q, o, m, r, h, out);
  UW12_LAUNCHED();
}

void sum_pairs(const double* Y, const double* Y2, long long size, long long a, long long c,
               long long k0, long long nk, long long n_pairs, double coef, double h,
               const double* S, double coef_s, double* out) {
  if (n_pairs <= 0 || size <= 0) return;
  PairRange g{};
  g.a = a;
  g.c = c;
  g.k0 = k0;
  g.nk = nk;
  g.i0 = std::max(k0, c) - c;
  g.core_pairs = a * std::max(0LL, std::min(k0 + nk, c) - k0);
  g.size = size;
  // four loads per thread and matrix, more only to keep the block count in 31 bits
  const bool vec = size % 2 == 0;  // every matrix of a 16-byte aligned buffer is aligned
  long long run = 4LL * kT * (vec ? 2 : 1);
  while (n_pairs * ((size + run - 1) / run) >= (1LL << 31)) run *= 2;
  const long long runs = (size + run - 1) / run;
  const dim3 grid(static_cast<unsigned>(n_pairs * runs));
  if (vec)
    launch_chained(k_sum_pairs<2>, grid, kT, 0, current_stream(), Y, Y2, g, run, runs, coef, h, S,
                   coef_s, out);
  else
    launch_chained(k_sum_pairs<1>, grid, kT, 0, current_stream(), Y, Y2, g, run, runs, coef, h, S,
                   coef_s, out);
  UW12_LAUNCHED();
}

void pack_sym_sum(const double* G, long long n, long long na, double* out, long long ldo,
                  double beta) {
  const long long total = n * (n + 1) / 2 * na;
  if (total <= 0) return;
  const long long np = n * (n + 1) / 2;
  if (small_index(std::max(total, n * n)))
    launch_chained(k_pack_sym_sum<unsigned>, grid_for(total), kT, 0, current_stream(), G,
                   static_cast<unsigned>(n), static_cast<unsigned>(np),
                   static_cast<unsigned>(total), out, ldo, beta);
  else
    launch_chained(k_pack_sym_sum<long long>, grid_for(total), kT, 0, current_stream(), G, n, np,
                   total, out, ldo, beta);
  UW12_LAUNCHED();
}

void perm_3el(const double* Z, double* out, long long rp, const PairColumns& q, double alpha) {
  if (rp <= 0 || q.a * q.nk <= 0) return;
  launch_chained(k_perm_3el, pair_blocks(q, q.a), kT, 0, current_stream(), Z, out, rp, q, alpha);
  UW12_LAUNCHED();
}

void perm_4el(const double* V, double* out, long long a, long long o, double alpha) {
  const long long total = a * o * a * o;
  if (total <= 0) return;
  if (small_index(total))
    launch_chained(k_perm_4el<unsigned>, grid_for(total), kT, 0, current_stream(), V, out, a, o,
                   alpha);
  else
    launch_chained(k_perm_4el<long long>, grid_for(total), kT, 0, current_stream(), V, out, a, o,
                   alpha);
  UW12_LAUNCHED();
}

void scale_pinv_cols(double* Q, long long n, const double* lambda, double tol) {
  if (n <= 0) return;
  launch_chained(k_scale_pinv_cols, grid_for(n * n), kT, 0, current_stream(), Q, n, lambda, tol);
  UW12_LAUNCHED();
}

void set_identity(double* A, long long n) {
  if (n <= 0) return;
  launch_chained(k_set_identity, grid_for(n * n), kT, 0, current_stream(), A, n);
  UW12_LAUNCHED();
}

void gather_scale_cols(const double* src, long long rows, const int* idx, const double* s,
                       long long nq, double* dst) {
  if (rows * nq <= 0) return;
  launch_chained(k_gather_scale_cols, grid_for(rows * nq), kT, 0, current_stream(), src, rows, idx,
                 s, nq, dst);
  UW12_LAUNCHED();
}

// out += sum of squares of the rows x cols block A (leading dimension lda):
// grid-stride partial sums, a warp-shuffle and shared-memory block reduction,
// one atomic add per block (summation order not fixed).
__global__ void k_sumsq_add(const double* A, long long lda, long long rows,
                            long long cols, double* out) {
  chain_wait();
  __shared__ double part[32];
  const long long total = rows * cols;
  double acc = 0.0;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const long long c = e / rows, r = e - c * rows;
    const double x = A[r + lda * c];
    acc = fma(x, x, acc);
  }
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) part[warp] = acc;
  __syncthreads();
  if (warp == 0) {
    acc = lane < (int)(blockDim.x >> 5) ? part[lane] : 0.0;
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) atomicAdd(out, acc);
  }
}

void sumsq_add(const double* A, long long lda, long long rows, long long cols, double* out,
               cudaStream_t s) {
  const long long total = rows * cols;
  if (total <= 0) return;
  launch_chained(k_sumsq_add, grid_for(total, 4), kT, 0, s, A, lda, rows, cols, out);
  UW12_LAUNCHED();
}

}  // namespace uw12b

// Streaming (HBM-bound) kernels of the UW12 schedule: packed-symmetric
// unpack/pack, diagonal scalings, strided copies, deterministic reductions
// and the permuted contractions of the same-spin energies.  All launch on
// current_stream().
#pragma once

#include "common.cuh"

namespace uw12b {

// out[i + ldo*j + so*c] = beta*out + alpha*S_c(i,j), S_c = square(P[:, c]) with
// P column-major (ldp), packed lower triangle row by row (idx = i(i+1)/2 + j).
void unpack_sym(const double* P, long long ldp, long long n, long long ncols, double* out,
                long long ldo, long long so, double alpha = 1.0, double beta = 0.0);

// d[idx(i,j)] = scale * (i != j ? 2 : 1) * sum_k C[i + ldc*k] C[j + ldc*k]
// (lower(scale * C C^T, 2) of libuw12's utils.hpp).
void pack_density(const double* C, long long ldc, long long n, long long nc, double scale,
                  double* d);

// Y[i + ldy*j] = alpha * r[i] * X[i + ldx*j] * c[j]   (r or c may be null = 1).
void scale_rc(const double* X, long long ldx, long long rows, long long cols, const double* r,
              const double* c, double alpha, double* Y, long long ldy);

// 3-D strided copy / scale: dst[i + d1*j + d2*l] = alpha * src[i + s1*j + s2*l]
// (+ beta * dst when beta != 0).
void copy3d(const double* src, long long s1, long long s2, double* dst, long long d1,
            long long d2, long long n0, long long n1, long long n2, double alpha = 1.0,
            double beta = 0.0);

// The distinct pairs (j, k) of a active orbitals j and the occupied orbitals k of
// [k0, k0 + nk), c of the occupied orbitals being core: (j, c + i) and (i, c + j) are one
// pair.  In column order: the range's core orbitals k ascending, j ascending within them;
// the range's active orbitals i0 + i with those up to themselves, triangle
// i (i + 1) / 2 + j - i0; then those with the active orbitals outside the range.  For a range
// from 0 to k this is the order of all pairs with j <= i.
struct PairColumns {
  long long a, c, k0, nk, nc, i0, ni;  // nc core, ni active orbitals of the range from i0

  __host__ __device__ static PairColumns of(long long a, long long c, long long k0, long long nk) {
    PairColumns q{};
    const long long k1 = k0 + nk;
    q.a = a;
    q.c = c;
    q.k0 = k0;
    q.nk = nk;
    q.nc = (k1 < c ? k1 : c) > k0 ? (k1 < c ? k1 : c) - k0 : 0;
    q.i0 = k0 > c ? k0 - c : 0;
    q.ni = (k1 > c ? k1 - c : 0) - q.i0;
    return q;
  }
  __host__ __device__ long long count() const {
    return a * nc + ni * (ni + 1) / 2 + (a - ni) * ni;
  }
  // whether (j, k) and its mirror image are two entries of the range
  __host__ __device__ bool mirrored(long long j, long long k) const {
    return k >= c && j >= i0 && j < i0 + ni && j != k - c;
  }
  __host__ __device__ long long column(long long j, long long k) const {
    if (k < c) return j + a * (k - k0);
    const long long i = k - c - i0, t = j - i0;
    if (t >= 0 && t < ni) {
      const long long hi = t > i ? t : i, lo = t > i ? i : t;
      return a * nc + hi * (hi + 1) / 2 + lo;
    }
    return a * nc + ni * (ni + 1) / 2 + (t < 0 ? j : j - ni) + (a - ni) * i;
  }
};

// Pairs (j, k) of active orbitals j and occupied orbitals k < k_end in pair order: k
// ascending and j ascending within it, every j for a core orbital, j <= k - c for
// an active one.
inline size_t pair_count(size_t a, size_t c, size_t k_end) {
  const size_t i = k_end > c ? k_end - c : 0;
  return a * (k_end < c ? k_end : c) + i * (i + 1) / 2;
}

// First occupied orbital of shard i of n (i = n: o = c + a): the shards' ranges have about
// the same number of pairs each, within the pairs of one orbital.  Even ranges of orbitals
// give the last of 8 shards 23 % of the pairs instead of 12.5 (no core).
inline size_t pair_bound(size_t a, size_t c, size_t i, size_t n) {
  const size_t o = c + a, total = pair_count(a, c, o) * i;
  size_t k = 0;
  while (k < o && pair_count(a, c, k) * n < total) ++k;
  if (k > 0 && pair_count(a, c, k) * n - total > total - pair_count(a, c, k - 1) * n) --k;
  return k;
}

// Sums of wdot, permdot_4el and permdot_3el: acc is a device array of
// kAccDoubles, zeroed before its first use; slots below kAccSlots hold sums, the
// last double is the ticket of the reductions' last block.
constexpr int kAccSlots = 8;
constexpr int kAccDoubles = kAccSlots + 1;

// acc[slot] += coef * sum_{i<rows, j<cols} x[i + ldx*j] * y[i + ldy*j] * rw[i] * cw[j]
// (rw / cw may be null).  Fixed-order reduction.
void wdot(const double* x, long long ldx, const double* y, long long ldy, long long rows,
          long long cols, const double* rw, const double* cw, double coef, double* acc, int slot);

// acc[slot_x] += sum_{s,q} cx[s + 2 q] <X[s], T[q]> and acc[slot_t] += sum_{s,q} ct[s + 2 q]
// <T[q], t[s]> over n elements, s, q < ns <= 2; terms with coefficient zero are left out.
void spin_dots(const double* const* X, const double* const* t, const double* const* T, int ns,
               long long n, const double* cx, const double* ct, double* acc, int slot_x,
               int slot_t);

// acc[slot] += coef * sum_{i,l<a; j,k<o} X[i + a*l + lda*(j + a*k)] * Y[i + a*k + lda*(j + a*l)]
// with lda = a*o: the same-spin four-electron energy over (ik|jl) blocks.
void permdot_4el(const double* X, const double* Y, long long a, long long o, double coef,
                 double* acc, int slot);

// acc[slot] += coef * sum_{p<rp; i,j<a; k of q} Y[p + rp*i + rp*a*col(j, k)]
//                                             * Z[p + rp*j + rp*a*col(i, k)]
// (Y, Z rp*a x q.count()): the same-spin three-electron energy.
void permdot_3el(const double* Y, const double* Z, long long rp, const PairColumns& q,
                 double coef, double* acc, int slot);

// F[i + ld*j] = 0.5 * (G[i + ldg*j] + G[j + ldg*i]) written into column-block
// sigma of the output; F may alias nothing in G.
void symmetrise(const double* G, long long ldg, long long n, double* F, long long ldf);

// max |A - A^T| and max |A| into out[0], out[1] (device), n x n column-major.
void symmetry_stats(const double* A, long long lda, long long n, double* out);
// *out += sum of squares of the rows x cols block A (leading dimension lda), on s.
void sumsq_add(const double* A, long long lda, long long rows, long long cols, double* out,
               cudaStream_t s);

// Y = sum_q coefT[q]*T[q] - r[i]*c[j]*sum_q coefX[q]*X[q], M x M, q < nq <= 2.
void combine_y(double* Y, long long m, const double* const* T, const double* coefT,
               const double* const* X, const double* coefX, int nq, const double* r,
               const double* c);

// V[:, s] = w .* sum_q coef[s*ns + q] * U[:, q], columns of length m (ns <= 2).
void combine_vecs(const double* U, long long m, int ns, const double* coef, const double* w,
                  double* V);

// P2 = Q * diag(pinv(lambda)) with |lambda| <= tol -> 0; in place on Q (n x n).
void scale_pinv_cols(double* Q, long long n, const double* lambda, double tol);
// Y (m x n, contiguous) = sum_q coef_q M_q, the terms with scaled_q != 0
// multiplied elementwise by r_i c_j (r, c may be null); at most kMaxLincomb terms.
constexpr int kMaxLincomb = 8;
void lincomb(double* Y, long long m, long long n, int nt, const double* const* mats,
             const double* coefs, const int* scaled, const double* r, const double* c);
// Gradient with respect to packed symmetric storage: out[:, a] (ldo >= n(n+1)/2)
// = beta * out[:, a] + the packed sum of the n x n matrix G[:, :, a]
// (consecutive, n*n apart), G_ij + G_ji off the diagonal, G_ii on it.
void pack_sym_sum(const double* G, long long n, long long na, double* out, long long ldo,
                  double beta = 0.0);

// out[p + rp*i + rp*a*col(j, k)] = alpha * (Z[p + rp*j + rp*a*col(i, k)] + the mirror
// image's) for p < rp, i < a and the pairs (j, k) of q: the active-orbital pair of a
// same-spin three-electron product (YW or ZV, rp*a x q.count()) exchanged and summed over
// both orders; out and Z distinct.
void perm_3el(const double* Z, double* out, long long rp, const PairColumns& q, double alpha);

// out[i + a*l + ao*(j + a*k)] = alpha * V[i + a*k + ao*(j + a*l)], ao = a*o:
// the occupied indices of an (ik|jl) matrix (ao x ao) exchanged between rows
// and columns; out and V distinct.
void perm_4el(const double* V, double* out, long long a, long long o, double alpha);

// out[col, A] (contiguous, q.count() x m) = r_A B2[j + a k, A] and, for mirrored pairs,
// r_A h (B2[j + a k, A] + B2[i + a (c + j), A]); B2 is (a o) x m, r may be null (ones).
void pack_pairs(const double* B2, const PairColumns& q, long long o, long long m, const double* r,
                double h, double* out);

// out[j + a k, A] = r_A h X[col, A] for mirrored pairs, r_A X[col, A] for the others, for
// every j and the range's k (out (a o) x m, X q.count() x m).
void unpack_pairs(const double* X, const PairColumns& q, long long o, long long m, const double* r,
                  double h, double* out);

// out[p] = coef (Y[j, k] + mirror image) + coef_s S[p], matrices of `size` elements, for the
// n_pairs pairs of the occupied orbitals [k0, k0 + nk) in the order of all pairs (every j for a
// core orbital k, j <= i for k = c + i); where there is a mirror image the sum of both is
// scaled by h.  Y[j, k] is matrix (k - k0) + nk j of Y, the mirror
// image Y[i, c + j] too where c + j >= k0, matrix j + i0 (i - i0) of Y2 before it (c + i0 the
// first active orbital of the range).  S may be null, or out itself.
void sum_pairs(const double* Y, const double* Y2, long long size, long long a, long long c,
               long long k0, long long nk, long long n_pairs, double coef, double h,
               const double* S, double coef_s, double* out);

// A = I (n x n, column-major).
void set_identity(double* A, long long n);

// Gather columns: dst[:, q] = src[:, idx[q]] * s[q] (idx, s on device).
void gather_scale_cols(const double* src, long long rows, const int* idx, const double* s,
                       long long nq, double* dst);

}  // namespace uw12b

// UW12 energy + Fock schedule on the device.
//
// Every contraction of libuw12's two-, three- and four-electron terms is
// restated as a handful of large FP64 GEMMs (gemm_f64.cu); the reference's
// per-aux-function parallel_for loops and per-orbital-pair parallel_sum_2d
// loops become batched / reduction-batched GEMMs.  Notation: N = n_ao,
// M = n_df, R = n_ri, R' = N + R, per spin o occupied, a active, c = o - a core.
//
//  T1  B1[mu + N k, A]  = sum_nu sq(J3_0[:,A])[mu,nu] Co[nu,k], then * P2
//      (transformations.hpp:33-54, integrals.cpp:213-248)
//  T2  Bri[nu + R i, A] = sum_mu J3ri_A[nu,mu] Ca[mu,i], then * P2
//      (transformations.hpp:130-158, integrals.cpp:250-287)
//  T3  B2[i + a k, A]   = sum_mu Ca[mu,i] B1[mu + N k, A]  (transformations.hpp:79-106)
//  Wst rows p + R' j: p < N -> B1 orbital c+j, p >= N -> Bri orbital j (the
//      AO-then-RI stacking of the ABS+ space), SV = (I_a (x) S^-1) Wst.
//  X_AB = Wst_W^T SV_V replaces the four calculate_xab_component loops
//      (direct_utils.cpp:31-133); t = B2_W^T B2_V, t~ = Lw t Lv
//      (four_electron_utils.cpp:33-79).
//  Fock pieces are accumulated unsymmetrised per spin and symmetrised once;
//  libuw12 symmetrises the three- and four-electron terms and its
//  two-electron pieces are symmetric by construction (utils.hpp:215-224).
#include <cusolverDn.h>

#include <algorithm>
#include <cstdint>
#include <exception>
#include <vector>
#include <thread>
#include <cstring>
#include <cmath>
#include <cstdio>
#include <map>
#include <mutex>
#include <string>

#include "engine.cuh"
#include "gemm_f64.cuh"
#include "kernels.cuh"
#include "ozaki.cuh"

namespace uw12b {

namespace {

void solver_check(cusolverStatus_t st, const char* what) {
  if (st != CUSOLVER_STATUS_SUCCESS)
    throw Error(kErrCuda, std::string(what) + ": cusolver status " + std::to_string(int(st)));
}

// Pinned chunks for host-to-device copies out of pageable memory: filled by
// several host threads at once while the previous chunk's DMA runs (a
// pageable cudaMemcpyAsync stages through the driver at ~10 GB/s).  One set
// per process, used under a mutex; an event per chunk guards its reuse.
struct Staging {
  static constexpr size_t kChunkBytes = size_t(64) << 20;
  static constexpr int kChunks = 4;
  std::mutex mu;
  char* buf[kChunks] = {};
  cudaEvent_t done[kChunks] = {};
  int device[kChunks] = {};
};

Staging& staging() {
  static Staging* st = new Staging();  // lives to process exit (pinned memory freed by it)
  return *st;
}

// memcpy of `bytes` split over up to `threads` host threads.
void parallel_memcpy(char* dst, const char* src, size_t bytes, unsigned threads) {
  const size_t per = (bytes + threads - 1) / threads;
  std::vector<std::thread> pool;
  for (unsigned t = 1; t < threads && t * per < bytes; ++t)
    pool.emplace_back([=] { std::memcpy(dst + t * per, src + t * per, std::min(per, bytes - t * per)); });
  std::memcpy(dst, src, std::min(per, bytes));
  for (auto& th : pool) th.join();
}

void upload_pageable(double* dst, const double* src, size_t n, cudaStream_t s) {
  Staging& st = staging();
  std::lock_guard<std::mutex> lk(st.mu);
  int dev = 0;
  UW12_CUDA(cudaGetDevice(&dev));
  for (int c = 0; c < Staging::kChunks; ++c) {
    if (!st.buf[c]) {
      UW12_CUDA(cudaMallocHost(reinterpret_cast<void**>(&st.buf[c]), Staging::kChunkBytes));
    }
    if (!st.done[c] || st.device[c] != dev) {
      if (st.done[c]) {
        UW12_CUDA(cudaEventSynchronize(st.done[c]));
        cudaEventDestroy(st.done[c]);
      }
      UW12_CUDA(cudaEventCreateWithFlags(&st.done[c], cudaEventDisableTiming));
      st.device[c] = dev;
    }
  }
  const unsigned threads = std::max(1u, std::min(8u, std::thread::hardware_concurrency() / 2));
  const char* from = reinterpret_cast<const char*>(src);
  char* to = reinterpret_cast<char*>(dst);
  const size_t bytes = n * sizeof(double);
  int c = 0;
  for (size_t off = 0; off < bytes; off += Staging::kChunkBytes, c = (c + 1) % Staging::kChunks) {
    const size_t len = std::min(Staging::kChunkBytes, bytes - off);
    UW12_CUDA(cudaEventSynchronize(st.done[c]));  // this chunk's previous copy is done
    parallel_memcpy(st.buf[c], from + off, len, threads);
    UW12_CUDA(cudaMemcpyAsync(to + off, st.buf[c], len, cudaMemcpyHostToDevice, s));
    UW12_CUDA(cudaEventRecord(st.done[c], s));
  }
  // the caller's buffer has been read; the chunks' copies finish in stream order
}

// n doubles to the device: device-to-device, a direct copy from pinned host
// memory, or the staged pipeline for large pageable host buffers.
void upload(double* dst, const double* src, size_t n, bool device_mem, cudaStream_t s) {
  if (!n) return;
  if (!device_mem && n * sizeof(double) >= (size_t(32) << 20)) {
    cudaPointerAttributes at{};
    const bool known = cudaPointerGetAttributes(&at, src) == cudaSuccess;
    if (!known) cudaGetLastError();  // clear the query's error
    if (!known || at.type == cudaMemoryTypeUnregistered) {
      upload_pageable(dst, src, n, s);
      return;
    }
  }
  UW12_CUDA(cudaMemcpyAsync(dst, src, n * sizeof(double),
                            device_mem ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, s));
}

// libuw12's linalg::is_symmetric(mat, 1e-10) (linalg.hpp:309-330), relative
// to max(1, max|A|).
void require_symmetric(const double* A, size_t n, const char* msg) {
  cudaStream_t s = current_stream();
  DevBuf st(2, s);
  symmetry_stats(A, n, n, st.get());
  double h[2];
  UW12_CUDA(cudaMemcpyAsync(h, st.get(), sizeof(h), cudaMemcpyDeviceToHost, s));
  UW12_CUDA(cudaStreamSynchronize(s));
  if (!(h[0] <= 1e-10 * std::max(1.0, h[1]))) throw_logic(msg);
}

// One cuSOLVER handle per host thread and device, created on first use.
cusolverDnHandle_t solver_handle() {
  struct Handles {
    std::map<int, cusolverDnHandle_t> h;
    ~Handles() {
      for (auto& kv : h) cusolverDnDestroy(kv.second);
    }
  };
  thread_local Handles handles;
  int dev = 0;
  UW12_CUDA(cudaGetDevice(&dev));
  auto it = handles.h.find(dev);
  if (it != handles.h.end()) return it->second;
  cusolverDnHandle_t h = nullptr;
  solver_check(cusolverDnCreate(&h), "cusolverDnCreate");
  handles.h[dev] = h;
  return h;
}

// Ascending eigenpairs of a symmetric n x n matrix, in place (A -> vectors).
void eigh(double* A, size_t n, double* w) {
  cudaStream_t s = current_stream();
  cusolverDnHandle_t h = solver_handle();
  solver_check(cusolverDnSetStream(h, s), "cusolverDnSetStream");
  int lwork = 0;
  solver_check(cusolverDnDsyevd_bufferSize(h, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER,
                                           static_cast<int>(n), A, static_cast<int>(n), w, &lwork),
               "cusolverDnDsyevd_bufferSize");
  DevBuf work(static_cast<size_t>(std::max(lwork, 1)), s);
  int* info = nullptr;
  UW12_CUDA(cudaMallocAsync(reinterpret_cast<void**>(&info), sizeof(int), s));
  solver_check(cusolverDnDsyevd(h, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER,
                                static_cast<int>(n), A, static_cast<int>(n), w, work.get(), lwork,
                                info),
               "cusolverDnDsyevd");
  UW12_LAUNCHED();
  int hinfo = 0;
  UW12_CUDA(cudaMemcpyAsync(&hinfo, info, sizeof(int), cudaMemcpyDeviceToHost, s));
  UW12_CUDA(cudaFreeAsync(info, s));
  UW12_CUDA(cudaStreamSynchronize(s));
  if (hinfo != 0) throw_runtime("eigen-decomposition failed");
}

// Chunk budget of one evaluation, in doubles: the caller's, or `fraction` (45% by
// default, at least 64 MiB) of its share of the device memory available now (free
// memory plus what the library's pool holds unused, over the evaluations that share
// it).  Re-read at the start of each chunked phase, after the phase's persistent
// intermediates are allocated.
//
// Asking for the free memory (cudaMemGetInfo) enters the kernel driver: 90 us on
// a quiet host, tens of milliseconds while other processes of the host are in
// it, against 2.5 us for a launch.  So:
//  * it is asked at most once per evaluation; afterwards the pool's own counters
//    say how much of that free memory the evaluation has taken.  Where the caller's code
//    runs inside the evaluation (producers, gradient sinks, the all-reduce) and may take
//    device memory itself, it is asked at every phase of an evaluation that is not
//    repeated when an allocation fails, or is the repeat;
//  * an evaluation whose chunks all fit whole in 64 MiB, or in 1/32 of the
//    device's memory where it may be repeated (assume_memory), asks nothing
//    (`need`: an upper bound of every size that is compared with a budget, so any
//    larger budget would give the same chunks).  Should an allocation of the
//    latter fail, the caller runs it again without the assumption.
class Budget {
 public:
  Budget(const FockRequest& rq, size_t need, bool callers_code)
      : requested_(rq.mem_budget), need_(need), sharers_(std::max<size_t>(1, rq.sharers)),
        callers_code_(callers_code && !rq.assume_memory) {
    if (!requested_ && rq.assume_memory) whole_ = std::max(whole_, assumed_doubles());
  }

  size_t doubles(double fraction = 0.45) {
    if (requested_)  // an explicit budget may be small (many small chunks)
      return std::max<size_t>(requested_, size_t(64) << 10) / sizeof(double);
    if (need_ <= whole_) return whole_;
    unsigned long long reserved = 0, used = 0;  // 64-bit pool attributes
    UW12_CUDA(cudaMemPoolGetAttribute(library_pool(), cudaMemPoolAttrReservedMemCurrent, &reserved));
    UW12_CUDA(cudaMemPoolGetAttribute(library_pool(), cudaMemPoolAttrUsedMemCurrent, &used));
    if (free0_ < 0.0 || callers_code_) {
      size_t free_b = 0, total_b = 0;
      UW12_CUDA(cudaMemGetInfo(&free_b, &total_b));
      free0_ = double(free_b);
      reserved0_ = double(reserved);
    }
    const double free_now = std::max(0.0, free0_ - (double(reserved) - reserved0_));
    const double avail = free_now + (reserved > used ? double(reserved - used) : 0.0);
    return std::max<size_t>(static_cast<size_t>(fraction * avail / double(sharers_)) / sizeof(double),
                            kFloor);
  }

 private:
  static constexpr size_t kFloor = (size_t(64) << 20) / sizeof(double);
  size_t requested_, need_, sharers_, whole_ = kFloor;
  bool callers_code_;
  double free0_ = -1.0, reserved0_ = 0.0;
};

inline long long LL(size_t v) { return static_cast<long long>(v); }

// Metric eigendecomposition (base_integrals.cpp:155-166): P2 = Q pinv(Lambda),
// df_vals = Lambda, after libuw12's symmetry check.
// A non-blocking stream that starts after the work already on `parent`;
// join() makes `parent` wait for it and waits for it on the host.  The
// destructor (also on an error path) waits for it before destroying it, so
// nothing it reads or writes is released while in flight.
class SideStream {
 public:
  explicit SideStream(cudaStream_t parent) : parent_(parent) {
    UW12_CUDA(cudaStreamCreateWithFlags(&s_, cudaStreamNonBlocking));
    UW12_CUDA(cudaEventCreateWithFlags(&ev_, cudaEventDisableTiming));
    UW12_CUDA(cudaEventRecord(ev_, parent_));
    UW12_CUDA(cudaStreamWaitEvent(s_, ev_, 0));
  }
  SideStream(const SideStream&) = delete;
  SideStream& operator=(const SideStream&) = delete;
  ~SideStream() {
    cudaStreamSynchronize(s_);
    cudaEventDestroy(ev_);
    cudaStreamDestroy(s_);
  }
  cudaStream_t get() const { return s_; }
  void join() {
    UW12_CUDA(cudaEventRecord(ev_, s_));
    UW12_CUDA(cudaStreamWaitEvent(parent_, ev_, 0));
    UW12_CUDA(cudaStreamSynchronize(s_));
  }

 private:
  cudaStream_t parent_ = nullptr, s_ = nullptr;
  cudaEvent_t ev_ = nullptr;
};

void setup_metric(IntegralsHandle* h, const double* X2, bool device_mem) {
  cudaStream_t s = current_stream();
  const size_t n_df = h->n_df;
  h->P2.alloc(n_df * n_df);
  upload(h->P2.get(), X2, n_df * n_df, device_mem, s);
  require_symmetric(h->P2.get(), n_df, "matrix must be symmetric");
  h->lam.alloc(n_df);
  eigh(h->P2.get(), n_df, h->lam.get());
  scale_pinv_cols(h->P2.get(), LL(n_df), h->lam.get(), 1e-10);
  h->lam_host.resize(n_df);
  UW12_CUDA(cudaMemcpyAsync(h->lam_host.data(), h->lam.get(), n_df * sizeof(double),
                            cudaMemcpyDeviceToHost, s));
  UW12_CUDA(cudaStreamSynchronize(s));
}

// Columns [a0, a0 + na) of X's AO (ri = false: Np rows) or RI (ri = true:
// R N rows) three-index tensor, column-major with leading dimension = rows: a
// pointer into the stored tensor, or the producer's output in `room`
// (integral-direct mode; rows * na doubles).
const double* aux_block(const IntegralsHandle& X, bool ri, size_t a0, size_t na, double* room) {
  const size_t rows = ri ? X.n_ri * X.n_ao : packed_size(X.n_ao);
  const DeviceArray& stored = ri ? X.J3_ri_0 : X.J3_0;
  if (stored.get()) return stored.get() + rows * a0;
  const AuxProducer& fn = ri ? X.ri_fn : X.ao_fn;
  if (!fn) throw_runtime(ri ? "J3_ri_0 not stored" : "J3_0 not stored");
  cudaStream_t s = current_stream();
  if (profile_enabled()) {
    cudaEvent_t a, b;
    UW12_CUDA(cudaEventCreate(&a));
    UW12_CUDA(cudaEventCreate(&b));
    UW12_CUDA(cudaEventRecord(a, s));
    fn(a0, na, room, rows, s);
    UW12_CUDA(cudaEventRecord(b, s));
    profile_record(kProfProducer, a, b, 8.0 * double(rows) * double(na),
                   std::string(ri ? "produce ri " : "produce ao ") + std::to_string(na));
  } else {
    fn(a0, na, room, rows, s);
  }
  return room;
}

// The same with the producer's output in `scratch`, which grows to hold it.
const double* aux_block(const IntegralsHandle& X, bool ri, size_t a0, size_t na,
                        DevBuf& scratch) {
  const size_t rows = ri ? X.n_ri * X.n_ao : packed_size(X.n_ao);
  if (!(ri ? X.J3_ri_0 : X.J3_0).get() && scratch.size() < rows * na) scratch.alloc(rows * na);
  return aux_block(X, ri, a0, na, scratch.get());
}

// Aux functions per block when looping over a tensor: all of them when it is
// stored (one block, the tensor itself), else as many as a quarter of the
// budget holds.
size_t aux_step(const IntegralsHandle& X, bool ri, size_t budget) {
  const DeviceArray& stored = ri ? X.J3_ri_0 : X.J3_0;
  if (stored.get()) return X.n_df;
  const size_t rows = ri ? X.n_ri * X.n_ao : packed_size(X.n_ao);
  return std::max<size_t>(1, std::min(X.n_df, budget / (4 * rows)));
}

}  // namespace

size_t assumed_doubles() {
  static std::mutex mu;
  static size_t total[64] = {};
  int dev = 0;
  UW12_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return 0;
  std::lock_guard<std::mutex> lk(mu);
  if (!total[dev]) {
    size_t free_b = 0;
    UW12_CUDA(cudaMemGetInfo(&free_b, &total[dev]));
  }
  return total[dev] / 32 / sizeof(double);
}

// --------------------------------------------------------------------------
// handles
// --------------------------------------------------------------------------
IntegralsHandle* integrals_create(const double* X3, const double* X2, const double* X3_ri,
                                  size_t n_ao, size_t n_df, size_t n_ri, bool device_mem) {
  if (n_ao == 0) throw_runtime("Number of ao orbitals is zero");
  if (n_df == 0) throw_runtime("Number of density-fitting basis functions is zero");
  if (!X3 || !X2) throw Error(kErrInvalid, "null integral pointer");
  if (X3_ri && n_ri == 0) throw_runtime("Three index ri integrals given but n_ri is zero");
  auto h = new IntegralsHandle();
  try {
    UW12_CUDA(cudaGetDevice(&h->device));
    cudaStream_t s = current_stream();
    h->n_ao = n_ao;
    h->n_df = n_df;
    h->n_ri = X3_ri ? n_ri : 0;
    const size_t np = packed_size(n_ao);
    h->J3_0.alloc(np * n_df);
    if (X3_ri) h->J3_ri_0.alloc(n_ri * n_ao * n_df);
    // The three-index copies run on a side stream (after the caller's work on
    // the current stream, which may have produced device inputs) while the
    // metric is diagonalised on the current stream; both are complete when
    // this returns.
    SideStream side(s);
    // host sources are read on a second host thread (a pageable source is
    // copied through pinned chunks by host threads), so the eigensolve runs
    // meanwhile
    std::exception_ptr upload_err;
    const int dev = h->device;
    std::thread up([&] {
      try {
        UW12_CUDA(cudaSetDevice(dev));
        upload(h->J3_0.get(), X3, np * n_df, device_mem, side.get());
        if (X3_ri) upload(h->J3_ri_0.get(), X3_ri, n_ri * n_ao * n_df, device_mem, side.get());
      } catch (...) {
        upload_err = std::current_exception();
      }
    });
    try {
      setup_metric(h, X2, device_mem);
    } catch (...) {
      up.join();
      throw;
    }
    up.join();
    if (upload_err) std::rethrow_exception(upload_err);
    side.join();
  } catch (...) {
    delete h;
    throw;
  }
  return h;
}

IntegralsHandle* integrals_create_producer(const double* X2, bool x2_device, AuxProducer ao_fn,
                                           AuxProducer ri_fn, size_t n_ao, size_t n_df,
                                           size_t n_ri, bool store_ao, bool store_ri) {
  if (n_ao == 0) throw_runtime("Number of ao orbitals is zero");
  if (n_df == 0) throw_runtime("Number of density-fitting basis functions is zero");
  if (!X2 || !ao_fn) throw Error(kErrInvalid, "null metric or three-index producer");
  if (ri_fn && n_ri == 0) throw_runtime("Three index ri integrals given but n_ri is zero");
  auto h = new IntegralsHandle();
  try {
    UW12_CUDA(cudaGetDevice(&h->device));
    cudaStream_t s = current_stream();
    h->n_ao = n_ao;
    h->n_df = n_df;
    h->n_ri = ri_fn ? n_ri : 0;
    setup_metric(h, X2, x2_device);
    const size_t np = packed_size(n_ao);
    if (store_ao) {
      h->J3_0.alloc(np * n_df);
      ao_fn(0, n_df, h->J3_0.get(), np, s);
    } else {
      h->ao_fn = std::move(ao_fn);
    }
    if (ri_fn) {
      if (store_ri) {
        h->J3_ri_0.alloc(n_ri * n_ao * n_df);
        ri_fn(0, n_df, h->J3_ri_0.get(), n_ri * n_ao, s);
      } else {
        h->ri_fn = std::move(ri_fn);
      }
    }
    UW12_CUDA(cudaStreamSynchronize(s));
  } catch (...) {
    delete h;
    throw;
  }
  return h;
}

IntegralsHandle* integrals_create_eigenbasis(const double* J3, const double* df_vals, size_t n_ao,
                                             size_t n_df, bool device_mem) {
  if (n_ao == 0) throw_runtime("Number of ao orbitals is zero");
  if (n_df == 0) throw_runtime("Number of density-fitting basis functions is zero");
  if (!J3 || !df_vals) throw Error(kErrInvalid, "null integral pointer");
  auto h = new IntegralsHandle();
  try {
    UW12_CUDA(cudaGetDevice(&h->device));
    cudaStream_t s = current_stream();
    h->n_ao = n_ao;
    h->n_df = n_df;
    const size_t np = packed_size(n_ao);
    h->J3_0.alloc(np * n_df);
    upload(h->J3_0.get(), J3, np * n_df, device_mem, s);
    h->P2.alloc(n_df * n_df);
    set_identity(h->P2.get(), LL(n_df));
    h->lam.alloc(n_df);
    upload(h->lam.get(), df_vals, n_df, device_mem, s);
    h->lam_host.resize(n_df);
    UW12_CUDA(cudaMemcpyAsync(h->lam_host.data(), h->lam.get(), n_df * sizeof(double),
                              cudaMemcpyDeviceToHost, s));
    UW12_CUDA(cudaStreamSynchronize(s));
  } catch (...) {
    delete h;
    throw;
  }
  return h;
}

AbsHandle* abs_create(const double* S, size_t n_ao, size_t n_ri, bool device_mem) {
  if (!S) throw Error(kErrInvalid, "null overlap pointer");
  const size_t n = n_ao + n_ri;
  if (n == 0) throw_runtime("Total number of basis functions is inconsistent");
  auto h = new AbsHandle();
  try {
    UW12_CUDA(cudaGetDevice(&h->device));
    cudaStream_t s = current_stream();
    h->n_ao = n_ao;
    h->n_ri = n_ri;
    DevBuf vecs(n * n, s);
    upload(vecs.get(), S, n * n, device_mem, s);
    require_symmetric(vecs.get(), n, "matrix must be symmetric");
    DevBuf vals(n, s);
    eigh(vecs.get(), n, vals.get());
    std::vector<double> lam(n);
    UW12_CUDA(cudaMemcpyAsync(lam.data(), vals.get(), n * sizeof(double), cudaMemcpyDeviceToHost,
                              s));
    UW12_CUDA(cudaStreamSynchronize(s));
    // eigen_decomposition(S, 1e-6, 1e-8) (linalg.hpp:1157-1197).
    double max_eig = 0.0;
    for (double v : lam) max_eig = std::max(max_eig, std::fabs(v));
    const double thr = std::max(max_eig * 1e-8, 1e-6);
    std::vector<int> keep;
    std::vector<double> inv;
    for (size_t i = 0; i < n; ++i)
      if (std::fabs(lam[i]) > thr) {
        if (!(lam[i] > 0.0)) throw_runtime("inv_sym_pd(): matrix is not positive definite");
        keep.push_back(static_cast<int>(i));
        inv.push_back(1.0 / lam[i]);
      }
    h->n_kept = keep.size();
    h->Sinv.alloc(n * n);
    const size_t r = keep.size();
    if (r == 0) {
      UW12_CUDA(cudaMemsetAsync(h->Sinv.get(), 0, n * n * sizeof(double), s));
    } else {
      int* d_idx = nullptr;
      UW12_CUDA(cudaMallocAsync(reinterpret_cast<void**>(&d_idx), r * sizeof(int), s));
      DevBuf d_inv(r, s), d_one(r, s), vk(n * r, s), vks(n * r, s);
      UW12_CUDA(cudaMemcpyAsync(d_idx, keep.data(), r * sizeof(int), cudaMemcpyHostToDevice, s));
      UW12_CUDA(cudaMemcpyAsync(d_inv.get(), inv.data(), r * sizeof(double),
                                cudaMemcpyHostToDevice, s));
      std::vector<double> ones(r, 1.0);
      UW12_CUDA(cudaMemcpyAsync(d_one.get(), ones.data(), r * sizeof(double),
                                cudaMemcpyHostToDevice, s));
      gather_scale_cols(vecs.get(), LL(n), d_idx, d_one.get(), LL(r), vk.get());
      gather_scale_cols(vecs.get(), LL(n), d_idx, d_inv.get(), LL(r), vks.get());
      GemmDesc g = gemm_nn(LL(n), LL(n), LL(r), 1.0, vks.get(), LL(n), vk.get(), LL(n), 0.0,
                           h->Sinv.get(), LL(n));
      g.b_ncontig = true;  // B = Vk^T
      gemm(g);
      UW12_CUDA(cudaFreeAsync(d_idx, s));
    }
    UW12_CUDA(cudaStreamSynchronize(s));
  } catch (...) {
    delete h;
    throw;
  }
  return h;
}

// --------------------------------------------------------------------------
// schedule helpers
// --------------------------------------------------------------------------
namespace {

// Phase timing: events recorded at phase boundaries while profiling is on.
std::mutex g_phase_mu;
std::map<std::string, double> g_phase_ms;

class PhaseClock {
 public:
  PhaseClock() : on_(profile_enabled()) {}
  ~PhaseClock() {
    if (!on_) return;
    for (auto& m : marks_) cudaEventDestroy(m.second);
  }
  void mark(const char* name) {
    if (!on_) return;
    cudaEvent_t e;
    UW12_CUDA(cudaEventCreate(&e));
    UW12_CUDA(cudaEventRecord(e, current_stream()));
    marks_.emplace_back(name, e);
  }
  // Accumulates the time from each mark to the next into its phase.
  void finish() {
    if (!on_ || marks_.size() < 2) return;
    UW12_CUDA(cudaEventSynchronize(marks_.back().second));
    std::lock_guard<std::mutex> lk(g_phase_mu);
    for (size_t i = 0; i + 1 < marks_.size(); ++i) {
      float ms = 0.f;
      UW12_CUDA(cudaEventElapsedTime(&ms, marks_[i].second, marks_[i + 1].second));
      g_phase_ms[marks_[i].first] += ms;
    }
  }

 private:
  bool on_;
  std::vector<std::pair<std::string, cudaEvent_t>> marks_;
};

enum Slot { kE2d = 0, kE2i = 1, kE3d = 2, kE3i = 3, kE4d = 4, kE4i = 5 };

double spin_factor(int ns, int s, int sp, double s_os, double s_ss) {
  // four_electron_utils.cpp:9-30
  if (ns == 1) return 2.0 * (s_os + s_ss);
  return (s == sp) ? s_ss : s_os;
}

// XDr (M x ns) = J3_0^T dmat: the unscaled fitted densities of libuw12's
// get_X_D (integrals.cpp:347-378), over aux blocks; only the rows of aux
// functions [a_lo, a_hi) are formed (the others are zero).
void fitted_density_raw(const IntegralsHandle& X, const double* dmat, int ns, double* XDr,
                        size_t budget, size_t a_lo = 0, size_t a_hi = SIZE_MAX) {
  const size_t M = X.n_df, np = packed_size(X.n_ao);
  a_hi = std::min(a_hi, M);
  if (a_lo > 0 || a_hi < M)
    UW12_CUDA(cudaMemsetAsync(XDr, 0, M * ns * sizeof(double), current_stream()));
  DevBuf scratch;
  const size_t step = aux_step(X, false, budget);
  for (size_t b0 = a_lo; b0 < a_hi; b0 += step) {
    const size_t nb = std::min(step, a_hi - b0);
    GemmDesc g = gemm_nn(LL(nb), ns, LL(np), 1.0, aux_block(X, false, b0, nb, scratch), LL(np),
                         dmat, LL(np), 0.0, XDr + b0, LL(M));
    g.a_kcontig = true;
    gemm(g);
  }
}

// Largest product (operations) of W and V in one launch, and largest evaluation (doubles of
// both potentials' transforms) that forms them side by side.  Closed-shell Fock matrices
// with 3 DF and 4 RI functions per AO, o = N / 10, in turn on one B200, with these limits / one
// after the other / side by side without limits: 0.26 / 0.31 / 0.26 ms at N = 24, 0.43 / 0.50
// / 0.43 at 61, 1.30 / 1.37 / 1.28 at 100, 2.32 / 2.38 / 2.28 at 120 (16 M doubles), 4.77 /
// 4.80 / 4.68 at 143, 6.98 / 7.00 / 6.89 at 160, 19.7 / 19.8 / 19.6 at 200: what lies above
// the limits gains 1 to 2 %, against twice the memory of the transforms.
constexpr double kJointFlops = 2e9;
constexpr size_t kJointDoubles = size_t(1) << 24;

// The same product for W and for V.  Small ones are bound by their launch and the
// latency of a k tile, so equal shapes run as two output batches of one launch, the
// batch strides being the distances between the operands (one B200, N=24 Fock 310 ->
// 270 us, open-shell energy at N=61 257 -> 231 us, N=120 Fock 2.38 -> 2.33 ms); larger
// ones fill the device by themselves, and split precision prepares its operands one by
// one.
void gemm_both(const GemmDesc& w, const GemmDesc& v) {
  const double flops = 2.0 * double(w.m) * double(w.n) * double(w.k) * double(w.nbo1) *
                       double(w.nbr1) * double(w.nbr2);
  const bool same = w.m == v.m && w.n == v.n && w.k == v.k && w.lda == v.lda && w.ldb == v.ldb &&
                    w.ldc == v.ldc && w.a_kcontig == v.a_kcontig && w.b_ncontig == v.b_ncontig &&
                    w.alpha == v.alpha && w.beta == v.beta && w.nbo1 == v.nbo1 && w.nbo2 == 1 &&
                    v.nbo2 == 1 && w.sAo1 == v.sAo1 && w.sBo1 == v.sBo1 && w.sCo1 == v.sCo1 &&
                    w.nbr1 == v.nbr1 && w.nbr2 == v.nbr2 && w.sAr1 == v.sAr1 &&
                    w.sAr2 == v.sAr2 && w.sBr1 == v.sBr1 && w.sBr2 == v.sBr2;
  if (!same || split_moduli() > 0 || flops > kJointFlops) {
    gemm(w);
    gemm(v);
    return;
  }
  auto distance = [](const double* from, const double* to) {
    return static_cast<long long>(reinterpret_cast<std::intptr_t>(to) -
                                  reinterpret_cast<std::intptr_t>(from)) /
           static_cast<long long>(sizeof(double));
  };
  GemmDesc g = w;
  g.nbo2 = 2;
  g.sAo2 = distance(w.A, v.A);
  g.sBo2 = distance(w.B, v.B);
  g.sCo2 = distance(w.C, v.C);
  gemm(g);
}

// H2 (R*na x (a_hi - a_lo)) = [J3_ri_0[:,A] (R x N) Cm] for A in [a_lo, a_hi)
// (transform_second_index, transformations.hpp:130-158), over aux blocks.
void ri_transform(const IntegralsHandle& X, const double* Cm, size_t na, double* H2,
                  size_t budget, size_t a_lo = 0, size_t a_hi = SIZE_MAX) {
  const size_t N = X.n_ao, R = X.n_ri;
  a_hi = std::min(a_hi, X.n_df);
  DevBuf scratch;
  const size_t step = aux_step(X, true, budget);
  for (size_t b0 = a_lo; b0 < a_hi; b0 += step) {
    const size_t nb = std::min(step, a_hi - b0);
    GemmDesc g = gemm_nn(LL(R), LL(na), LL(N), 1.0, aux_block(X, true, b0, nb, scratch), LL(R),
                         Cm, LL(N), 0.0, H2 + R * na * (b0 - a_lo), LL(R));
    g.nbo1 = LL(nb);
    g.sAo1 = LL(R * N);
    g.sCo1 = LL(R * na);
    gemm(g);
  }
}

// H (N*nc x (a_hi - a_lo)) = [sq(J3_0[:,A]) Cm] for A in [a_lo, a_hi), chunked
// over A.
void transform_ao(const IntegralsHandle& X, const double* Cm, size_t nc, double* H,
                  size_t budget, size_t a_lo = 0, size_t a_hi = SIZE_MAX) {
  const size_t N = X.n_ao, M = X.n_df, np = packed_size(N);
  a_hi = std::min(a_hi, M);
  if (nc == 0 || a_hi <= a_lo) return;
  const size_t ac =
      std::max<size_t>(1, std::min(a_hi - a_lo, budget / (N * N + (X.J3_0.get() ? 0 : np))));
  DevBuf U(N * N * ac), scratch;
  for (size_t a0 = a_lo; a0 < a_hi; a0 += ac) {
    const size_t na = std::min(ac, a_hi - a0);
    unpack_sym(aux_block(X, false, a0, na, scratch), LL(np), LL(N), LL(na), U.get(), LL(N),
               LL(N * N));
    GemmDesc g = gemm_nn(LL(N), LL(nc), LL(N), 1.0, U.get(), LL(N), Cm, LL(N), 0.0,
                         H + N * nc * (a0 - a_lo), LL(N));
    g.nbo1 = LL(na);
    g.sAo1 = LL(N * N);
    g.sCo1 = LL(N * nc);
    gemm(g);
  }
}

// Chunk size c <= max_chunk (in units of `unit` GEMM columns) for a loop over
// `total` units: the chunked GEMMs have n = unit * c columns, so c is chosen
// to fill 64-wide column tiles over the whole loop (fewest wasted columns, then
// the largest chunk).
size_t tile_chunk(size_t total, size_t unit, size_t max_chunk) {
  max_chunk = std::max<size_t>(1, std::min(max_chunk, total));
  auto tiles = [](size_t cols) { return (cols + 63) / 64; };
  size_t best = max_chunk;
  double best_fill = -1.0;
  for (size_t c = max_chunk; c >= std::max<size_t>(1, max_chunk / 2); --c) {
    const size_t full = total / c, rem = total % c;
    const size_t used = full * tiles(unit * c) + (rem ? tiles(unit * rem) : 0);
    const double fill = double(total * unit) / double(used * 64);
    if (fill > best_fill + 1e-9) {
      best_fill = fill;
      best = c;
    }
    if (c == 1) break;
  }
  return best;
}

struct SpinDims {
  size_t o = 0, a = 0, c = 0, ooff = 0, aoff = 0;
};

// Occupation-weighted occupied orbitals Co (utils.hpp:289-310) of both spins side
// by side (N x o_tot) and their active (last n_active) columns Ca (freeze_core,
// utils.hpp:235-253; N x a_tot), one after the other on the device.
void upload_orbitals(const FockRequest& rq, std::vector<SpinDims>& sd, size_t& o_tot,
                     size_t& a_tot, DevBuf& C) {
  const int ns = rq.n_spin;
  const size_t N = rq.n_ao;
  sd.assign(ns, SpinDims{});
  o_tot = a_tot = 0;
  for (int s = 0; s < ns; ++s) {
    sd[s].o = rq.n_occ[s];
    sd[s].a = rq.n_active[s];
    sd[s].c = sd[s].o - sd[s].a;
    sd[s].ooff = o_tot;
    sd[s].aoff = a_tot;
    o_tot += sd[s].o;
    a_tot += sd[s].a;
  }
  // [Co | Ca] is weighted on the host and copied at once
  std::vector<double> c(N * (o_tot + a_tot));
  const double per = (ns == 1) ? 2.0 : 1.0;
  for (int s = 0; s < ns; ++s)
    for (size_t k = 0; k < sd[s].o; ++k) {
      const double w = std::sqrt(rq.occ[s][k] / per);
      const double* src = rq.C[s] + rq.ldc[s] * k;
      double* dst = c.data() + N * (sd[s].ooff + k);
      for (size_t i = 0; i < N; ++i) dst[i] = w * src[i];
      if (k >= sd[s].c)
        std::copy(dst, dst + N, c.data() + N * (o_tot + sd[s].aoff + k - sd[s].c));
    }
  C.alloc(c.size());
  if (!c.empty())
    UW12_CUDA(cudaMemcpyAsync(C.get(), c.data(), c.size() * sizeof(double),
                              cudaMemcpyHostToDevice, current_stream()));
}

}  // namespace

// --------------------------------------------------------------------------
// form_fock
// --------------------------------------------------------------------------
namespace {
// Whether every three-index tensor that an evaluation reads is stored.
bool all_stored(const FockRequest& rq) {
  return rq.W->J3_0.get() && rq.V->J3_0.get() && rq.WV->J3_0.get() && rq.W->J3_ri_0.get() &&
         rq.V->J3_ri_0.get();
}

// Whether the t~ dX Fock term takes fewer operations over orbital pairs than over
// aux functions (halves of the FLOPs of both forms' products; a tie goes to
// the pairs).  Over aux functions: S^-1 G_W, and per spin J3^V T2^T and the sum
// over a.  Over pairs: S^-1 G_V and D, and without the same-spin terms (which
// form them anyway) G_W and G_V; with them Y_W is used twice and S^-1 Wst_W is
// not needed.  With 3 DF and 4 RI functions per AO and closed shell the pairs
// win in FP64 up to a o = 1.6 M without and 8 M with the same-spin terms.
// In split precision an operand element costs its preparation (8 bytes read twice and L
// residue bytes written at 5.8 TB/s) and a result element its reconstruction (L + 8
// bytes at 3.4 TB/s), in units of a multiply-add (L of them at 2.88 POPS): the forms'
// operations are equal at N=500, M=1500, R=2000, o=40/38, opposite spin, but the pairs
// prepare the three-index tensors once per spin: 338 ms, over aux functions 321 (in turn on
// one B200).  Every product is priced as if it ran split, which small and long ones
// do not; the routing rule has rates of its own (ozaki_profitable, where the reason stands).
//
// Unstored tensors are produced again for every chunk: V's over aux functions, W's and V's
// of every spin over pairs, where the same-spin terms do so anyway.  An element produced
// costs its 8 bytes at 2.9 TB/s on the device (a copy; slower producers would want aux
// functions earlier, but at 1 TB/s N=240, o=24/22 in split precision with a copying producer
// took 32.3 instead of 29.4 ms) or at 50 GB/s from the host, and the chunks are those that
// the budgets b_pairs and b_aux hold now.  Shards must agree on the form, whatever each has
// stored and free, so they leave this out.  N=160, M=480, R=640, o=16/15, opposite spin,
// host producers: 172 ms over pairs, 132 over aux functions.
bool pair_form_cheaper(const FockRequest& rq, const std::vector<SpinDims>& sd, bool same_spin,
                       double b_pairs, double b_aux) {
  const int ns = rq.n_spin;
  const double N = double(rq.n_ao), R = double(rq.W->n_ri), Rp = N + R;
  const double MW = double(rq.W->n_df), MV = double(rq.V->n_df);
  const double J = 0.5 * N * (N + 1.0) + R * N;  // rows of a three-index tensor
  const double L = split_moduli();
  const double prep = L > 0.0 ? 248.0 * (16.0 + L) / L : 0.0;
  const double crt = L > 0.0 ? 424.0 * (8.0 + L) / L : 0.0;
  auto product = [&](double m, double n, double k) {
    return m * n * k + prep * (m + n) * k + crt * m * n;
  };
  double aux = 0.0, pairs = 0.0, nq = 0.0;
  for (int sp = 0; sp < ns; ++sp) {
    bool any = false;
    for (int s = 0; s < ns; ++s)
      any = any || (spin_factor(ns, s, sp, rq.s_os, rq.s_ss) != 0.0 && sd[s].a > 0);
    if (any) nq += 1.0;
  }
  if (nq == 0.0) return false;
  aux = product(J, nq * MW, MV) + product(N, nq * N, Rp * MW) + nq * MW * MV * (MW + MV) +
        product(Rp, N * MW, Rp);
  for (int s = 0; s < ns; ++s) {
    const double a = double(sd[s].a), ap = double(pair_count(sd[s].a, sd[s].c, sd[s].o));
    pairs += product(Rp, N * ap, Rp) + (same_spin && ns == 1 ? 0.0 : product(N, N, Rp * ap));
    if (same_spin)
      aux += product(Rp * a, N * a, MW) + product(Rp, a * MW, Rp);
    else
      pairs += product(J, ap, MW) + product(J, ap, MV) + ap * (MW * MW + MV * MV);
  }
  // cost of producing what is not stored of X once
  const double per_second = L > 0.0 ? 1.44e15 / L : 16e12;
  auto once = [&](const IntegralsHandle& X) {
    const double elements =
        (X.J3_0.get() ? 0.0 : 0.5 * N * (N + 1.0)) + (X.J3_ri_0.get() ? 0.0 : R * N);
    return elements * double(X.n_df) * 8.0 / (X.host_producers ? 50e9 : 2.9e12) * per_second;
  };
  const double once_w = once(*rq.W), once_v = once(*rq.V);
  if (once_w + once_v > 0.0 && rq.n_shards <= 1) {
    const double np = 0.5 * N * (N + 1.0), gsz = Rp * N;
    auto chunks = [](double doubles, double budget) {
      return doubles > 0.0 ? std::ceil(doubles / budget) : 0.0;
    };
    // at most two eighths of the budget (a quarter and a sixteenth over aux functions) hold
    // the produced blocks
    auto pair_chunks = [&](const SpinDims& d, double n_s) {
      const double ap = double(pair_count(d.a, d.c, d.o));
      const double y = same_spin ? 2.0 * double(d.a) * double(d.o) : 0.0;
      return chunks(ap * ((1.0 + n_s) * gsz + np) + y * gsz, 0.75 * b_pairs);
    };
    aux += once_w + once_v * chunks(MW * ((1.0 + nq) * gsz + nq * np), 0.69 * b_aux);
    for (const SpinDims& d : sd) {
      pairs += pair_chunks(d, same_spin && ns == 2 ? 2.0 : 1.0) * (once_w + once_v);
      if (same_spin) aux += pair_chunks(d, 1.0) * (once_w + once_v);
    }
  }
  return pairs <= aux;
}
}  // namespace

size_t budget_need(const FockRequest& rq, bool adjoint, bool streamed) {
  const size_t N = rq.n_ao, np = packed_size(N), R = rq.W->n_ri, Rp = N + R;
  const size_t M = std::max({rq.W->n_df, rq.V->n_df, rq.WV->n_df});
  size_t o = 0, o1 = 0;  // occupied orbitals of all spins, of the larger spin
  for (size_t n : rq.n_occ) {
    o += n;
    o1 = std::max(o1, n);
  }
  // aux blocks of unstored tensors and of streamed gradients
  const size_t blocks = all_stored(rq) && !streamed ? 0 : 16 * (np + R * N) * M;
  size_t need = blocks + 2 * (N * N + np) * M;                           // unpacked AO blocks
  need = std::max(need, (2 * (N + o1) + 3 * Rp) * o * M);                // whole transforms
  if (rq.calc_fock) need = std::max(need, blocks + (4 * Rp * N + np + R * N) * M);
  if (rq.indirect) {
    need = std::max(need, (3 * Rp * o1 + M) * o1 * o1);                  // pair products of energies
  }
  if (rq.calc_fock) need = std::max(need, blocks + o1 * o1 * (5 * Rp * N + np));  // pair products
  if (adjoint)
    need = std::max({need, 2 * (N + R + 2 * (o1 + 2 * Rp)) * o * M, (4 * N * N + N * o) * M});
  return need;
}

void form_fock(const FockRequest& rq) {
  const IntegralsHandle& W = *rq.W;
  const IntegralsHandle& V = *rq.V;
  const IntegralsHandle& WV = *rq.WV;
  const AbsHandle& AB = *rq.abs;
  const int ns = rq.n_spin;
  const size_t N = rq.n_ao;
  const size_t np = packed_size(N);
  const size_t MW = W.n_df, MV = V.n_df, MX = WV.n_df;
  const size_t R = W.n_ri, Rp = N + R;
  const double s_os = rq.s_os, s_ss = rq.s_ss;
  const bool calc = rq.calc_fock;
  const bool do_ind = rq.indirect && s_ss != 0.0;
  const double half = (ns == 1) ? 0.5 : 1.0;
  const double two = (ns == 1) ? 2.0 : 1.0;
  const double kap4 = 2.0 * half;
  cudaStream_t st = current_stream();
  Budget budgets(rq, budget_need(rq, false, false), !all_stored(rq) || rq.n_shards > 1);
  size_t budget = budgets.doubles();
  // Sharding: aux functions and occupied orbitals are dealt out in
  // contiguous, balanced ranges (part).  The fitted densities, the MO
  // transforms and the 2-el Fock run over this shard's aux range, and the
  // partial intermediates (fitted densities, B1, the stacked RI rows) are
  // summed over the shards by rq.allreduce before use; X_AB and t are summed
  // from orbital ranges the same way.  The direct Fock and the same-spin 3-el
  // energy run over ranges of occupied k, the Fock terms over orbital pairs
  // over ranges of k with equal numbers of pairs (pair_bound), and t~ dX over
  // aux functions, where that form is the cheaper one, over a range of W's.
  // The energies built from the reduced intermediates and the same-spin 2-el /
  // 4-el terms come from shard 0.  The caller sums the partial energies and
  // Fock matrices over the shards.
  const size_t n_shards = std::max<size_t>(1, rq.n_shards);
  const size_t shard = rq.shard;
  const bool lead = shard == 0;
  const bool sharded = n_shards > 1;
  auto part = [&](size_t total) {
    return std::make_pair(total * shard / n_shards, total * (shard + 1) / n_shards);
  };
  if (sharded && !rq.allreduce)
    throw Error(kErrInvalid, "a sharded evaluation needs an all-reduce (uw12c_set_allreduce)");
  auto allreduce = [&](double* buf, size_t count) {
    if (!sharded || count == 0) return;
    if (rq.allreduce(buf, count, st, rq.allreduce_user) != 0)
      throw Error(kErrInvalid, "the all-reduce of a sharded evaluation failed");
  };

  std::vector<SpinDims> sd;
  size_t o_tot = 0, a_tot = 0;
  PhaseClock clock;
  clock.mark("orbitals");
  DevBuf orbs;
  upload_orbitals(rq, sd, o_tot, a_tot, orbs);
  const double* const Co = orbs.get();
  const double* const Ca = Co + N * o_tot;
  auto Ca_s = [&](int s) { return Ca + N * sd[s].aoff; };

  DevBuf acc(kAccDoubles);
  acc.zero();
  DevBuf Fall(N * N * ns);  // the spins' Fock matrices side by side
  Fall.zero();
  double* Fp[2] = {Fall.get(), Fall.get() + N * N};

  // =====================================================================
  // two-electron term (two_electron.cpp:11-153), WV integrals, active orbitals
  // =====================================================================
  clock.mark("two_electron");
  {
    // fitted densities and the 2-el Fock over this shard's aux range of WV
    const auto [xlo, xhi] = part(MX);
    DevBuf dmat(np * ns), XDr(MX * ns), XD(MX * ns);
    for (int s = 0; s < ns; ++s) pack_density(Ca_s(s), LL(N), LL(N), LL(sd[s].a), two, dmat.get() + np * s);
    fitted_density_raw(WV, dmat.get(), ns, XDr.get(), budget, xlo, xhi);
    allreduce(XDr.get(), MX * ns);
    GemmDesc g = gemm_nn(LL(MX), ns, LL(MX), 0.5 * ns, WV.P2.get(), LL(MX), XDr.get(), LL(MX), 0.0,
                         XD.get(), LL(MX));
    g.a_kcontig = true;
    gemm(g);
    double coef[4] = {0, 0, 0, 0};
    for (int s = 0; s < ns; ++s)
      for (int sp = 0; sp < ns; ++sp) {
        const double f = spin_factor(ns, s, sp, s_os, s_ss);
        if (f == 0.0) continue;
        if (lead)
          wdot(XD.get() + MX * s, LL(MX), XD.get() + MX * sp, LL(MX), LL(MX), 1, WV.lam.get(),
               nullptr, 0.5 * f, acc.get(), kE2d);
        coef[s * ns + sp] = 0.5 * ns * f;
      }
    if (calc) {
      DevBuf vc(MX * ns), u(MX * ns), gv(np * ns);
      combine_vecs(XD.get(), LL(MX), ns, coef, WV.lam.get(), vc.get());
      gemm(gemm_nn(LL(MX), ns, LL(MX), 1.0, WV.P2.get(), LL(MX), vc.get(), LL(MX), 0.0, u.get(),
                   LL(MX)));
      {
        // gv = J3_0 u over this shard's aux blocks
        DevBuf scratch;
        const size_t step = aux_step(WV, false, budget);
        if (xhi == xlo) gv.zero();
        for (size_t b0 = xlo; b0 < xhi; b0 += step) {
          const size_t nb = std::min(step, xhi - b0);
          gemm(gemm_nn(LL(np), ns, LL(nb), 1.0, aux_block(WV, false, b0, nb, scratch), LL(np),
                       u.get() + b0, LL(MX), b0 > xlo ? 1.0 : 0.0, gv.get(), LL(np)));
        }
      }
      for (int s = 0; s < ns; ++s)
        unpack_sym(gv.get() + np * s, LL(np), LL(N), 1, Fp[s], LL(N), 0, 1.0, 1.0);
    }
    if (do_ind && a_tot > 0) {
      // B1 of the active orbitals: the shard's aux range of sq(J3_0) Ca times
      // the matching rows of P2, summed over the shards
      DevBuf H(N * a_tot * (xhi - xlo));
      transform_ao(WV, Ca, a_tot, H.get(), budget / 2, xlo, xhi);
      for (int s = 0; s < ns; ++s) {
        const size_t a = sd[s].a;
        if (!a) continue;
        DevBuf B1(N * a * MX), B2(a * a * MX);
        gemm(gemm_nn(LL(N * a), LL(MX), LL(xhi - xlo), 1.0, H.get() + N * sd[s].aoff,
                     LL(N * a_tot), WV.P2.get() + xlo, LL(MX), 0.0, B1.get(), LL(N * a)));
        allreduce(B1.get(), N * a * MX);
        if (!lead) continue;
        GemmDesc g3 = gemm_nn(LL(a), LL(a * MX), LL(N), 1.0, Ca_s(s), LL(N), B1.get(), LL(N), 0.0,
                              B2.get(), LL(a));
        g3.a_kcontig = true;
        gemm(g3);
        wdot(B2.get(), LL(a * a), B2.get(), LL(a * a), LL(a * a), LL(MX), nullptr, WV.lam.get(),
             -0.5 * two, acc.get(), kE2i);
        if (calc) {
          DevBuf B1l(N * a * MX);
          scale_rc(B1.get(), LL(N * a), LL(N * a), LL(MX), nullptr, WV.lam.get(), 1.0, B1l.get(),
                   LL(N * a));
          GemmDesc gf = gemm_nn(LL(N), LL(N), LL(a * MX), -s_ss, B1.get(), LL(N), B1l.get(),
                                LL(N), 1.0, Fp[s], LL(N));
          gf.b_ncontig = true;
          gemm(gf);
        }
      }
    }
  }

  // =====================================================================
  // MO transforms for W and V (integrals.cpp:184-345)
  // =====================================================================
  clock.mark("transforms");
  struct PerX {
    std::vector<DevBuf> B1, B2, Wst, SV;
  };
  PerX XW, XV;
  // The t~ dX Fock term through orbital pairs (below) or aux functions; the
  // pairs need B2 whole.
  const bool pairs_cheaper =
      calc && (all_stored(rq) || sharded ? pair_form_cheaper(rq, sd, do_ind, 1.0, 1.0)
                              : pair_form_cheaper(rq, sd, do_ind, double(budgets.doubles()),
                                                  double(budgets.doubles(0.7))));
  const bool need_sv_w = calc && do_ind && !pairs_cheaper;
  // Without same-spin terms the stacked transforms serve only X_AB, t and the
  // direct Fock, which are sums over orbitals: when the whole intermediates
  // (B1, B2, Wst of W and V, S^-1 Wst_V) exceed the chunk budget they are
  // formed for a chunk of orbitals at a time instead (orbital_chunked).
  budget = budgets.doubles();
  size_t whole = 0;
  for (int s = 0; s < ns; ++s)
    whole += 2 * (N * sd[s].o * MW + sd[s].a * sd[s].o * MW) + 3 * Rp * sd[s].a * MW;
  bool orbital_chunked = !do_ind && whole > budget;
  if (sharded && !do_ind) {
    // every shard takes the same branch (the budgets may differ)
    DevBuf flag(1);
    const double one = orbital_chunked ? 1.0 : 0.0;
    UW12_CUDA(cudaMemcpyAsync(flag.get(), &one, sizeof(double), cudaMemcpyHostToDevice, st));
    allreduce(flag.get(), 1);
    double any = 0.0;
    UW12_CUDA(cudaMemcpyAsync(&any, flag.get(), sizeof(double), cudaMemcpyDeviceToHost, st));
    UW12_CUDA(cudaStreamSynchronize(st));
    orbital_chunked = any > 0.0;
  }
  const bool fold = pairs_cheaper && !orbital_chunked;
  // Small evaluations form W's and V's intermediates side by side, in joint launches: the
  // unpacked blocks and half transforms of both at once, so only within half of the chunk
  // budget, the share that the unpacked blocks have one after the other.
  const size_t side_by_side = 2 * (N * N + N * o_tot + R * a_tot) * MW;
  const bool joint = !sharded && MW == MV && W.J3_0.get() && V.J3_0.get() && W.J3_ri_0.get() &&
                     V.J3_ri_0.get() && split_moduli() == 0 &&
                     side_by_side <= std::min(kJointDoubles, budget / 2);
  for (int first = 0; first < 2 && !orbital_chunked; first += joint ? 2 : 1) {
    const int n_x = joint ? 2 : 1;
    const IntegralsHandle* Xs[2] = {first == 0 ? &W : &V, &V};
    PerX* Ps[2] = {first == 0 ? &XW : &XV, &XV};
    const size_t M = Xs[0]->n_df;
    auto each = [&](auto desc) {  // desc(q): the product of the group's potential q
      if (joint)
        gemm_both(desc(0), desc(1));
      else
        gemm(desc(0));
    };
    budget = budgets.doubles();
    // this shard's aux functions [xlo, xhi): B1 and the stacked RI rows are
    // partial products H[:, xlo:xhi] P2[xlo:xhi, :], summed over the shards
    const auto range = part(M);
    const size_t xlo = range.first, xhi = range.second;
    for (int q = 0; q < n_x; ++q) {
      Ps[q]->B1.resize(ns);
      Ps[q]->B2.resize(ns);
      Ps[q]->Wst.resize(ns);
      Ps[q]->SV.resize(ns);
      for (int s = 0; s < ns; ++s) Ps[q]->B1[s].alloc(N * sd[s].o * M);
    }
    {
      const size_t nh = N * o_tot * (xhi - xlo);
      DevBuf H(nh * n_x);
      if (joint) {
        DevBuf U(2 * N * N * M);
        for (int q = 0; q < 2; ++q)
          unpack_sym(Xs[q]->J3_0.get(), LL(np), LL(N), LL(M), U.get() + q * N * N * M, LL(N),
                     LL(N * N));
        GemmDesc g = gemm_nn(LL(N), LL(o_tot), LL(N), 1.0, U.get(), LL(N), Co, LL(N), 0.0, H.get(),
                             LL(N));
        g.nbo1 = LL(2 * M);
        g.sAo1 = LL(N * N);
        g.sCo1 = LL(N * o_tot);
        gemm(g);
      } else {
        transform_ao(*Xs[0], Co, o_tot, H.get(), budget / 2, xlo, xhi);
      }
      for (int s = 0; s < ns; ++s) {
        const size_t o = sd[s].o;
        if (!o) continue;
        each([&](int q) {
          return gemm_nn(LL(N * o), LL(M), LL(xhi - xlo), 1.0,
                         H.get() + nh * q + N * sd[s].ooff, LL(N * o_tot),
                         Xs[q]->P2.get() + xlo, LL(M), 0.0, Ps[q]->B1[s].get(), LL(N * o));
        });
        if (!joint) allreduce(Ps[0]->B1[s].get(), N * o * M);
      }
    }
    const size_t nh2 = R * a_tot * (xhi - xlo);
    DevBuf H2(nh2 * n_x);
    if (a_tot && joint) {
      each([&](int q) {
        GemmDesc g = gemm_nn(LL(R), LL(a_tot), LL(N), 1.0, Xs[q]->J3_ri_0.get(), LL(R), Ca, LL(N),
                             0.0, H2.get() + nh2 * q, LL(R));
        g.nbo1 = LL(M);
        g.sAo1 = LL(R * N);
        g.sCo1 = LL(R * a_tot);
        return g;
      });
    } else if (a_tot) {
      ri_transform(*Xs[0], Ca, a_tot, H2.get(), budget, xlo, xhi);
    }
    for (int s = 0; s < ns; ++s) {
      const size_t o = sd[s].o, a = sd[s].a, c = sd[s].c;
      if (!a) continue;
      for (int q = 0; q < n_x; ++q) {
        Ps[q]->B2[s].alloc(a * o * M);
        Ps[q]->Wst[s].alloc(Rp * a * M);
        if (sharded) Ps[q]->Wst[s].zero();  // AO rows stay zero through the sum
      }
      each([&](int q) {
        GemmDesc g3 = gemm_nn(LL(a), LL(o * M), LL(N), 1.0, Ca_s(s), LL(N), Ps[q]->B1[s].get(),
                              LL(N), 0.0, Ps[q]->B2[s].get(), LL(a));
        g3.a_kcontig = true;
        return g3;
      });
      each([&](int q) {
        GemmDesc g2 = gemm_nn(LL(R), LL(M), LL(xhi - xlo), 1.0,
                              H2.get() + nh2 * q + R * sd[s].aoff, LL(R * a_tot),
                              Xs[q]->P2.get() + xlo, LL(M), 0.0, Ps[q]->Wst[s].get() + N,
                              LL(Rp * a));
        g2.nbo1 = LL(a);
        g2.sAo1 = LL(R);
        g2.sCo1 = LL(Rp);
        return g2;
      });
      for (int q = 0; q < n_x; ++q) {
        PerX& P = *Ps[q];
        if (!joint) allreduce(P.Wst[s].get(), Rp * a * M);
        copy3d(P.B1[s].get() + N * c, LL(N), LL(N * o), P.Wst[s].get(), LL(Rp), LL(Rp * a), LL(N),
               LL(a), LL(M));
        if (first + q == 1 || need_sv_w) {
          // S^-1 Wst (R' x a M): this shard's aux columns, gathered by the sum
          P.SV[s].alloc(Rp * a * M);
          if (sharded) P.SV[s].zero();
          gemm(gemm_nn(LL(Rp), LL(a * (xhi - xlo)), LL(Rp), 1.0, AB.Sinv.get(), LL(Rp),
                       P.Wst[s].get() + Rp * a * xlo, LL(Rp), 0.0, P.SV[s].get() + Rp * a * xlo,
                       LL(Rp)));
          if (!joint) allreduce(P.SV[s].get(), Rp * a * M);
        }
      }
    }
  }

  // =====================================================================
  // X_AB, t, t~ and the direct energies (direct_utils.cpp:62-157,
  // four_electron.cpp:80-137)
  // =====================================================================
  clock.mark("xab_t_energies");
  std::vector<DevBuf> Xab(ns), tab(ns), ttl(ns);
  // B1 (N*nk x M) of occupied orbitals [k0, k0 + nk) of spin s for potential X:
  // sq(J3_0[:, A]) Co[:, k] P2.
  auto b1_chunk = [&](const IntegralsHandle& X, int s, size_t k0, size_t nk, DevBuf& out) {
    const size_t M = X.n_df;
    DevBuf H(N * nk * M);
    transform_ao(X, Co + N * (sd[s].ooff + k0), nk, H.get(), budget / 2);
    out.alloc(N * nk * M);
    gemm(gemm_nn(LL(N * nk), LL(M), LL(M), 1.0, H.get(), LL(N * nk), X.P2.get(), LL(M), 0.0,
                 out.get(), LL(N * nk)));
  };
  // occupied orbitals per chunk of the t and direct-Fock passes, active
  // orbitals per chunk of the X_AB pass
  // (per occupied orbital: B1 of W and V, the transform's output, Z or the two
  // B2 rows of its a active orbitals)
  // (the larger of the two potentials' aux counts sizes every buffer)
  const size_t Mmax = std::max(MW, MV);
  auto per_k = [&](int s) { return (4 * N + 2 * sd[s].a) * Mmax; };
  const size_t per_j = (N + R + 3 * Rp) * Mmax;
  if (orbital_chunked) {
    for (int s = 0; s < ns; ++s) {
      const size_t o = sd[s].o, a = sd[s].a, c = sd[s].c;
      Xab[s].alloc(MW * MV);
      tab[s].alloc(MW * MV);
      ttl[s].alloc(MW * MV);
      Xab[s].zero();
      tab[s].zero();
      if (a == 0) {
        ttl[s].zero();
        continue;
      }
      // X_AB = sum over active-orbital chunks of Wst_W[j]^T S^-1 Wst_V[j]
      // (this shard's orbitals; summed over the shards below)
      const auto [jlo, jhi] = part(a);
      const size_t jc = std::max<size_t>(1, std::min(jhi - jlo, budget / 2 / per_j));
      for (size_t j0 = jlo; j0 < jhi; j0 += jc) {
        const size_t nj = std::min(jc, jhi - j0);
        DevBuf St[2];
        for (int which = 0; which < 2; ++which) {
          const IntegralsHandle& X = which == 0 ? W : V;
          const size_t M = X.n_df;
          St[which].alloc(Rp * nj * M);
          // AO rows of orbital j: sq(J3_0) Co[:, c + j] P2, into rows [0, N) of its block
          DevBuf H(N * nj * M);
          transform_ao(X, Co + N * (sd[s].ooff + c + j0), nj, H.get(), budget / 2);
          GemmDesc ga = gemm_nn(LL(N), LL(M), LL(M), 1.0, H.get(), LL(N * nj), X.P2.get(), LL(M),
                                0.0, St[which].get(), LL(Rp * nj));
          ga.nbo1 = LL(nj);
          ga.sAo1 = LL(N);
          ga.sCo1 = LL(Rp);
          gemm(ga);
          // RI rows: J3ri_0[:, A] Ca[:, j] P2, into rows [N, R') of its block
          DevBuf H2(R * nj * M);
          ri_transform(X, Ca_s(s) + N * j0, nj, H2.get(), budget);
          GemmDesc gr = gemm_nn(LL(R), LL(M), LL(M), 1.0, H2.get(), LL(R * nj), X.P2.get(), LL(M),
                                0.0, St[which].get() + N, LL(Rp * nj));
          gr.nbo1 = LL(nj);
          gr.sAo1 = LL(R);
          gr.sCo1 = LL(Rp);
          gemm(gr);
        }
        DevBuf SVj(Rp * nj * MV);
        gemm(gemm_nn(LL(Rp), LL(nj * MV), LL(Rp), 1.0, AB.Sinv.get(), LL(Rp), St[1].get(),
                     LL(Rp), 0.0, SVj.get(), LL(Rp)));
        GemmDesc gx = gemm_nn(LL(MW), LL(MV), LL(Rp * nj), 1.0, St[0].get(), LL(Rp * nj),
                              SVj.get(), LL(Rp * nj), 1.0, Xab[s].get(), LL(MW));
        gx.a_kcontig = true;
        gemm(gx);
      }
      // t = sum over occupied-orbital chunks of B2_W[k]^T B2_V[k], B2 = Ca^T B1
      // (this shard's orbitals)
      const auto [klo, khi] = part(o);
      const size_t kc = std::max<size_t>(1, std::min(khi - klo, budget / 2 / per_k(s)));
      for (size_t k0 = klo; k0 < khi; k0 += kc) {
        const size_t nk = std::min(kc, khi - k0);
        DevBuf B1w, B1v, B2w(a * nk * MW), B2v(a * nk * MV);
        b1_chunk(W, s, k0, nk, B1w);
        b1_chunk(V, s, k0, nk, B1v);
        GemmDesc g3 = gemm_nn(LL(a), LL(nk * MW), LL(N), 1.0, Ca_s(s), LL(N), B1w.get(), LL(N),
                              0.0, B2w.get(), LL(a));
        g3.a_kcontig = true;
        gemm(g3);
        g3 = gemm_nn(LL(a), LL(nk * MV), LL(N), 1.0, Ca_s(s), LL(N), B1v.get(), LL(N), 0.0,
                     B2v.get(), LL(a));
        g3.a_kcontig = true;
        gemm(g3);
        GemmDesc gt = gemm_nn(LL(MW), LL(MV), LL(a * nk), 1.0, B2w.get(), LL(a * nk), B2v.get(),
                              LL(a * nk), 1.0, tab[s].get(), LL(MW));
        gt.a_kcontig = true;
        gemm(gt);
      }
      allreduce(Xab[s].get(), MW * MV);
      allreduce(tab[s].get(), MW * MV);
      scale_rc(tab[s].get(), LL(MW), LL(MW), LL(MV), W.lam.get(), V.lam.get(), 1.0,
               ttl[s].get(), LL(MW));
    }
  }
  for (int s = 0; s < ns && !orbital_chunked; ++s) {
    const size_t o = sd[s].o, a = sd[s].a;
    Xab[s].alloc(MW * MV);
    tab[s].alloc(MW * MV);
    ttl[s].alloc(MW * MV);
    if (a == 0) {
      Xab[s].zero();
      tab[s].zero();
      ttl[s].zero();
      continue;
    }
    // sums over this shard's orbitals (rows p + R' j of Wst / S^-1 Wst, rows
    // i + a k of B2), completed over the shards
    const auto [jlo, jhi] = part(a);
    const auto [klo, khi] = part(o);
    GemmDesc gx = gemm_nn(LL(MW), LL(MV), LL(Rp * (jhi - jlo)), 1.0, XW.Wst[s].get() + Rp * jlo,
                          LL(Rp * a), XV.SV[s].get() + Rp * jlo, LL(Rp * a), 0.0, Xab[s].get(),
                          LL(MW));
    gx.a_kcontig = true;
    gemm(gx);
    GemmDesc gt = gemm_nn(LL(MW), LL(MV), LL(a * (khi - klo)), 1.0, XW.B2[s].get() + a * klo,
                          LL(a * o), XV.B2[s].get() + a * klo, LL(a * o), 0.0, tab[s].get(),
                          LL(MW));
    gt.a_kcontig = true;
    gemm(gt);
    allreduce(Xab[s].get(), MW * MV);
    allreduce(tab[s].get(), MW * MV);
    scale_rc(tab[s].get(), LL(MW), LL(MW), LL(MV), W.lam.get(), V.lam.get(), 1.0, ttl[s].get(),
             LL(MW));
  }
  if (lead) {
    const double* X[2] = {};
    const double* t[2] = {};
    const double* T[2] = {};
    double cx[4] = {}, ct[4] = {};
    for (int s = 0; s < ns; ++s) {
      X[s] = Xab[s].get();
      t[s] = tab[s].get();
      T[s] = ttl[s].get();
      for (int sp = 0; sp < ns; ++sp) {
        const double f = spin_factor(ns, s, sp, s_os, s_ss);
        cx[s + 2 * sp] = -f;
        ct[s + 2 * sp] = 0.5 * f;
      }
    }
    spin_dots(X, t, T, ns, LL(MW * MV), cx, ct, acc.get(), kE3d, kE4d);
  }
  if (!do_ind && !orbital_chunked)  // the stacked transforms serve only X_AB and the same-spin terms
    for (int s = 0; s < ns; ++s) {
      XW.Wst[s].release();
      XW.SV[s].release();
      XV.Wst[s].release();
      XV.SV[s].release();
    }

  // =====================================================================
  // direct Fock: 4-el (four_electron.cpp:11-77) + 3-el X dt~ (direct_utils.cpp:164-204)
  // combined as sum_k w_k (B1_W Y)_k (x) (B1_V)_k, and 3-el t~ dX
  // (direct_utils.cpp:256-347) added to fock[sigma'] (three_electron.cpp:78)
  // =====================================================================
  if (calc) {
    clock.mark("direct_fock");
    for (int s = 0; s < ns; ++s) {
      const size_t o = sd[s].o, a = sd[s].a, c = sd[s].c;
      const auto [klo, khi] = part(o);  // this shard's occupied orbitals
      if (khi == klo) continue;
      const double* Tq[2] = {ttl[0].get(), ns > 1 ? ttl[1].get() : nullptr};
      const double* Xq[2] = {Xab[0].get(), ns > 1 ? Xab[1].get() : nullptr};
      double cT[2] = {0, 0}, cX[2] = {0, 0};
      for (int sp = 0; sp < ns; ++sp) {
        const double f = spin_factor(ns, s, sp, s_os, s_ss);
        cT[sp] = (f != 0.0) ? f * (a == 0 ? kap4 : 0.5 * kap4) : 0.0;
        cX[sp] = half * f;
      }
      DevBuf Y(MW * MV);
      combine_y(Y.get(), LL(MW), Tq, cT, Xq, cX, ns, W.lam.get(), V.lam.get());
      // whole B1 (rows of orbitals [klo, khi)), or B1 of W and V recomputed
      // for a chunk of occupied orbitals
      const size_t kc = orbital_chunked
                            ? std::max<size_t>(1, std::min(khi - klo, budget / 2 / per_k(s)))
                            : khi - klo;
      for (size_t k0 = klo; k0 < khi; k0 += kc) {
        const size_t nk = std::min(kc, khi - k0);
        DevBuf B1w, B1v, Z(N * nk * MV);
        if (orbital_chunked) {
          b1_chunk(W, s, k0, nk, B1w);
          b1_chunk(V, s, k0, nk, B1v);
        }
        const double* bw = orbital_chunked ? B1w.get() : XW.B1[s].get() + N * k0;
        const double* bv = orbital_chunked ? B1v.get() : XV.B1[s].get() + N * k0;
        const size_t ldb1 = orbital_chunked ? N * nk : N * o;
        gemm(gemm_nn(LL(N * nk), LL(MV), LL(MW), 1.0, bw, LL(ldb1), Y.get(), LL(MW), 0.0,
                     Z.get(), LL(N * nk)));
        // active orbitals (k >= c) weighted 2
        const size_t a0 = std::max(c, k0), a1 = k0 + nk;
        if (a > 0 && a1 > a0)
          copy3d(Z.get() + N * (a0 - k0), LL(N * nk), 0, Z.get() + N * (a0 - k0), LL(N * nk), 0,
                 LL(N * (a1 - a0)), LL(MV), 1, 2.0);
        GemmDesc gf = gemm_nn(LL(N), LL(N), LL(nk * MV), 1.0, Z.get(), LL(N), bv, LL(N), 1.0,
                              Fp[s], LL(N));
        gf.b_ncontig = true;
        if (ldb1 != N * nk) {
          // part of the whole B1: K = (k, A) as MV reduction batches of nk
          gf.k = LL(nk);
          gf.nbr1 = LL(MV);
          gf.sAr1 = LL(N * nk);
          gf.sBr1 = LL(ldb1);
        }
        gemm(gf);
      }
    }
    if (!do_ind && !orbital_chunked)  // B1 and B2 serve the direct Fock and the pair terms only
      for (int s = 0; s < ns; ++s) {
        XW.B1[s].release();
        XV.B1[s].release();
        if (fold) continue;
        XW.B2[s].release();
        XV.B2[s].release();
      }
    // t~ dX: F[sigma'] -= sum_ab T2[a,b] G_W[a]^T S^-1 G_V[b] with
    // T2 = P2_W Tc[sigma'] P2_V^T and G_X[a] = [sq(J3_0^X[:,a]); J3ri_0^X[:,a]]
    // (R' x N).  L[a] = S^-1 G_W[a] does not depend on sigma', so it is formed
    // once per aux chunk and contracted with H[a] = sum_b T2[a,b] G_V[b] of
    // every spin.
    if (!fold) clock.mark("tdx_fock");
    std::vector<int> tdx_spins;
    std::vector<DevBuf> T2s;
    for (int sp = 0; sp < ns && !fold; ++sp) {
      const double* Tq[2] = {ttl[0].get(), ns > 1 ? ttl[1].get() : nullptr};
      double cT[2] = {0, 0}, cX[2] = {0, 0};
      bool any = false;
      for (int s = 0; s < ns; ++s) {
        cT[s] = half * spin_factor(ns, s, sp, s_os, s_ss);
        any = any || (cT[s] != 0.0 && sd[s].a > 0);
      }
      if (!any) continue;
      DevBuf Tc(MW * MV), tmp(MW * MV), T2(MW * MV);
      combine_y(Tc.get(), LL(MW), Tq, cT, Tq, cX, ns, W.lam.get(), V.lam.get());
      gemm(gemm_nn(LL(MW), LL(MV), LL(MW), 1.0, W.P2.get(), LL(MW), Tc.get(), LL(MW), 0.0,
                   tmp.get(), LL(MW)));
      GemmDesc gt2 = gemm_nn(LL(MW), LL(MV), LL(MV), 1.0, tmp.get(), LL(MW), V.P2.get(), LL(MV),
                             0.0, T2.get(), LL(MW));
      gt2.b_ncontig = true;
      gemm(gt2);
      tdx_spins.push_back(sp);
      T2s.push_back(std::move(T2));
    }
    if (!tdx_spins.empty()) {
      // The chunk buffers are the only large allocations of this phase, so
      // it takes 70% of the available memory.  Unstored V blocks are
      // produced again for every chunk of W's aux functions: V's RI blocks
      // take up to a quarter of the budget (their aux functions are the
      // contraction length of the p GEMM, whose output is large), its AO
      // blocks up to a sixteenth, the chunk the rest.
      budget = budgets.doubles(0.7);
      const size_t vstep = aux_step(V, false, budget / 4), vrstep = aux_step(V, true, budget);
      const size_t vscr = (V.J3_0.get() ? 0 : np * vstep) + (V.J3_ri_0.get() ? 0 : R * N * vrstep);
      const size_t nq = tdx_spins.size(), gsz = Rp * N;
      const size_t per_a = (1 + nq) * gsz + nq * np;
      const size_t avail = budget > vscr ? budget - vscr : 0;
      const auto [alo, ahi] = part(MW);
      const size_t ac = tile_chunk(ahi - alo, 1,
                                   std::max<size_t>(1, std::min(ahi - alo, avail / per_a)));
      // T2 of the spins interleaved: row q + nq a, so that H[a] of all spins comes
      // out of one product and is one operand of the last
      DevBuf T2i;
      const double* T2 = T2s[0].get();
      if (nq > 1) {
        T2i.alloc(nq * MW * MV);
        for (size_t q = 0; q < nq; ++q)
          copy3d(T2s[q].get(), 1, LL(MW), T2i.get() + q, LL(nq), LL(nq * MW), 1, LL(MW), LL(MV));
        T2 = T2i.get();
      }
      // Per chunk of W's aux functions a: G = [sq(J3_0^W[:, a]); J3ri_0^W[:, a]]
      // (R' x N per a), L = S^-1 G, the packed columns s, and H (R' x N per a and
      // spin).  Stacked AO + RI operands and stacked spins prepare (in
      // split precision) and read every operand once per chunk, and each product
      // is written once: the opposite-spin Fock at N = 500, M = 1500, R = 2000, open
      // shell, 14 moduli 369 -> 332 ms.  What is larger per a makes chunks shorter and
      // the producers of V run more often, so memory is shared: W's blocks are produced
      // where L is written next, and H takes G's place, which only L reads.  Buffers for
      // each would be 28.0 instead of 15.1 M doubles per a at N = 1200, R = 4800 (closed
      // shell): 1.8 times the passes over V's integrals.
      DevBuf Lb(gsz * ac), H(gsz * ac * nq), sbuf(np * ac * nq), scrV, scrVr;
      double* const G = H.get();
      for (size_t a0 = alo; a0 < ahi; a0 += ac) {
        const size_t na = std::min(ac, ahi - a0);
        unpack_sym(aux_block(W, false, a0, na, Lb.get()), LL(np), LL(N), LL(na), G, LL(Rp),
                   LL(gsz));
        copy3d(aux_block(W, true, a0, na, Lb.get()), LL(R), LL(R * N), G + N, LL(Rp), LL(gsz),
               LL(R), LL(N), LL(na));
        gemm(gemm_nn(LL(Rp), LL(N * na), LL(Rp), 1.0, AB.Sinv.get(), LL(Rp), G, LL(Rp), 0.0,
                     Lb.get(), LL(Rp)));
        // s = J3_0^V T2^T and p = J3_ri_0^V T2^T, accumulated over V's aux blocks
        const double* t2 = T2 + nq * a0;
        for (size_t b0 = 0; b0 < MV; b0 += vstep) {
          const size_t nb = std::min(vstep, MV - b0);
          GemmDesc gs = gemm_nn(LL(np), LL(na * nq), LL(nb), 1.0,
                                aux_block(V, false, b0, nb, scrV), LL(np), t2 + nq * MW * b0,
                                LL(nq * MW), b0 ? 1.0 : 0.0, sbuf.get(), LL(np));
          gs.b_ncontig = true;
          gemm(gs);
        }
        unpack_sym(sbuf.get(), LL(np), LL(N), LL(na * nq), H.get(), LL(Rp), LL(gsz));
        for (size_t b0 = 0; b0 < MV; b0 += vrstep) {
          const size_t nb = std::min(vrstep, MV - b0);
          GemmDesc gp = gemm_nn(LL(R), LL(na * nq), LL(nb), 1.0,
                                aux_block(V, true, b0, nb, scrVr), LL(R * N), t2 + nq * MW * b0,
                                LL(nq * MW), b0 ? 1.0 : 0.0, H.get() + N, LL(gsz));
          gp.b_ncontig = true;
          gp.nbo1 = LL(N);
          gp.sAo1 = LL(R);
          gp.sCo1 = LL(Rp);
          gemm(gp);
        }
        // F[sigma'] -= sum_a L[a]^T H[a], the spins' Fock matrices side by side
        GemmDesc gf = gemm_nn(LL(N), LL(N * nq), LL(Rp), -1.0, Lb.get(), LL(Rp), H.get(), LL(Rp),
                              1.0, Fp[tdx_spins[0]], LL(N));
        gf.a_kcontig = true;
        gf.nbr1 = LL(na);
        gf.sAr1 = LL(gsz);
        gf.sBr1 = LL(gsz * nq);
        gemm(gf);
      }
    }
  }

  // =====================================================================
  // terms over orbital pairs: the same-spin (indirect) terms, and t~ dX when
  // it is cheaper there
  // =====================================================================
  if (do_ind || fold) {
    for (int s = 0; s < ns; ++s) {
      const size_t o = sd[s].o, a = sd[s].a, c = sd[s].c;
      if (a == 0 || o == 0) continue;
      const size_t ao = a * o, No = N * o;
      DevBuf b2wl, b2vl, b1wl, b1vl;
      if (do_ind) {
        b2wl.alloc(ao * MW);
        b2vl.alloc(ao * MV);
        scale_rc(XW.B2[s].get(), LL(ao), LL(ao), LL(MW), nullptr, W.lam.get(), 1.0, b2wl.get(),
                 LL(ao));
        scale_rc(XV.B2[s].get(), LL(ao), LL(ao), LL(MV), nullptr, V.lam.get(), 1.0, b2vl.get(),
                 LL(ao));
        clock.mark("ss_4el_energy");
        // ---- 4-el indirect energy (four_electron.cpp:143-179)
        if (lead) {
          DevBuf W4(ao * ao), V4(ao * ao);
          GemmDesc gw = gemm_nn(LL(ao), LL(ao), LL(MW), 1.0, b2wl.get(), LL(ao), XW.B2[s].get(),
                                LL(ao), 0.0, W4.get(), LL(ao));
          gw.b_ncontig = true;
          GemmDesc gv = gemm_nn(LL(ao), LL(ao), LL(MV), 1.0, b2vl.get(), LL(ao), XV.B2[s].get(),
                                LL(ao), 0.0, V4.get(), LL(ao));
          gv.b_ncontig = true;
          gemm_both(gw, gv);
          permdot_4el(W4.get(), V4.get(), LL(a), LL(o), -0.5 * two, acc.get(), kE4i);
        }
        clock.mark("ss_3el_energy");
        // ---- 3-el indirect energy (indirect_utils.cpp:101-133), chunked over k, YW and ZV
        // formed once per pair of a chunk (B2 is symmetric in the active pair): N=300 Fock
        // 129.5 -> 125.9 ms
        {
          budget = budgets.doubles();
          const size_t per_k = 2 * Rp * a * a + a * (MW + MV);
          const auto [klo, khi] = part(o);
          const size_t kc = tile_chunk(khi - klo, a,
                                       std::max<size_t>(1, std::min(khi - klo, budget / per_k)));
          DevBuf YW, ZV, b2p;
          for (size_t k0 = klo; k0 < khi; k0 += kc) {
            const PairColumns q = PairColumns::of(LL(a), LL(c), LL(k0), LL(std::min(kc, khi - k0)));
            const size_t n = static_cast<size_t>(q.count());
            if (YW.size() < Rp * a * n) {
              YW.alloc(Rp * a * n);
              ZV.alloc(Rp * a * n);
              b2p.alloc(n * (MW + MV));
            }
            double* b2v = b2p.get() + n * MW;
            pack_pairs(XW.B2[s].get(), q, LL(o), LL(MW), W.lam.get(), 0.5, b2p.get());
            pack_pairs(XV.B2[s].get(), q, LL(o), LL(MV), V.lam.get(), 0.5, b2v);
            GemmDesc gw = gemm_nn(LL(Rp * a), LL(n), LL(MW), 1.0, XW.Wst[s].get(), LL(Rp * a),
                                  b2p.get(), LL(n), 0.0, YW.get(), LL(Rp * a));
            gw.b_ncontig = true;
            GemmDesc gv = gemm_nn(LL(Rp * a), LL(n), LL(MV), 1.0, XV.SV[s].get(), LL(Rp * a), b2v,
                                  LL(n), 0.0, ZV.get(), LL(Rp * a));
            gv.b_ncontig = true;
            gemm_both(gw, gv);
            permdot_3el(YW.get(), ZV.get(), LL(Rp), q, two, acc.get(), kE3i);
          }
        }
        if (!calc) continue;
        b1wl.alloc(No * MW);
        b1vl.alloc(No * MV);
        scale_rc(XW.B1[s].get(), LL(No), LL(No), LL(MW), nullptr, W.lam.get(), 1.0, b1wl.get(),
                 LL(No));
        scale_rc(XV.B1[s].get(), LL(No), LL(No), LL(MV), nullptr, V.lam.get(), 1.0, b1vl.get(),
                 LL(No));
        clock.mark("ss_4el_fock");
        // ---- 4-el indirect Fock (four_electron.cpp:181-249)
        if (lead) {
          DevBuf W43(No * ao), V43(No * ao);
          GemmDesc gw = gemm_nn(LL(No), LL(ao), LL(MW), 1.0, b1wl.get(), LL(No), XW.B2[s].get(),
                                LL(ao), 0.0, W43.get(), LL(No));
          gw.b_ncontig = true;
          GemmDesc gv = gemm_nn(LL(No), LL(ao), LL(MV), 1.0, b1vl.get(), LL(No), XV.B2[s].get(),
                                LL(ao), 0.0, V43.get(), LL(No));
          gv.b_ncontig = true;
          gemm_both(gw, gv);
          GemmDesc gi = gemm_nn(LL(N), LL(N), LL(a), s_ss * (c > 0 ? -1.0 : -2.0),
                                W43.get() + N * c, LL(No), V43.get() + N * c, LL(N), 1.0,
                                Fp[s], LL(N));
          gi.b_ncontig = true;
          gi.nbr1 = LL(a);
          gi.nbr2 = LL(o);
          gi.sAr1 = LL(N);
          gi.sAr2 = LL(No * a);
          gi.sBr1 = LL(No);
          gi.sBr2 = LL(No * a);
          gemm(gi);
          if (c > 0) {
            GemmDesc gf = gemm_nn(LL(N), LL(N), LL(a), -s_ss, W43.get(), LL(No), V43.get(), LL(No),
                                  1.0, Fp[s], LL(N));
            gf.b_ncontig = true;
            gf.nbr1 = LL(o);
            gf.nbr2 = LL(o);
            gf.sAr1 = LL(N);
            gf.sAr2 = LL(No * a);
            gf.sBr1 = LL(No * a);
            gf.sBr2 = LL(N);
            gemm(gf);
          }
        }
      }
      clock.mark("pair_fock");
      // ---- Fock terms over pairs of an active orbital j and an occupied
      // orbital k, in chunks of k.  With G_X[jk] = sum_A [sq(J3_0^X[:,A]);
      // J3ri_0^X[:,A]] x^_X[A;jk], x^_X = P2_X L_X B2_X^T, and
      // Y_X[jk] = Wst_X[j] L_X B1_X[k]^T (both R' x N):
      //   same-spin 3-el (indirect_utils.cpp:139-345)
      //     s_ss sum_jk (G_W^T S^-1 Y_V + G_V^T S^-1 Y_W)
      //     + s_ss sum_ij Y_W[i,c+j]^T S^-1 Y_V[j,c+i]
      //   t~ dX (direct_utils.cpp:256-347), T2 = sum_s x^_W x^_V^T:
      //     F[sigma'] -= half f(s, sigma') D, D = sum_jk G_W^T S^-1 G_V.
      // t~ has the rank of the pairs, so D needs S^-1 on N a o columns instead
      // of S^-1 G_W on the N M of all aux functions and J3^V T2^T (M x M); with
      // the same-spin terms G_W and G_V are there already, S^-1 G_V also
      // replaces S^-1 Y_W (Y_W then serves the k-term as it is), and no
      // product has an aux x aux operand.  pair_form_cheaper counts both forms.
      // The integrals are symmetric, so x^ and G of the active pairs (j, c + i)
      // and (i, c + j) are the same: G, S^-1 G and the sums with them run over
      // the a c pairs with a core orbital and the a (a + 1) / 2 pairs j <= i, with
      // Y[j, c+i] + Y[i, c+j] beside G.  Only Y, which the k-term pairs with its
      // mirror image, is formed for both orders.
      // One B200, against the same sums over all a o pairs: closed shell N=300, M=900,
      // R=1200, o=30 in FP64 176 -> 130 ms, o=30/29 in split precision 186 -> 141; open
      // shell N=200, M=600, R=800, o=16/15 35.1 -> 26.7 ms.
      double cD[2] = {0.0, 0.0};
      for (int sp = 0; sp < ns && fold; ++sp) cD[sp] = half * spin_factor(ns, s, sp, s_os, s_ss);
      if (!do_ind && cD[0] == 0.0 && cD[1] == 0.0) continue;
      // x^ of the pairs, in pair order; twice the mean of the two orders for V, so that
      // S^-1 G_V carries the weight of a pair, the mean for W
      const size_t n_all = pair_count(a, c, o);
      DevBuf xhW(MW * n_all), xhV(MV * n_all);
      {
        DevBuf b2p(n_all * (MW + MV));
        double* b2v = b2p.get() + n_all * MW;
        const PairColumns all = PairColumns::of(LL(a), LL(c), 0, LL(o));
        pack_pairs(XW.B2[s].get(), all, LL(o), LL(MW), W.lam.get(), 0.5, b2p.get());
        pack_pairs(XV.B2[s].get(), all, LL(o), LL(MV), V.lam.get(), 1.0, b2v);
        GemmDesc gw = gemm_nn(LL(MW), LL(n_all), LL(MW), 1.0, W.P2.get(), LL(MW), b2p.get(),
                              LL(n_all), 0.0, xhW.get(), LL(MW));
        gw.b_ncontig = true;
        GemmDesc gv = gemm_nn(LL(MV), LL(n_all), LL(MV), 1.0, V.P2.get(), LL(MV), b2v, LL(n_all),
                              0.0, xhV.get(), LL(MV));
        gv.b_ncontig = true;
        gemm_both(gw, gv);
      }
      budget = budgets.doubles();
      // unstored W / V blocks (accumulated over, for every k chunk) take at
      // most an eighth of the budget each
      size_t xscr = 0;
      for (const IntegralsHandle* Xi : {&W, &V})
        xscr = std::max(xscr, (Xi->J3_0.get() ? 0 : np * aux_step(*Xi, false, budget / 2)) +
                                  (Xi->J3_ri_0.get() ? 0 : R * N * aux_step(*Xi, true, budget / 2)));
      const size_t pair = Rp * N;  // doubles of one pair's matrix
      const size_t klo = pair_bound(a, c, shard, n_shards);
      const size_t khi = pair_bound(a, c, shard + 1, n_shards);
      const size_t kavail = budget > xscr ? budget - xscr : 0;
      // A chunk of occupied orbitals [k0, k0 + nk): its pairs are [p0, p0 + np_) in
      // pair order.  Y of its pairs lies in two blocks: Y[j, k], j < nj, is matrix
      // (k - k0) + nk j; where the chunk's active orbitals are [i0, i1), the mirror
      // images Y[i, c + j], j < i0, are matrices j + i0 (i - i0) behind them.
      // Unless it takes every orbital, a chunk has core or active orbitals only.
      struct PairChunk {
        size_t k0, nk, p0, n_pairs, nj, i0, i1, n_y;
      };
      const size_t n_s = do_ind && fold && ns == 2 ? 2 : 1;
      const size_t n_g = joint && fold ? 2 : 1;  // G_V alone, or G_V and G_W at once
      auto pair_chunk = [&](size_t k0, size_t nk) {
        PairChunk q{};
        q.k0 = k0;
        q.nk = nk;
        q.p0 = pair_count(a, c, k0);
        q.n_pairs = pair_count(a, c, k0 + nk) - q.p0;
        q.i0 = std::max(k0, c) - c;
        q.i1 = std::max(k0 + nk, c) - c;
        q.nj = k0 < c ? a : q.i1;
        q.n_y = do_ind ? nk * q.nj + q.i0 * (q.i1 - q.i0) : 0;
        return q;
      };
      std::vector<PairChunk> chunks;
      size_t max_pairs = 0, max_y = 0;
      for (size_t k0 = klo; k0 < khi;) {
        PairChunk q = pair_chunk(k0, khi - k0);
        auto need = [&] {
          return pair * (q.n_pairs * (n_g + n_s) + 2 * q.n_y) + np * q.n_pairs * n_g;
        };
        if (q.nk < o || need() > kavail) {
          const size_t end = k0 < c ? std::min(c, khi) : khi;
          q = pair_chunk(k0, end - k0);
          while (q.nk > 1 && need() > kavail) q = pair_chunk(k0, q.nk - 1);
        }
        chunks.push_back(q);
        max_pairs = std::max(max_pairs, q.n_pairs);
        max_y = std::max(max_y, q.n_y);
        k0 += q.nk;
      }
      const size_t nbuf = pair * max_pairs;
      DevBuf gpk(np * max_pairs * n_g), bufG(nbuf * n_g), bufS(nbuf * n_s), bufY(pair * max_y),
          bufZ(pair * max_y), scrX, scrXr;
      // dst = G_X of the chunk's pairs, over X's aux blocks
      auto form_g = [&](const IntegralsHandle& X, const double* xh, const PairChunk& q,
                        double* dst) {
        const size_t M = X.n_df;
        const double* x = xh + M * q.p0;
        const size_t st_ao = aux_step(X, false, budget / 2);
        const size_t st_ri = aux_step(X, true, budget / 2);
        for (size_t b0 = 0; b0 < M; b0 += st_ao) {
          const size_t nb = std::min(st_ao, M - b0);
          gemm(gemm_nn(LL(np), LL(q.n_pairs), LL(nb), 1.0, aux_block(X, false, b0, nb, scrX),
                       LL(np), x + b0, LL(M), b0 ? 1.0 : 0.0, gpk.get(), LL(np)));
        }
        unpack_sym(gpk.get(), LL(np), LL(N), LL(q.n_pairs), dst, LL(Rp), LL(pair));
        for (size_t b0 = 0; b0 < M; b0 += st_ri) {
          const size_t nb = std::min(st_ri, M - b0);
          GemmDesc gr = gemm_nn(LL(R), LL(q.n_pairs), LL(nb), 1.0,
                                aux_block(X, true, b0, nb, scrXr), LL(R * N), x + b0, LL(M),
                                b0 ? 1.0 : 0.0, dst + N, LL(pair));
          gr.nbo1 = LL(N);
          gr.sAo1 = LL(R);
          gr.sCo1 = LL(Rp);
          gemm(gr);
        }
      };
      // G_V of the chunk's pairs and G_W behind it (stored integrals)
      auto form_g_both = [&](const PairChunk& q, double* dst) {
        auto ao_rows = [&](const IntegralsHandle& X, const double* xh, size_t at) {
          return gemm_nn(LL(np), LL(q.n_pairs), LL(X.n_df), 1.0, X.J3_0.get(), LL(np),
                         xh + X.n_df * q.p0, LL(X.n_df), 0.0, gpk.get() + np * at, LL(np));
        };
        auto ri_rows = [&](const IntegralsHandle& X, const double* xh, double* to) {
          GemmDesc gr = gemm_nn(LL(R), LL(q.n_pairs), LL(X.n_df), 1.0, X.J3_ri_0.get(), LL(R * N),
                                xh + X.n_df * q.p0, LL(X.n_df), 0.0, to + N, LL(pair));
          gr.nbo1 = LL(N);
          gr.sAo1 = LL(R);
          gr.sCo1 = LL(Rp);
          return gr;
        };
        gemm_both(ao_rows(V, xhV.get(), 0), ao_rows(W, xhW.get(), q.n_pairs));
        unpack_sym(gpk.get(), LL(np), LL(N), LL(2 * q.n_pairs), dst, LL(Rp), LL(pair));
        gemm_both(ri_rows(V, xhV.get(), dst), ri_rows(W, xhW.get(), dst + pair * q.n_pairs));
      };
      // block 0 (Y[j, k]) or 1 (the mirror images behind them) of dst = St[j] L B1[k]^T of
      // the chunk (St: R' a x M)
      auto y_block = [&](int b, const double* St, const double* b1l, size_t M,
                         const PairChunk& q, double* dst) {
        const size_t j0 = b ? q.i0 : 0, nj = b ? q.i1 - q.i0 : q.nj;
        const size_t k0 = b ? c : q.k0, nk = b ? q.i0 : q.nk;
        GemmDesc gy = gemm_nn(LL(Rp), LL(N * nk), LL(M), 1.0, St + Rp * j0, LL(Rp * a),
                              b1l + N * k0, LL(No), 0.0, dst + (b ? pair * q.nk * q.nj : 0),
                              LL(Rp));
        gy.b_ncontig = true;
        gy.nbo1 = LL(nj);
        gy.sAo1 = LL(Rp);
        gy.sCo1 = LL(pair * nk);
        return gy;
      };
      auto form_y = [&](const double* St, const double* b1l, size_t M, const PairChunk& q,
                        double* dst) {
        for (int b = 0; b < (q.i0 ? 2 : 1); ++b) gemm(y_block(b, St, b1l, M, q, dst));
      };
      // out = coef (Y[j, k] + Y[i, c + j]) + coef_s S per pair; the sum is scaled by
      // mirror where it has two terms
      auto sum_y = [&](const PairChunk& q, const double* Y, double coef, double mirror,
                       const double* S, double coef_s, double* dst) {
        sum_pairs(Y, Y + pair * q.nk * q.nj, LL(pair), LL(a), LL(c), LL(q.k0), LL(q.nk),
                  LL(q.n_pairs), coef, mirror, S, coef_s, dst);
      };
      // F += coef sum_pairs A[pair]^T B[pair]
      auto add_pairs = [&](double coef, const double* A, const double* B, size_t n_pairs,
                           double* F) {
        GemmDesc gf = gemm_nn(LL(N), LL(N), LL(Rp), coef, A, LL(Rp), B, LL(Rp), 1.0, F, LL(N));
        gf.a_kcontig = true;
        gf.nbr1 = LL(n_pairs);
        gf.sAr1 = LL(pair);
        gf.sBr1 = LL(pair);
        gemm(gf);
      };
      // k-term (fock_k): F += s_ss sum Y_W[i, c + j]^T Z[j, c + i] over the chunk's
      // active pairs, both orders
      auto k_term = [&](const PairChunk& q, const double* Yw, const double* Z) {
        const size_t ni = q.i1 - q.i0, i0 = q.i0, nk = q.nk;
        if (ni == 0) return;
        auto add = [&](size_t nj, const double* A, size_t sAi, size_t sAj, const double* B,
                       size_t sBi, size_t sBj) {
          if (nj == 0) return;
          GemmDesc fk = gemm_nn(LL(N), LL(N), LL(Rp), s_ss, A, LL(Rp), B, LL(Rp), 1.0, Fp[s],
                                LL(N));
          fk.a_kcontig = true;
          fk.nbr1 = LL(ni);
          fk.nbr2 = LL(nj);
          fk.sAr1 = LL(pair * sAi);
          fk.sAr2 = LL(pair * sAj);
          fk.sBr1 = LL(pair * sBi);
          fk.sBr2 = LL(pair * sBj);
          gemm(fk);
        };
        const size_t first = c + i0 - q.k0;  // orbital c + i0 in the chunk
        const size_t blk = pair * (first + nk * i0), back = pair * nk * q.nj;
        add(ni, Yw + blk, nk, 1, Z + blk, 1, nk);
        add(i0, Yw + back, i0, 1, Z + pair * first, 1, nk);
        add(i0, Yw + pair * first, 1, nk, Z + back, i0, 1);
      };
      for (const PairChunk& q : chunks) {
        const bool both = n_g == 2;
        const double* gw = bufG.get() + (both ? pair * q.n_pairs : 0);  // G_W
        if (both)
          form_g_both(q, bufG.get());
        else
          form_g(V, xhV.get(), q, bufG.get());
        if (both && do_ind)
          for (int b = 0; b < (q.i0 ? 2 : 1); ++b)
            gemm_both(y_block(b, XW.Wst[s].get(), b1wl.get(), MW, q, bufY.get()),
                      y_block(b, XV.SV[s].get(), b1vl.get(), MV, q, bufZ.get()));
        if (fold) {
          gemm(gemm_nn(LL(Rp), LL(N * q.n_pairs), LL(Rp), 1.0, AB.Sinv.get(), LL(Rp), bufG.get(),
                       LL(Rp), 0.0, bufS.get(), LL(Rp)));
          if (do_ind) {
            if (!both) form_y(XW.Wst[s].get(), b1wl.get(), MW, q, bufY.get());
            sum_y(q, bufY.get(), 1.0, 0.5, nullptr, 0.0, bufG.get());
            add_pairs(s_ss, bufS.get(), bufG.get(), q.n_pairs, Fp[s]);
          }
        } else {
          form_y(XW.SV[s].get(), b1wl.get(), MW, q, bufY.get());
          sum_y(q, bufY.get(), 1.0, 0.5, nullptr, 0.0, bufS.get());
          add_pairs(s_ss, bufG.get(), bufS.get(), q.n_pairs, Fp[s]);
          if (q.i1 > q.i0) form_y(XW.Wst[s].get(), b1wl.get(), MW, q, bufY.get());
        }
        if (!both) form_g(W, xhW.get(), q, bufG.get());
        if (do_ind) {
          if (!both) form_y(XV.SV[s].get(), b1vl.get(), MV, q, bufZ.get());
          k_term(q, bufY.get(), bufZ.get());
        }
        if (!fold) {
          sum_y(q, bufZ.get(), s_ss, 1.0, nullptr, 0.0, bufS.get());
          add_pairs(1.0, bufG.get(), bufS.get(), q.n_pairs, Fp[s]);
        } else if (ns == 1) {
          // one product for t~ dX and the same-spin term: G_W^T (s_ss S^-1 Y_V - cD S^-1 G_V)
          if (do_ind) sum_y(q, bufZ.get(), s_ss, 1.0, bufS.get(), -cD[0], bufS.get());
          add_pairs(do_ind ? 1.0 : -cD[0], gw, bufS.get(), q.n_pairs, Fp[s]);
        } else {
          // D and the same-spin term G_W^T S^-1 Y_V in one launch, G_W read once
          if (do_ind) sum_y(q, bufZ.get(), 1.0, 1.0, nullptr, 0.0, bufS.get() + nbuf);
          DevBuf D(2 * N * N);
          GemmDesc gd = gemm_nn(LL(N), LL(N), LL(Rp), 1.0, gw, LL(Rp), bufS.get(), LL(Rp), 0.0,
                                D.get(), LL(N));
          gd.a_kcontig = true;
          gd.nbr1 = LL(q.n_pairs);
          gd.sAr1 = LL(pair);
          gd.sBr1 = LL(pair);
          gd.nbo1 = do_ind ? 2 : 1;
          gd.sBo1 = LL(nbuf);
          gd.sCo1 = LL(N * N);
          gemm(gd);
          if (do_ind)
            copy3d(D.get() + N * N, LL(N), 0, Fp[s], LL(N), 0, LL(N), LL(N), 1, s_ss, 1.0);
          for (int sp = 0; sp < ns; ++sp)
            if (cD[sp] != 0.0)
              copy3d(D.get(), LL(N), 0, Fp[sp], LL(N), 0, LL(N), LL(N), 1, -cD[sp], 1.0);
        }
      }
    }
  }

  // =====================================================================
  // energies and the symmetrised Fock matrix
  // =====================================================================
  clock.mark("finish");
  double e[kAccSlots];
  UW12_CUDA(cudaMemcpyAsync(e, acc.get(), sizeof(e), cudaMemcpyDeviceToHost, st));
  if (rq.fock && calc) {
    double* dst = rq.fock;
    DevBuf out;
    if (!rq.fock_device) {
      out.alloc(N * N * ns);
      dst = out.get();
    }
    for (int s = 0; s < ns; ++s) symmetrise(Fp[s], LL(N), LL(N), dst + N * N * s, LL(N));
    if (!rq.fock_device)
      UW12_CUDA(cudaMemcpyAsync(rq.fock, dst, N * N * ns * sizeof(double), cudaMemcpyDeviceToHost,
                                st));
    UW12_CUDA(cudaStreamSynchronize(st));
  } else {
    if (rq.fock) {
      if (rq.fock_device)
        UW12_CUDA(cudaMemsetAsync(rq.fock, 0, N * N * ns * sizeof(double), st));
      else
        std::fill(rq.fock, rq.fock + N * N * ns, 0.0);
    }
    UW12_CUDA(cudaStreamSynchronize(st));
  }
  clock.mark("end");
  clock.finish();
  const double e2 = e[kE2d] + (do_ind ? s_ss * e[kE2i] : 0.0);
  const double e3 = e[kE3d] + (do_ind ? s_ss * e[kE3i] : 0.0);
  const double e4 = e[kE4d] + (do_ind ? s_ss * e[kE4i] : 0.0);
  const double total = e2 + e3 + e4;
  if (rq.energy) *rq.energy = total;
  if (rq.terms) {
    rq.terms[0] = e2;
    rq.terms[1] = e3;
    rq.terms[2] = e4;
  }
  if (rq.print_level > 0) {
    // print.hpp:13-42 formatting
    auto line = [](char ch) { for (int i = 0; i < 48; ++i) std::putchar(ch); std::putchar('\n'); };
    auto res = [](const char* s, double v) {
      std::string str(s);
      std::printf(" %s:%*s%12.6f\n", s, int(32 - str.size()), "", v);
    };
    if (rq.print_level > 2) {
      std::printf("\n");
      line('=');
      std::printf(" UW12 Calculation\n");
      line('=');
    }
    if (rq.print_level > 1) {
      res("Two electron energy", e2);
      res("Three electron energy", e3);
      res("Four electron energy", e4);
    }
    if (rq.print_level > 2) line('=');
    res("Total UW12 energy", total);
    std::fflush(stdout);
  }
}

// --------------------------------------------------------------------------
// reverse mode (direct terms, and the same-spin terms with indirect_term)
// --------------------------------------------------------------------------
// Energy of the direct terms, with f = f(s, s') the spin factor
// (four_electron_utils.cpp:9-30) and everything in the metric eigenbasis:
//   E = sum_{s,s'} f [ 1/2 X_D[s] . (L_WV X_D[s'])        (two_electron.cpp:37-81)
//                    + 1/2 < t~[s'], t[s] >               (four_electron.cpp:80-137)
//                    - < X[s], t~[s'] > ]                 (direct_utils.cpp:136-157)
// t = B2_W^T B2_V, t~ = L_W t L_V, X = Wst_W^T (I (x) S^-1) Wst_V.  Reverse sweep:
//   tbar[s] = sum_s' f (1/2 t~[s'] + L_W (1/2 t[s'] - X[s']) L_V),
//   Xbar[s] = -sum_s' f t~[s'];
//   B2bar_W = B2_V tbar^T, B2bar_V = B2_W tbar; Wstbar_W = SV_V Xbar^T,
//   Wstbar_V = SW_W Xbar (SW = (I (x) S^-1) Wst);
//   B1bar = Ca B2bar (+ the AO rows of Wstbar), Bribar = the RI rows of Wstbar;
//   B1bar_0 = B1bar P2^T, Bribar_0 = Bribar P2^T;
//   dE/dJ3_0[:, A] = packed-symmetric sum of B1bar_0[:, A] Co^T (N x N per A),
//   dE/dJ3_ri_0[:, A] = Bribar_0[:, A] Ca^T (R x N per A);
//   dE/dJ3_0^WV = 1/2 n_spin lower(D, 2) (P2 Xbar_D)^T, Xbar_D[s] = sum_s' f L X_D[s'].
// In the original aux basis E depends on each metric only through K = J2^-1
// (e.g. <t~[s'], t[s]> = tr(T0[s']^T K_W T0[s] K_V)), so dE/dJ2 = -K (dE/dK) K,
// which in the eigenbasis (Q = P2 L) reads
//   dE/dJ2_W  = -sym(Q_W [sum_s 1/2 T_s L_V t[s]^T - X[s] L_V T_s^T] Q_W^T),
//   dE/dJ2_V  = -sym(Q_V [sum_s 1/2 t[s]^T L_W T_s - T_s^T L_W X[s]] Q_V^T),
//   dE/dJ2_WV = -1/2 sum_{s,s'} f (Q X_D[s]) (Q X_D[s'])^T,
// with T_s = sum_s' f t[s'].  With indirect_term the same-spin energies
// (s_ss times E2-, E3-, E4-) add their own B2-bar, Wst-bar and metric terms
// (comment at the same-spin section below).
void form_fock_adjoint(const FockRequest& rq_in, const AdjointOutputs& out) {
  FockRequest rq = rq_in;
  if (rq.n_shards > 1) throw Error(kErrInvalid, "the adjoint evaluates unsharded");
  form_fock(rq);
  PhaseClock clock;
  clock.mark("adj_recompute");

  const IntegralsHandle& W = *rq.W;
  const IntegralsHandle& V = *rq.V;
  const IntegralsHandle& WV = *rq.WV;
  const AbsHandle& AB = *rq.abs;
  const int ns = rq.n_spin;
  const size_t N = rq.n_ao, np = packed_size(N);
  const size_t MW = W.n_df, MV = V.n_df, MX = WV.n_df;
  const size_t R = W.n_ri, Rp = N + R;
  const double two = (ns == 1) ? 2.0 : 1.0;
  cudaStream_t st = current_stream();
  const bool streamed = out.sink3[0] || out.sink3[1] || out.sink3[2] || out.sink3_ri[0] ||
                        out.sink3_ri[1];
  Budget budgets(rq, budget_need(rq, true, streamed), !all_stored(rq) || streamed);
  size_t budget = budgets.doubles();
  double F[2][2] = {{0, 0}, {0, 0}};
  for (int s = 0; s < ns; ++s)
    for (int sp = 0; sp < ns; ++sp) F[s][sp] = spin_factor(ns, s, sp, rq.s_os, rq.s_ss);

  std::vector<SpinDims> sd;
  size_t o_tot = 0, a_tot = 0;
  DevBuf orbs;
  upload_orbitals(rq, sd, o_tot, a_tot, orbs);
  const double* const Co = orbs.get();
  const double* const Ca = Co + N * o_tot;
  auto Ca_s = [&](int s) { return Ca + N * sd[s].aoff; };

  // output targets: the caller's device buffers, or device staging for host outputs
  std::vector<std::pair<DevBuf, double*>> staged;
  auto target = [&](double* user, size_t n) -> double* {
    if (!user) return nullptr;
    if (out.device_mem) return user;
    staged.emplace_back(DevBuf(n), user);
    return staged.back().first.get();
  };
  double* gJ3[3] = {target(out.dJ3[0], np * MW), target(out.dJ3[1], np * MV),
                    target(out.dJ3[2], np * MX)};
  double* gJ3ri[2] = {target(out.dJ3_ri[0], R * N * MW), target(out.dJ3_ri[1], R * N * MV)};
  double* gJ2[3] = {target(out.dJ2[0], MW * MW), target(out.dJ2[1], MV * MV),
                    target(out.dJ2[2], MX * MX)};

  // Without same-spin terms every recomputed intermediate enters the gradients
  // through sums over orbitals: X_AB and t over active / occupied orbitals,
  // B2-bar of occupied orbital k from the other potential's B2 of k alone, and
  // Wst-bar of active orbital j from the other potential's S^-1 Wst of j alone.
  // When the whole intermediates (B2, Wst and S^-1 Wst of W and V per spin,
  // and the transforms they come from) would not fit -- an explicit budget,
  // or 90 % of the free device memory -- they are formed for a chunk of
  // orbitals at a time instead (orbital_chunked), and only the gradient
  // factors B1-bar (N o x M) and, when the RI gradient is wanted, Bri-bar
  // (R a x M) are held whole.
  const bool same_spin = rq.indirect && rq.s_ss != 0.0;
  const size_t Mmax = std::max(MW, MV);
  size_t whole = (N * o_tot + R * a_tot) * Mmax;
  for (int s = 0; s < ns; ++s)
    whole += 2 * (sd[s].a * sd[s].o + 2 * Rp * sd[s].a) * Mmax;
  const bool orbital_chunked = !same_spin && whole > budgets.doubles(0.9);
  // B1 (N*nk x M) of occupied orbitals [k0, k0 + nk) of spin s for potential X:
  // sq(J3_0[:, A]) Co[:, k] P2
  auto b1_chunk = [&](const IntegralsHandle& X, int s, size_t k0, size_t nk, DevBuf& dst) {
    const size_t M = X.n_df;
    DevBuf H(N * nk * M);
    transform_ao(X, Co + N * (sd[s].ooff + k0), nk, H.get(), budget / 2);
    dst.alloc(N * nk * M);
    gemm(gemm_nn(LL(N * nk), LL(M), LL(M), 1.0, H.get(), LL(N * nk), X.P2.get(), LL(M), 0.0,
                 dst.get(), LL(N * nk)));
  };
  // Wst (R' nj x M) of active orbitals [j0, j0 + nj) of spin s for potential
  // X: per orbital the AO rows sq(J3_0) Co[:, c + j] P2, then the RI rows
  // J3ri_0 Ca[:, j] P2
  auto wst_chunk = [&](const IntegralsHandle& X, int s, size_t j0, size_t nj, double* St) {
    const size_t M = X.n_df;
    {
      DevBuf H(N * nj * M);
      transform_ao(X, Co + N * (sd[s].ooff + sd[s].c + j0), nj, H.get(), budget / 2);
      GemmDesc ga = gemm_nn(LL(N), LL(M), LL(M), 1.0, H.get(), LL(N * nj), X.P2.get(), LL(M),
                            0.0, St, LL(Rp * nj));
      ga.nbo1 = LL(nj);
      ga.sAo1 = LL(N);
      ga.sCo1 = LL(Rp);
      gemm(ga);
    }
    DevBuf H2(R * nj * M);
    ri_transform(X, Ca_s(s) + N * j0, nj, H2.get(), budget);
    GemmDesc gr = gemm_nn(LL(R), LL(M), LL(M), 1.0, H2.get(), LL(R * nj), X.P2.get(), LL(M), 0.0,
                          St + N, LL(Rp * nj));
    gr.nbo1 = LL(nj);
    gr.sAo1 = LL(R);
    gr.sCo1 = LL(Rp);
    gemm(gr);
  };
  // occupied orbitals per chunk (B1 and its transform, B2 of the chunk and its
  // adjoint) and active orbitals per chunk (the transforms, Wst of the chunk,
  // S^-1 Wst and Wst-bar), as in form_fock's chunked X_AB and t passes
  auto per_k = [&](int s) { return (4 * N + 2 * sd[s].a) * Mmax; };
  const size_t per_j = (N + R + 3 * Rp) * Mmax;

  // ---- forward intermediates (as in form_fock): B2, Wst, (I (x) S^-1) Wst per X, spin
  struct PerX {
    std::vector<DevBuf> B2, Wst, SW;
  };
  PerX XW, XV;
  for (int which = 0; which < 2 && !orbital_chunked; ++which) {
    const IntegralsHandle& X = which == 0 ? W : V;
    PerX& P = which == 0 ? XW : XV;
    const size_t M = X.n_df;
    P.B2.resize(ns);
    P.Wst.resize(ns);
    P.SW.resize(ns);
    budget = budgets.doubles();
    DevBuf H(N * o_tot * M);
    transform_ao(X, Co, o_tot, H.get(), budget / 2);
    DevBuf H2(R * a_tot * M);
    if (a_tot) ri_transform(X, Ca, a_tot, H2.get(), budget);
    for (int s = 0; s < ns; ++s) {
      const size_t o = sd[s].o, a = sd[s].a, c = sd[s].c;
      if (!a) continue;
      DevBuf B1(N * o * M);
      gemm(gemm_nn(LL(N * o), LL(M), LL(M), 1.0, H.get() + N * sd[s].ooff, LL(N * o_tot),
                   X.P2.get(), LL(M), 0.0, B1.get(), LL(N * o)));
      P.B2[s].alloc(a * o * M);
      GemmDesc g3 = gemm_nn(LL(a), LL(o * M), LL(N), 1.0, Ca_s(s), LL(N), B1.get(), LL(N), 0.0,
                            P.B2[s].get(), LL(a));
      g3.a_kcontig = true;
      gemm(g3);
      P.Wst[s].alloc(Rp * a * M);
      copy3d(B1.get() + N * c, LL(N), LL(N * o), P.Wst[s].get(), LL(Rp), LL(Rp * a), LL(N),
             LL(a), LL(M));
      GemmDesc g2 = gemm_nn(LL(R), LL(M), LL(M), 1.0, H2.get() + R * sd[s].aoff, LL(R * a_tot),
                            X.P2.get(), LL(M), 0.0, P.Wst[s].get() + N, LL(Rp * a));
      g2.nbo1 = LL(a);
      g2.sAo1 = LL(R);
      g2.sCo1 = LL(Rp);
      gemm(g2);
      P.SW[s].alloc(Rp * a * M);
      gemm(gemm_nn(LL(Rp), LL(a * M), LL(Rp), 1.0, AB.Sinv.get(), LL(Rp), P.Wst[s].get(),
                   LL(Rp), 0.0, P.SW[s].get(), LL(Rp)));
    }
  }
  // X, t, t~ per spin (zero for a spin without active orbitals)
  std::vector<DevBuf> Xab(ns), tab(ns), ttl(ns);
  for (int s = 0; s < ns; ++s) {
    const size_t o = sd[s].o, a = sd[s].a;
    Xab[s].alloc(MW * MV);
    tab[s].alloc(MW * MV);
    ttl[s].alloc(MW * MV);
    if (a == 0) {
      Xab[s].zero();
      tab[s].zero();
      ttl[s].zero();
      continue;
    }
    if (orbital_chunked) {
      // X_AB = sum over active-orbital chunks of Wst_W[j]^T S^-1 Wst_V[j];
      // t = sum over occupied-orbital chunks of B2_W[k]^T B2_V[k]
      Xab[s].zero();
      tab[s].zero();
      const size_t jc = std::max<size_t>(1, std::min(a, budget / 2 / per_j));
      for (size_t j0 = 0; j0 < a; j0 += jc) {
        const size_t nj = std::min(jc, a - j0);
        DevBuf Sw(Rp * nj * MW), SVj(Rp * nj * MV);
        {
          DevBuf Sv(Rp * nj * MV);
          wst_chunk(V, s, j0, nj, Sv.get());
          gemm(gemm_nn(LL(Rp), LL(nj * MV), LL(Rp), 1.0, AB.Sinv.get(), LL(Rp), Sv.get(),
                       LL(Rp), 0.0, SVj.get(), LL(Rp)));
        }
        wst_chunk(W, s, j0, nj, Sw.get());
        GemmDesc gx = gemm_nn(LL(MW), LL(MV), LL(Rp * nj), 1.0, Sw.get(), LL(Rp * nj), SVj.get(),
                              LL(Rp * nj), 1.0, Xab[s].get(), LL(MW));
        gx.a_kcontig = true;
        gemm(gx);
      }
      const size_t kc = std::max<size_t>(1, std::min(o, budget / 2 / per_k(s)));
      for (size_t k0 = 0; k0 < o; k0 += kc) {
        const size_t nk = std::min(kc, o - k0);
        DevBuf B2w(a * nk * MW), B2v(a * nk * MV);
        for (int which = 0; which < 2; ++which) {
          const IntegralsHandle& X = which == 0 ? W : V;
          DevBuf B1;
          b1_chunk(X, s, k0, nk, B1);
          GemmDesc g3 = gemm_nn(LL(a), LL(nk * X.n_df), LL(N), 1.0, Ca_s(s), LL(N), B1.get(),
                                LL(N), 0.0, (which == 0 ? B2w : B2v).get(), LL(a));
          g3.a_kcontig = true;
          gemm(g3);
        }
        GemmDesc gt = gemm_nn(LL(MW), LL(MV), LL(a * nk), 1.0, B2w.get(), LL(a * nk), B2v.get(),
                              LL(a * nk), 1.0, tab[s].get(), LL(MW));
        gt.a_kcontig = true;
        gemm(gt);
      }
      scale_rc(tab[s].get(), LL(MW), LL(MW), LL(MV), W.lam.get(), V.lam.get(), 1.0,
               ttl[s].get(), LL(MW));
      continue;
    }
    GemmDesc gx = gemm_nn(LL(MW), LL(MV), LL(Rp * a), 1.0, XW.Wst[s].get(), LL(Rp * a),
                          XV.SW[s].get(), LL(Rp * a), 0.0, Xab[s].get(), LL(MW));
    gx.a_kcontig = true;
    gemm(gx);
    GemmDesc gt = gemm_nn(LL(MW), LL(MV), LL(a * o), 1.0, XW.B2[s].get(), LL(a * o),
                          XV.B2[s].get(), LL(a * o), 0.0, tab[s].get(), LL(MW));
    gt.a_kcontig = true;
    gemm(gt);
    scale_rc(tab[s].get(), LL(MW), LL(MW), LL(MV), W.lam.get(), V.lam.get(), 1.0, ttl[s].get(),
             LL(MW));
  }

  clock.mark("adj_t_x");
  // ---- adjoints of t and X
  std::vector<DevBuf> tbar(ns), Xbar(ns);
  for (int s = 0; s < ns; ++s) {
    const double* mats[6];
    double coefs[6];
    int scaled[6];
    int nt = 0;
    for (int sp = 0; sp < ns; ++sp) {
      mats[nt] = ttl[sp].get(); coefs[nt] = 0.5 * F[s][sp]; scaled[nt++] = 0;
      mats[nt] = tab[sp].get(); coefs[nt] = 0.5 * F[sp][s]; scaled[nt++] = 1;
      mats[nt] = Xab[sp].get(); coefs[nt] = -F[sp][s]; scaled[nt++] = 1;
    }
    tbar[s].alloc(MW * MV);
    lincomb(tbar[s].get(), LL(MW), LL(MV), nt, mats, coefs, scaled, W.lam.get(), V.lam.get());
    nt = 0;
    for (int sp = 0; sp < ns; ++sp) {
      mats[nt] = ttl[sp].get(); coefs[nt] = -F[s][sp]; scaled[nt++] = 0;
    }
    Xbar[s].alloc(MW * MV);
    lincomb(Xbar[s].get(), LL(MW), LL(MV), nt, mats, coefs, scaled, nullptr, nullptr);
  }

  // ---- same-spin terms (indirect_term with s_ss != 0), energy s_ss E_ss:
  //   E3- = esf <YW, P3(ZV)>, YW = Wst_W L_W B2_W^T, ZV = SW_V L_V B2_V^T
  //   E4- = -1/2 esf <W4, P4(V4)>, W4 = B2_W L_W B2_W^T, V4 = B2_V L_V B2_V^T
  //   E2- = -1/2 esf <B2_WV L_WV, B2_WV> (WV over the active orbitals, below)
  // (esf = 2 closed shell, 1 open; P3, P4 the index exchanges of perm_3el,
  // perm_4el). Their B2-bar and Wst-bar join the direct ones before the
  // transforms are reversed; each L between eigenbasis factors adds
  // (left factor)^T G (right factor) to the metric's A matrix:
  //   G_Y = s esf P3(ZV), G_Z = s esf P3(YW) (chunks of occupied k),
  //   Wst_W-bar = (sum_k G_Y B2_W,k) L_W, B2_W,k-bar = (G_Y^T Wst_W) L_W,
  //   SW_V-bar = (sum_k G_Z B2_V,k) L_V -> Wst_V-bar = (I (x) S^-1) SW_V-bar,
  //   B2_V,k-bar = (G_Z^T SW_V) L_V;  A_W += Wst_W^T T_Y, A_V += SW_V^T T_Z;
  //   G_W4 = -1/2 s esf P4(V4): B2_W-bar += 2 (G_W4 B2_W) L_W,
  //   A_W += B2_W^T G_W4 B2_W (and W <-> V with P4(W4)).
  clock.mark("adj_same_spin");
  std::vector<DevBuf> ssB2b[2], ssWsb[2];
  DevBuf ssA[2];
  if (same_spin) {
    const double gs = two * rq.s_ss;
    ssA[0].alloc(MW * MW);
    ssA[0].zero();
    ssA[1].alloc(MV * MV);
    ssA[1].zero();
    for (int which = 0; which < 2; ++which) {
      ssB2b[which].resize(ns);
      ssWsb[which].resize(ns);
    }
    for (int s = 0; s < ns; ++s) {
      const size_t o = sd[s].o, a = sd[s].a;
      if (a == 0 || o == 0) continue;
      const size_t ao = a * o, Ra = Rp * a;
      ssB2b[0][s].alloc(ao * MW);
      ssB2b[1][s].alloc(ao * MV);
      DevBuf b2wl(ao * MW), b2vl(ao * MV);
      scale_rc(XW.B2[s].get(), LL(ao), LL(ao), LL(MW), nullptr, W.lam.get(), 1.0, b2wl.get(),
               LL(ao));
      scale_rc(XV.B2[s].get(), LL(ao), LL(ao), LL(MV), nullptr, V.lam.get(), 1.0, b2vl.get(),
               LL(ao));
      // three-electron, chunks of occupied orbitals k
      {
        budget = budgets.doubles();
        const size_t per_k = 3 * Ra * a + 2 * a * std::max(MW, MV);
        const size_t kc = tile_chunk(o, a, std::max<size_t>(1, std::min(o, budget / per_k)));
        const size_t c = o - a;
        // pairs of the largest chunk: fewer than a per orbital, and for whole sets half
        size_t most = 0;
        for (size_t k0 = 0; k0 < o; k0 += kc)
          most = std::max(most, static_cast<size_t>(PairColumns::of(LL(a), LL(c), LL(k0),
                                                                    LL(std::min(kc, o - k0)))
                                                        .count()));
        DevBuf TY(Ra * MW), TZ(Ra * MV), Tmp(Ra * most), GY(Ra * most), GZ(Ra * most),
            Bt(most * std::max(MW, MV)), b2p(most * std::max(MW, MV));
        // B2 is symmetric in the active pair, and so are the gradients that matter: a pair
        // of a chunk is formed once, G_Y and G_Z sum its two orders, and B2-bar of both
        // is half of the product (one B200, with the energy's: open shell N=200, M=600,
        // R=800, o=16/15 44.1 -> 42.7 ms, N=300, M=900, R=1200, o=30 in split precision
        // 103.0 -> 99.7)
        for (size_t k0 = 0; k0 < o; k0 += kc) {
          const double beta = k0 ? 1.0 : 0.0;
          const PairColumns q = PairColumns::of(LL(a), LL(c), LL(k0), LL(std::min(kc, o - k0)));
          const long long n = q.count();
          for (const bool is_w : {false, true}) {  // ZV and G_Y, then YW and G_Z
            const IntegralsHandle& X = is_w ? W : V;
            const double* St = is_w ? XW.Wst[s].get() : XV.SW[s].get();
            pack_pairs((is_w ? XW : XV).B2[s].get(), q, LL(o), LL(X.n_df), X.lam.get(), 0.5,
                       b2p.get());
            GemmDesc g = gemm_nn(LL(Ra), n, LL(X.n_df), 1.0, St, LL(Ra), b2p.get(), n, 0.0,
                                 Tmp.get(), LL(Ra));
            g.b_ncontig = true;
            gemm(g);
            perm_3el(Tmp.get(), (is_w ? GZ : GY).get(), LL(Rp), q, gs);
          }
          for (const bool is_w : {true, false}) {
            const IntegralsHandle& X = is_w ? W : V;
            const double* St = is_w ? XW.Wst[s].get() : XV.SW[s].get();
            const double* G = (is_w ? GY : GZ).get();
            pack_pairs((is_w ? XW : XV).B2[s].get(), q, LL(o), LL(X.n_df), nullptr, 0.5, b2p.get());
            gemm(gemm_nn(LL(Ra), LL(X.n_df), n, 1.0, G, LL(Ra), b2p.get(), n, beta,
                         (is_w ? TY : TZ).get(), LL(Ra)));
            GemmDesc g = gemm_nn(n, LL(X.n_df), LL(Ra), 1.0, G, LL(Ra), St, LL(Ra), 0.0, Bt.get(),
                                 n);
            g.a_kcontig = true;
            gemm(g);
            unpack_pairs(Bt.get(), q, LL(o), LL(X.n_df), X.lam.get(), 0.5,
                         ssB2b[is_w ? 0 : 1][s].get());
          }
        }
        Tmp = DevBuf();  // the chunk buffers are done: their memory goes to Wst-bar
        GY = DevBuf();
        GZ = DevBuf();
        Bt = DevBuf();
        GemmDesc g = gemm_nn(LL(MW), LL(MW), LL(Ra), 1.0, XW.Wst[s].get(), LL(Ra), TY.get(),
                             LL(Ra), 1.0, ssA[0].get(), LL(MW));
        g.a_kcontig = true;
        gemm(g);
        g = gemm_nn(LL(MV), LL(MV), LL(Ra), 1.0, XV.SW[s].get(), LL(Ra), TZ.get(), LL(Ra), 1.0,
                    ssA[1].get(), LL(MV));
        g.a_kcontig = true;
        gemm(g);
        // Wst_W-bar = T_Y L_W in place; Wst_V-bar = (I (x) S^-1) (T_Z L_V)
        scale_rc(TY.get(), LL(Ra), LL(Ra), LL(MW), nullptr, W.lam.get(), 1.0, TY.get(), LL(Ra));
        ssWsb[0][s] = std::move(TY);
        scale_rc(TZ.get(), LL(Ra), LL(Ra), LL(MV), nullptr, V.lam.get(), 1.0, TZ.get(), LL(Ra));
        ssWsb[1][s].alloc(Ra * MV);
        gemm(gemm_nn(LL(Rp), LL(a * MV), LL(Rp), 1.0, AB.Sinv.get(), LL(Rp), TZ.get(), LL(Rp),
                     0.0, ssWsb[1][s].get(), LL(Rp)));
        TZ = DevBuf();
      }
      // four-electron
      {
        DevBuf W4(ao * ao), V4(ao * ao), G4(ao * ao), T4(ao * std::max(MW, MV));
        GemmDesc g = gemm_nn(LL(ao), LL(ao), LL(MW), 1.0, b2wl.get(), LL(ao), XW.B2[s].get(),
                             LL(ao), 0.0, W4.get(), LL(ao));
        g.b_ncontig = true;
        gemm(g);
        g = gemm_nn(LL(ao), LL(ao), LL(MV), 1.0, b2vl.get(), LL(ao), XV.B2[s].get(), LL(ao), 0.0,
                    V4.get(), LL(ao));
        g.b_ncontig = true;
        gemm(g);
        for (int which = 0; which < 2; ++which) {
          const size_t M = which == 0 ? MW : MV;
          const DevBuf& B2 = which == 0 ? XW.B2[s] : XV.B2[s];
          const double* lam = which == 0 ? W.lam.get() : V.lam.get();
          perm_4el(which == 0 ? V4.get() : W4.get(), G4.get(), LL(a), LL(o), -0.5 * gs);
          gemm(gemm_nn(LL(ao), LL(M), LL(ao), 1.0, G4.get(), LL(ao), B2.get(), LL(ao), 0.0,
                       T4.get(), LL(ao)));
          GemmDesc ga = gemm_nn(LL(M), LL(M), LL(ao), 1.0, B2.get(), LL(ao), T4.get(), LL(ao),
                                1.0, ssA[which].get(), LL(M));
          ga.a_kcontig = true;
          gemm(ga);
          const double* mats[2] = {ssB2b[which][s].get(), T4.get()};
          const double coefs[2] = {1.0, 2.0};
          const int scaled[2] = {0, 1};
          lincomb(ssB2b[which][s].get(), LL(ao), LL(M), 2, mats, coefs, scaled, nullptr, lam);
        }
      }
    }
  }

  clock.mark("adj_three_index");
  // ---- dE/dJ3_0 and dE/dJ3_ri_0 of W and V, orbital-chunked: B2-bar of
  // occupied orbitals k (B2-bar_W = B2_V t-bar^T, B2-bar_V = B2_W t-bar) and
  // Wst-bar of active orbitals j (Wst-bar_W = S^-1 Wst_V X-bar^T,
  // Wst-bar_V = S^-1 Wst_W X-bar) from the other potential's intermediates of
  // those orbitals, formed afresh per chunk, into the whole B1-bar (and
  // Bri-bar); then B1-bar P2^T per block of aux functions
  for (int which = 0; which < 2 && orbital_chunked; ++which) {
    const IntegralsHandle& X = which == 0 ? W : V;
    const IntegralsHandle& Y = which == 0 ? V : W;  // the other potential
    const size_t M = X.n_df, MY = Y.n_df;
    double* g3 = gJ3[which];
    double* g3ri = gJ3ri[which];
    const GradSink& s3 = out.sink3[which];
    const GradSink& s3ri = out.sink3_ri[which];
    const bool want3 = g3 || s3, want_ri = g3ri || s3ri;
    if (!want3 && !want_ri) continue;
    DevBuf Bb1(N * o_tot * M), Bbri;
    Bb1.zero();  // the columns of spins without active orbitals stay zero
    if (want_ri && a_tot) Bbri.alloc(R * a_tot * M);
    budget = budgets.doubles();
    for (int s = 0; s < ns; ++s) {
      const size_t o = sd[s].o, a = sd[s].a, c = sd[s].c;
      if (!a) continue;
      // B1-bar[:, k] = Ca B2-bar[:, k] over chunks of occupied k (written)
      const size_t kc = std::max<size_t>(1, std::min(o, budget / 2 / per_k(s)));
      for (size_t k0 = 0; k0 < o; k0 += kc) {
        const size_t nk = std::min(kc, o - k0);
        DevBuf B2y(a * nk * MY), B2b(a * nk * M);
        {
          DevBuf B1y;
          b1_chunk(Y, s, k0, nk, B1y);
          GemmDesc g3y = gemm_nn(LL(a), LL(nk * MY), LL(N), 1.0, Ca_s(s), LL(N), B1y.get(),
                                 LL(N), 0.0, B2y.get(), LL(a));
          g3y.a_kcontig = true;
          gemm(g3y);
        }
        GemmDesc gb = gemm_nn(LL(a * nk), LL(M), LL(MY), 1.0, B2y.get(), LL(a * nk),
                              tbar[s].get(), LL(MW), 0.0, B2b.get(), LL(a * nk));
        gb.b_ncontig = which == 0;  // t-bar is MW x MV
        gemm(gb);
        GemmDesc g1 = gemm_nn(LL(N), LL(nk), LL(a), 1.0, Ca_s(s), LL(N), B2b.get(), LL(a), 0.0,
                              Bb1.get() + N * (sd[s].ooff + k0), LL(N));
        g1.nbo1 = LL(M);
        g1.sBo1 = LL(a * nk);
        g1.sCo1 = LL(N * o_tot);
        gemm(g1);
      }
      // Wst-bar of active orbitals j: AO rows added to B1-bar[:, c + j], RI
      // rows into Bri-bar[:, j]
      const size_t jc = std::max<size_t>(1, std::min(a, budget / 2 / per_j));
      for (size_t j0 = 0; j0 < a; j0 += jc) {
        const size_t nj = std::min(jc, a - j0);
        DevBuf SYj(Rp * nj * MY);
        {
          DevBuf Sy(Rp * nj * MY);
          wst_chunk(Y, s, j0, nj, Sy.get());
          gemm(gemm_nn(LL(Rp), LL(nj * MY), LL(Rp), 1.0, AB.Sinv.get(), LL(Rp), Sy.get(),
                       LL(Rp), 0.0, SYj.get(), LL(Rp)));
        }
        DevBuf Wsb(Rp * nj * M);
        GemmDesc gw = gemm_nn(LL(Rp * nj), LL(M), LL(MY), 1.0, SYj.get(), LL(Rp * nj),
                              Xbar[s].get(), LL(MW), 0.0, Wsb.get(), LL(Rp * nj));
        gw.b_ncontig = which == 0;  // X-bar is MW x MV
        gemm(gw);
        copy3d(Wsb.get(), LL(Rp), LL(Rp * nj), Bb1.get() + N * (sd[s].ooff + c + j0), LL(N),
               LL(N * o_tot), LL(N), LL(nj), LL(M), 1.0, 1.0);
        if (Bbri.size())
          copy3d(Wsb.get() + N, LL(Rp), LL(Rp * nj), Bbri.get() + R * (sd[s].aoff + j0), LL(R),
                 LL(R * a_tot), LL(R), LL(nj), LL(M));
      }
    }
    if (want3) {
      // per block of aux functions: B1-bar_0 = B1-bar P2^T (the block's
      // columns), then per aux function the packed symmetric sum of B1-bar_0 Co^T
      const size_t ac = std::max<size_t>(1, std::min(M, budget / (2 * N * N + N * o_tot)));
      DevBuf Bb10(N * o_tot * ac), G(N * N * ac), Pk;
      if (!g3) Pk.alloc(np * ac);  // one streamed block
      for (size_t a0 = 0; a0 < M; a0 += ac) {
        const size_t na = std::min(ac, M - a0);
        GemmDesc gp = gemm_nn(LL(N * o_tot), LL(na), LL(M), 1.0, Bb1.get(), LL(N * o_tot),
                              X.P2.get() + a0, LL(M), 0.0, Bb10.get(), LL(N * o_tot));
        gp.b_ncontig = true;
        gemm(gp);
        GemmDesc g = gemm_nn(LL(N), LL(N), LL(o_tot), 1.0, Bb10.get(), LL(N), Co, LL(N), 0.0,
                             G.get(), LL(N));
        g.b_ncontig = true;
        g.nbo1 = LL(na);
        g.sAo1 = LL(N * o_tot);
        g.sCo1 = LL(N * N);
        gemm(g);
        pack_sym_sum(G.get(), LL(N), LL(na), g3 ? g3 + np * a0 : Pk.get(), LL(np));
        if (!g3) s3(a0, na, Pk.get(), np, st);
      }
    }
    if (want_ri) {
      // as in the whole form: one batched GEMM into the whole gradient, or
      // aux blocks of at most a quarter of the budget when streamed
      const size_t rows = R * N;
      const size_t step = g3ri ? M : std::max<size_t>(1, std::min(M, budget / (4 * rows)));
      DevBuf Rk;
      if (!g3ri) Rk.alloc(rows * step);
      if (a_tot == 0) {
        if (g3ri) {
          UW12_CUDA(cudaMemsetAsync(g3ri, 0, R * N * M * sizeof(double), st));
        } else {
          Rk.zero();
          for (size_t b0 = 0; b0 < M; b0 += step) s3ri(b0, std::min(step, M - b0), Rk.get(), rows, st);
        }
      } else {
        DevBuf Bbri0(R * a_tot * M);
        GemmDesc gp = gemm_nn(LL(R * a_tot), LL(M), LL(M), 1.0, Bbri.get(), LL(R * a_tot),
                              X.P2.get(), LL(M), 0.0, Bbri0.get(), LL(R * a_tot));
        gp.b_ncontig = true;
        gemm(gp);
        Bbri = DevBuf();
        for (size_t b0 = 0; b0 < M; b0 += step) {
          const size_t nb = std::min(step, M - b0);
          GemmDesc g = gemm_nn(LL(R), LL(N), LL(a_tot), 1.0, Bbri0.get() + R * a_tot * b0, LL(R),
                               Ca, LL(N), 0.0, g3ri ? g3ri + rows * b0 : Rk.get(), LL(R));
          g.b_ncontig = true;
          g.nbo1 = LL(nb);
          g.sAo1 = LL(R * a_tot);
          g.sCo1 = LL(R * N);
          gemm(g);
          if (!g3ri) s3ri(b0, nb, Rk.get(), rows, st);
        }
      }
    }
  }
  // ---- dE/dJ3_0 and dE/dJ3_ri_0 of W and V, whole intermediates
  for (int which = 0; which < 2 && !orbital_chunked; ++which) {
    const IntegralsHandle& X = which == 0 ? W : V;
    const size_t M = X.n_df;
    double* g3 = gJ3[which];
    double* g3ri = gJ3ri[which];
    const GradSink& s3 = out.sink3[which];
    const GradSink& s3ri = out.sink3_ri[which];
    if (!g3 && !g3ri && !s3 && !s3ri) continue;
    budget = budgets.doubles();
    DevBuf Bb1(N * o_tot * M), Bbri(R * a_tot * M);
    Bb1.zero();
    for (int s = 0; s < ns; ++s) {
      const size_t o = sd[s].o, a = sd[s].a, c = sd[s].c;
      if (!a) continue;
      // B2bar (a*o x M)
      DevBuf B2b(a * o * M);
      if (which == 0) {
        GemmDesc g = gemm_nn(LL(a * o), LL(MW), LL(MV), 1.0, XV.B2[s].get(), LL(a * o),
                             tbar[s].get(), LL(MW), 0.0, B2b.get(), LL(a * o));
        g.b_ncontig = true;
        gemm(g);
      } else {
        gemm(gemm_nn(LL(a * o), LL(MV), LL(MW), 1.0, XW.B2[s].get(), LL(a * o), tbar[s].get(),
                     LL(MW), 0.0, B2b.get(), LL(a * o)));
      }
      if (same_spin && ssB2b[which][s].size()) {
        const double* mats[2] = {B2b.get(), ssB2b[which][s].get()};
        const double coefs[2] = {1.0, 1.0};
        lincomb(B2b.get(), LL(a * o), LL(M), 2, mats, coefs, nullptr, nullptr, nullptr);
      }
      // B1bar_A (N x o) = Ca_s B2bar_A, into the spin block of Bb1
      GemmDesc g1 = gemm_nn(LL(N), LL(o), LL(a), 1.0, Ca_s(s), LL(N), B2b.get(), LL(a), 0.0,
                            Bb1.get() + N * sd[s].ooff, LL(N));
      g1.nbo1 = LL(M);
      g1.sBo1 = LL(a * o);
      g1.sCo1 = LL(N * o_tot);
      gemm(g1);
      // Wstbar (R'a x M)
      DevBuf Wsb(Rp * a * M);
      if (which == 0) {
        GemmDesc g = gemm_nn(LL(Rp * a), LL(MW), LL(MV), 1.0, XV.SW[s].get(), LL(Rp * a),
                             Xbar[s].get(), LL(MW), 0.0, Wsb.get(), LL(Rp * a));
        g.b_ncontig = true;
        gemm(g);
      } else {
        gemm(gemm_nn(LL(Rp * a), LL(MV), LL(MW), 1.0, XW.SW[s].get(), LL(Rp * a), Xbar[s].get(),
                     LL(MW), 0.0, Wsb.get(), LL(Rp * a)));
      }
      if (same_spin && ssWsb[which][s].size()) {
        const double* mats[2] = {Wsb.get(), ssWsb[which][s].get()};
        const double coefs[2] = {1.0, 1.0};
        lincomb(Wsb.get(), LL(Rp * a), LL(M), 2, mats, coefs, nullptr, nullptr, nullptr);
      }
      // AO rows -> active orbitals of B1bar; RI rows -> Bribar
      copy3d(Wsb.get(), LL(Rp), LL(Rp * a), Bb1.get() + N * (sd[s].ooff + c), LL(N),
             LL(N * o_tot), LL(N), LL(a), LL(M), 1.0, 1.0);
      copy3d(Wsb.get() + N, LL(Rp), LL(Rp * a), Bbri.get() + R * sd[s].aoff, LL(R),
             LL(R * a_tot), LL(R), LL(a), LL(M));
    }
    if (g3 || s3) {
      // B1bar_0 = B1bar P2^T, then per aux function the packed symmetric sum of B1bar_0 Co^T
      DevBuf Bb10(N * o_tot * M);
      GemmDesc gp = gemm_nn(LL(N * o_tot), LL(M), LL(M), 1.0, Bb1.get(), LL(N * o_tot),
                            X.P2.get(), LL(M), 0.0, Bb10.get(), LL(N * o_tot));
      gp.b_ncontig = true;
      gemm(gp);
      const size_t ac = std::max<size_t>(1, std::min(M, budget / (2 * N * N)));
      DevBuf G(N * N * ac), Pk;
      if (!g3) Pk.alloc(np * ac);  // one streamed block
      for (size_t a0 = 0; a0 < M; a0 += ac) {
        const size_t na = std::min(ac, M - a0);
        GemmDesc g = gemm_nn(LL(N), LL(N), LL(o_tot), 1.0, Bb10.get() + N * o_tot * a0, LL(N),
                             Co, LL(N), 0.0, G.get(), LL(N));
        g.b_ncontig = true;
        g.nbo1 = LL(na);
        g.sAo1 = LL(N * o_tot);
        g.sCo1 = LL(N * N);
        gemm(g);
        pack_sym_sum(G.get(), LL(N), LL(na), g3 ? g3 + np * a0 : Pk.get(), LL(np));
        if (!g3) s3(a0, na, Pk.get(), np, st);
      }
    }
    if (g3ri || s3ri) {
      // stored: one batched GEMM into the whole gradient; streamed: aux blocks
      // of at most a quarter of the budget
      const size_t rows = R * N;
      const size_t step = g3ri ? M : std::max<size_t>(1, std::min(M, budget / (4 * rows)));
      DevBuf Rk;
      if (!g3ri) Rk.alloc(rows * step);
      if (a_tot == 0) {
        if (g3ri) {
          UW12_CUDA(cudaMemsetAsync(g3ri, 0, R * N * M * sizeof(double), st));
        } else {
          Rk.zero();
          for (size_t b0 = 0; b0 < M; b0 += step) s3ri(b0, std::min(step, M - b0), Rk.get(), rows, st);
        }
      } else {
        DevBuf Bbri0(R * a_tot * M);
        GemmDesc gp = gemm_nn(LL(R * a_tot), LL(M), LL(M), 1.0, Bbri.get(), LL(R * a_tot),
                              X.P2.get(), LL(M), 0.0, Bbri0.get(), LL(R * a_tot));
        gp.b_ncontig = true;
        gemm(gp);
        for (size_t b0 = 0; b0 < M; b0 += step) {
          const size_t nb = std::min(step, M - b0);
          GemmDesc g = gemm_nn(LL(R), LL(N), LL(a_tot), 1.0, Bbri0.get() + R * a_tot * b0, LL(R),
                               Ca, LL(N), 0.0, g3ri ? g3ri + rows * b0 : Rk.get(), LL(R));
          g.b_ncontig = true;
          g.nbo1 = LL(nb);
          g.sAo1 = LL(R * a_tot);
          g.sCo1 = LL(R * N);
          gemm(g);
          if (!g3ri) s3ri(b0, nb, Rk.get(), rows, st);
        }
      }
    }
  }

  clock.mark("adj_metric");
  // ---- metric gradients of W and V: -sym(Q A Q^T), Q = P2 L
  for (int which = 0; which < 2; ++which) {
    double* g2 = gJ2[which];
    if (!g2) continue;
    const IntegralsHandle& X = which == 0 ? W : V;
    const IntegralsHandle& Y = which == 0 ? V : W;  // the other potential
    const size_t M = X.n_df;
    DevBuf Amat(M * M), Ts(M * M), tmp(M * M);
    Amat.zero();
    for (int s = 0; s < ns; ++s) {
      const double* mats[2];
      double coefs[2];
      for (int sp = 0; sp < ns; ++sp) {
        mats[sp] = tab[sp].get();
        coefs[sp] = F[s][sp];
      }
      lincomb(Ts.get(), LL(MW), LL(MV), ns, mats, coefs, nullptr, nullptr, nullptr);
      if (which == 0) {
        // A_W += 1/2 T_s L_V t[s]^T - X[s] L_V T_s^T
        scale_rc(Ts.get(), LL(MW), LL(MW), LL(MV), nullptr, Y.lam.get(), 1.0, tmp.get(), LL(MW));
        GemmDesc g = gemm_nn(LL(MW), LL(MW), LL(MV), 0.5, tmp.get(), LL(MW), tab[s].get(), LL(MW),
                             1.0, Amat.get(), LL(MW));
        g.b_ncontig = true;
        gemm(g);
        scale_rc(Xab[s].get(), LL(MW), LL(MW), LL(MV), nullptr, Y.lam.get(), 1.0, tmp.get(),
                 LL(MW));
        g = gemm_nn(LL(MW), LL(MW), LL(MV), -1.0, tmp.get(), LL(MW), Ts.get(), LL(MW), 1.0,
                    Amat.get(), LL(MW));
        g.b_ncontig = true;
        gemm(g);
      } else {
        // A_V += 1/2 t[s]^T L_W T_s - T_s^T L_W X[s]
        scale_rc(Ts.get(), LL(MW), LL(MW), LL(MV), Y.lam.get(), nullptr, 1.0, tmp.get(), LL(MW));
        GemmDesc g = gemm_nn(LL(MV), LL(MV), LL(MW), 0.5, tab[s].get(), LL(MW), tmp.get(), LL(MW),
                             1.0, Amat.get(), LL(MV));
        g.a_kcontig = true;
        gemm(g);
        scale_rc(Xab[s].get(), LL(MW), LL(MW), LL(MV), Y.lam.get(), nullptr, 1.0, tmp.get(),
                 LL(MW));
        g = gemm_nn(LL(MV), LL(MV), LL(MW), -1.0, Ts.get(), LL(MW), tmp.get(), LL(MW), 1.0,
                    Amat.get(), LL(MV));
        g.a_kcontig = true;
        gemm(g);
      }
    }
    if (same_spin) {
      const double* mats[2] = {Amat.get(), ssA[which].get()};
      const double coefs[2] = {1.0, 1.0};
      lincomb(Amat.get(), LL(M), LL(M), 2, mats, coefs, nullptr, nullptr, nullptr);
    }
    DevBuf Q(M * M), QA(M * M);
    scale_rc(X.P2.get(), LL(M), LL(M), LL(M), nullptr, X.lam.get(), 1.0, Q.get(), LL(M));
    gemm(gemm_nn(LL(M), LL(M), LL(M), 1.0, Q.get(), LL(M), Amat.get(), LL(M), 0.0, QA.get(),
                 LL(M)));
    GemmDesc g = gemm_nn(LL(M), LL(M), LL(M), -1.0, QA.get(), LL(M), Q.get(), LL(M), 0.0,
                         tmp.get(), LL(M));
    g.b_ncontig = true;
    gemm(g);
    symmetrise(tmp.get(), LL(M), LL(M), g2, LL(M));
  }

  // ---- WV: dE/dJ3_0 and dE/dJ2 through the fitted density, and through the
  // same-spin exchange E2- = -1/2 esf <B2 L, B2> (B2 = Ca^T B1, B1 of the
  // active orbitals, two_electron.cpp:87-132): B2-bar = -s esf B2 L,
  // B1-bar = Ca B2-bar, then P2^T and the packed symmetric sum per aux
  // function with Ca; A_WV = -1/2 s esf B2^T B2
  clock.mark("adj_wv");
  const GradSink& s3x = out.sink3[2];
  std::vector<DevBuf> ssX10(ns);  // B1-bar_0 of WV per spin (N a x MX)
  DevBuf ssAX;
  if (same_spin && (gJ3[2] || s3x || gJ2[2])) {
    const double gs = two * rq.s_ss;
    ssAX.alloc(MX * MX);
    ssAX.zero();
    budget = budgets.doubles();
    DevBuf H(N * a_tot * MX);
    transform_ao(WV, Ca, a_tot, H.get(), budget / 2);
    for (int s = 0; s < ns; ++s) {
      const size_t a = sd[s].a;
      if (!a) continue;
      DevBuf B1(N * a * MX), B2(a * a * MX), B2b(a * a * MX), B1b(N * a * MX);
      gemm(gemm_nn(LL(N * a), LL(MX), LL(MX), 1.0, H.get() + N * sd[s].aoff, LL(N * a_tot),
                   WV.P2.get(), LL(MX), 0.0, B1.get(), LL(N * a)));
      GemmDesc g2 = gemm_nn(LL(a), LL(a * MX), LL(N), 1.0, Ca_s(s), LL(N), B1.get(), LL(N), 0.0,
                            B2.get(), LL(a));
      g2.a_kcontig = true;
      gemm(g2);
      GemmDesc ga = gemm_nn(LL(MX), LL(MX), LL(a * a), -0.5 * gs, B2.get(), LL(a * a), B2.get(),
                            LL(a * a), 1.0, ssAX.get(), LL(MX));
      ga.a_kcontig = true;
      gemm(ga);
      scale_rc(B2.get(), LL(a * a), LL(a * a), LL(MX), nullptr, WV.lam.get(), -gs, B2b.get(),
               LL(a * a));
      GemmDesc g1 = gemm_nn(LL(N), LL(a), LL(a), 1.0, Ca_s(s), LL(N), B2b.get(), LL(a), 0.0,
                            B1b.get(), LL(N));
      g1.nbo1 = LL(MX);
      g1.sBo1 = LL(a * a);
      g1.sCo1 = LL(N * a);
      gemm(g1);
      ssX10[s].alloc(N * a * MX);
      GemmDesc gp = gemm_nn(LL(N * a), LL(MX), LL(MX), 1.0, B1b.get(), LL(N * a), WV.P2.get(),
                            LL(MX), 0.0, ssX10[s].get(), LL(N * a));
      gp.b_ncontig = true;
      gemm(gp);
    }
  }
  // adds the same-spin part of dE/dJ3_0^WV for aux functions [b0, b0 + nb)
  // to dst (packed rows, leading dimension np)
  auto add_ss_wv = [&](size_t b0, size_t nb, double* dst) {
    if (!same_spin) return;
    const size_t ac = std::max<size_t>(1, std::min(nb, budget / (4 * N * N)));
    DevBuf G(N * N * ac);
    for (int s = 0; s < ns; ++s) {
      const size_t a = sd[s].a;
      if (!a) continue;
      for (size_t c0 = 0; c0 < nb; c0 += ac) {
        const size_t nc = std::min(ac, nb - c0);
        GemmDesc g = gemm_nn(LL(N), LL(N), LL(a), 1.0, ssX10[s].get() + N * a * (b0 + c0), LL(N),
                             Ca_s(s), LL(N), 0.0, G.get(), LL(N));
        g.b_ncontig = true;
        g.nbo1 = LL(nc);
        g.sAo1 = LL(N * a);
        g.sCo1 = LL(N * N);
        gemm(g);
        pack_sym_sum(G.get(), LL(N), LL(nc), dst + np * c0, LL(np), 1.0);
      }
    }
  };
  if (gJ3[2] || s3x || gJ2[2]) {
    DevBuf dmat(np * ns), XDr(MX * ns), XD(MX * ns), XDb(MX * ns), vb(MX * ns);
    for (int s = 0; s < ns; ++s)
      pack_density(Ca_s(s), LL(N), LL(N), LL(sd[s].a), two, dmat.get() + np * s);
    fitted_density_raw(WV, dmat.get(), ns, XDr.get(), budget);
    GemmDesc g = gemm_nn(LL(MX), ns, LL(MX), 0.5 * ns, WV.P2.get(), LL(MX), XDr.get(), LL(MX),
                         0.0, XD.get(), LL(MX));
    g.a_kcontig = true;
    gemm(g);
    double coef[4] = {0, 0, 0, 0};
    for (int s = 0; s < ns; ++s)
      for (int sp = 0; sp < ns; ++sp) coef[s * ns + sp] = F[s][sp];
    if (gJ3[2] || s3x) {
      // Xbar_D[s] = L sum_s' f X_D[s'];  dJ3 = 1/2 n_spin dmat (P2 Xbar_D)^T
      combine_vecs(XD.get(), LL(MX), ns, coef, WV.lam.get(), XDb.get());
      gemm(gemm_nn(LL(MX), ns, LL(MX), 1.0, WV.P2.get(), LL(MX), XDb.get(), LL(MX), 0.0, vb.get(),
                   LL(MX)));
      // whole, or in aux blocks of at most a quarter of the budget when streamed
      const size_t step = gJ3[2] ? MX : std::max<size_t>(1, std::min(MX, budget / (4 * np)));
      DevBuf Xk;
      if (!gJ3[2]) Xk.alloc(np * step);
      for (size_t b0 = 0; b0 < MX; b0 += step) {
        const size_t nb = std::min(step, MX - b0);
        double* dst = gJ3[2] ? gJ3[2] + np * b0 : Xk.get();
        GemmDesc gd = gemm_nn(LL(np), LL(nb), ns, 0.5 * ns, dmat.get(), LL(np), vb.get() + b0,
                              LL(MX), 0.0, dst, LL(np));
        gd.b_ncontig = true;
        gemm(gd);
        add_ss_wv(b0, nb, dst);
        if (!gJ3[2]) s3x(b0, nb, Xk.get(), np, st);
      }
    }
    if (gJ2[2]) {
      // U = Q X_D = P2 (L X_D); dJ2 = -1/2 U (U F)^T
      DevBuf LX(MX * ns), U(MX * ns), UF(MX * ns);
      scale_rc(XD.get(), LL(MX), LL(MX), ns, WV.lam.get(), nullptr, 1.0, LX.get(), LL(MX));
      gemm(gemm_nn(LL(MX), ns, LL(MX), 1.0, WV.P2.get(), LL(MX), LX.get(), LL(MX), 0.0, U.get(),
                   LL(MX)));
      for (int s = 0; s < ns; ++s) {
        const double* mats[2] = {U.get(), U.get() + MX};
        double coefs[2] = {F[s][0], ns > 1 ? F[s][1] : 0.0};
        lincomb(UF.get() + MX * s, LL(MX), 1, ns, mats, coefs, nullptr, nullptr, nullptr);
      }
      GemmDesc gd = gemm_nn(LL(MX), LL(MX), ns, -0.5, U.get(), LL(MX), UF.get(), LL(MX), 0.0,
                            gJ2[2], LL(MX));
      gd.b_ncontig = true;
      gemm(gd);
      if (same_spin) {
        // += -Q A_WV Q^T (A_WV symmetric), Q = P2 L
        DevBuf Q(MX * MX), QA(MX * MX);
        scale_rc(WV.P2.get(), LL(MX), LL(MX), LL(MX), nullptr, WV.lam.get(), 1.0, Q.get(),
                 LL(MX));
        gemm(gemm_nn(LL(MX), LL(MX), LL(MX), 1.0, Q.get(), LL(MX), ssAX.get(), LL(MX), 0.0,
                     QA.get(), LL(MX)));
        GemmDesc gq = gemm_nn(LL(MX), LL(MX), LL(MX), -1.0, QA.get(), LL(MX), Q.get(), LL(MX),
                              1.0, gJ2[2], LL(MX));
        gq.b_ncontig = true;
        gemm(gq);
      }
    }
  }

  clock.mark("adj_copy_out");
  for (auto& sg : staged)
    UW12_CUDA(cudaMemcpyAsync(sg.second, sg.first.get(), sg.first.size() * sizeof(double),
                              cudaMemcpyDeviceToHost, st));
  clock.mark("adj_end");
  UW12_CUDA(cudaStreamSynchronize(st));
  clock.finish();
}

std::string phase_profile_read() {
  std::lock_guard<std::mutex> lk(g_phase_mu);
  std::string out;
  for (const auto& kv : g_phase_ms) out += kv.first + "=" + std::to_string(kv.second) + ";";
  g_phase_ms.clear();
  return out;
}

}  // namespace uw12b

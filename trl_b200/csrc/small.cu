// Small bs x bs block operations and the projected eigenproblem of the restart.
//
// The projected matrix T (N = nblk*bs <= a few thousand) stays on the device: it is
// assembled dense from its lower triangle (the reference's Eigen solver reads the lower
// triangle only, evp_base.hh:95), diagonalised by cuSOLVER's symmetric divide-and-conquer
// (syevd), re-ordered by decreasing |theta| (evp_base.hh:101-103) into the block layout,
// and the Ritz estimates ||beta * y_last|| / max(|theta|, eps) (evp_base.hh:124-151) are
// counted on the device. Only the eigenvalues and the converged count come back to the host.
#include "common.cuh"
#include "orthonormal_limit.h"
#include "tridiag_schedule.h"

#include <cooperative_groups.h>
#include <cusolverDn.h>

#include <cfloat>
#include <cstring>
#include <mutex>

namespace {

struct DiagValues {
  double v[16];
};

__global__ void k_mb_copy(double* __restrict__ dst, const double* __restrict__ src, int bs, int transpose)
{
  ::trl_detail::pdl_enter();
  const int e = threadIdx.x;
  if (e >= bs * bs) return;
  const int i = e / bs, j = e % bs;
  dst[e] = transpose ? src[j * bs + i] : src[e];
}

__global__ void k_mb_mult(const double* __restrict__ A, const double* __restrict__ B, double* __restrict__ C, int bs)
{
  ::trl_detail::pdl_enter();
  const int e = threadIdx.x;
  if (e >= bs * bs) return;
  const int i = e / bs, j = e % bs;
  double s = 0.0;
  for (int k = 0; k < bs; ++k) s = fma(A[i * bs + k], B[k * bs + j], s);
  C[e] = s;
}

__global__ void k_mb_set_diag(double* __restrict__ dst, DiagValues d, int bs)
{
  ::trl_detail::pdl_enter();
  const int i = threadIdx.x;
  if (i < bs) dst[i * bs + i] = d.v[i];
}

// max |T_ij| over the block matrix into *out, which holds zero before: non-negative doubles order
// like their bit patterns. Spread over the SMs (one CTA took 27 us for 384 x 384 entries).
__global__ void __launch_bounds__(256) k_max_abs(const double* __restrict__ T, int64_t count, unsigned long long* __restrict__ out)
{
  ::trl_detail::pdl_enter();
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  double m = 0.0;
#pragma unroll 4
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < count; e += stride) m = fmax(m, fabs(T[e]));
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0 && m > 0.0) atomicMax(out, static_cast<unsigned long long>(__double_as_longlong(m)));
}

// Entries below kFlushRel * max|T| are set to zero when the dense copy is assembled: they
// change no eigenvalue by more than N * 1e-30 * ||T||, far below rounding, while leaving
// them in lets their squares underflow inside the Householder reduction (a converged Ritz
// pair's coupling in a thick-restart matrix can be ~1e-160 next to entries of order 10);
// a reflector built from an underflowed norm is not orthogonal, and the computed spectrum is
// then wrong (cuSOLVER's syevd on the GPU fails the same way on such matrices).
constexpr double kFlushRel = 1e-30;

// 2^-e with 2^(e-1) <= tmax < 2^e: an exact scale that brings max|T| into [0.5, 1), so that
// squares and products of the scaled entries neither overflow nor underflow
__device__ __forceinline__ int scale_exponent(double tmax)
{
  if (!(tmax > 0.0) || isinf(tmax)) return 0;
  const int e = ilogb(tmax) + 1;
  return e < -1000 ? -1000 : (e > 1000 ? 1000 : e);
}

// dense column-major A (N x N) from the lower triangle of the block matrix T; `scaled`:
// times 2^-scale_exponent(max|T|)
__global__ void k_assemble_dense(const double* __restrict__ T, int nblk, int bs, const double* __restrict__ tmax, int scaled, double* __restrict__ A)
{
  ::trl_detail::pdl_enter();
  const int N = nblk * bs;
  const int64_t total = static_cast<int64_t>(N) * N;
  const double floor = kFlushRel * *tmax;
  const double scale = scaled ? scalbn(1.0, -scale_exponent(*tmax)) : 1.0;
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < total; e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(e / N), r = static_cast<int>(e % N); // A[c*N + r] = M(r, c)
    const int hi = r > c ? r : c, lo = r > c ? c : r;
    const int bi = hi / bs, ri = hi % bs, bj = lo / bs, cj = lo % bs;
    const double v = T[(static_cast<int64_t>(bi) * nblk + bj) * bs * bs + ri * bs + cj];
    A[e] = fabs(v) < floor ? 0.0 : v * scale;
  }
}

// rank of each eigenvalue in decreasing |theta| order (ties keep ascending index); tmax: w is
// that of a matrix scaled by 2^-scale_exponent(*tmax) (null: not scaled)
__global__ void k_rank(const double* __restrict__ w, int N, const double* __restrict__ tmax, int* __restrict__ perm, double* __restrict__ evals_sorted,
                       const int* __restrict__ syevd_info, int* status)
{
  ::trl_detail::pdl_enter();
  const double unscale = tmax ? scalbn(1.0, scale_exponent(*tmax)) : 1.0;
  if (blockIdx.x == 0 && threadIdx.x == 0 && *syevd_info != 0) atomicOr(status, TRL_DEV_EIGEN);
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int i = blockIdx.x * nw + (threadIdx.x >> 5); i < N; i += gridDim.x * nw) { // a warp per eigenvalue
    // |w| ordered by bit pattern: the order of the values, and a permutation even with NaNs
    const long long ai = __double_as_longlong(fabs(w[i]));
    int r = 0;
    for (int j = lane; j < N; j += 32) {
      const long long aj = __double_as_longlong(fabs(w[j]));
      r += (aj > ai) || (aj == ai && j < i);
    }
    r = __reduce_add_sync(0xffffffffu, r);
    if (lane == 0) {
      perm[r] = i;
      evals_sorted[r] = w[i] * unscale;
    }
  }
}

__global__ void k_scatter_evecs(const double* __restrict__ A, const int* __restrict__ perm, int nblk, int bs, double* __restrict__ Y)
{
  ::trl_detail::pdl_enter();
  const int N = nblk * bs;
  const int64_t total = static_cast<int64_t>(N) * N;
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < total; e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    // Y in block layout: e = ((bi*nblk + bj)*bs + ri)*bs + cj
    const int cj = static_cast<int>(e % bs);
    const int64_t q = e / bs;
    const int ri = static_cast<int>(q % bs);
    const int64_t blk = q / bs;
    const int bj = static_cast<int>(blk % nblk), bi = static_cast<int>(blk / nblk);
    const int row = bi * bs + ri, col = bj * bs + cj;
    Y[e] = A[static_cast<int64_t>(perm[col]) * N + row];
  }
}

__global__ void k_count_converged(const double* __restrict__ A, const int* __restrict__ perm, const double* __restrict__ evals_sorted, const double* __restrict__ beta, int nblk,
                                  int bs, int ncheck, double tol, int* __restrict__ count)
{
  ::trl_detail::pdl_enter();
  const int N = nblk * bs;
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int c = blockIdx.x * nw + (threadIdx.x >> 5); c < ncheck; c += gridDim.x * nw) { // a warp per pair, a lane per entry of beta y
    const double* y = A + static_cast<int64_t>(perm[c]) * N + (nblk - 1) * bs;
    double v = 0.0;
    if (lane < bs)
      for (int k = 0; k < bs; ++k) v = fma(beta[lane * bs + k], y[k], v);
    double nrm2 = v * v;
    for (int o = 16; o > 0; o >>= 1) nrm2 += __shfl_xor_sync(0xffffffffu, nrm2, o);
    const double denom = fmax(fabs(evals_sorted[c]), DBL_EPSILON);
    if (lane == 0 && sqrt(nrm2) / denom < tol) atomicAdd(count, 1);
  }
}

} // namespace

using namespace trl_detail;

namespace trl_detail {

void destroy_solver(trl_cuda_context* h)
{
  if (h->solver) cusolverDnDestroy(static_cast<cusolverDnHandle_t>(h->solver));
  if (h->syevd_work) cudaFree(h->syevd_work);
  h->solver = nullptr;
  h->syevd_work = nullptr;
  h->syevd_work_bytes = 0;
}

} // namespace trl_detail

extern "C" {

int trl_cuda_mb_copy(trl_cuda_handle h, double* dst, const double* src, int bs, int transpose)
{
  TRL_CHECK_HANDLE(h);
  if (!valid_bs(bs) || !dst || !src) return set_error(h, TRL_EINVAL, "bad block copy arguments");
  if (dst == src && !transpose) return TRL_OK;
  if (dst == src) return set_error(h, TRL_EINVAL, "in-place transpose not supported");
  ProfScope prof(h, PROF_BLOCK_OPS, 16.0 * bs * bs);
  launch(k_mb_copy, 1, bs * bs, 0, h->stream, dst, src, bs, transpose);
  return after_launch(h, "mb_copy");
}

int trl_cuda_mb_zero(trl_cuda_handle h, double* dst, int bs)
{
  TRL_CHECK_HANDLE(h);
  if (!valid_bs(bs) || !dst) return set_error(h, TRL_EINVAL, "bad block zero arguments");
  ProfScope prof(h, PROF_BLOCK_OPS, 8.0 * bs * bs);
  return trl_cuda_memset_zero(h, dst, sizeof(double) * bs * bs);
}

int trl_cuda_mb_mult(trl_cuda_handle h, const double* A, const double* B, double* C, int bs)
{
  TRL_CHECK_HANDLE(h);
  if (!valid_bs(bs) || !A || !B || !C) return set_error(h, TRL_EINVAL, "bad block mult arguments");
  if (C == A || C == B) return set_error(h, TRL_EINVAL, "block mult output must not alias an input");
  ProfScope prof(h, PROF_BLOCK_OPS, 24.0 * bs * bs, 2.0 * bs * bs * bs);
  launch(k_mb_mult, 1, bs * bs, 0, h->stream, A, B, C, bs);
  return after_launch(h, "mb_mult");
}

int trl_cuda_mb_set_diagonal(trl_cuda_handle h, double* dst, const double* host_values, int bs)
{
  TRL_CHECK_HANDLE(h);
  if (!valid_bs(bs) || !dst || !host_values) return set_error(h, TRL_EINVAL, "bad set_diagonal arguments");
  ProfScope prof(h, PROF_BLOCK_OPS, 8.0 * bs);
  DiagValues d{};
  for (int i = 0; i < bs; ++i) d.v[i] = host_values[i];
  launch(k_mb_set_diag, 1, 32, 0, h->stream, dst, d, bs);
  return after_launch(h, "mb_set_diagonal");
}

int trl_cuda_small_eigen(trl_cuda_handle h, const double* T, int nblk, int bs, const double* beta, int nev, double tol, double* evals, double* evecs, double* host_evals,
                         int* host_nconv)
{
  TRL_CHECK_HANDLE(h);
  if (!valid_bs(bs) || nblk <= 0 || !T || !beta || !evals || !evecs || !host_evals || !host_nconv) return set_error(h, TRL_EINVAL, "bad small_eigen arguments");
  const int N = nblk * bs;
  if (N > 8192) return set_error(h, TRL_EINVAL, "projected problem too large (%d)", N);
  ProfScope prof(h, PROF_SMALL_EIGEN, 16.0 * N * N);
  cusolverStatus_t cs;
  if (!h->solver) {
    cusolverDnHandle_t sh;
    if (cusolverDnCreate(&sh) != CUSOLVER_STATUS_SUCCESS) return set_error(h, TRL_ECUDA, "cusolverDnCreate failed");
    h->solver = sh;
  }
  auto sh = static_cast<cusolverDnHandle_t>(h->solver);
  cusolverDnSetStream(sh, h->stream);

  // workspace: A (N*N) | w (N) | evals scratch | perm (N ints) | info | count
  const size_t a_bytes = sizeof(double) * static_cast<size_t>(N) * N;
  const size_t w_bytes = sizeof(double) * N;
  const size_t off_w = a_bytes;
  const size_t off_perm = off_w + w_bytes;
  const size_t off_info = off_perm + sizeof(int) * N + 64;
  const size_t off_tmax = (off_info + 64 + 15) / 16 * 16; // a double: 8-byte aligned whatever N is
  const size_t total = off_tmax + 64;
  char* ws = static_cast<char*>(workspace(h, total));
  if (!ws) return TRL_ENOMEM;
  double* A = reinterpret_cast<double*>(ws);
  double* w = reinterpret_cast<double*>(ws + off_w);
  int* perm = reinterpret_cast<int*>(ws + off_perm);
  int* info = reinterpret_cast<int*>(ws + off_info);
  int* count = info + 1;
  double* tmax = reinterpret_cast<double*>(ws + off_tmax);

  int lwork = 0;
  cs = cusolverDnDsyevd_bufferSize(sh, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, N, A, N, w, &lwork);
  if (cs != CUSOLVER_STATUS_SUCCESS) return set_error(h, TRL_ECUDA, "syevd_bufferSize failed (%d)", static_cast<int>(cs));
  const size_t need = sizeof(double) * static_cast<size_t>(lwork);
  if (need > h->syevd_work_bytes) {
    cudaStreamSynchronize(h->stream);
    if (h->syevd_work) cudaFree(h->syevd_work);
    h->syevd_work = nullptr;
    h->syevd_work_bytes = 0;
    if (cudaMalloc(&h->syevd_work, need) != cudaSuccess) {
      cudaGetLastError();
      return set_error(h, TRL_ENOMEM, "syevd workspace allocation failed");
    }
    h->syevd_work_bytes = need;
  }

  const unsigned g = grid_for(h, static_cast<int64_t>(N) * N, 256, 4);
  cudaMemsetAsync(tmax, 0, sizeof *tmax, h->stream);
  launch(k_max_abs, grid_for(h, static_cast<int64_t>(N) * N, 1024, 1), 256, 0, h->stream, T, static_cast<int64_t>(N) * N, reinterpret_cast<unsigned long long*>(tmax));
  launch(k_assemble_dense, g, 256, 0, h->stream, T, nblk, bs, tmax, 0, A);
  if (int st = after_launch(h, "assemble")) return st;
  cs = cusolverDnDsyevd(sh, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, N, A, N, w, static_cast<double*>(h->syevd_work), lwork, info);
  if (cs != CUSOLVER_STATUS_SUCCESS) return set_error(h, TRL_ECUDA, "syevd failed (%d)", static_cast<int>(cs));
  launch(k_rank, (N + 7) / 8, 256, 0, h->stream, w, N, static_cast<const double*>(nullptr), perm, evals, info, h->d_status);
  if (int st = after_launch(h, "rank")) return st;
  launch(k_scatter_evecs, g, 256, 0, h->stream, A, perm, nblk, bs, evecs);
  if (int st = after_launch(h, "scatter")) return st;
  cudaMemsetAsync(count, 0, sizeof(int), h->stream);
  const int ncheck = nev < N ? nev : N;
  if (ncheck > 0) {
    launch(k_count_converged, (ncheck + 3) / 4, 128, 0, h->stream, A, perm, evals, beta, nblk, bs, ncheck, tol, count);
    if (int st = after_launch(h, "count")) return st;
  }
  char* pin = static_cast<char*>(pinned(h, w_bytes + 64));
  if (!pin) return TRL_ENOMEM;
  cudaMemcpyAsync(pin, evals, w_bytes, cudaMemcpyDeviceToHost, h->stream);
  cudaMemcpyAsync(pin + w_bytes, count, sizeof(int), cudaMemcpyDeviceToHost, h->stream);
  int st = trl_cuda_synchronize(h);
  if (st) return st;
  std::memcpy(host_evals, pin, w_bytes);
  std::memcpy(host_nconv, pin + w_bytes, sizeof(int));
  return TRL_OK;
}

} // extern "C"

// ---- the projected eigenproblem for the eigenvectors the restart keeps ------------------
//
// trl_cuda_small_eigen_partial returns every eigenvalue but only the first kvec eigenvectors
// (|theta| descending), which is all the driver reads (the kept blocks, lanczos.hh:105-131).
// For 3 <= N <= kTriMaxN and kvec <= kTriMaxVec it runs without cuSOLVER:
//  1. k_tridiag: Householder tridiagonalisation Q^T A Q = T in ONE thread-block cluster of 16
//     CTAs that exchange one column per step through distributed shared memory.
//     (cuSOLVER's tridiagonalisation of the same matrix is a sequence of small kernels, about
//     3.7 ms at N = 384 on B200.)
//  2. k_bisect: all eigenvalues of T by bisection on Sturm counts, a CTA per eigenvalue whose
//     threads evaluate one of 64 points of the interval each per round (multisection).
//  3. k_tri_vectors, k_gs_apply: eigenvectors of T for the kvec selected
//     eigenvalues by inverse iteration (partial-pivoting LU of T - lambda I, tiny pivots
//     replaced by eps * ||T||), all vectors at once. A solve shrinks the component along an
//     eigenvalue at distance g by eps * ||T|| / g relative to the wanted one; the wanted end of
//     a Lanczos T is one tight cluster (48 values within 5e-4 ||T|| at the 96^3 workload), so
//     vectors are not iterated one after another but orthonormalised at the end (k_tri_cluster).
//  4. k_wy_factor / k_backtransform: x = Q z with the stored reflectors in compact WY
//     chunks (Q restricted to a chunk = I - V T V^T).
// Otherwise it falls back to trl_cuda_small_eigen and zeroes the columns from kvec on.

namespace {

// The tridiagonalisation runs in one thread-block cluster of 16 CTAs (a non-portable cluster
// size): N <= kTriMaxReg with the rows in registers (k_tridiag); beyond that, or where the
// device cannot hold such a cluster, in shared memory (N <= kTriMaxShared) or in global memory
// (k_tridiag_mem).
constexpr int kTriThreads = 512;
constexpr double kTinyNorm2 = 1e-290; // squared column norms below this are treated as zero (entries are at most 1)
constexpr int kTriMaxReg = 512;
constexpr int kTriMaxShared = 624; // 39 rows and 7 vectors of N doubles in one CTA
constexpr int kTriMaxN = 1024;
constexpr int kTriMaxVec = 256;    // vectors by inverse iteration
constexpr int kTriIters = 3;       // inverse-iteration sweeps

enum TriRows { kTriRegs, kTriShared, kTriGlobal };

size_t tridiag_smem(int N, int C, TriRows rows)
{
  // {t, a} x 2, then v x 2 and w where the CTA shares them, then its rows
  return sizeof(double) * static_cast<size_t>(N) * ((rows == kTriRegs ? 4 : 7) + (rows == kTriShared ? (N + C - 1) / C : 0));
}

__device__ __forceinline__ double warp_sum(double v)
{
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// block sum over the CTA; `red` holds 32 doubles; all threads get the result
__device__ double block_sum(double v, double* red)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_sum(v);
  __syncthreads(); // red may still be read from a previous call
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double s = 0.0;
  if (warp == 0) {
    s = lane < static_cast<int>(blockDim.x >> 5) ? red[lane] : 0.0;
    s = warp_sum(s);
    if (lane == 0) red[0] = s;
  }
  __syncthreads();
  return red[0];
}

// dst[i] = src[i], i < count, by all threads of the CTA with kStageBatch global loads in
// flight per thread (a plain copy loop waits for each load before its store)
constexpr int kStageBatch = 8;

__device__ __forceinline__ void stage(double* dst, const double* __restrict__ src, int count)
{
  const int step = static_cast<int>(blockDim.x);
  for (int base = threadIdx.x; base < count; base += step * kStageBatch) {
    double v[kStageBatch];
#pragma unroll
    for (int u = 0; u < kStageBatch; ++u) {
      const int i = base + u * step;
      v[u] = i < count ? src[i] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kStageBatch; ++u) {
      const int i = base + u * step;
      if (i < count) dst[i] = v[u];
    }
  }
}

// 16-byte store {a, b} into shared memory of another CTA of the cluster (dst, bar: shared::cluster
// addresses of that CTA), counted as 16 bytes on its mbarrier: the data is visible to whoever
// sees the barrier's phase complete, without a cluster barrier or a fence on either side.
__device__ __forceinline__ void st_async_pair(uint32_t dst, double a, double b, uint32_t bar)
{
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(dst), "l"(__double_as_longlong(a)), "l"(__double_as_longlong(b)),
               "r"(bar)
               : "memory");
}

// address in CTA `rank` of the cluster of the shared variable at `addr` of this CTA
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank)
{
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

// mbar_wait (common.cuh) for a phase that other CTAs of the cluster complete
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, int* status, uint32_t limit = (1u << 24))
{
  const uint32_t a = smem_addr(bar);
  for (uint32_t it = 0; it < limit; ++it) {
    uint32_t done;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(done)
                 : "r"(a), "r"(parity)
                 : "memory");
    if (done) return true;
  }
  atomicOr(status, TRL_DEV_TIMEOUT);
  return false;
}

// Householder tridiagonalisation. A: N x N symmetric (full storage, max|A| in [0.5, 1)).
// Outputs: d[N], e[N-1] of Q^T A Q with Q = H_0 ... H_{N-3}, H_k = I - tau_k u_k u_k^T, u_k
// stored in refl[k*ld + k+1 .. N-1] (not normalised).
//
// One cluster of kTriC CTAs of kTriW warps; row g belongs to CTA g % 16 and there to warp
// (g / 16) % 8, which holds it in registers (lane l: columns l, l + 32, ...): row i of a warp
// lies in [128 i, 128 i + 127]. The chain of N steps is bound by latency, so a step is one
// exchange between the CTAs and two sums over a warp, and every warp runs it for itself, with no
// barrier over the CTA or the cluster:
//  - step s starts with each warp sending {t_g, a_gs} of its rows g >= s to every CTA, t = A u_{s-1}
//    and a_gs the row's entry in column s before the update of step s - 1, as one 16-byte
//    asynchronous store that counts on the receiver's mbarrier (every CTA that still has a row
//    beyond s and so waits for the step: tri_sends);
//  - with all pairs there, every warp of every CTA forms w = tau t - K u, column s after the
//    rank-2 update (x = a - u w_s - w u_s), and u_s from x. They compute from the same operands in
//    the same order, so all hold the same bits, and the column's norm needs no second exchange;
//  - it updates its own rows, and multiplies them by u_s. The only entry of u_s that depends on the
//    norm is the first, so that product and its sum run beside the norm's:
//    t = sum_{j > s+1} a_j x_j + a_{s+1} u_{s+1}. tau is not needed before the next exchange.
// Buffers and barriers alternate by step: a warp sends step s + 1 only after it has read step
// s, and step s + 2 needs every row's data of step s + 1, so nothing is overwritten unread. A
// warp leaves when its last row has been sent; the warp with the CTA's last row arms the
// barrier of each step. Steps [128 F, 128 F + 127] run a body of their own without the rows
// and columns before 128 F, so that the body has no branches and its chains overlap.
// Measured on B200 (ncu, us a launch): N = 384 535, N = 512 965, N = 160 120. The kernel before
// this one (rows in shared memory, two cluster barriers and three CTA barriers a step, the
// sums over all CTAs' partials): 1,719, 2,604, 480. At N = 384 a step is about 2,300 cycles:
// sending and waiting 660, reading the pairs and the first sum 440, rows and columns 750, the
// second sum and the norm 410.
constexpr int kTriW = 8;
constexpr int kTriStride = kTriC * kTriW; // rows of one warp are this far apart

template <int RPW>
struct TriState {
  static constexpr int Q = 4 * RPW; // column groups of 32
  double a[RPW][Q], u[Q], ug[RPW], t[RPW], col[RPW];
  double us, half, dprev, eprev; // u_{s-1}[s]; (u . u) / 2 of u_{s-1} (0: no reflector); d, e of step s - 1
  int s;
};

struct TriArgs {
  int N, ld, g0, glast; // matrix size, length of a reflector's row; this warp's first and last row
  bool keeper;
  uint32_t to_pairs, to_bar; // lane q: addresses in CTA q
  const double2* pairs;
  uint64_t* bars;
  double *dout, *eout, *tau_out, *refl;
  int* status;
};

// Steps 128 F ... 128 F + 127 (fewer at the end). false: this warp is done.
template <int RPW, int F>
__device__ __forceinline__ bool tri_steps(TriState<RPW>& st, const TriArgs& k)
{
  constexpr int Q = TriState<RPW>::Q, Q0 = 4 * F;
  const int lane = threadIdx.x & 31, N = k.N;
  for (; st.s < kTriStride * (F + 1); ++st.s) {
    const int s = st.s, cur = s & 1;
    if (s < N - 1) {
#pragma unroll
      for (int i = F; i < RPW; ++i) {
        const int g = k.g0 + i * kTriStride;
        if (tri_sends(N, g, lane, s))
          st_async_pair(k.to_pairs + static_cast<uint32_t>((cur * N + g) * 16), st.t[i], st.col[i], k.to_bar + static_cast<uint32_t>(cur * 8));
      }
    }
    const double tau = st.half > 0.0 ? 1.0 / st.half : 0.0;
    if (s > 0 && (s & (kTriStride - 1)) == k.g0) { // the owner of row s writes reflector s - 1
      if (s < N - 1) {
#pragma unroll
        for (int q = Q0; q < Q; ++q) {
          const int j = q * 32 + lane;
          if (j >= s && j < N) k.refl[static_cast<size_t>(s - 1) * k.ld + j] = st.u[q];
        }
      }
      if (lane == 0) {
        k.dout[s - 1] = st.dprev;
        k.eout[s - 1] = st.eprev;
        k.tau_out[s - 1] = tau;
      }
    }
    if (s == k.glast) {
      if (s == N - 1 && lane == 0) { // the last diagonal entry is not sent: nobody needs it
#pragma unroll
        for (int i = F; i < RPW; ++i)
          if (k.g0 + i * kTriStride == s) k.dout[s] = st.col[i];
      }
      return false;
    }
    if (k.keeper && lane == 0) mbar_arrive_expect_tx(&k.bars[cur], static_cast<uint32_t>(N - s) * 16u);
    const bool late = !mbar_wait_cluster(&k.bars[cur], static_cast<uint32_t>(s >> 1) & 1u, k.status);
    if (__any_sync(0xffffffffu, late)) return false; // whole warp: gives up, the status word says why
    // ---- w = tau t - K u with K = tau^2 (t . u) / 2; x: column s after the update
    const double2* pc = k.pairs + cur * N;
    const double us = st.us;
    // four rows of 16 column groups leave no registers for the t_j as well: they are read again
    constexpr bool kReload = RPW - F >= 4;
    double w[Q], x[Q];
    double k4[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int q = Q0; q < Q; ++q) {
      const int j = q * 32 + lane;
      double2 p = make_double2(0.0, 0.0);
      if (j >= s && j < N) p = pc[j];
      w[q] = p.x;
      x[q] = p.y;
      k4[q & 3] = fma(p.x, st.u[q], k4[q & 3]);
    }
    const double2 ps = pc[s];
    // tau times the sum first: tau is up to 1e290, and tau^2 alone may be out of range
    const double K = 0.5 * tau * (tau * warp_sum((k4[0] + k4[1]) + (k4[2] + k4[3])));
    const double ws = fma(-K, us, tau * ps.x);
    st.dprev = fma(-2.0 * ws, us, ps.y);
    if constexpr (kReload) asm volatile("" ::: "memory");
    // ... column by column, with this warp's rows: update, product with x, entry of column s + 1
    double wg[RPW], t2[RPW][2];
#pragma unroll
    for (int i = F; i < RPW; ++i) {
      wg[i] = fma(-K, st.ug[i], tau * st.t[i]);
      t2[i][0] = t2[i][1] = 0.0;
    }
    double xg[RPW];
#pragma unroll
    for (int i = F; i < RPW; ++i) xg[i] = st.col[i] - fma(st.ug[i], ws, wg[i] * us);
    double n4[4] = {0.0, 0.0, 0.0, 0.0};
    double x0 = 0.0;
#pragma unroll
    for (int q = Q0; q < Q; ++q) {
      const int j = q * 32 + lane;
      if constexpr (kReload) w[q] = j >= s && j < N ? pc[j].x : 0.0;
      const double wq = fma(-K, st.u[q], tau * w[q]);
      const double uq = st.u[q];
      double xq = x[q] - fma(uq, ws, wq * us);
      if (j == s + 1) x0 = xq;
      if (j <= s + 1) xq = 0.0;
      n4[q & 3] = fma(xq, xq, n4[q & 3]);
#pragma unroll
      for (int i = F; i < RPW; ++i) {
        // the two products summed before they are subtracted: subtracted one after the other
        // they lose half a digit of the eigenvalues where A is near a multiple of I
        const double aq = st.a[i][q] - fma(st.ug[i], wq, wg[i] * uq);
        st.a[i][q] = aq;
        t2[i][q & 1] = fma(aq, xq, t2[i][q & 1]);
        if (q == Q0) st.col[i] = aq;
        else st.col[i] = j == s + 1 ? aq : st.col[i];
      }
      st.u[q] = xq;
    }
    double tn[RPW];
#pragma unroll
    for (int i = F; i < RPW; ++i) {
      tn[i] = t2[i][0] + t2[i][1];
      st.ug[i] = xg[i];
    }
    double xnorm2 = (n4[0] + n4[1]) + (n4[2] + n4[3]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      xnorm2 += __shfl_xor_sync(0xffffffffu, xnorm2, o);
#pragma unroll
      for (int i = F; i < RPW; ++i) tn[i] += __shfl_xor_sync(0xffffffffu, tn[i], o);
    }
    x0 = __shfl_sync(0xffffffffu, x0, (s + 1) & 31);
    // ---- reflector s: u = x + copysign(||x||, x_{s+1}) e_{s+1}, tau = 2 / (u . u)
    // a column whose squares underflow is left as it is (H = I): a reflector built from a
    // norm computed in the subnormal range would not be orthogonal
    const double norm2 = fma(x0, x0, xnorm2);
    const double norm = (xnorm2 > 0.0 && norm2 > kTinyNorm2) ? sqrt(norm2) : 0.0;
    const double beta = norm > 0.0 ? -copysign(norm, x0) : x0;
    st.us = x0 - beta;
#pragma unroll
    for (int q = Q0; q < Q; ++q)
      if (q * 32 + lane == s + 1) st.u[q] = st.us;
#pragma unroll
    for (int i = F; i < RPW; ++i) {
      st.col[i] = __shfl_sync(0xffffffffu, st.col[i], (s + 1) & 31);
      st.t[i] = fma(st.col[i], st.us, tn[i]);
      if (k.g0 + i * kTriStride == s + 1) st.ug[i] = st.us;
    }
    st.half = norm > 0.0 ? 0.5 * fma(st.us, st.us, xnorm2) : 0.0;
    st.eprev = beta;
  }
  return true;
}

template <int RPW, int F>
__device__ __forceinline__ void tri_phases(TriState<RPW>& st, const TriArgs& k)
{
  if constexpr (F < RPW) {
    if (tri_steps<RPW, F>(st, k)) tri_phases<RPW, F + 1>(st, k);
  }
}

template <int RPW>
__global__ void __launch_bounds__(kTriW * 32, 1)
    k_tridiag(double* __restrict__ A, int N, int ld, double* __restrict__ dout, double* __restrict__ eout, double* __restrict__ tau_out,
              double* __restrict__ refl, int* status)
{
  ::trl_detail::pdl_enter();
  namespace cg = cooperative_groups;
  constexpr int Q = TriState<RPW>::Q;
  cg::cluster_group cluster = cg::this_cluster();
  const int r = static_cast<int>(cluster.block_rank());
  extern __shared__ __align__(16) double sm[]; // [2][N] pairs {t, a}
  __shared__ __align__(8) uint64_t bars[2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    mbar_init_fence();
  }
  TriArgs k;
  k.N = N;
  k.ld = ld;
  k.g0 = r + kTriC * warp;
  k.glast = k.g0 < N ? k.g0 + (N - 1 - k.g0) / kTriStride * kTriStride : -1;
  k.keeper = k.glast >= 0 && k.glast == tri_last_row(N, r);
  // lane q < 16 sends to CTA q
  k.to_pairs = cluster_addr(smem_addr(sm), lane < kTriC ? lane : 0);
  k.to_bar = cluster_addr(smem_addr(&bars[0]), lane < kTriC ? lane : 0);
  k.pairs = reinterpret_cast<const double2*>(sm);
  k.bars = bars;
  k.dout = dout;
  k.eout = eout;
  k.tau_out = tau_out;
  k.refl = refl;
  k.status = status;
  TriState<RPW> st;
#pragma unroll
  for (int i = 0; i < RPW; ++i) {
    const int g = k.g0 + i * kTriStride;
#pragma unroll
    for (int q = 0; q < Q; ++q) st.a[i][q] = (g < N && q * 32 + lane < N) ? A[static_cast<size_t>(g) * N + q * 32 + lane] : 0.0;
    st.col[i] = __shfl_sync(0xffffffffu, st.a[i][0], 0);
    st.ug[i] = st.t[i] = 0.0;
  }
#pragma unroll
  for (int q = 0; q < Q; ++q) st.u[q] = 0.0;
  st.us = st.half = st.dprev = st.eprev = 0.0;
  st.s = 0;
  cluster.sync(); // every CTA's barriers exist before any store counts on them
  if (k.glast >= 0) tri_phases<RPW, 0>(st, k);
  // Every store sent to a CTA is one its keeper waits for, so none is under way when the keepers are
  // here; the barrier keeps the shared memory of the CTAs in place until then.
  cluster.sync();
}

// The same reduction for matrices whose rows do not fit the cluster's registers, or where a
// cluster of 16 CTAs cannot be resident: rows in the owner's shared memory, or in global memory
// (A itself, L2-resident), updated in place by the lanes of the owning warp; v normalised to v_k[k+1] = 1; the CTA's threads
// share the vectors, thread t holding entries t + 512 e, and the sums are over the CTA.
// RPW: rows a warp owns at most, ceil(ceil(N / C) / 16).
// N = 576 (shared memory) and N = 640, 768, 1024 (global): see kTriVariants.
constexpr int kTriEntries = kTriMaxN / kTriThreads;

// Sum over the CTA of kTriThreads threads, all threads get it: one shuffle tree, one barrier,
// the warps' partials re-read by everyone in one order. `slot` (16 doubles) may be reused
// after one more barrier.
__device__ __forceinline__ double tri_block_sum(double v, double* slot)
{
  constexpr int NW = kTriThreads / 32;
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) slot[threadIdx.x >> 5] = v;
  __syncthreads();
  double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int q = 0; q < NW; ++q) s[q & 3] += slot[q];
  return (s[0] + s[1]) + (s[2] + s[3]);
}

template <int C, int RPW, bool kGlobalRows>
__global__ void __launch_bounds__(kTriThreads, 1)
    k_tridiag_mem(double* __restrict__ A, int N, int ld, double* __restrict__ dout, double* __restrict__ eout, double* __restrict__ tau_out,
                  double* __restrict__ refl, int* status)
{
  ::trl_detail::pdl_enter();
  namespace cg = cooperative_groups;
  constexpr int NW = kTriThreads / 32;
  constexpr int E = kTriEntries;
  cg::cluster_group cluster = cg::this_cluster();
  const int r = static_cast<int>(cluster.block_rank());
  const int RB = (N + C - 1) / C;
  extern __shared__ __align__(16) double sm[];
  __shared__ __align__(16) double red[2][NW];
  __shared__ double x0s;
  __shared__ __align__(8) uint64_t bars[2];
  double* const pa = sm;                 // [2][N] pairs {p, a}, written by the rows' owners
  double* const vbuf = pa + 4 * N;       // [2][N] v_k by parity of k
  double* const wbuf = vbuf + 2 * N;     // [N] w_{k-1}
  double* const rows = wbuf + N;         // RB x N, local row l = global row r + C * l
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  if (!kGlobalRows)
    for (int l = 0; l < RB; ++l)
      if (r + C * l < N) stage(rows + l * N, A + static_cast<size_t>(r + C * l) * N, N);
  if (tid == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    mbar_init_fence();
  }
  for (int j = tid; j < 3 * N; j += kTriThreads) vbuf[j] = 0.0; // v, w
  // lane q < C sends to CTA q
  const uint32_t to_pa = cluster_addr(smem_addr(pa), lane < C ? lane : 0);
  const uint32_t to_bar = cluster_addr(smem_addr(&bars[0]), lane < C ? lane : 0);
  cluster.sync(); // every CTA's barriers exist before any store counts on them

  double tau = 0.0;
  double vj[E]; // v_k[tid + 512 e]
#pragma unroll
  for (int e = 0; e < E; ++e) vj[e] = 0.0;
  for (int k = -1; k <= N - 2; ++k) { // step k: d[k+1], e[k+1], reflector k+1
    const int s = k + 1;
    const int cur = s & 1; // buffers of v_k, of this step's exchange; the other one holds v_{k-1}
    const double* v = vbuf + cur * N;
    const double* vp = vbuf + (cur ^ 1) * N;
    if (tid == 0) mbar_arrive_expect_tx(&bars[cur], static_cast<uint32_t>(N - s) * 16u);
    // ---- rows g > k: rank-2 update of step k - 1, p = tau A v, entry of column k + 1
    const int l0 = s - r > 0 ? (s - r + C - 1) / C : 0; // first local row >= s
    const int lw = l0 + (warp + NW - l0 % NW) % NW;     // this warp's first one
    {
      double acc[RPW], col[RPW], vg[RPW], wg[RPW];
      double* rl[RPW];
      bool on[RPW];
#pragma unroll
      for (int i = 0; i < RPW; ++i) {
        const int l = lw + i * NW, g = r + C * l;
        on[i] = l < RB && g < N;
        rl[i] = kGlobalRows ? A + static_cast<size_t>(on[i] ? g : 0) * N : rows + static_cast<size_t>(on[i] ? l : 0) * N;
        vg[i] = on[i] ? vp[g] : 0.0;
        wg[i] = on[i] ? wbuf[g] : 0.0;
        acc[i] = col[i] = 0.0;
      }
      const int q0 = s & ~31; // columns from the multiple of 32 at or below k + 1 (v, vp, w are zero or unused before it)
      for (int j = q0 + lane; j < N; j += 32) {
        const double vjj = v[j], vpj = vp[j], wpj = wbuf[j];
        double a[RPW];
#pragma unroll
        for (int i = 0; i < RPW; ++i) a[i] = on[i] ? rl[i][j] : 0.0;
#pragma unroll
        for (int i = 0; i < RPW; ++i)
          if (on[i]) {
            a[i] -= fma(vg[i], wpj, wg[i] * vpj);
            rl[i][j] = a[i];
            acc[i] = fma(a[i], vjj, acc[i]);
            if (j == s) col[i] = a[i];
          }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < RPW; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
#pragma unroll
      for (int i = 0; i < RPW; ++i) {
        col[i] = __shfl_sync(0xffffffffu, col[i], s & 31);
        if (on[i] && lane < C) {
          const int g = r + C * (lw + i * NW);
          st_async_pair(to_pa + static_cast<uint32_t>((cur * N + g) * 16), tau * acc[i], col[i], to_bar + static_cast<uint32_t>(cur * 8));
        }
      }
    }
    const bool late = !mbar_wait_cluster(&bars[cur], static_cast<uint32_t>(s >> 1) & 1u, status);
    // ---- w_k = p - K v, K = tau (p . v) / 2
    const double2* pc = reinterpret_cast<const double2*>(pa) + cur * N;
    double p[E], a[E];
    double pv = 0.0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int j = tid + e * kTriThreads;
      const double2 q = j >= s && j < N ? pc[j] : make_double2(0.0, 0.0);
      p[e] = q.x;
      a[e] = q.y;
      pv = fma(q.x, vj[e], pv);
    }
    const double p1 = pc[s].x;
    if (__syncthreads_or(late)) break; // whole CTA: give up, the status word says why
    const double K = 0.5 * tau * tri_block_sum(pv, red[0]);
    const double w1 = p1 - K; // v_k[k+1] = 1
    // ---- column k + 1 after step k: its diagonal entry and x below it
    double x[E], w[E];
    double ssq = 0.0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int j = tid + e * kTriThreads;
      w[e] = k >= 0 ? p[e] - K * vj[e] : 0.0;
      x[e] = k >= 0 ? a[e] - (vj[e] * w1 + w[e]) : a[e];
      if (j == s && r == 0) dout[s] = x[e];
      if (j == s + 1) x0s = x[e];
      if (j > s + 1 && j < N) ssq = fma(x[e], x[e], ssq);
    }
    const double xnorm2 = tri_block_sum(ssq, red[1]);
    if (s == N - 1) break; // d[N-1] was the last
    const double x0 = x0s;
    double beta = x0, scale = 0.0;
    tau = 0.0;
    if (xnorm2 > 0.0 && x0 * x0 + xnorm2 > kTinyNorm2) { // as in k_tridiag
      beta = -copysign(sqrt(x0 * x0 + xnorm2), x0);
      tau = (beta - x0) / beta;
      scale = 1.0 / (x0 - beta);
    }
    double* vn = vbuf + (cur ^ 1) * N; // v_{k+1}; all of this step's reads of v_{k-1} and w_{k-1} are behind the barriers above
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int j = tid + e * kTriThreads;
      vj[e] = j > s + 1 ? x[e] * scale : (j == s + 1 ? 1.0 : 0.0);
      if (j < N) {
        vn[j] = vj[e];
        wbuf[j] = w[e];
        if (r == s % C && j > s && s < N - 2) refl[static_cast<size_t>(s) * ld + j] = vj[e];
      }
    }
    if (r == 0 && tid == 0) {
      eout[s] = beta;
      tau_out[s] = tau;
    }
    __syncthreads();
  }
  cluster.sync(); // every CTA waited for every step's stores; its shared memory stays until all have sent
}

// ---- eigenvalues of the tridiagonal by bisection on Sturm counts
// The number of eigenvalues below sigma is the number of negative pivots of T - sigma I, that is of
// sign changes in p_j = (d_j - sigma) p_{j-1} - e_{j-1}^2 p_{j-2} (the pivots are p_j / p_{j-1}).
// The products need no division, which leaves one dependent FMA per row (17 cycles, against
// about 190 for a row of pivots), and are kept in range by powers of two. Elimination runs from
// both ends to row h = N / 2 at once, whose pivot is
// (d_h - sigma) - e_{h-1}^2 p_{h-2} / p_{h-1} - (the same from below).
// Where they vanish all the same (a pivot of exactly zero beside a zero coupling, or several
// minute ones in a row), the pivots themselves are counted.
constexpr double kPivMin = 0x1p-900; // smallest pivot of the division form

// number of eigenvalues below sigma, counted on pivots; row j = (d_j, e_{j-1}^2)
__device__ __noinline__ int sturm_count_pivots(const double2* up, const double2* down, int N, double sigma)
{
  const int h = N / 2;
  double q = 1.0;
  int c = 0;
  for (int j = 0; j < N; ++j) {
    const double d = j < h ? up[j].x : (j == h ? up[h].x : down[N - 1 - j].x);
    const double e2 = j <= h ? up[j].y : down[N - j].y; // coupling to row j - 1
    q = (d - sigma) - (j > 0 ? e2 / q : 0.0);
    if (fabs(q) < kPivMin) q = -kPivMin;
    c += q < 0.0;
  }
  return c;
}

// One step of the recurrence for row r = (d, e^2 to the row before): p1 the newest product, whose
// sign goes into the lowest bit of signs
__device__ __forceinline__ void sturm_step(double2 r, double sigma, double& p1, double& p0, unsigned& signs)
{
  const double p = fma(r.x - sigma, p1, -(r.y * p0));
  signs = __funnelshift_l(static_cast<unsigned>(__double2hiint(p)), signs, 1);
  p0 = p1;
  p1 = p;
}

// sign changes within the last `rows` products and the one before them
__device__ __forceinline__ int sturm_changes(unsigned signs, int rows) { return __popc((signs ^ (signs >> 1)) & ((1u << rows) - 1u)); }

__device__ __forceinline__ int sturm_top(double p1, double p0) { return max(__double2hiint(p1) & 0x7fffffff, __double2hiint(p0) & 0x7fffffff); } // exponent in the upper 11 bits
constexpr int kSturmRows = 8; // rows between looks at the range (4 / 8 / 16: the call at N = 384 852 / 832 / 824 us; 16 leaves equal diagonals to the pivots)
constexpr int kSturmLow = (1023 - 300) << 20, kSturmHigh = (1023 + 300) << 20;

// Brings a pair of products to the middle of the range, both by the same power of two (their signs
// and ratio stay). Sets `lost` where they are too small to tell.
__device__ __forceinline__ void sturm_rescale(double& p1, double& p0, bool& lost)
{
  const int top = sturm_top(p1, p0);
  lost |= top < ((1023 - 900) << 20);
  const int exponent = min(max(top >> 20, 1), 2045);
  const double by = __hiloint2double((2046 - exponent) << 20, 0);
  p1 *= by;
  p0 *= by;
}

// number of eigenvalues below sigma. up[j] = (d_j, e_{j-1}^2) for rows 0 .. h from the top,
// down[i] = (d, e^2 to the row below) of row N - 1 - i for rows N - 1 .. h + 1 from the bottom
// (down[N - 1 - h].y: the coupling of rows h and h + 1).
__device__ __forceinline__ int sturm_count(const double2* up, const double2* down, int N, double sigma)
{
  const int h = N / 2, m = N - 1 - h; // rows from the top, from the bottom: h = m or m + 1
  double p1 = 1.0, p0 = 0.0, r1 = 1.0, r0 = 0.0;
  unsigned ps = 0, rs = 0;
  int c = 0;
  bool lost = false;
  int j = 0;
  // A row grows the products by less than 2^24 (entries below 1, N <= 1024), so kSturmRows of them
  // stay far from an overflow; what falls too low is noticed (`lost`)
  for (; j + kSturmRows <= m; j += kSturmRows) {
#pragma unroll
    for (int u = 0; u < kSturmRows; ++u) {
      sturm_step(up[j + u], sigma, p1, p0, ps);
      sturm_step(down[j + u], sigma, r1, r0, rs);
    }
    c += sturm_changes(ps, kSturmRows) + sturm_changes(rs, kSturmRows);
    constexpr unsigned kRange = kSturmHigh - kSturmLow;
    if (static_cast<unsigned>(sturm_top(p1, p0) - kSturmLow) > kRange || static_cast<unsigned>(sturm_top(r1, r0) - kSturmLow) > kRange) {
      sturm_rescale(p1, p0, lost);
      sturm_rescale(r1, r0, lost);
    }
  }
  for (; j < m; ++j) {
    sturm_step(up[j], sigma, p1, p0, ps);
    sturm_step(down[j], sigma, r1, r0, rs);
    c += sturm_changes(ps, 1) + sturm_changes(rs, 1);
  }
  if (j < h) {
    sturm_step(up[j], sigma, p1, p0, ps);
    c += sturm_changes(ps, 1);
  }
  sturm_rescale(p1, p0, lost);
  sturm_rescale(r1, r0, lost);
  // pivot of row h times p1 r1
  const double g = fma((up[h].x - sigma) * p1, r1, -fma(up[h].y * p0, r1, down[m].y * r0 * p1));
  if (lost || !(fabs(p1) > 0.0) || !(fabs(r1) > 0.0) || !(fabs(g) > 0.0)) return sturm_count_pivots(up, down, N, sigma);
  return c + static_cast<int>(static_cast<unsigned>(__double2hiint(g) ^ __double2hiint(p1) ^ __double2hiint(r1)) >> 31);
}

// w[i] = i-th smallest eigenvalue of the tridiagonal (d, e): a CTA of two warps per eigenvalue,
// which evaluates the count at 64 points of the interval at a time (multisection). Bound by the
// latency of the recurrence: N / 2 rows x 9 rounds.
// Measured on B200: N = 384 94 us, N = 512 123 us (before, on pivots from one end, one warp and 32
// points per eigenvalue, and the Gershgorin bounds summed by one thread: 427 and 568 us); with signs
// shifted into a word and the range looked at every eight rows instead of four N = 384 72 us, and the
// whole call 844 -> 818 and, N = 512, 1,359 -> 1,324 us.
constexpr int kBisectPoints = 64;

__global__ void __launch_bounds__(kBisectPoints) k_bisect(const double* __restrict__ dg, const double* __restrict__ eg, int N, double* __restrict__ w)
{
  ::trl_detail::pdl_enter();
  extern __shared__ __align__(16) double2 rows[]; // up: N / 2 + 1, then down: N - N / 2
  __shared__ double red[3][2];
  __shared__ unsigned above[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int h = N / 2;
  double2* up = rows;
  double2* down = rows + h + 1;
  double lo = INFINITY, hi = -INFINITY;
  for (int j = tid; j < N; j += kBisectPoints) {
    const double d = dg[j], eb = j > 0 ? fabs(eg[j - 1]) : 0.0, ea = j + 1 < N ? fabs(eg[j]) : 0.0;
    if (j <= h) up[j] = make_double2(d, eb * eb);
    if (j >= h) down[N - 1 - j] = make_double2(d, ea * ea);
    lo = fmin(lo, d - (eb + ea));
    hi = fmax(hi, d + (eb + ea));
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if (lane == 0) {
    red[0][warp] = lo;
    red[1][warp] = hi;
  }
  __syncthreads();
  lo = fmin(red[0][0], red[0][1]);
  hi = fmax(red[1][0], red[1][1]);
  const double margin = 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)) * N + kPivMin;
  lo -= margin;
  hi += margin;
  const int i = blockIdx.x;
  for (int it = 0; it < 64; ++it) {
    const double width = hi - lo;
    if (width <= 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)) + 2.0 * kPivMin) break;
    constexpr double parts = kBisectPoints + 1;
    const double sigma = lo + width * (tid + 1) / parts;
    const int c = sturm_count(up, down, N, sigma);
    const unsigned mask = __ballot_sync(0xffffffffu, c > i);
    if (lane == 0) above[warp] = mask;
    __syncthreads();
    // smallest point with more than i eigenvalues below it
    const int q = above[0] ? __ffs(above[0]) - 1 : (above[1] ? 31 + __ffs(above[1]) : kBisectPoints);
    __syncthreads();
    const double nlo = q == 0 ? lo : lo + width * q / parts;
    const double nhi = q == kBisectPoints ? hi : lo + width * (q + 1) / parts;
    if (!(nhi < hi || nlo > lo)) break; // no progress in floating point
    lo = nlo;
    hi = nhi;
  }
  if (tid == 0) w[i] = 0.5 * (lo + hi);
}

__device__ __forceinline__ double hash_unit(unsigned a, unsigned b)
{
  unsigned x = a * 0x9E3779B1u ^ (b + 0x7F4A7C15u) * 0x85EBCA77u;
  x ^= x >> 15;
  x *= 0x2C1B3C6Du;
  x ^= x >> 12;
  x *= 0x297A2D39u;
  x ^= x >> 15;
  return (static_cast<double>(x) / 4294967295.0) * 2.0 - 1.0;
}

// Inverse iteration for the eigenvectors of the tridiagonal (d, e) at the K eigenvalues
// w[sel[t]] (sel ascending): a warp per vector t, kTriIters solves with T - lambda_t I from a random
// start, into Z[t * N + i] (not scaled; k_tri_cluster does that).
// Elimination with partial pivoting runs from both ends to the middle at once, lane 0 from row 0
// and lane 1 from row N - 1 (a side sees the matrix in its own order, so both run the same
// code), and leaves two equations in the two middle unknowns; substitution runs outwards. The
// recurrences are chains of one reciprocal (factorisation) or one FMA (substitution) per row;
// everything else is prepared by all lanes. Pivots below eps * ||T|| are replaced by +-eps * ||T||,
// and the vector is brought to the middle of the range after each solve.
// Position i of side s is stored at 2 i + s.
// Measured on B200 (K = 40, N = 384 / K = 112, N = 512): 51 / 63 us (before,
// one lane from one end, a kernel for the factors and one per solve: 177 / 227 us).
constexpr int kVectorArrays = 5; // diagonal -> U1, coupling -> U2, multiplier, 1 / pivot, vector

size_t vectors_smem(int N) { return (sizeof(double) * kVectorArrays + 1) * static_cast<size_t>(N + 1); }

__global__ void __launch_bounds__(32) k_tri_vectors(const double* __restrict__ dg, const double* __restrict__ eg, int N, const double* __restrict__ w, const int* __restrict__ sel,
                                                    double* __restrict__ Z)
{
  ::trl_detail::pdl_enter();
  extern __shared__ __align__(16) double vs[];
  const int M = N + 1; // odd N: side 1 is one shorter
  double* U1 = vs;          // diagonal; then the pivot row's next entry times 1 / pivot
  double* U2 = vs + M;      // coupling to the next position; then the entry after it, times 1 / pivot
  double* F = vs + 2 * M;   // multiplier
  double* RP = vs + 3 * M;  // 1 / pivot
  double* X = vs + 4 * M;   // right-hand side, solution
  unsigned char* SW = reinterpret_cast<unsigned char*>(vs + 5 * M); // rows exchanged
  const int t = blockIdx.x, lane = threadIdx.x;
  const int h0 = (N + 1) / 2, h1 = N / 2;
  const double lam = w[sel[t]];
  double nrm = 0.0;
  for (int i = lane; i < N; i += 32) {
    const double eb = i > 0 ? eg[i - 1] : 0.0, ea = i + 1 < N ? eg[i] : 0.0, d = dg[i];
    nrm = fmax(nrm, fabs(d) + fabs(eb) + fabs(ea));
    const int at = i < h0 ? 2 * i : 2 * (N - 1 - i) + 1;
    U1[at] = d - lam;
    U2[at] = i < h0 ? ea : eb;
    X[at] = hash_unit(static_cast<unsigned>(t), static_cast<unsigned>(i));
  }
  for (int o = 16; o > 0; o >>= 1) nrm = fmax(nrm, __shfl_xor_sync(0xffffffffu, nrm, o));
  if (!(nrm > 0.0)) nrm = 1.0;
  const double tiny = DBL_EPSILON * nrm;
  const auto floored = [tiny](double p) { return fabs(p) < tiny ? (p < 0.0 ? -tiny : tiny) : p; };
  // whether the row below is the pivot row: not for an entry below the floor, which stands for zero (taken as
  // a pivot it would multiply what is behind it by 1e25 and more, a vector out of range after a few)
  const auto below = [tiny](double own, double other) { return fabs(own) < fabs(other) && fabs(other) >= tiny; };
  __syncwarp();
  const int side = lane & 1, len = side ? h1 : h0;
  double D = 0.0, U = 0.0, c = 0.0; // the equation carried along: D x_i + U x_{i+1} = c
  if (lane < 2) { // factorisation, with the first forward elimination
    D = U1[side];
    U = U2[side];
    c = X[side];
    double d1 = U1[2 + side], e1 = U2[2 + side], b1 = X[2 + side]; // (position 1; read past the side's end where len is 1, not used)
    double L = U;
    for (int i = 0; i + 1 < len; ++i) {
      const int at = 2 * i + side;
      const int nx = i + 2 < len ? at + 4 : at + 2;
      const double d2 = U1[nx], e2 = U2[nx], b2 = X[nx]; // the next round's row
      const bool sw = below(D, L);
      const double piv = sw ? L : floored(D);
      const double rp = 1.0 / piv;
      const double f = (sw ? D : L) * rp;
      const double u1 = sw ? d1 : U, u2 = sw ? e1 : 0.0, y = sw ? b1 : c;
      c = fma(-f, y, sw ? c : b1);
      D = fma(-f, u1, sw ? U : d1);
      U = sw ? -f * e1 : e1;
      L = e1;
      F[at] = f;
      RP[at] = rp;
      U1[at] = u1;
      U2[at] = u2;
      X[at] = y;
      SW[at] = sw;
      d1 = d2;
      e1 = e2;
      b1 = b2;
    }
  }
  // the two middle equations D x_own + U x_other = c, eliminated with pivoting on x of side 0
  const double D0 = __shfl_sync(0xffffffffu, D, 0), U0 = __shfl_sync(0xffffffffu, U, 0);
  const double D1 = __shfl_sync(0xffffffffu, D, 1), V1 = __shfl_sync(0xffffffffu, U, 1);
  const bool mid = below(D0, V1); // the equation of side 1 is the pivot row
  const double mr = 1.0 / (mid ? V1 : floored(D0));
  const double mf = (mid ? D0 : V1) * mr;
  const double mu = mid ? D1 : U0; // the pivot row's entry of x of side 1
  const double ms = 1.0 / floored(fma(-mf, mu, mid ? U0 : D1));
  __syncwarp();
  for (int at = lane; at < N + 1; at += 32) // entries of positions without a pivot are not read
    if (at / 2 + 1 < ((at & 1) ? h1 : h0)) {
      const double rp = RP[at];
      U1[at] *= rp;
      U2[at] *= rp;
    }
  __syncwarp();
  for (int it = 0; it < kTriIters; ++it) {
    if (it > 0 && lane < 2) { // forward elimination
      c = X[side];
      int i = 0;
      for (; i + 4 < len; i += 4) {
        double f[4], b[4];
        unsigned char sw[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int at = 2 * (i + u) + side;
          f[u] = F[at];
          sw[u] = SW[at];
          b[u] = X[at + 2];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const double y = sw[u] ? b[u] : c;
          c = fma(-f[u], y, sw[u] ? c : b[u]);
          X[2 * (i + u) + side] = y;
        }
      }
      for (; i + 1 < len; ++i) {
        const int at = 2 * i + side;
        const double b = X[at + 2];
        const bool sw = SW[at];
        const double y = sw ? b : c;
        c = fma(-F[at], y, sw ? c : b);
        X[at] = y;
      }
    }
    const double c0 = __shfl_sync(0xffffffffu, c, 0), c1 = __shfl_sync(0xffffffffu, c, 1);
    const double xb = fma(-mf, mid ? c1 : c0, mid ? c0 : c1) * ms; // x of side 1
    const double xa = fma(-mu, xb, mid ? c1 : c0) * mr;            // x of side 0
    if (lane < 2) { // substitution, outwards
      double x1 = side ? xb : xa, x2 = side ? xa : xb; // x_{i+1}, x_{i+2}
      X[2 * (len - 1) + side] = x1;
      int i = len - 2;
      for (; i >= 3; i -= 4) {
        double y[4], a[4], b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int at = 2 * (i - u) + side;
          y[u] = X[at] * RP[at];
          a[u] = U1[at];
          b[u] = U2[at];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const double v = fma(-a[u], x1, fma(-b[u], x2, y[u]));
          X[2 * (i - u) + side] = v;
          x2 = x1;
          x1 = v;
        }
      }
      for (; i >= 0; --i) {
        const int at = 2 * i + side;
        const double v = fma(-U1[at], x1, fma(-U2[at], x2, X[at] * RP[at]));
        X[at] = v;
        x2 = x1;
        x1 = v;
      }
    }
    __syncwarp();
    double mx = 0.0;
    for (int at = lane; at < N + 1; at += 32)
      if (at / 2 < ((at & 1) ? h1 : h0)) mx = fmax(mx, fabs(X[at]));
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const double by = scalbn(1.0, -scale_exponent(mx));
    for (int at = lane; at < N + 1; at += 32) X[at] *= by;
    __syncwarp();
  }
  for (int i = lane; i < N; i += 32) Z[static_cast<size_t>(t) * N + i] = X[i < h0 ? 2 * i : 2 * (N - 1 - i) + 1];
}

// Orthonormalisation of the K vectors (rows of Z, ascending eigenvalues). Inverse iteration
// leaves an overlap of about eps ||T|| / gap between two vectors, so the vectors of eigenvalues
// further apart than kClusterGap ||T|| are orthogonal to 1e-5, and one step
//   z_j <- z_j - (E_jj / 2) z_j - sum_{i<j} E_ij z_i,   E = Z Z^T - I,
// which is Gram-Schmidt in this order to first order, squares what is left: two steps reach
// rounding. They are matrix products spread over the SMs, where Gram-Schmidt vector by vector
// is a chain of K steps in one CTA (B200, N = 384, K = 40: 165 us in shared memory; N = 512, K =
// 112: 3,610 us in global memory; now 38 and 59 us in all).
//  1. k_tri_cluster: Gram-Schmidt twice within each group of closer eigenvalues, a CTA per group;
//     it also scales every vector to unit length;
//  2. k_gs_gram, k_gs_apply twice;
//  3. k_tri_gs, where the first step left more than the second may be given (gs_limit; never
//     seen): Gram-Schmidt twice over all vectors.
constexpr double kClusterGap = 1e-10;

// Gram-Schmidt twice of z_j against z_first .. z_{j-1}, then unit length, by one CTA; coef: K
// doubles of shared memory
__device__ void gs_column(int N, int first, int j, double* __restrict__ Z, double* coef, double* red)
{
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  double* zj = Z + static_cast<size_t>(j) * N;
  for (int pass = 0; pass < 2 && j > first; ++pass) {
    for (int i = first + warp; i < j; i += nw) {
      const double* zi = Z + static_cast<size_t>(i) * N;
      double s = 0.0;
      for (int n = lane; n < N; n += 32) s = fma(zi[n], zj[n], s);
      s = warp_sum(s);
      if (lane == 0) coef[i - first] = s;
    }
    __syncthreads();
    for (int n = tid; n < N; n += blockDim.x) {
      double v = zj[n];
      for (int i = first; i < j; ++i) v = fma(-coef[i - first], Z[static_cast<size_t>(i) * N + n], v);
      zj[n] = v;
    }
    __syncthreads();
  }
  double s = 0.0;
  for (int n = tid; n < N; n += blockDim.x) s = fma(zj[n], zj[n], s);
  s = block_sum(s, red);
  const double inv = s > 0.0 ? 1.0 / sqrt(s) : 0.0;
  for (int n = tid; n < N; n += blockDim.x) zj[n] *= inv;
  __syncthreads();
}

constexpr int kClusterThreads = 256;

__global__ void __launch_bounds__(kClusterThreads) k_tri_cluster(int N, int K, const double* __restrict__ w, const int* __restrict__ sel, double* __restrict__ Z)
{
  ::trl_detail::pdl_enter();
  __shared__ double coef[kTriMaxVec];
  __shared__ double red[32];
  const int t = blockIdx.x;
  const double tol = kClusterGap * fmax(fabs(w[0]), fabs(w[N - 1]));
  if (t > 0 && w[sel[t]] - w[sel[t - 1]] <= tol) return; // in the group of the vector before
  gs_column(N, t, t, Z, coef, red);
  for (int j = t + 1; j < K && w[sel[j]] - w[sel[j - 1]] <= tol; ++j) gs_column(N, t, j, Z, coef, red);
}

// E(i, j) = z_i . z_j - delta_ij (row-major K x K) for the 8 x 8 tiles on and above the
// diagonal: a CTA per tile, its 8 warps take every 8th group of 4 entries of the vectors
// (DMMA), summed in warp order. emax (may be null): the largest |E| as an ordered bit pattern.
__global__ void __launch_bounds__(256) k_gs_gram(int N, int K, const double* __restrict__ Z, double* __restrict__ E, unsigned long long* emax)
{
  ::trl_detail::pdl_enter();
  __shared__ double part[8][64];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  int tj = 0, ti = blockIdx.x; // tile (ti <= tj): column tj holds tj + 1 tiles
  while (ti > tj) ti -= ++tj;
  const int i = ti * 8 + g, j = tj * 8 + g;
  const double* zi = Z + static_cast<size_t>(i < K ? i : 0) * N;
  const double* zj = Z + static_cast<size_t>(j < K ? j : 0) * N;
  double d0[2] = {0.0, 0.0}, d1[2] = {0.0, 0.0};
  constexpr int U = 4; // loads in flight
  for (int n0 = warp * 4; n0 < N; n0 += 32 * U) {
    double a[U], b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int n = n0 + u * 32 + t4;
      a[u] = (n < N && i < K) ? zi[n] : 0.0;
      b[u] = (n < N && j < K) ? zj[n] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) dmma_m8n8k4(d0[u & 1], d1[u & 1], a[u], b[u]);
  }
  part[warp][g * 8 + 2 * t4] = d0[0] + d0[1];
  part[warp][g * 8 + 2 * t4 + 1] = d1[0] + d1[1];
  __syncthreads();
  if (tid < 64) {
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) s += part[q][tid];
    const int ei = ti * 8 + (tid >> 3), ej = tj * 8 + (tid & 7);
    double big = 0.0;
    if (ei < K && ej < K) {
      if (ei == ej) s -= 1.0;
      E[static_cast<size_t>(ei) * K + ej] = s;
      if (ei <= ej) big = fabs(s);
    }
    for (int o = 16; o > 0; o >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
    if (emax && (tid & 31) == 0) atomicMax(emax, static_cast<unsigned long long>(__double_as_longlong(big)));
  }
}

// out_j = z_j - (E_jj / 2) z_j - sum_{i<j} E_ij z_i: a warp per 8 vectors x 32 entries (DMMA).
// With emax above the limit: out = z.
__global__ void __launch_bounds__(128) k_gs_apply(int N, int K, const double* __restrict__ Z, const double* __restrict__ E, const unsigned long long* emax, double limit, double* __restrict__ out)
{
  ::trl_detail::pdl_enter();
  const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int j0 = blockIdx.x * 8, n0 = (blockIdx.y * 4 + (threadIdx.x >> 5)) * 32;
  if (n0 >= N) return;
  const int iend = (emax && __longlong_as_double(static_cast<long long>(*emax)) > limit) ? 0 : min(j0 + 8, K);
  double d0[4] = {0.0, 0.0, 0.0, 0.0}, d1[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
  for (int i0 = 0; i0 < iend; i0 += 4) {
    const int i = i0 + t4, j = j0 + g; // A(g, t4) = -U(i, j), B(t4, g) = z_i[n]
    double a = (i < iend && j < K && i <= j) ? -E[static_cast<size_t>(i) * K + j] : 0.0;
    if (i == j) a *= 0.5;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int n = n0 + c * 8 + g;
      const double b = (i < iend && n < N) ? Z[static_cast<size_t>(i) * N + n] : 0.0;
      dmma_m8n8k4(d0[c], d1[c], a, b);
    }
  }
  const int j = j0 + g;
  if (j >= K) return;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int n = n0 + c * 8 + 2 * t4;
    if (n < N) out[static_cast<size_t>(j) * N + n] = Z[static_cast<size_t>(j) * N + n] + d0[c];
    if (n + 1 < N) out[static_cast<size_t>(j) * N + n + 1] = Z[static_cast<size_t>(j) * N + n + 1] + d1[c];
  }
}

// Gram-Schmidt twice over all vectors, one CTA, if *emax is above the limit
__global__ void __launch_bounds__(kTriThreads) k_tri_gs(int N, int K, double* __restrict__ Z, const unsigned long long* emax, double limit)
{
  ::trl_detail::pdl_enter();
  if (!(__longlong_as_double(static_cast<long long>(*emax)) > limit)) return;
  __shared__ double coef[kTriMaxVec];
  __shared__ double red[32];
  for (int j = 0; j < K; ++j) gs_column(N, 0, j, Z, coef, red);
}

// Back-transform X = Q Z, Q = H_0 ... H_{N-3}, in chunks of kWyRows reflectors: a chunk
// H_a ... H_b equals I - V T V^T (compact WY form, T upper triangular: T_ii = tau_i,
// T[0:i, i] = -tau_i T[0:i, 0:i] V[:, 0:i]^T v_i), so a chunk is three small matrix
// products on the vectors instead of kWyRows dependent reflector applications. Reflectors are
// rows of `ld` doubles (an even number: 16-byte aligned rows).
constexpr int kWyRows = 16;
constexpr int kWyThreads = 256;
constexpr size_t kWyStageMax = 200 * 1024; // two chunks of reflectors in shared memory, or one

__host__ __device__ __forceinline__ int refl_ld(int N) { return N + (N & 1); }

// T of chunk c (reflectors c * kWyRows ...) into Tw[c][kWyRows][kWyRows], and the zeros of the
// chunk's reflectors up to their first entry (from the multiple of 32 at or below it) into refl
__global__ void __launch_bounds__(kWyThreads) k_wy_factor(double* __restrict__ refl, const double* __restrict__ tau, int N, int ld, double* __restrict__ Tw)
{
  ::trl_detail::pdl_enter();
  constexpr int NW = kWyThreads / 32;
  __shared__ double part[NW][3][64];
  __shared__ double G[kWyRows][kWyRows + 1];
  const int R = N - 2;
  const int k0 = blockIdx.x * kWyRows;
  const int b = R - k0 < kWyRows ? R - k0 : kWyRows;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  const int start = k0 & ~31;
  for (int rr = warp; rr < b; rr += NW)
    for (int i = start + lane; i <= k0 + rr; i += 32) refl[static_cast<size_t>(k0 + rr) * ld + i] = 0.0;
  // G = V^T V: tiles (0, 0), (0, 1), (1, 1) of 8 x 8 on the tensor cores, entries split over the warps
  double d0[3] = {0.0, 0.0, 0.0}, d1[3] = {0.0, 0.0, 0.0};
  const double* v0 = refl + static_cast<size_t>(k0 + (g < b ? g : 0)) * ld;
  const double* v1 = refl + static_cast<size_t>(k0 + (g + 8 < b ? g + 8 : 0)) * ld;
#pragma unroll 4
  for (int n0 = start + warp * 4; n0 < N; n0 += NW * 4) {
    const int n = n0 + t4;
    const double a0 = (g < b && n > k0 + g && n < N) ? v0[n] : 0.0; // v_k is zero up to entry k
    const double a1 = (g + 8 < b && n > k0 + g + 8 && n < N) ? v1[n] : 0.0;
    dmma_m8n8k4(d0[0], d1[0], a0, a0);
    dmma_m8n8k4(d0[1], d1[1], a0, a1);
    dmma_m8n8k4(d0[2], d1[2], a1, a1);
  }
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    part[warp][q][g * 8 + 2 * t4] = d0[q];
    part[warp][q][g * 8 + 2 * t4 + 1] = d1[q];
  }
  __syncthreads();
  if (tid < 192) {
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < NW; ++q) s += part[q][tid >> 6][tid & 63];
    const int tile = tid >> 6, e = tid & 63;
    G[(tile == 2 ? 8 : 0) + (e >> 3)][(tile == 0 ? 0 : 8) + (e & 7)] = s;
  }
  __syncthreads();
  if (warp == 0 && lane < kWyRows) { // lane j: row j of T
    double row[kWyRows];
#pragma unroll
    for (int i = 0; i < kWyRows; ++i) {
      const double ti = i < b ? tau[k0 + i] : 0.0;
      double s4[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int m = 0; m < i; ++m) s4[m & 3] = fma(row[m], G[m][i], s4[m & 3]); // row[m] = 0 for m < lane
      const double s = (s4[0] + s4[1]) + (s4[2] + s4[3]);
      row[i] = i < lane || i >= b ? 0.0 : (i == lane ? ti : -ti * s);
      Tw[(static_cast<size_t>(blockIdx.x) * kWyRows + lane) * kWyRows + i] = row[i];
    }
  }
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}

// One vector per CTA (the chunks are a chain, so the vectors spread over the SMs). While a chunk
// is applied, the next one's reflectors arrive in the other half of the stage.
// Measured on B200 with k_wy_factor (K = 40, N = 384 / K = 112, N = 512): 72 / 98 us
// (before, each chunk loaded after the last was applied and T applied between barriers: 208 /
// 315 us).
__global__ void __launch_bounds__(kWyThreads) k_backtransform(const double* __restrict__ Z, int N, int ld, int stages, const double* __restrict__ refl, const double* __restrict__ Tw,
                                                              double* __restrict__ X)
{
  ::trl_detail::pdl_enter();
  extern __shared__ __align__(16) double sm[]; // stages x kWyRows x ld reflectors | vector
  constexpr int NW = kWyThreads / 32;
  __shared__ double W[kWyRows], W2[NW][kWyRows];
  double* const xs = sm + static_cast<size_t>(stages) * kWyRows * ld;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < N; i += kWyThreads) xs[i] = Z[static_cast<size_t>(blockIdx.x) * N + i];
  const int R = N - 2;
  const int nch = (R + kWyRows - 1) / kWyRows;
  const auto fetch = [&](int c) { // chunk c's rows, entries from the multiple of 32 below its first
    const int k0 = c * kWyRows, b = R - k0 < kWyRows ? R - k0 : kWyRows, start = k0 & ~31;
    double* to = sm + static_cast<size_t>(c % stages) * kWyRows * ld;
    for (int rr = warp; rr < b; rr += NW)
      for (int i = start + 2 * lane; i < ld; i += 64) cp_async16(to + static_cast<size_t>(rr) * ld + i, refl + static_cast<size_t>(k0 + rr) * ld + i);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (stages > 1) fetch(nch - 1);
  for (int c = nch - 1; c >= 0; --c) {
    const int k0 = c * kWyRows, b = R - k0 < kWyRows ? R - k0 : kWyRows, start = k0 & ~31;
    if (stages > 1 && c > 0) {
      fetch(c - 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    }
    else {
      if (stages == 1) fetch(c);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    double tr[kWyRows]; // lane m < 16: row m of T
#pragma unroll
    for (int q = 0; q < kWyRows; ++q) tr[q] = lane < kWyRows ? __ldg(Tw + (static_cast<size_t>(c) * kWyRows + lane) * kWyRows + q) : 0.0;
    __syncthreads(); // the chunk is there for all; the vector is as the last chunk left it
    const double* vs = sm + static_cast<size_t>(c % stages) * kWyRows * ld;
    // W = V^T x: warp w takes rows w and w + 8
    {
      const double* va = vs + static_cast<size_t>(warp) * ld;
      const double* vb = vs + static_cast<size_t>(warp + NW) * ld;
      const bool oka = warp < b, okb = warp + NW < b;
      double sa0 = 0.0, sa1 = 0.0, sb0 = 0.0, sb1 = 0.0;
      int i = start + lane;
#pragma unroll 2
      for (; i + 32 < N; i += 64) {
        const double x0 = xs[i], x1 = xs[i + 32];
        sa0 = fma(oka ? va[i] : 0.0, x0, sa0);
        sb0 = fma(okb ? vb[i] : 0.0, x0, sb0);
        sa1 = fma(oka ? va[i + 32] : 0.0, x1, sa1);
        sb1 = fma(okb ? vb[i + 32] : 0.0, x1, sb1);
      }
      if (i < N) {
        sa0 = fma(oka ? va[i] : 0.0, xs[i], sa0);
        sb0 = fma(okb ? vb[i] : 0.0, xs[i], sb0);
      }
      double s0 = sa0 + sa1, s1 = sb0 + sb1;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        s0 += __shfl_xor_sync(0xffffffffu, s0, o);
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
      }
      if (lane == 0) {
        W[warp] = s0;
        W[warp + NW] = s1;
      }
    }
    __syncthreads();
    { // W2 = T W, by every warp for itself
      double s4[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int q = 0; q < kWyRows; ++q) s4[q & 3] = fma(tr[q], W[q], s4[q & 3]);
      if (lane < kWyRows) W2[warp][lane] = (s4[0] + s4[1]) + (s4[2] + s4[3]);
      __syncwarp();
    }
    for (int i = start + tid; i < N; i += kWyThreads) { // x -= V W2
      double s4[4] = {xs[i], 0.0, 0.0, 0.0};
#pragma unroll
      for (int rr = 0; rr < kWyRows; ++rr)
        if (rr < b) s4[rr & 3] = fma(-vs[static_cast<size_t>(rr) * ld + i], W2[warp][rr], s4[rr & 3]);
      xs[i] = (s4[0] + s4[1]) + (s4[2] + s4[3]);
    }
    __syncthreads(); // done with the stage and with W
  }
  for (int i = tid; i < N; i += kWyThreads) X[static_cast<size_t>(blockIdx.x) * N + i] = xs[i];
}

// selected ascending indices: sel[t] (ascending), slot[c] = t for rank c < K
__global__ void k_select(const int* __restrict__ perm, int K, int* __restrict__ sel, int* __restrict__ slot)
{
  ::trl_detail::pdl_enter();
  const int c = threadIdx.x;
  if (c >= K) return;
  const int a = perm[c];
  int t = 0;
  for (int q = 0; q < K; ++q) t += perm[q] < a;
  sel[t] = a;
  slot[c] = t;
}

// Y in block layout: column c < K is X[slot[c]], the rest zero
__global__ void k_scatter_partial(const double* __restrict__ X, const int* __restrict__ slot, int nblk, int bs, int K, double* __restrict__ Y)
{
  ::trl_detail::pdl_enter();
  const int N = nblk * bs;
  const int64_t total = static_cast<int64_t>(N) * N;
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < total; e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int cj = static_cast<int>(e % bs);
    const int64_t q = e / bs;
    const int ri = static_cast<int>(q % bs);
    const int64_t blk = q / bs;
    const int bj = static_cast<int>(blk % nblk), bi = static_cast<int>(blk / nblk);
    const int row = bi * bs + ri, col = bj * bs + cj;
    Y[e] = col < K ? X[static_cast<int64_t>(slot[col]) * N + row] : 0.0;
  }
}

__global__ void k_count_partial(const double* __restrict__ X, const int* __restrict__ slot, const double* __restrict__ evals_sorted, const double* __restrict__ beta, int nblk, int bs,
                                int ncheck, double tol, int* __restrict__ count)
{
  ::trl_detail::pdl_enter();
  const int N = nblk * bs;
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int c = blockIdx.x * nw + (threadIdx.x >> 5); c < ncheck; c += gridDim.x * nw) { // a warp per pair, a lane per entry of beta y
    const double* y = X + static_cast<int64_t>(slot[c]) * N + (nblk - 1) * bs;
    double v = 0.0;
    if (lane < bs)
      for (int k = 0; k < bs; ++k) v = fma(beta[lane * bs + k], y[k], v);
    double nrm2 = v * v;
    for (int o = 16; o > 0; o >>= 1) nrm2 += __shfl_xor_sync(0xffffffffu, nrm2, o);
    const double denom = fmax(fabs(evals_sorted[c]), DBL_EPSILON);
    if (lane == 0 && sqrt(nrm2) / denom < tol) atomicAdd(count, 1);
  }
}

// zero the block-layout columns >= K of Y
__global__ void k_zero_cols(double* __restrict__ Y, int nblk, int bs, int K)
{
  ::trl_detail::pdl_enter();
  const int N = nblk * bs;
  const int64_t total = static_cast<int64_t>(N) * N;
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < total; e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int cj = static_cast<int>(e % bs);
    const int bj = static_cast<int>((e / (static_cast<int64_t>(bs) * bs)) % nblk);
    if (bj * bs + cj >= K) Y[e] = 0.0;
  }
}

using TriKernel = void (*)(double*, int, int, double*, double*, double*, double*, int*);

struct TriVariant {
  TriKernel fn;
  int C;       // CTAs in the cluster
  int threads;
  TriRows rows;
  int max_n;
};

constexpr TriVariant kTriVariants[] = {
    {k_tridiag<1>, kTriC, kTriW * 32, kTriRegs, 128},
    {k_tridiag<2>, kTriC, kTriW * 32, kTriRegs, 256},
    {k_tridiag<3>, kTriC, kTriW * 32, kTriRegs, 384},
    {k_tridiag<4>, kTriC, kTriW * 32, kTriRegs, kTriMaxReg},
    {k_tridiag_mem<16, 3, false>, 16, kTriThreads, kTriShared, kTriMaxShared},
    {k_tridiag_mem<16, 4, true>, 16, kTriThreads, kTriGlobal, kTriMaxN},
    {k_tridiag_mem<8, 8, true>, 8, kTriThreads, kTriGlobal, kTriMaxN},
};
constexpr int kNumTriVariants = sizeof(kTriVariants) / sizeof(kTriVariants[0]);

void tri_config(const TriVariant& v, int N, cudaStream_t stream, cudaLaunchConfig_t& cfg, cudaLaunchAttribute& attr)
{
  cfg = cudaLaunchConfig_t{};
  cfg.gridDim = dim3(v.C);
  cfg.blockDim = dim3(v.threads);
  cfg.dynamicSmemBytes = tridiag_smem(N, v.C, v.rows);
  cfg.stream = stream;
  attr = cudaLaunchAttribute{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = v.C;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
}

// The first variant that takes N and can be resident on `device`, or null. Checked once per
// device: function attributes belong to the current device.
const TriVariant* tri_variant(int device, int N)
{
  static int ok[64][kNumTriVariants];
  static bool checked[64];
  static std::mutex lock;
  std::lock_guard<std::mutex> g(lock);
  if (!checked[device]) {
    checked[device] = true;
    const bool common = cudaFuncSetAttribute(k_backtransform, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kWyStageMax + sizeof(double) * kTriMaxN)) == cudaSuccess;
    for (int i = 0; i < kNumTriVariants && common; ++i) {
      const TriVariant& v = kTriVariants[i];
      if (cudaFuncSetAttribute(v.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(tridiag_smem(v.max_n, v.C, v.rows))) != cudaSuccess) continue;
      if (v.C > 8 && cudaFuncSetAttribute(v.fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) continue;
      cudaLaunchConfig_t cfg{};
      cudaLaunchAttribute attr{};
      tri_config(v, v.max_n, nullptr, cfg, attr);
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, v.fn, &cfg) == cudaSuccess && clusters > 0) ok[device][i] = 1;
    }
    cudaGetLastError();
  }
  for (int i = 0; i < kNumTriVariants; ++i)
    if (ok[device][i] && N <= kTriVariants[i].max_n) return &kTriVariants[i];
  return nullptr;
}

} // namespace

extern "C" int trl_cuda_small_eigen_partial(trl_cuda_handle h, const double* T, int nblk, int bs, const double* beta, int nev, double tol, int kvec, double* evals, double* evecs,
                                            double* host_evals, int* host_nconv)
{
  TRL_CHECK_HANDLE(h);
  if (!valid_bs(bs) || nblk <= 0 || !T || !beta || !evals || !evecs || !host_evals || !host_nconv) return set_error(h, TRL_EINVAL, "bad small_eigen arguments");
  const int N = nblk * bs;
  if (kvec < 0 || kvec > N) return set_error(h, TRL_EINVAL, "kvec %d outside [0, %d]", kvec, N);
  if (h->device < 0 || h->device >= 64) return set_error(h, TRL_EINVAL, "device index %d", h->device);
  const TriVariant* tv = tri_variant(h->device, N);
  if (N < 3 || kvec > kTriMaxVec || !tv) {
    if (int st = trl_cuda_small_eigen(h, T, nblk, bs, beta, nev, tol, evals, evecs, host_evals, host_nconv)) return st;
    launch(k_zero_cols, grid_for(h, static_cast<int64_t>(N) * N, 256, 4), 256, 0, h->stream, evecs, nblk, bs, kvec);
    return after_launch(h, "zero columns");
  }
  ProfScope prof(h, PROF_SMALL_EIGEN, 16.0 * N * N);
  const int K = kvec > 0 ? kvec : 1;
  // workspace: refl (N*ld) | A (N*N) | d | e | tau | w (N each) | Z (N*K) | X (N*K) |
  // E (K*K overlaps) | perm, sel, slot (N ints each) | max|T|, largest overlap, flags
  const size_t NN = static_cast<size_t>(N) * N, NK = static_cast<size_t>(N) * K;
  const size_t nchunks = static_cast<size_t>(N - 2 + kWyRows - 1) / kWyRows;
  const int ld = refl_ld(N);
  const size_t doubles = NN + static_cast<size_t>(N) * ld + 4 * static_cast<size_t>(N) + 2 * NK + static_cast<size_t>(K) * K + nchunks * kWyRows * kWyRows;
  const size_t ints = 3 * static_cast<size_t>(N);
  char* ws = static_cast<char*>(workspace(h, sizeof(double) * (doubles + 1) + sizeof(int) * ints + 256));
  if (!ws) return TRL_ENOMEM;
  double* refl = reinterpret_cast<double*>(ws);
  double* A = refl + static_cast<size_t>(N) * ld;
  double* d = A + NN;
  double* e = d + N;
  double* tau = e + N;
  double* w = tau + N;
  double* Z = w + N;
  double* X = Z + NK;
  double* E = X + NK;
  double* Tw = E + static_cast<size_t>(K) * K;
  int* perm = reinterpret_cast<int*>(Tw + nchunks * kWyRows * kWyRows);
  int* sel = perm + N;
  int* slot = sel + N;
  double* tmax = reinterpret_cast<double*>(ws + (sizeof(double) * doubles + sizeof(int) * ints + 15) / 16 * 16);
  auto* emax = reinterpret_cast<unsigned long long*>(tmax + 1);
  int* flags = reinterpret_cast<int*>(tmax + 2); // [0] = 0 (no solver error), [1] = converged count

  const unsigned g = grid_for(h, static_cast<int64_t>(N) * N, 256, 4);
  cudaMemsetAsync(tmax, 0, 2 * sizeof(double) + 2 * sizeof(int), h->stream); // tmax, emax, flags
  launch(k_max_abs, grid_for(h, static_cast<int64_t>(N) * N, 1024, 1), 256, 0, h->stream, T, static_cast<int64_t>(N) * N, reinterpret_cast<unsigned long long*>(tmax));
  launch(k_assemble_dense, g, 256, 0, h->stream, T, nblk, bs, tmax, 1, A);
  if (int st = after_launch(h, "assemble")) return st;
  {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    tri_config(*tv, N, h->stream, cfg, attr);
    cudaLaunchKernelEx(&cfg, tv->fn, A, N, ld, d, e, tau, refl, h->d_status);
    if (int st = after_launch(h, "tridiagonalise")) return st;
  }
  launch(k_bisect, N, kBisectPoints, sizeof(double2) * (N + 1), h->stream, d, e, N, w);
  if (int st = after_launch(h, "bisect")) return st;
  launch(k_rank, (N + 7) / 8, 256, 0, h->stream, w, N, tmax, perm, evals, flags, h->d_status);
  if (int st = after_launch(h, "rank")) return st;
  launch(k_select, 1, kTriMaxVec, 0, h->stream, perm, K, sel, slot);
  if (int st = after_launch(h, "select")) return st;
  launch(k_tri_vectors, K, 32, vectors_smem(N), h->stream, d, e, N, w, sel, Z);
  if (int st = after_launch(h, "inverse iteration")) return st;
  launch(k_tri_cluster, K, kClusterThreads, 0, h->stream, N, K, w, sel, Z);
  if (int st = after_launch(h, "gram-schmidt")) return st;
  const int kt = (K + 7) / 8;
  const dim3 apply_grid(kt, (N + 127) / 128);
  for (int round = 0; round < 2; ++round) {
    double* from = round == 0 ? Z : X;
    double* to = round == 0 ? X : Z;
    unsigned long long* check = round == 0 ? nullptr : emax;
    launch(k_gs_gram, kt * (kt + 1) / 2, 256, 0, h->stream, N, K, from, E, check);
    if (int st = after_launch(h, "overlaps")) return st;
    launch(k_gs_apply, apply_grid, 128, 0, h->stream, N, K, from, E, check, gs_limit(K), to);
    if (int st = after_launch(h, "orthogonalise")) return st;
  }
  launch(k_tri_gs, 1, kTriThreads, 0, h->stream, N, K, Z, emax, gs_limit(K));
  if (int st = after_launch(h, "gram-schmidt")) return st;
  const int nch = (N - 2 + kWyRows - 1) / kWyRows;
  launch(k_wy_factor, nch, kWyThreads, 0, h->stream, refl, tau, N, ld, Tw);
  if (int st = after_launch(h, "wy factor")) return st;
  const size_t chunk = sizeof(double) * kWyRows * ld;
  const int stages = 2 * chunk <= kWyStageMax ? 2 : 1;
  launch(k_backtransform, K, kWyThreads, stages * chunk + sizeof(double) * N, h->stream, Z, N, ld, stages, refl, Tw, X);
  if (int st = after_launch(h, "back-transform")) return st;
  launch(k_scatter_partial, g, 256, 0, h->stream, X, slot, nblk, bs, kvec, evecs);
  if (int st = after_launch(h, "scatter")) return st;
  const int ncheck = nev < kvec ? nev : kvec;
  if (ncheck > 0) {
    launch(k_count_partial, (ncheck + 3) / 4, 128, 0, h->stream, X, slot, evals, beta, nblk, bs, ncheck, tol, flags + 1);
    if (int st = after_launch(h, "count")) return st;
  }
  const size_t w_bytes = sizeof(double) * N;
  char* pin = static_cast<char*>(pinned(h, w_bytes + 64));
  if (!pin) return TRL_ENOMEM;
  cudaMemcpyAsync(pin, evals, w_bytes, cudaMemcpyDeviceToHost, h->stream);
  cudaMemcpyAsync(pin + w_bytes, flags + 1, sizeof(int), cudaMemcpyDeviceToHost, h->stream);
  int st = trl_cuda_synchronize(h);
  if (st) return st;
  std::memcpy(host_evals, pin, w_bytes);
  std::memcpy(host_nconv, pin + w_bytes, sizeof(int));
  return TRL_OK;
}

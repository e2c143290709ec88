// Block-vector kernels of the backend: elementwise ops, the multi-block inner product
// (block dot), the tall-skinny block GEMM behind mult / mult_transpose / mult_add /
// subtract_product / the CGS projection update / the thick-restart rotation, and
// Cholesky-QR. Contractions run on the FP64 tensor cores (DMMA m8n8k4); FP32 storage is
// widened to FP64 in registers, so products are exact and sums are FP64.
//
// Layout: a block vector is n x BS row-major; block j of a multivector at base + j*n*BS.
#include "common.cuh"

#include <cmath>
#include <cstdio>
#include <cstdlib>

namespace {

constexpr int kThreads = 256; // 8 warps per CTA for every kernel in this file
constexpr int kWarps = kThreads / 32;

// ---------------------------------------------------------------- elementwise
template <typename T>
struct Vec16;
template <>
struct Vec16<double> {
  using type = double2;
  static constexpr int width = 2;
};
template <>
struct Vec16<float> {
  using type = float4;
  static constexpr int width = 4;
};

template <typename T>
__device__ __forceinline__ void vsub(typename Vec16<T>::type& a, const typename Vec16<T>::type& b);
template <>
__device__ __forceinline__ void vsub<double>(double2& a, const double2& b)
{
  a.x -= b.x;
  a.y -= b.y;
}
template <>
__device__ __forceinline__ void vsub<float>(float4& a, const float4& b)
{
  a.x -= b.x;
  a.y -= b.y;
  a.z -= b.z;
  a.w -= b.w;
}

// X -= Y over `count` elements; vectorised when both pointers are 16-byte aligned.
template <typename T>
__global__ void __launch_bounds__(kThreads) k_sub(T* __restrict__ X, const T* __restrict__ Y, int64_t count, int vec_ok)
{
  ::trl_detail::pdl_enter();
  const int64_t tid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  using V = typename Vec16<T>::type;
  constexpr int W = Vec16<T>::width;
  int64_t done = 0;
  if (vec_ok) {
    const int64_t nv = count / W;
    V* xv = reinterpret_cast<V*>(X);
    const V* yv = reinterpret_cast<const V*>(Y);
    for (int64_t i = tid; i < nv; i += stride) {
      V a = xv[i];
      vsub<T>(a, yv[i]);
      xv[i] = a;
    }
    done = nv * W;
  }
  for (int64_t i = done + tid; i < count; i += stride) X[i] -= Y[i];
}

template <typename D, typename S>
__global__ void __launch_bounds__(kThreads) k_convert(D* __restrict__ dst, const S* __restrict__ src, int64_t count)
{
  ::trl_detail::pdl_enter();
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += stride) dst[i] = static_cast<D>(src[i]);
}

// ---------------------------------------------------------------- sums over the CTAs of a kernel
// A kernel that leaves one row of LEN partial sums per CTA can also add them up: the CTA that
// finishes last does it, found by ticket counters (zero between launches), so the short
// results of single-block dots and Grams need no second launch. The rows are added in groups of
// kTicketGroup, each by the last CTA of its group, and the groups' sums by the last group's: two
// rounds of loads, however many CTAs there are. Which CTA adds depends on scheduling, the order
// of the additions does not.
constexpr int kTicketGroup = 32;
constexpr int kTickets = 128; // counters of a handle: one for the groups, one per group

struct Tickets {
  unsigned* count; // [kTickets]
  double* groups;  // [number of groups][LEN]
};

// sum[e] = sum of a[r * LEN + e] over the rows r < rows, by a CTA of kThreads; scratch: kThreads doubles
template <int LEN>
__device__ __forceinline__ void sum_rows(const double* a, int rows, double* sum, double* scratch)
{
  constexpr int SL = LEN >= kThreads ? 1 : (kThreads / LEN < 16 ? kThreads / LEN : 16); // threads per entry
  constexpr int U = 8;                                    // loads in flight
  const int tid = threadIdx.x;
  for (int e = SL > 1 ? (tid < LEN * SL ? tid % LEN : LEN) : tid; e < LEN; e += kThreads) {
    double t[U];
#pragma unroll
    for (int u = 0; u < U; ++u) t[u] = 0.0;
    for (int r = tid / LEN; r < rows; r += U * SL) {
#pragma unroll
      for (int u = 0; u < U; ++u) t[u] += r + u * SL < rows ? __ldcg(a + static_cast<int64_t>(r + u * SL) * LEN + e) : 0.0; // L2: other CTAs wrote it
    }
    const double v = ((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7]));
    if constexpr (SL == 1) sum[e] = v;
    else scratch[tid] = v;
  }
  if constexpr (SL > 1) {
    __syncthreads();
    if (tid < LEN) {
      double v = 0.0;
#pragma unroll
      for (int q = 0; q < SL; ++q) v += scratch[q * LEN + tid];
      sum[tid] = v;
    }
  }
  __syncthreads();
}

// Called by every CTA after it wrote its row `chunk` of partial[chunks][LEN]; true in the one CTA
// that then has the totals in sum[LEN] (shared memory, as scratch).
template <int LEN>
__device__ __forceinline__ bool last_cta_sum(const double* partial, int chunks, int chunk, const Tickets& t, double* sum, double* scratch)
{
  __shared__ int last;
  const int group = chunk / kTicketGroup, ngroups = (chunks + kTicketGroup - 1) / kTicketGroup;
  const int members = min(kTicketGroup, chunks - group * kTicketGroup);
  // the barrier and thread 0's fence order this CTA's row before its ticket, and the rows of
  // the CTAs that came before it after the ticket
  const auto take = [](unsigned* counter, int count) {
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      last = atomicAdd(counter, 1u) == static_cast<unsigned>(count - 1);
      __threadfence();
    }
    __syncthreads();
    return last != 0;
  };
  if (!take(&t.count[1 + group], members)) return false;
  sum_rows<LEN>(partial + static_cast<int64_t>(group) * kTicketGroup * LEN, members, sum, scratch);
  if (threadIdx.x == 0) t.count[1 + group] = 0u;
  if (ngroups == 1) return true;
  for (int e = threadIdx.x; e < LEN; e += kThreads) t.groups[static_cast<int64_t>(group) * LEN + e] = sum[e];
  if (!take(&t.count[0], ngroups)) return false;
  sum_rows<LEN>(t.groups, ngroups, sum, scratch);
  if (threadIdx.x == 0) t.count[0] = 0u;
  return true;
}

// What the last CTA does with the totals (all its threads call it).
struct FinishNone { // partial sums only
  static constexpr bool kOn = false;
  __device__ void operator()(const double*) const {}
};

template <int LEN>
struct FinishStore {
  static constexpr bool kOn = true;
  double* out;
  __device__ void operator()(const double* sum) const
  {
    for (int e = threadIdx.x; e < LEN; e += kThreads) out[e] = sum[e];
  }
};

// Gram matrix of an updated block, and (flag) the DGKS criterion (Daniel, Gragg, Kaufman &
// Stewart 1976): a second Gram-Schmidt pass is needed when some column kept less than eta of
// its norm through the first pass.
template <int BS>
struct FinishGram {
  static constexpr bool kOn = true;
  double* G;
  const double* before; // Gram matrix before the pass
  double eta2;
  int* flag; // null: no test
  __device__ void operator()(const double* sum) const
  {
    for (int e = threadIdx.x; e < BS * BS; e += kThreads) G[e] = sum[e];
    if (flag && threadIdx.x < 32) {
      const int c = threadIdx.x;
      const bool lost = c < BS && sum[c * BS + c] < eta2 * before[c * BS + c];
      const unsigned any = __ballot_sync(0xffffffffu, lost);
      if (c == 0) *flag = any != 0;
    }
  }
};

// sum = [E; G] = [S, W]^T W. flag = ||E||_F^2 > thr2 * trace(G): the sketch S^T W says W's components
// along the basis exceed thr relative to W's norm. With `pair` (a word kept across calls), a step
// whose test fired also projects the next one: pair = this step's test. G goes to both outputs
// (G: the answer unless a pass runs; before: what the DGKS test compares with), and flag2 (the
// second pass) is cleared, since the first pass may not run.
template <int BS>
struct FinishSketch {
  static constexpr bool kOn = true;
  double *G, *before;
  double thr2;
  int *flag, *flag2, *pair;
  __device__ void operator()(const double* sum) const
  {
    constexpr int BB = BS * BS;
    for (int e = threadIdx.x; e < BB; e += kThreads) G[e] = before[e] = sum[BB + e];
    if (threadIdx.x < 32) {
      const int lane = threadIdx.x;
      double e2 = 0.0, tr = 0.0;
      for (int e = lane; e < BB; e += 32) e2 = fma(sum[e], sum[e], e2);
      for (int c = lane; c < BS; c += 32) tr += sum[BB + c * BS + c];
      for (int o = 16; o > 0; o >>= 1) {
        e2 += __shfl_xor_sync(0xffffffffu, e2, o);
        tr += __shfl_xor_sync(0xffffffffu, tr, o);
      }
      if (lane == 0) {
        const int fired = !(e2 <= thr2 * tr); // NaN counts as loss
        int f = fired;
        if (pair) {
          f |= (*pair != 0) ? 2 : 0; // bit 1: forced by the previous step
          *pair = fired;
        }
        *flag = f;
        *flag2 = 0;
      }
    }
  }
};

// ---------------------------------------------------------------- block dot
// C_j = V_j^T W, j < nblk. Grid: x = chunk of JC blocks, y = chunk of rows.
// A warp takes G groups of 4 rows per iteration. All operand loads of the iteration are
// issued before the first DMMA (block indices beyond nblk are clamped to a valid block and
// their products discarded), so each warp keeps G*(JC+1)*NT 256-byte loads in flight.
// Per group: one DMMA m8n8k4 per (j, 8x8 output tile). Per-CTA sums go to
// partial[row_chunk][j][BS*BS]; k_reduce_partials adds the row chunks in a fixed order, or (Fin,
// nblk = JC, one chunk of blocks) the last CTA does.
template <typename T, int BS, int JC, int G, class Fin>
__global__ void __launch_bounds__(kThreads) k_block_dot(const T* __restrict__ V, int64_t vstride, int nblk, const T* __restrict__ W, int64_t n, int64_t rows_per_cta,
                                                        double* __restrict__ partial, const int* __restrict__ cond, Tickets tickets, Fin fin)
{
  ::trl_detail::pdl_enter();
  if (cond && *cond == 0) return; // device-side skip (uniform over the grid)
  constexpr int NT = (BS + 7) / 8;
  constexpr int BB = BS * BS;
  __shared__ double red[kWarps][NT * NT * 64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int j0 = blockIdx.x * JC;
  const int64_t rb = static_cast<int64_t>(blockIdx.y) * rows_per_cta;
  const int64_t re = min(n, rb + rows_per_cta);

  double acc[JC][NT][NT][2];
#pragma unroll
  for (int jj = 0; jj < JC; ++jj)
#pragma unroll
    for (int a = 0; a < NT; ++a)
#pragma unroll
      for (int b = 0; b < NT; ++b) acc[jj][a][b][0] = acc[jj][a][b][1] = 0.0;

  const T* Vb[JC];
#pragma unroll
  for (int jj = 0; jj < JC; ++jj) Vb[jj] = V + static_cast<int64_t>(min(j0 + jj, nblk - 1)) * vstride;

  for (int64_t r0 = rb + warp * 4 * G; r0 < re; r0 += kWarps * 4 * G) {
    double bf[G][NT];
    double av[G][JC][NT];
#pragma unroll
    for (int q = 0; q < G; ++q) {
      const int64_t row = r0 + q * 4 + t4;
      const bool rok = row < re;
#pragma unroll
      for (int tk = 0; tk < NT; ++tk) {
        const int col = tk * 8 + g;
        bf[q][tk] = (rok && col < BS) ? ld_widen(W + row * BS + col) : 0.0;
      }
#pragma unroll
      for (int jj = 0; jj < JC; ++jj)
#pragma unroll
        for (int ti = 0; ti < NT; ++ti) {
          const int col = ti * 8 + g;
          av[q][jj][ti] = (rok && col < BS) ? ld_widen(Vb[jj] + row * BS + col) : 0.0;
        }
    }
#pragma unroll
    for (int q = 0; q < G; ++q)
#pragma unroll
      for (int jj = 0; jj < JC; ++jj) {
        if (j0 + jj < nblk) {
#pragma unroll
          for (int ti = 0; ti < NT; ++ti)
#pragma unroll
            for (int tk = 0; tk < NT; ++tk) dmma_m8n8k4(acc[jj][ti][tk][0], acc[jj][ti][tk][1], av[q][jj][ti], bf[q][tk]);
        }
      }
  }

  // cross-warp reduction, one block j at a time
#pragma unroll
  for (int jj = 0; jj < JC; ++jj) {
    if (j0 + jj >= nblk) break;
#pragma unroll
    for (int ti = 0; ti < NT; ++ti)
#pragma unroll
      for (int tk = 0; tk < NT; ++tk) {
        red[warp][(ti * NT + tk) * 64 + g * 8 + 2 * t4 + 0] = acc[jj][ti][tk][0];
        red[warp][(ti * NT + tk) * 64 + g * 8 + 2 * t4 + 1] = acc[jj][ti][tk][1];
      }
    __syncthreads();
    for (int e = threadIdx.x; e < NT * NT * 64; e += kThreads) {
      const int tile = e >> 6, within = e & 63;
      const int row = (tile / NT) * 8 + (within >> 3);
      const int col = (tile % NT) * 8 + (within & 7);
      if (row < BS && col < BS) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) s += red[w][e];
        partial[(static_cast<int64_t>(blockIdx.y) * nblk + j0 + jj) * BB + row * BS + col] = s;
      }
    }
    __syncthreads();
  }
  if constexpr (Fin::kOn) {
    constexpr int LEN = JC * BB;
    static_assert(LEN + kThreads <= kWarps * NT * NT * 64, "totals and scratch fit the reduction buffer");
    double* sum = &red[0][0];
    if (last_cta_sum<LEN>(partial, static_cast<int>(gridDim.y), static_cast<int>(blockIdx.y), tickets, sum, sum + LEN)) fin(sum);
  }
}

// ---------------------------------------------------------------- block dot, bulk-copy pipeline
// Same result as k_block_dot, for BS*sizeof(T) a multiple of 16 bytes. The CTA walks its
// row range in tiles of R rows (2 to 8 KB per block tile). Thread 0 streams the W tile and the
// tiles of the JC blocks of V into an S-stage shared-memory ring with 1-D bulk copies that
// complete on a per-stage "full" mbarrier; the 8 warps read DMMA fragments from shared
// memory and release the stage on its "empty" mbarrier. HBM traffic is a continuous stream
// of copies, independent of register pressure and of the element width.
// Waits are bounded (mbar_wait): on a timeout the status word records TRL_DEV_TIMEOUT, the
// threads leave the tile loop, and thread 0 waits (bounded) for the copies it issued.
template <typename T, int BS, int TB>
struct BulkTile {
  static constexpr int R = TB / (BS * static_cast<int>(sizeof(T))); // rows per tile (TB bytes per block tile)
  // Rows of 128 bytes: the four rows of a fragment load would share their shared-memory banks (4-way
  // conflicts, a wavefront per cycle at the DMMA's full rate). They are taken from SUB pieces of the tile
  // instead, which lie 32 bytes apart modulo 128 (B200, 300,001 x 16 FP64, 12 blocks: 110 -> 90 us; the
  // bytes take 76).
  static constexpr int SUB = BS * sizeof(T) >= 128 ? 4 : 1;
  static constexpr int SROWS = R / SUB; // rows per piece
  static constexpr int PIECE = SROWS * BS + (SUB > 1 ? 32 / static_cast<int>(sizeof(T)) : 0);
  static constexpr int ELEMS = SUB * PIECE;
};

template <typename T, int BS, int JC, int S, int TB>
__global__ void __launch_bounds__(kThreads) k_block_dot_bulk(const T* __restrict__ V, int64_t vstride, int nblk, const T* __restrict__ W, int64_t n, int64_t rows_per_cta,
                                                             double* __restrict__ partial, int* status, const int* __restrict__ cond)
{
  ::trl_detail::pdl_enter();
  if (cond && *cond == 0) return; // device-side skip (uniform over the grid)
  constexpr int NT = (BS + 7) / 8;
  constexpr int BB = BS * BS;
  constexpr int R = BulkTile<T, BS, TB>::R;
  constexpr int TILE = BulkTile<T, BS, TB>::ELEMS;
  constexpr int SUB = BulkTile<T, BS, TB>::SUB, SROWS = BulkTile<T, BS, TB>::SROWS, PIECE = BulkTile<T, BS, TB>::PIECE;
  constexpr int GPW = R / (kWarps * 4); // 4-row groups per warp per tile
  static_assert(GPW >= 1 && R % (kWarps * 4) == 0, "tile rows must cover the CTA's warps");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  T* tiles = reinterpret_cast<T*>(smem_raw); // [S][JC + 1][TILE]: slot 0 is W
  uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw + static_cast<size_t>(S) * (JC + 1) * TILE * sizeof(T));
  uint64_t* empty = full + S;
  __shared__ double red[kWarps][NT * NT * 64];

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int j0 = blockIdx.x * JC;
  const int jn = min(JC, nblk - j0);
  const int64_t rb = static_cast<int64_t>(blockIdx.y) * rows_per_cta;
  const int64_t re = min(n, rb + rows_per_cta);
  const int ntiles = re > rb ? static_cast<int>((re - rb + R - 1) / R) : 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kWarps);
    }
    mbar_init_fence();
  }
  __syncthreads();

  // one thread starts a tile's copies; with SUB pieces per block it is a warp (100,003 x 16 FP64, 20 blocks:
  // 53 us, by one thread 61)
  const bool issuer = SUB > 1 ? warp == 0 : threadIdx.x == 0;
  int issued = 0; // by the issuer: tiles whose copies were started
  auto issue = [&](int t) {
    const int s = t % S;
    const int64_t r0 = rb + static_cast<int64_t>(t) * R;
    const int rows = static_cast<int>(min(static_cast<int64_t>(R), re - r0));
    const uint32_t bytes = static_cast<uint32_t>(rows * BS * sizeof(T));
    T* st = tiles + static_cast<size_t>(s) * (JC + 1) * TILE;
    if (threadIdx.x == 0) mbar_arrive_expect_tx(&full[s], bytes * static_cast<uint32_t>(jn + 1));
    if constexpr (SUB == 1) {
      bulk_g2s(st, W + r0 * BS, bytes, &full[s]);
      for (int jj = 0; jj < jn; ++jj) bulk_g2s(st + (jj + 1) * TILE, V + static_cast<int64_t>(j0 + jj) * vstride + r0 * BS, bytes, &full[s]);
    }
    else {
      __syncwarp();
      for (int e = lane; e < (jn + 1) * SUB; e += 32) {
        const int jj = e / SUB - 1, first = e % SUB * SROWS;
        const T* from = jj < 0 ? W : V + static_cast<int64_t>(j0 + jj) * vstride;
        if (first < rows) bulk_g2s(st + (jj + 1) * TILE + e % SUB * PIECE, from + (r0 + first) * BS, static_cast<uint32_t>(min(SROWS, rows - first) * BS * sizeof(T)), &full[s]);
      }
    }
    issued = t + 1;
  };
  if (issuer)
    for (int t = 0; t < min(S - 1, ntiles); ++t) issue(t);

  double acc[JC][NT][NT][2];
#pragma unroll
  for (int jj = 0; jj < JC; ++jj)
#pragma unroll
    for (int a = 0; a < NT; ++a)
#pragma unroll
      for (int b = 0; b < NT; ++b) acc[jj][a][b][0] = acc[jj][a][b][1] = 0.0;

  int consumed = 0;
  for (int t = 0; t < ntiles; ++t) {
    if (issuer && t + S - 1 < ntiles) {
      const int tn = t + S - 1; // refill the slot that tile t-1 used
      bool vacant = tn < S || mbar_wait(&empty[tn % S], static_cast<uint32_t>((tn - S) / S) & 1u, status);
      if constexpr (SUB > 1) vacant = __all_sync(0xffffffffu, vacant);
      if (vacant) issue(tn);
    }
    const int s = t % S;
    bool there = mbar_wait(&full[s], static_cast<uint32_t>(t / S) & 1u, status);
    if constexpr (SUB > 1) there = __all_sync(0xffffffffu, there); // the whole warp leaves or none of it: it issues together
    if (!there) break;
    const T* st = tiles + static_cast<size_t>(s) * (JC + 1) * TILE;
    const int rows = static_cast<int>(min(static_cast<int64_t>(R), re - (rb + static_cast<int64_t>(t) * R)));
#pragma unroll
    for (int q = 0; q < GPW; ++q) {
      const int lr = SUB > 1 ? t4 * SROWS + warp * GPW + q : (warp * GPW + q) * 4 + t4;
      const int at = SUB > 1 ? t4 * PIECE + (warp * GPW + q) * BS : lr * BS;
      const bool rok = lr < rows;
      double bf[NT];
#pragma unroll
      for (int tk = 0; tk < NT; ++tk) {
        const int col = tk * 8 + g;
        bf[tk] = (rok && col < BS) ? static_cast<double>(st[at + col]) : 0.0;
      }
#pragma unroll
      for (int jj = 0; jj < JC; ++jj) {
        if (jj < jn) {
#pragma unroll
          for (int ti = 0; ti < NT; ++ti) {
            const int col = ti * 8 + g;
            const double a = (rok && col < BS) ? static_cast<double>(st[(jj + 1) * TILE + at + col]) : 0.0;
#pragma unroll
            for (int tk = 0; tk < NT; ++tk) dmma_m8n8k4(acc[jj][ti][tk][0], acc[jj][ti][tk][1], a, bf[tk]);
          }
        }
      }
    }
    __syncwarp(); // the DMMAs above consumed every lane's shared-memory reads
    if (lane == 0) mbar_arrive(&empty[s]);
    consumed = t + 1;
  }
  if (threadIdx.x == 0) // after an aborted loop: let the copies already started land
    for (int t = consumed; t < issued; ++t) mbar_wait(&full[t % S], static_cast<uint32_t>(t / S) & 1u, status, 1u << 20);

#pragma unroll
  for (int jj = 0; jj < JC; ++jj) {
    if (jj >= jn) break;
#pragma unroll
    for (int ti = 0; ti < NT; ++ti)
#pragma unroll
      for (int tk = 0; tk < NT; ++tk) {
        red[warp][(ti * NT + tk) * 64 + g * 8 + 2 * t4 + 0] = acc[jj][ti][tk][0];
        red[warp][(ti * NT + tk) * 64 + g * 8 + 2 * t4 + 1] = acc[jj][ti][tk][1];
      }
    __syncthreads();
    for (int e = threadIdx.x; e < NT * NT * 64; e += kThreads) {
      const int tile = e >> 6, within = e & 63;
      const int row = (tile / NT) * 8 + (within >> 3);
      const int col = (tile % NT) * 8 + (within & 7);
      if (row < BS && col < BS) {
        double sum = 0.0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) sum += red[w][e];
        partial[(static_cast<int64_t>(blockIdx.y) * nblk + j0 + jj) * BB + row * BS + col] = sum;
      }
    }
    __syncthreads();
  }
}

// Sum of partial[c][e] over the chunks c = s, s + SL, s + 2 SL, ... of one slice. Eight
// loads are issued before the adds that consume them (a thread issues in order, so each
// batch is one dependent memory round: ~600 partials take 3 rounds, not 5); eight
// accumulators, combined in a fixed tree, so the result does not depend on scheduling.
template <int SL>
__device__ __forceinline__ double slice_sum(const double* __restrict__ partial, int chunks, int64_t len, int64_t e, int s)
{
  constexpr int U = 8;
  double a[U];
#pragma unroll
  for (int u = 0; u < U; ++u) a[u] = 0.0;
  for (int c = s; c < chunks; c += U * SL) {
    double v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int cu = c + u * SL;
      v[u] = cu < chunks ? partial[static_cast<int64_t>(cu) * len + e] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) a[u] += v[u];
  }
  return ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]));
}

// out[e] = sum_c partial[c][e]: OPC outputs per CTA, SL = 1024 / OPC slices of the chunk
// range per output (slice_sum); the slices are combined in a fixed order, so the result
// does not depend on scheduling. OPC = 32 for long outputs (one warp per slice, coalesced);
// OPC = 8 for short ones (the b x b blocks of one or a few basis blocks): eight times the
// CTAs and a quarter of the loads per thread, so that ~600 partials take one memory round.
constexpr int kRedThreads = 1024;
template <int OPC>
__global__ void __launch_bounds__(kRedThreads) k_reduce_partials(const double* __restrict__ partial, int chunks, int64_t len, double* __restrict__ out,
                                                                 const int* __restrict__ cond)
{
  ::trl_detail::pdl_enter();
  if (cond && *cond == 0) return;
  constexpr int SL = kRedThreads / OPC;
  __shared__ double part[SL][OPC + 1];
  const int o = threadIdx.x % OPC, s = threadIdx.x / OPC;
  const int64_t e = static_cast<int64_t>(blockIdx.x) * OPC + o;
  part[s][o] = e < len ? slice_sum<SL>(partial, chunks, len, e, s) : 0.0;
  __syncthreads();
  if (s == 0 && e < len) {
    double t = 0.0;
#pragma unroll 8
    for (int q = 0; q < SL; ++q) t += part[q][o];
    out[e] = t;
  }
}

// Launches the fixed-order reduction of `chunks` partial rows of `len` doubles into out.
inline cudaError_t launch_reduce(cudaStream_t stream, const double* partial, int64_t chunks, int64_t len, double* out, const int* cond)
{
  if (len <= 1024 && chunks > 128)
    return ::trl_detail::launch(k_reduce_partials<8>, static_cast<unsigned>((len + 7) / 8), kRedThreads, 0, stream, partial, static_cast<int>(chunks), len, out, cond);
  return ::trl_detail::launch(k_reduce_partials<32>, static_cast<unsigned>((len + 31) / 32), kRedThreads, 0, stream, partial, static_cast<int>(chunks), len, out, cond);
}

// ---------------------------------------------------------------- block GEMM
// out_j = (accumulate ? out_j : 0) + sign * sum_{i<MB} in_i * Coef(i, j)   for j < NB <= NBMAX
// Coef(i, j) = coef + (i*ldc + j)*BS*BS (row-major BS x BS, or its transpose).
// A warp owns RT 8-row tiles at a time and walks the input blocks U at a time: the
// A-fragment loads of U blocks x RT tiles (from `in`, HBM) are all issued before the DMMAs
// that consume them (indices past MB are clamped and their products skipped). B fragments
// come from the tiny coefficient array (L1-resident) and are shared by the RT tiles.
// `in` and `out` may alias when MB = NB = 1 (in-place X <- X U^{-1}): a warp reads all its
// rows before it writes them, and no other warp touches those rows.
template <typename T, int BS, int NBMAX, int RT, int U>
__global__ void __launch_bounds__(kThreads) k_block_gemm(const T* in, int64_t istride, int MB, const double* __restrict__ coef, int ldc, int transpose_coef, T* out,
                                                         int64_t ostride, int NB, int64_t n, int accumulate, double sign)
{
  ::trl_detail::pdl_enter();
  constexpr int NT = (BS + 7) / 8;
  constexpr int KS = (BS + 3) / 4;
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2, t4 = lane & 3;
  const int64_t warp_global = static_cast<int64_t>(blockIdx.x) * kWarps + (threadIdx.x >> 5);
  const int64_t warp_stride = static_cast<int64_t>(gridDim.x) * kWarps;

  for (int64_t r0 = warp_global * 8 * RT; r0 < n; r0 += warp_stride * 8 * RT) {
    double acc[RT][NBMAX][NT][2];
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      const int64_t row = r0 + r * 8 + g;
      const bool rok = row < n;
#pragma unroll
      for (int jb = 0; jb < NBMAX; ++jb)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int col = t * 8 + 2 * t4 + i;
            acc[r][jb][t][i] = (accumulate && jb < NB && rok && col < BS) ? static_cast<double>(out[jb * ostride + row * BS + col]) : 0.0;
          }
    }

    for (int ib0 = 0; ib0 < MB; ib0 += U) {
      double a[U][RT][KS];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const T* A = in + static_cast<int64_t>(min(ib0 + u, MB - 1)) * istride;
#pragma unroll
        for (int r = 0; r < RT; ++r) {
          const int64_t row = r0 + r * 8 + g;
#pragma unroll
          for (int ks = 0; ks < KS; ++ks) {
            const int kcol = ks * 4 + t4;
            a[u][r][ks] = (row < n && kcol < BS) ? static_cast<double>(A[row * BS + kcol]) : 0.0;
          }
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (ib0 + u < MB) {
          const double* Crow = coef + static_cast<int64_t>(ib0 + u) * ldc * (BS * BS);
#pragma unroll
          for (int ks = 0; ks < KS; ++ks)
#pragma unroll
            for (int jb = 0; jb < NBMAX; ++jb) {
              if (jb < NB) {
                const double* Cb = Crow + jb * (BS * BS);
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                  const int krow = ks * 4 + t4, ncol = t * 8 + g;
                  double b = 0.0;
                  if (krow < BS && ncol < BS) b = sign * __ldg(transpose_coef ? Cb + ncol * BS + krow : Cb + krow * BS + ncol);
#pragma unroll
                  for (int r = 0; r < RT; ++r) dmma_m8n8k4(acc[r][jb][t][0], acc[r][jb][t][1], a[u][r][ks], b);
                }
              }
            }
        }
      }
    }

#pragma unroll
    for (int r = 0; r < RT; ++r) {
      const int64_t row = r0 + r * 8 + g;
#pragma unroll
      for (int jb = 0; jb < NBMAX; ++jb)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int col = t * 8 + 2 * t4 + i;
            if (jb < NB && row < n && col < BS) out[jb * ostride + row * BS + col] = static_cast<T>(acc[r][jb][t][i]);
          }
    }
  }
}

// ---------------------------------------------------------------- restart rotation
// W_j = sum_{i<m} V_i Y(i,j) for the output columns [c0, c0 + 8*NTC) of the N = k*BS columns
// (one chunk of output columns per launch). As a GEMM, out[rows x N] = V[rows x K] * Yhat[K x N]
// with K = m*BS: 2*n*K*N flops over (K + N)*n elements, ~9 flop/B at the thick restart's
// shapes, so the kernel is bound by the FP64 DMMA rate rather than by HBM.
// The chunk of Yhat lives in shared memory in DMMA B-fragment order (for every k-step of 4
// rows and n-tile of 8 columns the 32 values in lane order: one conflict-free 256-byte load
// per fragment) and is loaded once per CTA. Each warp owns RT tiles of 8 rows and streams the
// m input blocks through a register ring D blocks deep, so every load is issued D blocks
// before the DMMAs that consume it.
constexpr int kRotThreads = 512;

template <typename T, int BS, int NTC, int RT, int D>
__global__ void __launch_bounds__(kRotThreads, 1) k_rotate(const T* __restrict__ V, int64_t vstride, int m, const double* __restrict__ Y, int ldy, int N, int c0,
                                                           T* __restrict__ W, int64_t wstride, int64_t n)
{
  ::trl_detail::pdl_enter();
  constexpr int KSB = BS / 4; // k-steps per input block
  extern __shared__ double sY[];
  const int ks_total = m * KSB;
  for (int idx = threadIdx.x; idx < ks_total * NTC * 32; idx += blockDim.x) {
    const int ln = idx & 31, f = idx >> 5;
    const int nt = f % NTC, ks = f / NTC;
    const int krow = ks * 4 + (ln & 3), col = c0 + nt * 8 + (ln >> 2);
    double v = 0.0;
    if (col < N) {
      const int i = krow / BS, r = krow % BS, j = col / BS, cc = col % BS;
      v = Y[(static_cast<int64_t>(i) * ldy + j) * (BS * BS) + r * BS + cc];
    }
    sY[idx] = v;
  }
  __syncthreads();

  const int lane = threadIdx.x & 31;
  const int g = lane >> 2, t4 = lane & 3;
  const int64_t warp = static_cast<int64_t>(blockIdx.x) * (kRotThreads / 32) + (threadIdx.x >> 5);
  const int64_t nwarps = static_cast<int64_t>(gridDim.x) * (kRotThreads / 32);

  for (int64_t r0 = warp * 8 * RT; r0 < n; r0 += nwarps * 8 * RT) {
    double acc[RT][NTC][2];
#pragma unroll
    for (int rt = 0; rt < RT; ++rt)
#pragma unroll
      for (int nt = 0; nt < NTC; ++nt) acc[rt][nt][0] = acc[rt][nt][1] = 0.0;

    double a[D][RT][KSB];
    auto load = [&](double(&dst)[RT][KSB], int blk) {
#pragma unroll
      for (int rt = 0; rt < RT; ++rt) {
        const int64_t row = r0 + rt * 8 + g;
#pragma unroll
        for (int ks = 0; ks < KSB; ++ks)
          dst[rt][ks] = (blk < m && row < n) ? static_cast<double>(V[static_cast<int64_t>(blk) * vstride + row * BS + ks * 4 + t4]) : 0.0;
      }
    };
#pragma unroll
    for (int d = 0; d < D; ++d) load(a[d], d);

    for (int ib = 0; ib < m; ib += D) {
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const int i = ib + d;
        if (i < m) {
#pragma unroll
          for (int ks = 0; ks < KSB; ++ks) {
            const double* bf = sY + static_cast<size_t>((i * KSB + ks) * NTC) * 32 + lane;
#pragma unroll
            for (int nt = 0; nt < NTC; ++nt) {
              const double b = bf[nt * 32];
#pragma unroll
              for (int rt = 0; rt < RT; ++rt) dmma_m8n8k4(acc[rt][nt][0], acc[rt][nt][1], a[d][rt][ks], b);
            }
          }
        }
        load(a[d], i + D);
      }
    }

#pragma unroll
    for (int rt = 0; rt < RT; ++rt) {
      const int64_t row = r0 + rt * 8 + g;
      if (row >= n) continue;
#pragma unroll
      for (int nt = 0; nt < NTC; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int col = c0 + nt * 8 + 2 * t4 + e;
          if (col < N) W[static_cast<int64_t>(col / BS) * wstride + row * BS + (col % BS)] = static_cast<T>(acc[rt][nt][e]);
        }
    }
  }
}

// KS adjacent elements p[0..KS) (p aligned to KS * sizeof(T) when that is 8 or 16 bytes),
// in as few loads as possible; columns past BS are never requested.
template <typename T, int KS>
__device__ __forceinline__ void load_cols(const T* p, T (&v)[KS])
{
  if constexpr (sizeof(T) == 8 && KS == 2) {
    const double2 q = *reinterpret_cast<const double2*>(p);
    v[0] = q.x;
    v[1] = q.y;
  }
  else if constexpr (sizeof(T) == 8 && KS == 4) {
    const double2 q0 = *reinterpret_cast<const double2*>(p), q1 = *reinterpret_cast<const double2*>(p + 2);
    v[0] = q0.x;
    v[1] = q0.y;
    v[2] = q1.x;
    v[3] = q1.y;
  }
  else if constexpr (sizeof(T) == 4 && KS == 2) {
    const float2 q = *reinterpret_cast<const float2*>(p);
    v[0] = q.x;
    v[1] = q.y;
  }
  else if constexpr (sizeof(T) == 4 && KS == 4) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    v[0] = q.x;
    v[1] = q.y;
    v[2] = q.z;
    v[3] = q.w;
  }
  else {
#pragma unroll
    for (int i = 0; i < KS; ++i) v[i] = p[i];
  }
}

// ---------------------------------------------------------------- update + Gram in one pass
// out = (accumulate ? out : 0) + sign * sum_{i<MB} in_i Coef(i),  Coef(i) = coef + i*BS*BS,
// and in the same pass the Gram matrix out^T out of the values as stored (rounded to T):
// each warp stages its finished rows in shared memory, re-reads them in DMMA fragment
// layout (k = rows) and accumulates the BS x BS Gram; per-CTA sums go to
// gram_partial[blockIdx.x][BS*BS], added up by the last CTA. When cond is given and *cond == 0
// the kernel does nothing (a device-side decision: no host round trip).
template <typename T, int BS, int RT, int U, class Fin>
__global__ void __launch_bounds__(kThreads, BS == 16 ? 2 : 0) k_update_gram(const T* in, int64_t istride, int MB, const double* __restrict__ coef, T* out, int64_t n,
                                                          int accumulate, double sign, double* __restrict__ gram_partial, const int* __restrict__ cond, Tickets tickets, Fin fin)
{
  ::trl_detail::pdl_enter();
  if (cond && *cond == 0) return;
  // input blocks per loop body, without which ptxas picks worse ones from kernel to kernel.
  // Measured on B200 (one projection, 884,736 rows, 2 / 3 blocks): FP64 bs 2 175 / 183 us, 4 285 / 319, 8
  // 462 / 511; FP32 bs 1 195 / 182, 2 415 / 393, 4 265 / 220, 8 286 / 295; FP64 bs 1, 24 blocks (3 / 4) 258 / 225.
  // ptxas's schedule hangs on the form of this loop: with `accumulate`, `sign` and U, which have one value each,
  // taken out, FP64 bs 2 and 24 blocks took 377 us in place of 218, bs 4 322 in place of 259.
  constexpr int kUnroll = sizeof(T) == 4 ? (BS <= 4 ? 3 : 2) : (BS == 1 ? 4 : 2);
  constexpr int NT = (BS + 7) / 8;
  constexpr int KS = (BS + 3) / 4;
  __shared__ double stage[kWarps][RT * 8 * BS];
  __shared__ double red[kWarps][NT * NT * 64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int64_t warp_global = static_cast<int64_t>(blockIdx.x) * kWarps + warp;
  const int64_t warp_stride = static_cast<int64_t>(gridDim.x) * kWarps;
  double gacc[NT][NT][2];
#pragma unroll
  for (int a = 0; a < NT; ++a)
#pragma unroll
    for (int b = 0; b < NT; ++b) gacc[a][b][0] = gacc[a][b][1] = 0.0;

  for (int64_t r0 = warp_global * 8 * RT; r0 < n; r0 += warp_stride * 8 * RT) {
    double acc[RT][NT][2];
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      const int64_t row = r0 + r * 8 + g;
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int col = t * 8 + 2 * t4 + i;
          acc[r][t][i] = (accumulate && row < n && col < BS) ? static_cast<double>(out[row * BS + col]) : 0.0;
        }
    }
#pragma unroll(kUnroll)
    for (int ib0 = 0; ib0 < MB; ib0 += U) {
      // k is permuted so that lane t4 owns the KS adjacent columns t4*KS .. t4*KS+KS-1 of
      // its row (one vector load); the values stay in the storage type until the DMMA
      T a[U][RT][KS];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const T* A = in + static_cast<int64_t>(min(ib0 + u, MB - 1)) * istride;
#pragma unroll
        for (int r = 0; r < RT; ++r) {
          const int64_t row = r0 + r * 8 + g;
          if (row < n && t4 * KS < BS) load_cols<T, KS>(A + row * BS + t4 * KS, a[u][r]);
          else
#pragma unroll
            for (int ks = 0; ks < KS; ++ks) a[u][r][ks] = T(0);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (ib0 + u < MB) {
          const double* Cb = coef + static_cast<int64_t>(ib0 + u) * (BS * BS);
#pragma unroll
          for (int ks = 0; ks < KS; ++ks)
#pragma unroll
            for (int t = 0; t < NT; ++t) {
              const int krow = t4 * KS + ks, ncol = t * 8 + g;
              const double b = (krow < BS && ncol < BS) ? sign * __ldg(Cb + krow * BS + ncol) : 0.0;
#pragma unroll
              for (int r = 0; r < RT; ++r) dmma_m8n8k4(acc[r][t][0], acc[r][t][1], static_cast<double>(a[u][r][ks]), b);
            }
        }
      }
    }
    // store, and stage the stored values for the Gram
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      const int64_t row = r0 + r * 8 + g;
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int col = t * 8 + 2 * t4 + i;
          if (col < BS) {
            const T v = static_cast<T>(acc[r][t][i]);
            if (row < n) out[row * BS + col] = v;
            stage[warp][(r * 8 + g) * BS + col] = row < n ? static_cast<double>(v) : 0.0;
          }
        }
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 2 * RT; ++q) { // groups of 4 staged rows = the DMMA k dimension
      const int lr = q * 4 + t4;
      double bf[NT];
#pragma unroll
      for (int tk = 0; tk < NT; ++tk) bf[tk] = (tk * 8 + g < BS) ? stage[warp][lr * BS + tk * 8 + g] : 0.0;
#pragma unroll
      for (int ti = 0; ti < NT; ++ti) {
        const double av = (ti * 8 + g < BS) ? stage[warp][lr * BS + ti * 8 + g] : 0.0;
#pragma unroll
        for (int tk = 0; tk < NT; ++tk) dmma_m8n8k4(gacc[ti][tk][0], gacc[ti][tk][1], av, bf[tk]);
      }
    }
    __syncwarp();
  }
  // cross-warp reduction of the Gram
#pragma unroll
  for (int ti = 0; ti < NT; ++ti)
#pragma unroll
    for (int tk = 0; tk < NT; ++tk) {
      red[warp][(ti * NT + tk) * 64 + g * 8 + 2 * t4 + 0] = gacc[ti][tk][0];
      red[warp][(ti * NT + tk) * 64 + g * 8 + 2 * t4 + 1] = gacc[ti][tk][1];
    }
  __syncthreads();
  for (int e = threadIdx.x; e < NT * NT * 64; e += kThreads) {
    const int tile = e >> 6, within = e & 63;
    const int row = (tile / NT) * 8 + (within >> 3);
    const int col = (tile % NT) * 8 + (within & 7);
    if (row < BS && col < BS) {
      double s = 0.0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) s += red[w][e];
      gram_partial[static_cast<int64_t>(blockIdx.x) * BS * BS + row * BS + col] = s;
    }
  }
  __syncthreads();
  static_assert(BS * BS + kThreads <= kWarps * NT * NT * 64, "totals and scratch fit the reduction buffer");
  double* sum = &red[0][0];
  if (last_cta_sum<BS * BS>(gram_partial, static_cast<int>(gridDim.x), static_cast<int>(blockIdx.x), tickets, sum, sum + BS * BS)) fin(sum);
}

// ---------------------------------------------------------------- Cholesky-QR
// Shared memory of the factorisation: [G | I] under elimination, L, and the pivots' square roots.
template <int BS>
struct FactorSpace {
  double A[BS][2 * BS + 1];
  double L[BS][BS + 1];
  double root[BS];
};

// By the whole CTA: G = L L^T (reading the lower triangle), Ui = L^{-T}; L is left in f. Gaussian
// elimination of [G | I] without pivoting (the pivots d are those of Cholesky, L = (unit lower factor)
// D^{1/2}) gives the factor and its inverse in one chain of a division per column, a matrix entry or
// two per thread; the square roots come at the end, all at once. Rolled loops: the code runs once
// per CTA, and by one warp, unrolled, with a chain of its own for the inverse, it took 4,500 / 9,200
// / 20,500 cycles for 4 / 8 / 16 columns, most of them waiting for instructions; now 2,500
// / 4,100 / 9,200 (with a division per entry in place of the reciprocal: 2,600 / 4,400 / 10,800, and twice
// that where the code is cold).
// A row and column whose diagonal entry is below 2^-800 are scaled by 2^400 and the factor scaled back:
// a pivot's reciprocal would be out of range (columns of norm below 7e-155).
// false (uniform): a pivot was <= 0 or NaN; Ui is then the identity, which leaves an apply a no-op.
template <int BS>
__device__ __forceinline__ bool cta_factor(const double* G, FactorSpace<BS>& f, double* Ui)
{
  constexpr int COLS = 2 * BS;
  constexpr int PER = (BS * COLS + kThreads - 1) / kThreads; // entries per thread
  const auto minute = [&](int k) { return G[k * (BS + 1)] < 0x1p-800; };
  for (int e = threadIdx.x; e < BS * BS; e += kThreads) {
    const int r = e / BS, k = e % BS;
    f.A[r][k] = (k <= r ? G[e] : G[k * BS + r]) * (minute(r) ? 0x1p400 : 1.0) * (minute(k) ? 0x1p400 : 1.0);
    f.A[r][BS + k] = r == k ? 1.0 : 0.0;
  }
  bool ok = true;
  __syncthreads();
#pragma unroll 1
  for (int j = 0; j < BS; ++j) { // row j and column j are final: nobody writes them in this round
    const double d = f.A[j][j];
    ok = ok && d > 0.0;
    const double piv = d > 0.0 ? d : 1.0, inv = 1.0 / piv;
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const int e = threadIdx.x + q * kThreads, i = e / COLS, k = e % COLS;
      if (i > j && i < BS && k != j) {
        const double a = f.A[i][j];
        double m = a * inv;
        m = fma(fma(-m, piv, a), inv, m); // a / piv with its remainder added back
        f.A[i][k] = fma(-m, f.A[j][k], f.A[i][k]);
      }
      if (k == j && i < BS) f.L[i][j] = i < j ? 0.0 : (i == j ? piv : f.A[i][j]);
    }
    __syncthreads();
  }
  if (threadIdx.x < BS) f.root[threadIdx.x] = sqrt(f.L[threadIdx.x][threadIdx.x]); // the pivots
  __syncthreads();
  for (int e = threadIdx.x; e < BS * BS; e += kThreads) {
    const int r = e / BS, k = e % BS; // row r, column k of L, and of L^{-1}
    f.L[r][k] = (r == k ? f.root[k] : f.L[r][k] / f.root[k]) * (minute(r) ? 0x1p-400 : 1.0);
    Ui[k * BS + r] = ok ? (k <= r ? f.A[r][BS + k] / f.root[r] * (minute(k) ? 0x1p400 : 1.0) : 0.0) : (r == k ? 1.0 : 0.0);
  }
  __syncthreads();
  return ok;
}

// The factor's outputs, by the same CTA: Ui to global memory, and R <- L^T (first pass) or
// R <- L^T R (X_in = X_out R across passes). A breakdown leaves R and records TRL_DEV_CHOLESKY.
template <int BS>
__device__ __forceinline__ void cta_factor_store(bool ok, FactorSpace<BS>& f, const double* Ui, double* Uout, double* R, bool first, int* status)
{
  for (int e = threadIdx.x; e < BS * BS; e += kThreads) {
    Uout[e] = Ui[e];
    f.A[e / BS][e % BS] = first ? 0.0 : __ldcg(R + e); // R before (L2: another CTA may have written it)
  }
  if (!ok) {
    if (threadIdx.x == 0) atomicOr(status, TRL_DEV_CHOLESKY);
    return;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < BS * BS; e += kThreads) {
    const int i = e / BS, c = e % BS;
    double v = first && i <= c ? f.L[c][i] : 0.0;
    if (!first)
      for (int k = i; k <= c; ++k) v = fma(f.L[k][i], f.A[k][c], v);
    R[e] = v;
  }
}

// KS adjacent columns of a row in as few stores as possible (the counterpart of load_cols)
template <typename T, int KS>
__device__ __forceinline__ void store_cols(T* p, const T (&v)[KS])
{
  constexpr int VEC = KS * sizeof(T) > 16 ? 16 / static_cast<int>(sizeof(T)) : KS;
#pragma unroll
  for (int c = 0; c < KS; c += VEC) {
    T part[VEC];
#pragma unroll
    for (int i = 0; i < VEC; ++i) part[i] = v[c + i];
    ::trl_detail::store_vec<T, VEC>(p + c, part);
  }
}

// X's rows as a warp holds them: lane (g, t4) columns 8 t + 2 t4 and the next one of row g of an
// 8-row tile, which is at once the accumulator layout of a DMMA and, with the k dimension
// permuted, its A operand: the product with a factor feeds the next one without a move.
template <typename T, int BS>
struct CholTile {
  static constexpr int NT = (BS + 7) / 8;
  // pairs: X is aligned to two elements, so that a lane's two columns are one load
  static __device__ __forceinline__ void load(const T* X, int64_t row, int64_t n, int t4, bool pairs, double (&x)[NT][2])
  {
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const int col = t * 8 + 2 * t4;
      x[t][0] = x[t][1] = 0.0;
      if (row < n && col < BS) {
        if constexpr (BS >= 2) {
          T v[2];
          if (pairs) load_cols<T, 2>(X + row * BS + col, v);
          else {
            v[0] = X[row * BS + col];
            v[1] = X[row * BS + col + 1];
          }
          x[t][0] = static_cast<double>(v[0]);
          x[t][1] = static_cast<double>(v[1]);
        }
        else
          x[t][0] = static_cast<double>(X[row]);
      }
    }
  }
  // this lane's fragments of a factor U (shared memory, row-major)
  static __device__ __forceinline__ void fragments(const double* U, int g, int t4, double (&b)[NT][2][NT])
  {
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int c = 0; c < NT; ++c) {
          const int k = t * 8 + 2 * t4 + i, col = c * 8 + g;
          b[t][i][c] = (k < BS && col < BS) ? U[k * BS + col] : 0.0;
        }
  }
  // x <- x U, rounded to T as a stored block would be
  static __device__ __forceinline__ void apply(double (&x)[NT][2], const double (&b)[NT][2][NT])
  {
    double acc[NT][2];
#pragma unroll
    for (int c = 0; c < NT; ++c) acc[c][0] = acc[c][1] = 0.0;
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int c = 0; c < NT; ++c) dmma_m8n8k4(acc[c][0], acc[c][1], x[t][i], b[t][i][c]);
#pragma unroll
    for (int c = 0; c < NT; ++c) {
      x[c][0] = static_cast<double>(static_cast<T>(acc[c][0]));
      x[c][1] = static_cast<double>(static_cast<T>(acc[c][1]));
    }
  }
};

constexpr int kCholMaxPasses = 4;

// CholQR without storing the block between passes: the factors so far, U_0 ... U_{nf-1}, are applied to
// each row tile in registers (rounded to T after each, so the values are those of a stored
// block). With G0, nf is 1 and every CTA factors G0 for itself first (a few microseconds in
// place of a launch); CTA 0 keeps the outputs.
// GRAM: forms the Gram matrix of the result, and the last CTA factors it into U_nf. Otherwise the
// result is stored in place, and CholQR2 has read the block twice and written it once.
// Measured on B200, CholQR2 of 884,736 x 8 FP64 / 100,003 x 16 FP32: 34 / 33 us (before, with a
// launch per factor and the block stored between the passes: 57 / 61 us).
template <typename T, int BS, int RT, bool GRAM>
__global__ void __launch_bounds__(kThreads) k_cholqr(T* X, int64_t n, const double* __restrict__ G0, int nf, double* U, double* R, int* status, double* __restrict__ partial,
                                                     Tickets tickets)
{
  ::trl_detail::pdl_enter();
  using Tile = CholTile<T, BS>;
  constexpr int NT = Tile::NT;
  constexpr int BB = BS * BS;
  __shared__ double Us[kCholMaxPasses][BB];
  __shared__ FactorSpace<BS> fs;
  __shared__ double stage[GRAM ? kWarps : 1][GRAM ? RT * 8 * BS : 1];
  __shared__ double red[GRAM ? kWarps : 1][GRAM ? NT * NT * 64 : BB];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  if (G0) {
    double* Gs = &red[0][0];
    for (int e = threadIdx.x; e < BB; e += kThreads) Gs[e] = G0[e];
    __syncthreads();
    const bool ok = cta_factor<BS>(Gs, fs, Us[0]);
    if (blockIdx.x == 0) cta_factor_store<BS>(ok, fs, Us[0], U, R, true, status);
  }
  else
    for (int e = threadIdx.x; e < nf * BB; e += kThreads) Us[e / BB][e % BB] = U[e];
  __syncthreads();
  const bool pairs = reinterpret_cast<uintptr_t>(X) % (2 * sizeof(T)) == 0;
  double b0[NT][2][NT], b1[NT][2][NT]; // the first two factors in registers
  Tile::fragments(Us[0], g, t4, b0);
  if (nf > 1) Tile::fragments(Us[1], g, t4, b1);

  double gacc[NT][NT][2];
#pragma unroll
  for (int a = 0; a < NT; ++a)
#pragma unroll
    for (int b = 0; b < NT; ++b) gacc[a][b][0] = gacc[a][b][1] = 0.0;
  const int64_t warp_stride = static_cast<int64_t>(gridDim.x) * kWarps * 8 * RT;
  for (int64_t r0 = (static_cast<int64_t>(blockIdx.x) * kWarps + warp) * 8 * RT; r0 < n; r0 += warp_stride) {
    double x[RT][NT][2];
#pragma unroll
    for (int r = 0; r < RT; ++r) Tile::load(X, r0 + r * 8 + g, n, t4, pairs, x[r]);
#pragma unroll
    for (int r = 0; r < RT; ++r) Tile::apply(x[r], b0);
    if (nf > 1) {
#pragma unroll
      for (int r = 0; r < RT; ++r) Tile::apply(x[r], b1);
    }
    for (int f = 2; f < nf; ++f) {
      double bf[NT][2][NT];
      Tile::fragments(Us[f], g, t4, bf);
#pragma unroll
      for (int r = 0; r < RT; ++r) Tile::apply(x[r], bf);
    }
    if constexpr (!GRAM) {
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        const int64_t row = r0 + r * 8 + g;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const int col = t * 8 + 2 * t4;
          if (row < n && col < BS) {
            if constexpr (BS >= 2) {
              const T v[2] = {static_cast<T>(x[r][t][0]), static_cast<T>(x[r][t][1])};
              if (pairs) ::trl_detail::store_vec<T, 2>(X + row * BS + col, v);
              else {
                X[row * BS + col] = v[0];
                X[row * BS + col + 1] = v[1];
              }
            }
            else
              X[row] = static_cast<T>(x[r][t][0]);
          }
        }
      }
    }
    else {
      // rows past n are zero: they add nothing to the Gram
#pragma unroll
      for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int col = t * 8 + 2 * t4 + i;
            if (col < BS) stage[warp][(r * 8 + g) * BS + col] = x[r][t][i];
          }
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 2 * RT; ++q) { // groups of 4 staged rows = the DMMA k dimension
        const int lr = q * 4 + t4;
        double bf[NT];
#pragma unroll
        for (int tk = 0; tk < NT; ++tk) bf[tk] = (tk * 8 + g < BS) ? stage[warp][lr * BS + tk * 8 + g] : 0.0;
#pragma unroll
        for (int ti = 0; ti < NT; ++ti)
#pragma unroll
          for (int tk = 0; tk < NT; ++tk) dmma_m8n8k4(gacc[ti][tk][0], gacc[ti][tk][1], bf[ti], bf[tk]);
      }
      __syncwarp();
    }
  }
  if constexpr (GRAM) {
    __syncthreads(); // red held G0
#pragma unroll
    for (int ti = 0; ti < NT; ++ti)
#pragma unroll
      for (int tk = 0; tk < NT; ++tk) {
        red[warp][(ti * NT + tk) * 64 + g * 8 + 2 * t4 + 0] = gacc[ti][tk][0];
        red[warp][(ti * NT + tk) * 64 + g * 8 + 2 * t4 + 1] = gacc[ti][tk][1];
      }
    __syncthreads();
    for (int e = threadIdx.x; e < NT * NT * 64; e += kThreads) {
      const int tile = e >> 6, within = e & 63;
      const int row = (tile / NT) * 8 + (within >> 3);
      const int col = (tile % NT) * 8 + (within & 7);
      if (row < BS && col < BS) {
        double v = 0.0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) v += red[w][e];
        partial[static_cast<int64_t>(blockIdx.x) * BB + row * BS + col] = v;
      }
    }
    __syncthreads();
    double* sum = &red[0][0];
    if (last_cta_sum<BB>(partial, static_cast<int>(gridDim.x), static_cast<int>(blockIdx.x), tickets, sum, sum + BB)) {
      const bool ok = cta_factor<BS>(sum, fs, Us[0]);
      cta_factor_store<BS>(ok, fs, Us[0], U + nf * BB, R, false, status);
    }
  }
}

// The same for rows of up to 16 bytes: a thread per row, since of the 32 lanes that hold 8 rows above
// half or more would have nothing to load. Only the lower triangle of the Gram matrix is formed.
// Measured on B200, us, k_cholqr / this, two passes: 100,003 x 1 FP64 11.1 / 8.5, x 2 FP32 13.7 / 10.9, x 4 FP32
// 14.7 / 12.8; 884,736 x 2 FP32 32.9 / 13.9, x 4 FP32 34.9 / 24.5. (Rows of 32 bytes: 884,736 x 4 FP64
// 27.8 / 29.5, 5,000 x 4 9.1 / 10.0; a factor per launch and the block stored between the passes: 100,003 x 1
// 11.4, x 2 FP32 12.7, 884,736 x 2 FP32 31.3.)
template <typename T, int BS, int R, bool GRAM>
__global__ void __launch_bounds__(kThreads) k_cholqr_narrow(T* X, int64_t n, const double* __restrict__ G0, int nf, double* U, double* R_out, int* status,
                                                            double* __restrict__ partial, Tickets tickets)
{
  ::trl_detail::pdl_enter();
  constexpr int BB = BS * BS, TRI = BS * (BS + 1) / 2;
  __shared__ double Us[kCholMaxPasses][BB];
  __shared__ FactorSpace<BS> fs;
  __shared__ double Gs[BB];
  __shared__ double red[TRI + kThreads]; // totals, scratch
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (G0) {
    for (int e = tid; e < BB; e += kThreads) Gs[e] = G0[e];
    __syncthreads();
    const bool ok = cta_factor<BS>(Gs, fs, Us[0]);
    if (blockIdx.x == 0) cta_factor_store<BS>(ok, fs, Us[0], U, R_out, true, status);
  }
  else
    for (int e = tid; e < nf * BB; e += kThreads) Us[e / BB][e % BB] = U[e];
  __syncthreads();
  const bool whole = reinterpret_cast<uintptr_t>(X) % (BS * sizeof(T) < 16 ? BS * sizeof(T) : 16) == 0; // rows in as few loads as possible
  double gram[TRI];
#pragma unroll
  for (int e = 0; e < TRI; ++e) gram[e] = 0.0;
  const int64_t step = static_cast<int64_t>(gridDim.x) * kThreads * R;
  for (int64_t r0 = static_cast<int64_t>(blockIdx.x) * kThreads * R + tid; r0 < n; r0 += step) {
    T v[R][BS];
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int64_t row = r0 + q * kThreads;
#pragma unroll
      for (int c = 0; c < BS; ++c) v[q][c] = T(0);
      if (row < n) {
        if (whole) load_cols<T, BS>(X + row * BS, v[q]);
        else
#pragma unroll
          for (int c = 0; c < BS; ++c) v[q][c] = X[row * BS + c];
      }
    }
    for (int f = 0; f < nf; ++f) {
#pragma unroll
      for (int c = BS - 1; c >= 0; --c) { // the factor is upper triangular: column c needs the first c + 1
        double u[BS];
#pragma unroll
        for (int k = 0; k <= c; ++k) u[k] = Us[f][k * BS + c];
#pragma unroll
        for (int q = 0; q < R; ++q) {
          double s = 0.0;
#pragma unroll
          for (int k = 0; k <= c; ++k) s = fma(static_cast<double>(v[q][k]), u[k], s);
          v[q][c] = static_cast<T>(s); // rounded to T as a stored block would be
        }
      }
    }
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int64_t row = r0 + q * kThreads;
      if constexpr (GRAM) { // rows past n are zero
#pragma unroll
        for (int i = 0; i < BS; ++i)
#pragma unroll
          for (int k = 0; k <= i; ++k) gram[i * (i + 1) / 2 + k] = fma(static_cast<double>(v[q][i]), static_cast<double>(v[q][k]), gram[i * (i + 1) / 2 + k]);
      }
      else if (row < n) {
        if (whole) store_cols<T, BS>(X + row * BS, v[q]);
        else
#pragma unroll
          for (int c = 0; c < BS; ++c) X[row * BS + c] = v[q][c];
      }
    }
  }
  if constexpr (GRAM) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int e = 0; e < TRI; ++e) gram[e] += __shfl_xor_sync(0xffffffffu, gram[e], o);
    if (lane == 0)
#pragma unroll
      for (int e = 0; e < TRI; ++e) red[warp * TRI + e] = gram[e];
    __syncthreads();
    if (tid < TRI) {
      double v = 0.0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) v += red[w * TRI + tid];
      partial[static_cast<int64_t>(blockIdx.x) * TRI + tid] = v;
    }
    __syncthreads();
    if (last_cta_sum<TRI>(partial, static_cast<int>(gridDim.x), static_cast<int>(blockIdx.x), tickets, red, red + TRI)) {
      if (tid < BB) Gs[tid] = tid / BS >= tid % BS ? red[tid / BS * (tid / BS + 1) / 2 + tid % BS] : 0.0; // the factorisation reads the lower triangle
      __syncthreads();
      const bool ok = cta_factor<BS>(Gs, fs, Us[0]);
      cta_factor_store<BS>(ok, fs, Us[0], U + nf * BB, R_out, false, status);
    }
  }
}

// ---------------------------------------------------------------- projection in one launch
// W -= V (V^T W) against nblk blocks, the Gram matrix of the result, and a second time where a column
// kept less than eta of its norm, by one cooperative launch of a CTA per SM: CTA r owns a range of
// rows, and the sums over the CTAs go through global memory between grid-wide barriers. The separate
// kernels (dot, its reduction, update; each twice, and launched also when the sketch asks for nothing)
// cost more in launches than in work on small bases, and stream faster on large ones.
// cond: the sketch's decision. before: the Gram matrix before the pass.
// one_launch_projects has the times on both sides. (project_out always runs and keeps to the separate
// kernels, so that its modes agree to the last bit.)
constexpr int kProjThreads = 512;
constexpr int kProjWarps = kProjThreads / 32;
constexpr int kProjMaxEntries = 8192; // coefficients, nblk BS^2, in shared memory

template <typename T, int BS>
__global__ void __launch_bounds__(kProjThreads, 1) k_project(const T* V, int nblk, T* W, int64_t n, int64_t rows_per_cta, const int* __restrict__ cond,
                                                             const double* __restrict__ before, double eta2, double* __restrict__ G, double* partial, double* total,
                                                             double* gpartial, unsigned* bar, int* status)
{
  ::trl_detail::pdl_enter();
  if (*cond == 0) return; // the whole grid
  constexpr int NT = (BS + 7) / 8, KS = (BS + 3) / 4, BB = BS * BS;
  constexpr int JC = BS >= 16 ? 2 : 4; // blocks a warp takes at a time in the dots
  extern __shared__ __align__(16) double sm[];
  double* coef = sm;                             // [nblk BB]
  double* stage = coef + nblk * BB;              // [kProjWarps][8 BS]
  double* red = stage + kProjWarps * 8 * BS;     // [kProjWarps][NT NT 64]
  __shared__ double Gs[BB], G0[BB];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  const int64_t vstride = n * BS;
  const int64_t rb = min(n, static_cast<int64_t>(blockIdx.x) * rows_per_cta), re = min(n, rb + rows_per_cta);
  const int ncta = static_cast<int>(gridDim.x);

  // sum over the CTAs of src[c * stride + e], e = e0 .. e0 + 7, for a warp: lane (q, i) adds every 4th CTA's
  // entry e0 + i, eight loads in flight; lanes 0 .. 7 return the totals. One order of additions.
  const auto sum_ctas = [&](const double* src, int stride, int e0, int count) {
    const int i = lane & 7, q = lane >> 3;
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = 0.0;
    for (int c = q; c < ncta; c += 32)
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] += (c + 4 * u < ncta && e0 + i < count) ? __ldcg(src + static_cast<int64_t>(c + 4 * u) * stride + e0 + i) : 0.0;
    double t = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
    t += __shfl_xor_sync(0xffffffffu, t, 8);
    t += __shfl_xor_sync(0xffffffffu, t, 16);
    return t;
  };
  // total = V^T W. The CTA's warps are split into groups of up to JC blocks each, and what is left of
  // them over the rows.
  const auto dots = [&]() {
    const int len = nblk * BB;
    const int groups = min(kProjWarps, (nblk + JC - 1) / JC), splits = kProjWarps / groups;
    const int jg = warp % groups, rs = warp / groups; // warps with rs >= splits only join the barriers
    constexpr int BUF = NT * NT * 64;
    for (int j0 = 0; j0 < nblk; j0 += groups * JC) { // block j0 + jg + q * groups, q < JC
      double acc[JC][NT][NT][2];
#pragma unroll
      for (int q = 0; q < JC; ++q)
#pragma unroll
        for (int a = 0; a < NT; ++a)
#pragma unroll
          for (int b = 0; b < NT; ++b) acc[q][a][b][0] = acc[q][a][b][1] = 0.0;
      const T* Vb[JC];
      bool on[JC];
#pragma unroll
      for (int q = 0; q < JC; ++q) {
        const int j = j0 + jg + q * groups;
        on[q] = j < nblk && rs < splits;
        Vb[q] = V + static_cast<int64_t>(min(j, nblk - 1)) * vstride;
      }
      if (on[0]) {
#pragma unroll 4
        for (int64_t r0 = rb + 4 * rs; r0 < re; r0 += 4 * splits) {
          const int64_t row = r0 + t4;
          double bf[NT], av[JC][NT];
#pragma unroll
          for (int t = 0; t < NT; ++t) {
            const int col = t * 8 + g;
            const bool ok = row < re && col < BS;
            bf[t] = ok ? static_cast<double>(W[row * BS + col]) : 0.0;
#pragma unroll
            for (int q = 0; q < JC; ++q) av[q][t] = ok && on[q] ? static_cast<double>(Vb[q][row * BS + col]) : 0.0;
          }
#pragma unroll
          for (int q = 0; q < JC; ++q)
            if (on[q])
#pragma unroll
              for (int a = 0; a < NT; ++a)
#pragma unroll
                for (int b = 0; b < NT; ++b) dmma_m8n8k4(acc[q][a][b][0], acc[q][a][b][1], av[q][a], bf[b]);
        }
      }
      // over the row splits, one of the JC blocks of every group at a time
#pragma unroll
      for (int q = 0; q < JC; ++q) {
        if (j0 + q * groups >= nblk) break;
#pragma unroll
        for (int a = 0; a < NT; ++a)
#pragma unroll
          for (int b = 0; b < NT; ++b) {
            red[warp * BUF + (a * NT + b) * 64 + g * 8 + 2 * t4] = acc[q][a][b][0];
            red[warp * BUF + (a * NT + b) * 64 + g * 8 + 2 * t4 + 1] = acc[q][a][b][1];
          }
        __syncthreads();
        for (int e = tid; e < groups * BUF; e += kProjThreads) {
          const int gr = e / BUF, w = e % BUF, j = j0 + gr + q * groups;
          const int row = (w >> 6) / NT * 8 + ((w & 63) >> 3), col = (w >> 6) % NT * 8 + (w & 7);
          if (j < nblk && row < BS && col < BS) {
            double v = 0.0;
            for (int k = 0; k < splits; ++k) v += red[(k * groups + gr) * BUF + w];
            partial[static_cast<int64_t>(blockIdx.x) * len + j * BB + row * BS + col] = v;
          }
        }
        __syncthreads();
      }
    }
    if (!grid_barrier(bar, gridDim.x, status)) return false;
    for (int e0 = (static_cast<int>(blockIdx.x) * kProjWarps + warp) * 8; e0 < len; e0 += ncta * kProjWarps * 8) {
      const double t = sum_ctas(partial, len, e0, len);
      if (lane < 8 && e0 + lane < len) total[e0 + lane] = t;
    }
    return grid_barrier(bar, gridDim.x, status);
  };
  // W -= sum_j V_j C_j over this CTA's rows, and Gs = the Gram matrix of the result over all rows
  const auto update = [&]() {
    for (int e = tid; e < nblk * BB; e += kProjThreads) coef[e] = __ldcg(total + e);
    __syncthreads();
    double gacc[NT][NT][2];
#pragma unroll
    for (int a = 0; a < NT; ++a)
#pragma unroll
      for (int b = 0; b < NT; ++b) gacc[a][b][0] = gacc[a][b][1] = 0.0;
    double* st = stage + warp * 8 * BS;
    for (int64_t r0 = rb + warp * 8; r0 < re; r0 += kProjWarps * 8) {
      const int64_t row = r0 + g;
      double acc[NT][2];
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int col = t * 8 + 2 * t4 + i;
          acc[t][i] = (row < re && col < BS) ? static_cast<double>(W[row * BS + col]) : 0.0;
        }
#pragma unroll 8
      for (int j = 0; j < nblk; ++j) {
        T a[KS];
        const T* Vj = V + static_cast<int64_t>(j) * vstride;
        if (row < re && t4 * KS < BS) load_cols<T, KS>(Vj + row * BS + t4 * KS, a);
        else
#pragma unroll
          for (int ks = 0; ks < KS; ++ks) a[ks] = T(0);
#pragma unroll
        for (int ks = 0; ks < KS; ++ks)
#pragma unroll
          for (int t = 0; t < NT; ++t) {
            const int krow = t4 * KS + ks, col = t * 8 + g;
            const double b = (krow < BS && col < BS) ? -coef[j * BB + krow * BS + col] : 0.0;
            dmma_m8n8k4(acc[t][0], acc[t][1], static_cast<double>(a[ks]), b);
          }
      }
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int col = t * 8 + 2 * t4 + i;
          if (col < BS) {
            const T v = static_cast<T>(acc[t][i]);
            if (row < re) W[row * BS + col] = v;
            st[g * BS + col] = row < re ? static_cast<double>(v) : 0.0;
          }
        }
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int lr = q * 4 + t4;
        double f[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t) f[t] = (t * 8 + g < BS) ? st[lr * BS + t * 8 + g] : 0.0;
#pragma unroll
        for (int a = 0; a < NT; ++a)
#pragma unroll
          for (int b = 0; b < NT; ++b) dmma_m8n8k4(gacc[a][b][0], gacc[a][b][1], f[a], f[b]);
      }
      __syncwarp();
    }
#pragma unroll
    for (int a = 0; a < NT; ++a)
#pragma unroll
      for (int b = 0; b < NT; ++b) {
        red[warp * (NT * NT * 64) + (a * NT + b) * 64 + g * 8 + 2 * t4] = gacc[a][b][0];
        red[warp * (NT * NT * 64) + (a * NT + b) * 64 + g * 8 + 2 * t4 + 1] = gacc[a][b][1];
      }
    __syncthreads();
    for (int e = tid; e < NT * NT * 64; e += kProjThreads) {
      const int row = (e >> 6) / NT * 8 + ((e & 63) >> 3), col = (e >> 6) % NT * 8 + (e & 7);
      if (row < BS && col < BS) {
        double v = 0.0;
#pragma unroll
        for (int w = 0; w < kProjWarps; ++w) v += red[w * (NT * NT * 64) + e];
        gpartial[static_cast<int64_t>(blockIdx.x) * BB + row * BS + col] = v;
      }
    }
    if (!grid_barrier(bar, gridDim.x, status)) return false;
    for (int e0 = warp * 8; e0 < BB; e0 += kProjWarps * 8) { // every CTA for itself: the decision needs no barrier
      const double t = sum_ctas(gpartial, BB, e0, BB);
      if (lane < 8 && e0 + lane < BB) Gs[e0 + lane] = t;
    }
    __syncthreads();
    return true;
  };

  for (int e = tid; e < BB; e += kProjThreads) G0[e] = before[e];
  for (int pass = 0; pass < 2; ++pass) {
    if (!dots() || !update()) return;
    if (blockIdx.x == 0)
      for (int e = tid; e < BB; e += kProjThreads) G[e] = Gs[e];
    bool again = false; // the same in every CTA
    for (int c = 0; c < BS; ++c) again |= Gs[c * BS + c] < eta2 * G0[c * BS + c];
    if (!again) return;
  }
}

} // namespace

using namespace trl_detail;

// ---------------------------------------------------------------- launchers
namespace trl_detail {

// Workspace of a kernel whose last CTA adds up `chunks` rows of `len` partial sums; null on failure.
inline double* ticket_workspace(trl_cuda_context* h, int64_t chunks, int64_t len, Tickets& t)
{
  const int64_t groups = (chunks + kTicketGroup - 1) / kTicketGroup;
  if (groups + 1 > kTickets) return nullptr;
  double* partial = static_cast<double*>(workspace(h, static_cast<size_t>(chunks + groups) * len * sizeof(double)));
  t.count = reinterpret_cast<unsigned*>(h->d_small + kSmallTickets);
  t.groups = partial ? partial + chunks * len : nullptr;
  return partial;
}

// Row chunks of the register-fed dot: about 4 CTAs per SM in total, 512+ rows per CTA.
template <int G>
int64_t dot_chunks(int num_sms, int gj, int64_t n, int64_t& rows_per_cta)
{
  int64_t chunks = static_cast<int64_t>(num_sms) * 4 / gj;
  const int64_t max_chunks = (n + 511) / 512;
  if (chunks > max_chunks) chunks = max_chunks;
  if (chunks < 1) chunks = 1;
  rows_per_cta = (n + chunks - 1) / chunks;
  constexpr int step = kWarps * 4 * G; // rows one CTA iteration covers
  rows_per_cta = (rows_per_cta + step - 1) / step * step;
  return (n + rows_per_cta - 1) / rows_per_cta;
}

// C = [V_0, V_vstride, ...]^T W for JC blocks `vstride` elements apart, reading W once; fin gets the
// JC * BS * BS totals in the same launch.
template <typename T, int BS, int JC, int G, class Fin>
int launch_block_dot_finish(trl_cuda_context* h, const T* V, int64_t vstride, const T* W, int64_t n, const int* cond, const Fin& fin)
{
  int64_t rows_per_cta = 0;
  const int64_t chunks = dot_chunks<G>(h->num_sms, 1, n, rows_per_cta);
  Tickets t{};
  double* partial = ticket_workspace(h, chunks, static_cast<int64_t>(JC) * BS * BS, t);
  if (!partial) return TRL_ENOMEM;
  launch(k_block_dot<T, BS, JC, G, Fin>, dim3(1, static_cast<unsigned>(chunks)), kThreads, 0, h->stream, V, vstride, JC, W, n, rows_per_cta, partial, cond, t, fin);
  return after_launch(h, "block_dot");
}

template <typename T, int BS, int JC, int G>
int launch_block_dot_jc(trl_cuda_context* h, const T* V, int nblk, const T* W, int64_t n, double* C, const int* cond)
{
  const int64_t len = static_cast<int64_t>(nblk) * BS * BS;
  const int gj = (nblk + JC - 1) / JC;
  int64_t rows_per_cta = 0;
  const int64_t chunks = dot_chunks<G>(h->num_sms, gj, n, rows_per_cta);
  double* partial = static_cast<double*>(workspace(h, static_cast<size_t>(chunks) * len * sizeof(double)));
  if (!partial) return TRL_ENOMEM;
  launch(k_block_dot<T, BS, JC, G, FinishNone>, dim3(gj, static_cast<unsigned>(chunks)), kThreads, 0, h->stream, V, n * BS, nblk, W, n, rows_per_cta, partial, cond, Tickets{},
         FinishNone{});
  int st = after_launch(h, "block_dot");
  if (st) return st;
  launch_reduce(h->stream, partial, chunks, len, C, cond);
  return after_launch(h, "block_dot reduce");
}

template <typename T, int BS, int JC, int S, int TB>
int launch_block_dot_bulk(trl_cuda_context* h, const T* V, int nblk, const T* W, int64_t n, double* C, const int* cond)
{
  constexpr int R = BulkTile<T, BS, TB>::R;
  constexpr size_t smem = static_cast<size_t>(S) * (JC + 1) * BulkTile<T, BS, TB>::ELEMS * sizeof(T) + 2 * S * sizeof(uint64_t);
  // the shared-memory attribute belongs to the current device: set it on every call
  if (cudaFuncSetAttribute(k_block_dot_bulk<T, BS, JC, S, TB>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) != cudaSuccess) {
    cudaGetLastError();
    return set_error(h, TRL_ECUDA, "block dot: %zu bytes of shared memory refused", smem);
  }
  const int resident = resident_ctas<k_block_dot_bulk<T, BS, JC, S, TB>>(h->device, kThreads, smem, 1);
  const int64_t len = static_cast<int64_t>(nblk) * BS * BS;
  const int gj = (nblk + JC - 1) / JC;
  int64_t chunks = static_cast<int64_t>(h->num_sms) * resident / gj;
  if (chunks < 1) chunks = 1;
  constexpr int kLeast = TB > 4096 ? 1 : 2; // tiles per CTA at least
  const int64_t max_chunks = (n + kLeast * R - 1) / (kLeast * R);
  if (chunks > max_chunks) chunks = max_chunks;
  int64_t rows_per_cta = (n + chunks - 1) / chunks;
  rows_per_cta = (rows_per_cta + R - 1) / R * R;
  chunks = (n + rows_per_cta - 1) / rows_per_cta;
  double* partial = static_cast<double*>(workspace(h, static_cast<size_t>(chunks) * len * sizeof(double)));
  if (!partial) return TRL_ENOMEM;
  launch(k_block_dot_bulk<T, BS, JC, S, TB>, dim3(gj, static_cast<unsigned>(chunks)), kThreads, smem, h->stream, V, n * BS, nblk, W, n, rows_per_cta, partial, h->d_status, cond);
  int st = after_launch(h, "block_dot");
  if (st) return st;
  launch_reduce(h->stream, partial, chunks, len, C, cond);
  return after_launch(h, "block_dot reduce");
}

constexpr int64_t kTicketDotRows = 131072;

// Bulk-copy pipeline when a row of the block is a whole number of 16-byte units; otherwise
// the register-prefetch kernel with JC blocks and G row groups per warp iteration (about
// 16-20 independent loads in flight per warp).
template <typename T, int BS>
int launch_block_dot(trl_cuda_context* h, const T* V, int nblk, const T* W, int64_t n, double* C, const int* cond = nullptr)
{
  if (n == 0 && !cond) {
    cudaMemsetAsync(C, 0, static_cast<size_t>(nblk) * BS * BS * sizeof(double), h->stream);
    return TRL_OK;
  }
  // Shapes measured on B200 for the 884,736 x 8 blocks of the 96^3 workload (GB/s of
  // algorithmic bytes; the STREAM copy reference is 6,552): FP64 with 2 KB tiles, JC=8, S=3
  // gives 6,835 (24 blocks) and 6,921 (48 blocks); FP32 with 4 KB tiles gives 5,176 (8 blocks,
  // JC=8) and with JC=4 5,849 (24) and 5,831 (48).
  // A single block (the driver's T_ii = V_i^T W, both operands usually still in L2 from the
  // SpMM): the register-fed kernel with 8 (FP64) / 4 (FP32) row groups per warp and 4 CTAs
  // per SM measured 6,851 / 5,682 GB/s against 4,759 / 4,562 for the bulk pipeline.
  // Up to kTicketDotRows rows its last CTA adds the partial sums up (B200, 16,384 x 8 FP64: 10.0 -> 7.3 us,
  // the second launch's host time); beyond that the wider second kernel is faster (884,736 x 8: FP64
  // 20.8 against 19.6 us, FP32 15.5 against 12.0).
  if (nblk == 1 && BS <= 8) {
    constexpr int G1 = sizeof(T) == 8 ? 8 : 4;
    if (n <= kTicketDotRows) return launch_block_dot_finish<T, BS, 1, G1>(h, V, n * BS, W, n, cond, FinishStore<BS * BS>{C});
    return launch_block_dot_jc<T, BS, 1, G1>(h, V, nblk, W, n, C, cond);
  }
  if constexpr ((BS * sizeof(T)) % 16 == 0) {
    if constexpr (BS == 16) {
      // 8 KB tiles, stages for the same shared memory: a copy's start costs its thread as much as 4 KB
      // of data (B200, 300,001 rows, 4 KB -> 8 KB tiles: 1 block FP64 22 -> 17 us, FP32 14 -> 13; 4 blocks 54 -> 40,
      // 45 -> 29; 8 blocks FP32 53 -> 48; 24 blocks FP32, from 2 KB, 162 -> 127)
      if (nblk == 1) return launch_block_dot_bulk<T, BS, 1, 4, 8192>(h, V, nblk, W, n, C, cond);
      if (nblk == 2) return launch_block_dot_bulk<T, BS, 2, 3, 8192>(h, V, nblk, W, n, C, cond);
      return launch_block_dot_bulk<T, BS, 4, 2, 8192>(h, V, nblk, W, n, C, cond);
    }
    else {
      if (nblk == 1) return launch_block_dot_bulk<T, BS, 1, 8, 4096>(h, V, nblk, W, n, C, cond);
      if (nblk == 2) return launch_block_dot_bulk<T, BS, 2, 6, 4096>(h, V, nblk, W, n, C, cond);
      if (nblk <= 4) return launch_block_dot_bulk<T, BS, 4, 4, 4096>(h, V, nblk, W, n, C, cond);
      if constexpr (sizeof(T) == 8) return launch_block_dot_bulk<T, BS, 8, 3, 2048>(h, V, nblk, W, n, C, cond);
      if (nblk <= 8) return launch_block_dot_bulk<T, BS, 8, 3, 4096>(h, V, nblk, W, n, C, cond);
      return launch_block_dot_bulk<T, BS, 4, 3, 4096>(h, V, nblk, W, n, C, cond);
    }
  }
  if (nblk == 1) return launch_block_dot_jc<T, BS, 1, 8>(h, V, nblk, W, n, C, cond);
  if (nblk == 2) return launch_block_dot_jc<T, BS, 2, 4>(h, V, nblk, W, n, C, cond);
  if (nblk <= 4) return launch_block_dot_jc<T, BS, 4, 4>(h, V, nblk, W, n, C, cond);
  return launch_block_dot_jc<T, BS, 8, 2>(h, V, nblk, W, n, C, cond);
}

// out -= V C over MB blocks and the Gram matrix of the result, which fin gets
template <typename T, int BS, int RT, class Fin>
int launch_update_gram_rt(trl_cuda_context* h, const T* in, int MB, const double* coef, T* out, int64_t n, const int* cond, const Fin& fin)
{
  // Measured on B200 (24 blocks of 884,736 x 8, GB/s of algorithmic bytes; copy peak
  // 6,539): one input block per loop iteration (U = 1) beats explicit multi-block register
  // prefetch (U = 4: FP64 6,075, FP32 3,860), and 8-row tiles per warp RT = 4 (FP64, 6,784)
  // and RT = 2 (FP32, 5,439) with two resident waves of CTAs do best.
  const int resident = resident_ctas<k_update_gram<T, BS, RT, 1, Fin>>(h->device, kThreads, 0, 4);
  const unsigned grid = grid_for(h, (n + 8 * RT - 1) / (8 * RT), kWarps, 2 * resident);
  Tickets t{};
  double* partial = ticket_workspace(h, grid, BS * BS, t);
  if (!partial) return TRL_ENOMEM;
  launch(k_update_gram<T, BS, RT, 1, Fin>, grid, kThreads, 0, h->stream, in, n * BS, MB, coef, out, n, 1, -1.0, partial, cond, t, fin);
  return after_launch(h, "update_gram");
}

// 16 columns: two tiles of columns take each coefficient load to 2 RT products, and with RT = 1 the loads
// bound the kernel. With 24 rows per warp and registers for two CTAs per SM (RT = 1 -> 3, one projection less
// its dot): 300,001 rows, 24 blocks FP32 285 -> 166 us (the products take 103), 12 blocks FP64 196 -> 156 (the
// bytes 82); 20,000 rows, 30 blocks 44 -> 37 and 51 -> 41. Up to kFewRows rows single tiles give
// more warps (RT = 1 / 3, FP32 and FP64: 1,500 rows 13.9 / 16.5 and 20.2 / 23.5 us, 3,500 22.3 / 25.9 and
// 23.8 / 27.0; 4,096 33.7 / 30.8 and 36.7 / 31.8).
constexpr int64_t kFewRows = 3584;

template <typename T, int BS, class Fin>
int launch_update_gram(trl_cuda_context* h, const T* in, int MB, const double* coef, T* out, int64_t n, const int* cond, const Fin& fin)
{
  if constexpr (BS == 16) {
    if (n <= kFewRows) return launch_update_gram_rt<T, BS, 1>(h, in, MB, coef, out, n, cond, fin);
    return launch_update_gram_rt<T, BS, 3>(h, in, MB, coef, out, n, cond, fin);
  }
  else {
    return launch_update_gram_rt<T, BS, (sizeof(T) == 8 ? 4 : 2)>(h, in, MB, coef, out, n, cond, fin);
  }
}

// Where the projection is one launch. A sketch that asks for nothing is 8 - 10 us there and 18 - 19 us in
// separate kernels, at every size; one that asks for a projection is faster in separate kernels by an
// amount that grows with the rows and, in narrow or FP32 blocks, with their number. The line lies where
// that amount would make the call slower than it was with a kernel for each test, flag and sum (29 - 34 us
// at least). us, that / one launch / separate kernels: FP32 16,384 x 4, 20 blocks 34 / 31 / 25, 40 blocks 35 / 38 /
// 28; 24,576 x 4, 16 blocks 32 / 33 / 26; FP64 16,384 x 4, 40 blocks 35 / 34 / 32; 32,768 x 8, 24 blocks 42 / 41 / 38;
// 49,152 x 8, 4 blocks 31 / 33 / 27; 24,576 x 1, 40 blocks 38 / 39 / 18; 16 columns FP32, 24,576 rows, 2 blocks 38 / 42 /
// 34, 16 blocks 63 / 59 / 53; 32,768 rows, 8 blocks 49 / 52 / 45; 4,096 rows, 2 blocks 34 / 29 / 23.
template <typename T, int BS>
bool one_launch_projects(int64_t n, int nblk)
{
  if (nblk * BS * BS > kProjMaxEntries || nblk * n * BS * static_cast<int64_t>(sizeof(T)) > (int64_t(64) << 20)) return false; // (half of L2)
  if (BS == 16) return n <= 4096 || (n <= 24576 && nblk > 2);
  return n <= 32768 && ((BS > 1 && sizeof(T) == 8) || nblk * n <= 350000);
}

// True if the projection ran in one launch (st: its status), false if the separate kernels have to.
template <typename T, int BS>
bool launch_project(trl_cuda_context* h, const T* V, int nblk, T* W, int64_t n, const int* cond, const double* before, double eta2, double* G, int& st)
{
  constexpr int BB = BS * BS, NT = (BS + 7) / 8;
  if (!one_launch_projects<T, BS>(n, nblk)) return false;
  const auto kern = k_project<T, BS>;
  const auto smem = [](int entries) { return sizeof(double) * (entries + static_cast<size_t>(kProjWarps) * (8 * BS + NT * NT * 64)); };
  static std::atomic<int> usable[64]; // per device: 1 the kernel can be launched with the most shared memory, -1 it cannot
  int ok = usable[h->device & 63];
  if (ok == 0) {
    int resident = 0, coop = 0;
    const size_t most = smem(kProjMaxEntries);
    const bool fits = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, h->device) == cudaSuccess && coop &&
                      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(most)) == cudaSuccess &&
                      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kern, kProjThreads, most) == cudaSuccess && resident > 0;
    cudaGetLastError();
    usable[h->device & 63] = ok = fits ? 1 : -1;
  }
  if (ok < 0) return false;
  // a CTA per SM, each with 16 rows (two tiles) at least
  int64_t rows = (n + h->num_sms - 1) / h->num_sms;
  rows = rows < 16 ? 16 : (rows + 7) / 8 * 8;
  const int64_t ctas = (n + rows - 1) / rows;
  const size_t len = static_cast<size_t>(nblk) * BB;
  double* partial = static_cast<double*>(workspace(h, sizeof(double) * ((ctas + 1) * len + ctas * BB)));
  if (!partial) {
    st = TRL_ENOMEM;
    return true;
  }
  double* total = partial + ctas * len;
  cudaLaunchAttribute attr[1] = {};
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(ctas));
  cfg.blockDim = dim3(kProjThreads);
  cfg.dynamicSmemBytes = smem(nblk * BB);
  cfg.stream = h->stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, V, nblk, W, n, rows, cond, before, eta2, G, partial, total, total + len, reinterpret_cast<unsigned*>(h->d_small + kSmallCounters) + 2, h->d_status);
  st = after_launch(h, "project");
  return true;
}

constexpr int64_t kCholStream = int64_t(64) << 20; // bytes of a block that comes from memory (about half of L2)

// One pass of k_cholqr over the block: GRAM factors the Gram matrix of X U_0 ... U_{nf-1}, otherwise
// X <- X U_0 ... U_{nf-1}.
template <typename T, int BS, bool GRAM>
int launch_cholqr(trl_cuda_context* h, T* X, int64_t n, const double* G0, int nf, double* U, double* R)
{
  const auto run = [&](auto kernel, unsigned grid) {
    Tickets t{};
    double* partial = nullptr;
    if (GRAM && !(partial = ticket_workspace(h, grid, BS * BS, t))) return static_cast<int>(TRL_ENOMEM);
    launch(kernel.fn, grid, kThreads, 0, h->stream, X, n, G0, nf, U, R, h->d_status, partial, t);
    return after_launch(h, "cholqr");
  };
  if constexpr (BS * sizeof(T) <= 16) {
    constexpr int ROWS = 4;
    unsigned grid = grid_for(h, n, kThreads * ROWS, 2);
    if (GRAM && grid > kTicketGroup && grid <= 2 * kTicketGroup) grid = kTicketGroup; // one round of sums
    return run(KernelOf<k_cholqr_narrow<T, BS, ROWS, GRAM>>{}, grid);
  }
  else {
    // one resident wave: every CTA prepares its factors once
    const auto tiles = [&](auto rt) {
      constexpr int RT = decltype(rt)::value;
      return run(KernelOf<k_cholqr<T, BS, RT, GRAM>>{}, grid_for(h, n, kWarps * 8 * RT, resident_ctas<k_cholqr<T, BS, RT, GRAM>>(h->device, kThreads, 0, 4)));
    };
    // 16 columns in FP32 from memory: more warps with a tile each (us, 4,194,304 rows, two tiles / one: 1 pass 218
    // / 174, 2 passes 494 / 405, 4 passes 1,231 / 1,134; from L2 two are better, 300,001 rows, 4 passes 126 / 137)
    if constexpr (BS == 16 && sizeof(T) == 4)
      if (n * BS * static_cast<int64_t>(sizeof(T)) > kCholStream) return tiles(std::integral_constant<int, 1>{});
    return tiles(std::integral_constant<int, (BS > 8 ? 2 : 4)>{});
  }
}

template <typename T, int BS, int NBMAX>
void launch_gemm_nb(trl_cuda_context* h, const T* in, int MB, const double* coef, int ldc, int transpose, T* out, int nb, int64_t n, int accumulate, double sign)
{
  constexpr int NT = (BS + 7) / 8;
  constexpr int KS = (BS + 3) / 4;
  constexpr int RT = (NBMAX * NT >= 8) ? 1 : 2; // keep the accumulators within ~64 registers
  constexpr int U = (KS >= 4) ? 2 : 4;
  const unsigned grid = grid_for(h, (n + 8 * RT - 1) / (8 * RT), kWarps, 8);
  if (MB == 1) // a single input block: no point loading it U times
    launch(k_block_gemm<T, BS, NBMAX, RT, 1>, grid, kThreads, 0, h->stream, in, n * BS, MB, coef, ldc, transpose, out, n * BS, nb, n, accumulate, sign);
  else
    launch(k_block_gemm<T, BS, NBMAX, RT, U>, grid, kThreads, 0, h->stream, in, n * BS, MB, coef, ldc, transpose, out, n * BS, nb, n, accumulate, sign);
}

template <typename T, int BS>
int launch_block_gemm(trl_cuda_context* h, const T* in, int MB, const double* coef, int ldc, int transpose, T* out, int NB, int64_t n, int accumulate, double sign)
{
  if (n == 0 || NB == 0) return TRL_OK;
  constexpr int NBCAP = (BS >= 16) ? 4 : 16;
  for (int j0 = 0; j0 < NB; j0 += NBCAP) {
    const int nb = (NB - j0) < NBCAP ? (NB - j0) : NBCAP;
    const double* cj = coef + static_cast<int64_t>(j0) * BS * BS;
    T* oj = out + static_cast<int64_t>(j0) * n * BS;
    if (nb == 1)
      launch_gemm_nb<T, BS, 1>(h, in, MB, cj, ldc, transpose, oj, nb, n, accumulate, sign);
    else if (nb <= 2)
      launch_gemm_nb<T, BS, 2>(h, in, MB, cj, ldc, transpose, oj, nb, n, accumulate, sign);
    else if (nb <= 4)
      launch_gemm_nb<T, BS, 4>(h, in, MB, cj, ldc, transpose, oj, nb, n, accumulate, sign);
    else if (nb <= 8)
      launch_gemm_nb<T, BS, 8>(h, in, MB, cj, ldc, transpose, oj, nb, n, accumulate, sign);
    else
      launch_gemm_nb<T, BS, NBCAP>(h, in, MB, cj, ldc, transpose, oj, nb, n, accumulate, sign);
    int st = after_launch(h, "block_gemm");
    if (st) return st;
  }
  return TRL_OK;
}


// Restart rotation through k_rotate: the output columns are processed in chunks of at most 6
// n-tiles whose Yhat fragments fit in shared memory. Returns -1 (nothing launched) for block
// sizes below 4 or bases too deep for one k-step column of fragments; the caller then uses
// k_block_gemm.
template <typename T, int BS, int NTC>
int launch_rotate_chunk(trl_cuda_context* h, const T* V, int m, const double* Y, int ldy, int N, int c0, T* W, int64_t n, size_t smem)
{
  constexpr int RT = 2;
  constexpr int D = (BS >= 16) ? 2 : (BS == 8 ? 4 : 8);
  auto kern = k_rotate<T, BS, NTC, RT, D>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) != cudaSuccess)
    return set_error(h, TRL_ECUDA, "rotation: %zu bytes of shared memory refused", smem);
  const int64_t tiles = (n + 8 * RT - 1) / (8 * RT);
  int64_t grid = h->num_sms;
  const int64_t need = (tiles + kRotThreads / 32 - 1) / (kRotThreads / 32);
  if (grid > need) grid = need;
  if (grid < 1) grid = 1;
  launch(kern, static_cast<unsigned>(grid), kRotThreads, smem, h->stream, V, n * BS, m, Y, ldy, N, c0, W, n * BS, n);
  return after_launch(h, "rotate");
}

template <typename T, int BS>
int launch_rotate(trl_cuda_context* h, const T* V, int m, const double* Y, int ldy, int k, T* W, int64_t n)
{
  if constexpr (BS < 4) {
    return -1;
  }
  else {
    constexpr size_t kSmemMax = 200 * 1024;
    const size_t frag_bytes = static_cast<size_t>(m) * (BS / 4) * 32 * sizeof(double); // one n-tile column
    int ntc_max = static_cast<int>(kSmemMax / frag_bytes);
    if (ntc_max > 6) ntc_max = 6; // beyond 6 n-tiles the accumulators spill at 128 registers
    if (ntc_max < 1) return -1;
    const int N = k * BS;
    const int tiles = (N + 7) / 8;
    const int passes = (tiles + ntc_max - 1) / ntc_max;
    const int per = (tiles + passes - 1) / passes;
    for (int t0 = 0; t0 < tiles; t0 += per) {
      const int ntc = (tiles - t0) < per ? (tiles - t0) : per;
      const size_t smem = frag_bytes * ntc;
      int st = TRL_OK;
      switch (ntc) {
      case 1: st = launch_rotate_chunk<T, BS, 1>(h, V, m, Y, ldy, N, t0 * 8, W, n, smem); break;
      case 2: st = launch_rotate_chunk<T, BS, 2>(h, V, m, Y, ldy, N, t0 * 8, W, n, smem); break;
      case 3: st = launch_rotate_chunk<T, BS, 3>(h, V, m, Y, ldy, N, t0 * 8, W, n, smem); break;
      case 4: st = launch_rotate_chunk<T, BS, 4>(h, V, m, Y, ldy, N, t0 * 8, W, n, smem); break;
      case 5: st = launch_rotate_chunk<T, BS, 5>(h, V, m, Y, ldy, N, t0 * 8, W, n, smem); break;
      default: st = launch_rotate_chunk<T, BS, 6>(h, V, m, Y, ldy, N, t0 * 8, W, n, smem); break;
      }
      if (st) return st;
    }
    return TRL_OK;
  }
}

} // namespace trl_detail

static int check_common(trl_cuda_context* h, int dtype, int64_t n, int bs)
{
  if (!valid_dtype(dtype)) return set_error(h, TRL_ENOTSUP, "unsupported dtype %d", dtype);
  if (!valid_bs(bs)) return set_error(h, TRL_ENOTSUP, "unsupported block size %d", bs);
  if (n < 0) return set_error(h, TRL_EINVAL, "negative row count");
  return TRL_OK;
}

static size_t elt_size(int dtype) { return dtype == TRL_F64 ? sizeof(double) : sizeof(float); }

extern "C" {

int trl_cuda_bv_zero(trl_cuda_handle h, int dtype, void* X, int64_t n, int bs)
{
  TRL_CHECK_HANDLE(h);
  if (int st = check_common(h, dtype, n, bs)) return st;
  ProfScope prof(h, PROF_COPY, static_cast<double>(n) * bs * elt_size(dtype));
  return trl_cuda_memset_zero(h, X, static_cast<size_t>(n) * bs * elt_size(dtype));
}

int trl_cuda_bv_copy(trl_cuda_handle h, int dtype, void* X, const void* Y, int64_t n, int bs)
{
  TRL_CHECK_HANDLE(h);
  if (int st = check_common(h, dtype, n, bs)) return st;
  if (X == Y) return TRL_OK;
  ProfScope prof(h, PROF_COPY, 2.0 * n * bs * elt_size(dtype));
  return trl_cuda_memcpy(h, X, Y, static_cast<size_t>(n) * bs * elt_size(dtype), TRL_D2D);
}

int trl_cuda_bv_sub(trl_cuda_handle h, int dtype, void* X, const void* Y, int64_t n, int bs)
{
  TRL_CHECK_HANDLE(h);
  if (int st = check_common(h, dtype, n, bs)) return st;
  const int64_t count = n * bs;
  if (count == 0) return TRL_OK;
  if (!X || !Y) return set_error(h, TRL_EINVAL, "null pointer");
  ProfScope prof(h, PROF_SUB, 3.0 * count * elt_size(dtype));
  const int vec_ok = ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(Y)) & 15) == 0;
  const unsigned grid = grid_for(h, count / 4 + 1, kThreads, 8);
  TRL_DISPATCH_DT(dtype, launch(k_sub<T>, grid, kThreads, 0, h->stream, static_cast<T*>(X), static_cast<const T*>(Y), count, vec_ok));
  return after_launch(h, "bv_sub");
}

int trl_cuda_convert(trl_cuda_handle h, int dst_dtype, void* dst, int src_dtype, const void* src, int64_t count)
{
  TRL_CHECK_HANDLE(h);
  if (!valid_dtype(dst_dtype) || !valid_dtype(src_dtype)) return set_error(h, TRL_ENOTSUP, "unsupported dtype");
  if (count < 0) return set_error(h, TRL_EINVAL, "negative count");
  if (count == 0) return TRL_OK;
  if (!dst || !src) return set_error(h, TRL_EINVAL, "null pointer");
  ProfScope prof(h, PROF_COPY, static_cast<double>(count) * (elt_size(dst_dtype) + elt_size(src_dtype)));
  if (dst_dtype == src_dtype) return trl_cuda_memcpy(h, dst, src, static_cast<size_t>(count) * elt_size(dst_dtype), TRL_D2D);
  const unsigned grid = grid_for(h, count, kThreads * 4, 8);
  if (dst_dtype == TRL_F64)
    launch(k_convert<double, float>, grid, kThreads, 0, h->stream, static_cast<double*>(dst), static_cast<const float*>(src), count);
  else
    launch(k_convert<float, double>, grid, kThreads, 0, h->stream, static_cast<float*>(dst), static_cast<const double*>(src), count);
  return after_launch(h, "convert");
}

int trl_cuda_bv_mult(trl_cuda_handle h, int dtype, int mode, const void* X, const double* W, void* Y, int64_t n, int bs)
{
  TRL_CHECK_HANDLE(h);
  if (int st = check_common(h, dtype, n, bs)) return st;
  if (n == 0) return TRL_OK;
  if (!X || !W || !Y) return set_error(h, TRL_EINVAL, "null pointer");
  int transpose = 0, accumulate = 0;
  double sign = 1.0;
  switch (mode) {
  case TRL_MULT: break;
  case TRL_MULT_TRANSPOSE: transpose = 1; break;
  case TRL_MULT_ADD: accumulate = 1; break;
  case TRL_SUBTRACT:
    accumulate = 1;
    sign = -1.0;
    break;
  case TRL_SUBTRACT_TRANSPOSE:
    accumulate = 1;
    sign = -1.0;
    transpose = 1;
    break;
  default: return set_error(h, TRL_EINVAL, "bad mult mode %d", mode);
  }
  if (X == Y && accumulate) return set_error(h, TRL_EINVAL, "accumulating mult requires distinct input and output");
  ProfScope prof(h, PROF_MULT, (accumulate ? 3.0 : 2.0) * n * bs * elt_size(dtype), 2.0 * n * bs * bs);
  int st = TRL_OK;
  TRL_DISPATCH_DT(dtype, TRL_DISPATCH_BS(bs, st = launch_block_gemm<T, BS>(h, static_cast<const T*>(X), 1, W, 1, transpose, static_cast<T*>(Y), 1, n, accumulate, sign)));
  return st;
}

int trl_cuda_block_dot(trl_cuda_handle h, int dtype, const void* V, int nblk, const void* W, int64_t n, int bs, double* C)
{
  TRL_CHECK_HANDLE(h);
  if (int st = check_common(h, dtype, n, bs)) return st;
  if (nblk <= 0) return set_error(h, TRL_EINVAL, "nblk must be positive");
  if (!C) return set_error(h, TRL_EINVAL, "null pointer");
  if (n == 0) return trl_cuda_memset_zero(h, C, sizeof(double) * nblk * bs * bs); // empty sum
  if (!V || !W) return set_error(h, TRL_EINVAL, "null pointer");
  ProfScope prof(h, PROF_DOT, (nblk + 1.0) * n * bs * elt_size(dtype), 2.0 * nblk * n * bs * bs);
  int st = TRL_OK;
  TRL_DISPATCH_DT(dtype, TRL_DISPATCH_BS(bs, st = launch_block_dot<T, BS>(h, static_cast<const T*>(V), nblk, static_cast<const T*>(W), n, C)));
  return st;
}

int trl_cuda_block_update(trl_cuda_handle h, int dtype, void* W, const void* V, int nblk, const double* C, int64_t n, int bs)
{
  TRL_CHECK_HANDLE(h);
  if (int st = check_common(h, dtype, n, bs)) return st;
  if (nblk <= 0) return set_error(h, TRL_EINVAL, "nblk must be positive");
  if (n == 0) return TRL_OK;
  if (!V || !W || !C) return set_error(h, TRL_EINVAL, "null pointer");
  ProfScope prof(h, PROF_UPDATE, (nblk + 2.0) * n * bs * elt_size(dtype), 2.0 * nblk * n * bs * bs);
  int st = TRL_OK;
  // Coef(i, 0) = C + i*bs*bs  ->  ldc = 1
  TRL_DISPATCH_DT(dtype, TRL_DISPATCH_BS(bs, st = launch_block_gemm<T, BS>(h, static_cast<const T*>(V), nblk, C, 1, 0, static_cast<T*>(W), 1, n, 1, -1.0)));
  return st;
}

int trl_cuda_block_rotate(trl_cuda_handle h, int dtype, const void* V, int m, const double* Y, int ldy, int k, void* W, int64_t n, int bs)
{
  TRL_CHECK_HANDLE(h);
  if (int st = check_common(h, dtype, n, bs)) return st;
  if (m <= 0 || k <= 0 || ldy < k) return set_error(h, TRL_EINVAL, "bad rotation shape m=%d k=%d ldy=%d", m, k, ldy);
  if (n == 0) return TRL_OK;
  if (!V || !Y || !W) return set_error(h, TRL_EINVAL, "null pointer");
  const size_t es = elt_size(dtype);
  const char* v0 = static_cast<const char*>(V);
  const char* v1 = v0 + static_cast<size_t>(m) * n * bs * es;
  const char* w0 = static_cast<const char*>(W);
  const char* w1 = w0 + static_cast<size_t>(k) * n * bs * es;
  if (w0 < v1 && v0 < w1) return set_error(h, TRL_EINVAL, "rotation output overlaps its input");
  ProfScope prof(h, PROF_ROTATE, (static_cast<double>(m) + k) * n * bs * es, 2.0 * n * m * k * bs * bs);
  int st = TRL_OK;
  TRL_DISPATCH_DT(dtype, TRL_DISPATCH_BS(bs, {
    st = launch_rotate<T, BS>(h, static_cast<const T*>(V), m, Y, ldy, k, static_cast<T*>(W), n);
    if (st == -1) st = launch_block_gemm<T, BS>(h, static_cast<const T*>(V), m, Y, ldy, 0, static_cast<T*>(W), k, n, 0, 1.0);
  }));
  return st;
}

int trl_cuda_cholqr(trl_cuda_handle h, int dtype, void* X, int64_t n, int bs, int passes, double* R)
{
  TRL_CHECK_HANDLE(h);
  if (int st = check_common(h, dtype, n, bs)) return st;
  if (passes < 1 || passes > 4) return set_error(h, TRL_EINVAL, "passes must be in [1, 4]");
  if (!X || !R) return set_error(h, TRL_EINVAL, "null pointer");
  double* G = h->d_small;
  ProfScope prof(h, PROF_CHOLQR, 3.0 * passes * n * bs * elt_size(dtype), 4.0 * passes * n * bs * bs);
  int st = trl_cuda_block_dot(h, dtype, X, 1, X, n, bs, G);
  if (st) return st;
  return trl_cuda_cholqr_gram(h, dtype, X, n, bs, passes, R, G);
}

// passes - 1 launches that each add a factor (the first one factors G0 too), and one that applies
// them all.
int trl_cuda_cholqr_gram(trl_cuda_handle h, int dtype, void* X, int64_t n, int bs, int passes, double* R, const double* G0)
{
  TRL_CHECK_HANDLE(h);
  if (!G0) return trl_cuda_cholqr(h, dtype, X, n, bs, passes, R);
  if (int st = check_common(h, dtype, n, bs)) return st;
  if (passes < 1 || passes > kCholMaxPasses) return set_error(h, TRL_EINVAL, "passes must be in [1, 4]");
  if (!X || !R) return set_error(h, TRL_EINVAL, "null pointer");
  double* U = h->d_small + kSmallFactors;
  // R over G0 (the factor in place of its Gram matrix): every CTA of the first launch reads G0 while CTA 0
  // writes R, so they read a copy
  const size_t block = sizeof(double) * bs * bs;
  const auto at = [](const double* p) { return reinterpret_cast<uintptr_t>(p); };
  if (at(R) < at(G0) + block && at(G0) < at(R) + block) {
    if (int st = trl_cuda_memcpy(h, h->d_small, G0, block, TRL_D2D)) return st;
    G0 = h->d_small;
  }
  ProfScope prof(h, PROF_CHOLQR, 2.0 * passes * n * bs * elt_size(dtype), 4.0 * passes * n * bs * bs);
  int st = TRL_OK;
  TRL_DISPATCH_DT(dtype, TRL_DISPATCH_BS(bs, {
    T* Xt = static_cast<T*>(X);
    for (int q = 1; q < passes && !st; ++q) st = launch_cholqr<T, BS, true>(h, Xt, n, q == 1 ? G0 : nullptr, q, U, R);
    if (!st) st = launch_cholqr<T, BS, false>(h, Xt, n, passes == 1 ? G0 : nullptr, passes, U, R);
  }));
  return st;
}

int trl_cuda_project_out(trl_cuda_handle h, int dtype, const void* V, int nblk, void* W, int64_t n, int bs, int mode, double eta, double* G)
{
  TRL_CHECK_HANDLE(h);
  if (int st = check_common(h, dtype, n, bs)) return st;
  if (nblk <= 0 || !G) return set_error(h, TRL_EINVAL, "bad project_out arguments");
  if (mode != TRL_CGS_ONE && mode != TRL_CGS_TWO && mode != TRL_CGS_IFNEEDED) return set_error(h, TRL_EINVAL, "bad project_out mode %d", mode);
  const int BB = bs * bs;
  if (n == 0) return trl_cuda_memset_zero(h, G, sizeof(double) * BB);
  if (!V || !W) return set_error(h, TRL_EINVAL, "null pointer");
  const size_t es = elt_size(dtype);
  // coefficient storage: C1 (nblk+1 blocks) | C2 (nblk blocks) | Gw0 | flag
  double* base = static_cast<double*>(workspace2(h, sizeof(double) * (static_cast<size_t>(2 * nblk + 2) * BB) + 64));
  if (!base) return TRL_ENOMEM;
  double* C1 = base;
  double* C2 = C1 + static_cast<size_t>(nblk + 1) * BB;
  double* Gw0 = C2 + static_cast<size_t>(nblk) * BB;
  int* flag = reinterpret_cast<int*>(Gw0 + BB);
  const bool contiguous = static_cast<const char*>(W) == static_cast<const char*>(V) + static_cast<size_t>(nblk) * n * bs * es;
  int st = TRL_OK;
  TRL_DISPATCH_DT(dtype, TRL_DISPATCH_BS(bs, {
    const T* Vt = static_cast<const T*>(V);
    T* Wt = static_cast<T*>(W);
    // pass 1: C1 = V^T w (and w^T w, for free when w is the block right after V)
    {
      ProfScope prof(h, PROF_DOT, (nblk + (contiguous ? 1.0 : 2.0)) * n * bs * es, 2.0 * (nblk + 1) * n * bs * bs);
      st = launch_block_dot<T, BS>(h, Vt, nblk + (contiguous ? 1 : 0), Wt, n, C1);
      if (contiguous) Gw0 = C1 + static_cast<size_t>(nblk) * BB;
      else if (!st) st = launch_block_dot<T, BS>(h, Wt, 1, Wt, n, Gw0);
    }
    if (st) return st;
    {
      ProfScope prof(h, PROF_UPDATE, (nblk + 2.0) * n * bs * es, 2.0 * nblk * n * bs * bs + 2.0 * n * bs * bs);
      st = launch_update_gram<T, BS>(h, Vt, nblk, C1, Wt, n, nullptr, FinishGram<BS>{G, Gw0, eta * eta, mode == TRL_CGS_IFNEEDED ? flag : nullptr});
    }
    if (st || mode == TRL_CGS_ONE) return st;
    // pass 2, always or only where the flag is set (decided on the device; its bytes are not
    // credited to the profile because the host does not know whether it ran)
    {
      ProfScope prof(h, PROF_REORTH2, 0.0);
      const int* cond = mode == TRL_CGS_IFNEEDED ? flag : nullptr;
      st = launch_block_dot<T, BS>(h, Vt, nblk, Wt, n, C2, cond);
      if (!st) st = launch_update_gram<T, BS>(h, Vt, nblk, C2, Wt, n, cond, FinishGram<BS>{G, nullptr, 0.0, nullptr});
    }
  }));
  return st;
}

int trl_cuda_project_out_sketch(trl_cuda_handle h, int dtype, const void* V, int nblk, void* W, int64_t n, int bs, const void* S, double thr, double eta, double* G,
                                int* pair_state)
{
  TRL_CHECK_HANDLE(h);
  if (int st = check_common(h, dtype, n, bs)) return st;
  if (nblk <= 0 || !G || !(thr >= 0.0)) return set_error(h, TRL_EINVAL, "bad project_out_sketch arguments");
  const int BB = bs * bs;
  if (n == 0) return trl_cuda_memset_zero(h, G, sizeof(double) * BB);
  if (!V || !W || !S) return set_error(h, TRL_EINVAL, "null pointer");
  // coefficient storage: C1 (nblk blocks) | C2 (nblk blocks) | Gw0 | flags
  double* base = static_cast<double*>(workspace2(h, sizeof(double) * (static_cast<size_t>(2 * nblk + 1) * BB) + 64));
  if (!base) return TRL_ENOMEM;
  double* C1 = base;
  double* C2 = C1 + static_cast<size_t>(nblk) * BB;
  double* Gw0 = C2 + static_cast<size_t>(nblk) * BB;
  int* flag1 = reinterpret_cast<int*>(Gw0 + BB);
  int* flag2 = flag1 + 1;
  const size_t es = elt_size(dtype);
  int st = TRL_OK;
  TRL_DISPATCH_DT(dtype, TRL_DISPATCH_BS(bs, {
    const T* Vt = static_cast<const T*>(V);
    const T* St = static_cast<const T*>(S);
    T* Wt = static_cast<T*>(W);
    {
      ProfScope prof(h, PROF_DOT, 3.0 * n * bs * es, 4.0 * n * bs * bs);
      // [E; G] = [S, W]^T W in one pass over W, the decision, and G = W^T W as it stands
      st = launch_block_dot_finish<T, BS, 2, 4>(h, St, Wt - St, Wt, n, nullptr, FinishSketch<BS>{G, Gw0, thr * thr, flag1, flag2, pair_state});
    }
    if (st) return st;
    // both passes only where flagged (decided on the device; their bytes are not credited
    // to the profile because the host does not know whether they ran)
    {
      ProfScope prof(h, PROF_REORTH2, 0.0);
      if (launch_project<T, BS>(h, Vt, nblk, Wt, n, flag1, Gw0, eta * eta, G, st)) return st;
      st = launch_block_dot<T, BS>(h, Vt, nblk, Wt, n, C1, flag1);
      if (!st) st = launch_update_gram<T, BS>(h, Vt, nblk, C1, Wt, n, flag1, FinishGram<BS>{G, Gw0, eta * eta, flag2});
      if (!st) st = launch_block_dot<T, BS>(h, Vt, nblk, Wt, n, C2, flag2);
      if (!st) st = launch_update_gram<T, BS>(h, Vt, nblk, C2, Wt, n, flag2, FinishGram<BS>{G, nullptr, 0.0, nullptr});
    }
#ifdef TRL_DEBUG_TRACE
    // debug builds (-DTRL_DEBUG_TRACE) with TRL_PARTIAL_TRACE set: one stderr line per call
    // (synchronises; diagnostics only)
    static const bool trace = std::getenv("TRL_PARTIAL_TRACE") != nullptr;
    if (!st && trace) {
      int fl[2];
      cudaMemcpyAsync(fl, flag1, sizeof(int) * 2, cudaMemcpyDeviceToHost, h->stream);
      cudaStreamSynchronize(h->stream);
      std::fprintf(stderr, "partial nblk %d projected %d forced %d second %d\n", nblk, fl[0] & 1, (fl[0] >> 1) & 1, fl[1]);
    }
#endif
  }));
  return st;
}

} // extern "C"

namespace {
__global__ void __launch_bounds__(kThreads) k_unblock(const double* __restrict__ X, int64_t n, int bs, int ncols, double* __restrict__ out)
{
  ::trl_detail::pdl_enter();
  const int64_t total = n * ncols;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < total; e += stride) {
    const int64_t r = e / ncols;
    const int c = static_cast<int>(e % ncols);
    out[e] = X[static_cast<int64_t>(c / bs) * n * bs + r * bs + (c % bs)];
  }
}
} // namespace

extern "C" int trl_cuda_unblock(trl_cuda_handle h, const double* X, int64_t n, int bs, int ncols, double* out)
{
  TRL_CHECK_HANDLE(h);
  if (!valid_bs(bs) || n < 0 || ncols < 0) return set_error(h, TRL_EINVAL, "bad unblock arguments");
  if (n == 0 || ncols == 0) return TRL_OK;
  if (!X || !out) return set_error(h, TRL_EINVAL, "null pointer");
  ProfScope prof(h, PROF_COPY, 16.0 * n * ncols);
  launch(k_unblock, grid_for(h, n * ncols, kThreads * 4, 8), kThreads, 0, h->stream, X, n, bs, ncols, out);
  return after_launch(h, "unblock");
}

// ---------------------------------------------------------------- allocation-free block dot
// trl_cuda_block_dot_noalloc: the multi-block inner product for callers that must not
// allocate device memory. Its per-chunk partial sums live in the fixed array below instead
// of a handle's workspace. One copy of the array (2 MiB) exists on every GPU that loads this
// library and stays there until the process exits.
#include <mutex>

static constexpr int64_t kNoAllocScratchDoubles = int64_t(1) << 18; // 2 MiB of FP64 partials
static constexpr int kNoAllocMaxDevices = 64;
static __device__ __align__(256) double g_noalloc_partials[kNoAllocScratchDoubles];

static std::mutex g_noalloc_mutex;
static double* g_noalloc_ptr[kNoAllocMaxDevices] = {};
static int g_noalloc_sms[kNoAllocMaxDevices] = {};

// Resolves the device address of the scratch array on the current device (once per device).
static int noalloc_scratch(int device, double** ptr, int* sms)
{
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_noalloc_ptr[device]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_partials);
    if (e != cudaSuccess || !p) {
      cudaGetLastError();
      return TRL_ECUDA;
    }
    int count = 0;
    if (cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || count <= 0) {
      cudaGetLastError();
      return TRL_ECUDA;
    }
    g_noalloc_sms[device] = count;
    g_noalloc_ptr[device] = static_cast<double*>(p);
  }
  *ptr = g_noalloc_ptr[device];
  *sms = g_noalloc_sms[device];
  return TRL_OK;
}

template <typename T, int BS, int JC, int G>
static int noalloc_dot(cudaStream_t stream, int sms, double* partial, const T* V, int nblk, const T* W, int64_t n, double* C)
{
  const int64_t len = static_cast<int64_t>(nblk) * BS * BS;
  const int gj = (nblk + JC - 1) / JC;
  int64_t chunks = static_cast<int64_t>(sms) * 4 / gj;
  const int64_t fit = kNoAllocScratchDoubles / len; // chunks whose partials fit the array
  if (chunks > fit) chunks = fit;
  const int64_t max_chunks = (n + 511) / 512;
  if (chunks > max_chunks) chunks = max_chunks;
  if (chunks < 1) chunks = 1;
  int64_t rows_per_cta = (n + chunks - 1) / chunks;
  constexpr int step = kWarps * 4 * G;
  rows_per_cta = (rows_per_cta + step - 1) / step * step;
  chunks = (n + rows_per_cta - 1) / rows_per_cta;
  // every (chunk, block) entry of the partials is written before it is read in this call,
  // so nothing left in the array by an earlier call is used and nothing needs clearing
  launch(k_block_dot<T, BS, JC, G, FinishNone>, dim3(gj, static_cast<unsigned>(chunks)), kThreads, 0, stream, V, n * BS, nblk, W, n, rows_per_cta, partial, nullptr, Tickets{},
         FinishNone{});
  if (cudaGetLastError() != cudaSuccess) return TRL_ECUDA;
  launch_reduce(stream, partial, chunks, len, C, nullptr);
  if (cudaGetLastError() != cudaSuccess) return TRL_ECUDA;
  return TRL_OK;
}

template <typename T, int BS>
static int noalloc_dot_dispatch(cudaStream_t stream, int sms, double* partial, const T* V, int nblk, const T* W, int64_t n, double* C)
{
  if (nblk == 1) return noalloc_dot<T, BS, 1, 8>(stream, sms, partial, V, nblk, W, n, C);
  if (nblk == 2) return noalloc_dot<T, BS, 2, 4>(stream, sms, partial, V, nblk, W, n, C);
  if (nblk <= 4) return noalloc_dot<T, BS, 4, (BS >= 16 ? 2 : 4)>(stream, sms, partial, V, nblk, W, n, C);
  return noalloc_dot<T, BS, (BS >= 16 ? 4 : 8), 2>(stream, sms, partial, V, nblk, W, n, C);
}

extern "C" int trl_cuda_block_dot_noalloc(void* stream, int dtype, const void* V, int nblk, const void* W, int64_t n, int bs, double* C)
{
  if (!valid_dtype(dtype) || !valid_bs(bs)) return TRL_ENOTSUP;
  if (nblk <= 0 || n < 0 || !C) return TRL_EINVAL;
  if (static_cast<int64_t>(nblk) * bs * bs > TRL_CUDA_NOALLOC_MAX_ENTRIES) return TRL_EINVAL; // the output would not fit the partial-sum array
  auto s = static_cast<cudaStream_t>(stream);
  if (n == 0) return cudaMemsetAsync(C, 0, sizeof(double) * nblk * bs * bs, s) == cudaSuccess ? TRL_OK : TRL_ECUDA;
  if (!V || !W) return TRL_EINVAL;
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kNoAllocMaxDevices) {
    cudaGetLastError();
    return TRL_ECUDA;
  }
  double* partial = nullptr;
  int sms = 0;
  if (int st = noalloc_scratch(device, &partial, &sms)) return st;
  int st = TRL_OK;
  trl_cuda_context* h = nullptr; // only for the dispatch macros' error path
  TRL_DISPATCH_DT(dtype, TRL_DISPATCH_BS(bs, st = noalloc_dot_dispatch<T, BS>(s, sms, partial, static_cast<const T*>(V), nblk, static_cast<const T*>(W), n, C)));
  return st;
}

namespace {

// FP64 tensor-core (DMMA m8n8k4) issue rate: every warp runs kDmmaChains independent
// accumulator chains for `iters` rounds; the result is written so that nothing is elided.
constexpr int kDmmaChains = 8;

__global__ void __launch_bounds__(256) k_dmma_rate(int iters, double* __restrict__ out)
{
  ::trl_detail::pdl_enter();
  double d0[kDmmaChains], d1[kDmmaChains];
  const double a = 1.0 + 1e-9 * threadIdx.x, b = 1.0 - 1e-9 * blockIdx.x;
#pragma unroll
  for (int c = 0; c < kDmmaChains; ++c) d0[c] = d1[c] = 0.0;
  for (int i = 0; i < iters; ++i)
#pragma unroll
    for (int c = 0; c < kDmmaChains; ++c) dmma_m8n8k4(d0[c], d1[c], a, b);
  double s = 0.0;
#pragma unroll
  for (int c = 0; c < kDmmaChains; ++c) s += d0[c] + d1[c];
  if (s == 12345.678) out[0] = s; // never true; keeps the chains alive
}

} // namespace

extern "C" int trl_cuda_measure_dmma_rate(trl_cuda_handle h, double* host_tflops)
{
  TRL_CHECK_HANDLE(h);
  if (!host_tflops) return set_error(h, TRL_EINVAL, "null output");
  double* out = h->d_small;
  const int iters = 4096;
  const unsigned grid = static_cast<unsigned>(h->num_sms) * 8;
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  launch(k_dmma_rate, grid, 256, 0, h->stream, iters, out); // warm-up
  cudaEventRecord(a, h->stream);
  launch(k_dmma_rate, grid, 256, 0, h->stream, iters, out);
  cudaEventRecord(b, h->stream);
  const cudaError_t e = cudaEventSynchronize(b);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, a, b);
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  if (e != cudaSuccess) return set_error(h, TRL_ECUDA, "dmma rate: %s", cudaGetErrorString(e));
  if (int st = after_launch(h, "dmma rate")) return st;
  const double flops = 2.0 * 8 * 8 * 4 * kDmmaChains * static_cast<double>(iters) * grid * (256 / 32);
  *host_tflops = flops / (ms * 1e-3) / 1e12;
  return TRL_OK;
}

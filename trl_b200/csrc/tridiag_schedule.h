// Who takes part in which step of the cluster tridiagonalisation (k_tridiag): plain functions, so
// that the host can check them too. Row g of the matrix belongs to CTA g % kTriC; step s sends a
// pair of numbers per row g >= s to CTAs of the cluster with asynchronous stores.
#ifndef TRL_TRIDIAG_SCHEDULE_H
#define TRL_TRIDIAG_SCHEDULE_H

#ifdef __CUDACC__
#define TRL_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define TRL_HOST_DEVICE inline
#endif

namespace trl_detail {

constexpr int kTriC = 16; // CTAs in the cluster

// last row of CTA `cta`, -1 if there is no such CTA or it has no row (N < kTriC)
TRL_HOST_DEVICE int tri_last_row(int N, int cta) { return cta < kTriC && cta < N ? cta + ((N - 1 - cta) & ~(kTriC - 1)) : -1; }

// The warp with a CTA's last row arms the CTA's barrier for step s and waits for the pairs of all
// rows g >= s until that row is sent; after that nobody there waits.
TRL_HOST_DEVICE bool tri_waits(int N, int cta, int s) { return s < tri_last_row(N, cta); }

// Whether row g's pair of step s goes to CTA `cta`. Only to one that waits for it: an asynchronous
// store is complete for nobody but the receiver that sees its mbarrier's phase end (the cluster
// barrier at the kernel's end orders ordinary accesses), so one that nobody waits for might land in
// the shared memory of a CTA that has left.
TRL_HOST_DEVICE bool tri_sends(int N, int g, int cta, int s) { return g >= s && g < N && tri_waits(N, cta, s); }

} // namespace trl_detail

#endif

// Two kernels of one type ask for their CTAs per SM, without a device: each gets its own answer (its
// fallback), and keeps it.
#include "common.cuh"

#include <cstdio>

template <int N>
__global__ void k_nothing(int*)
{
}

int main()
{
  using trl_detail::resident_ctas;
  std::printf("%d", resident_ctas<k_nothing<1>>(0, 256, 0, 4));
  std::printf(" %d", resident_ctas<k_nothing<2>>(0, 256, 0, 2));
  std::printf(" %d", resident_ctas<k_nothing<1>>(0, 256, 0, 7));
  std::printf(" %d", resident_ctas<k_nothing<2>>(0, 256, 0, 7));
  std::printf(" %d\n", resident_ctas<k_nothing<1>>(1, 256, 0, 3)); // another device
}

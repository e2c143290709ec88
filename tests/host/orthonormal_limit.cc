// Prints, for numbers of vectors, the largest overlap that the second step is given.
#include "orthonormal_limit.h"

#include <cstdio>
#include <initializer_list>

int main()
{
  for (int K : {1, 2, 8, 40, 112, 256}) std::printf("%d %.17g\n", K, trl_detail::gs_limit(K));
}

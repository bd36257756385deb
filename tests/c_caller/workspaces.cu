// Prints, for every n of 3 .. 2048, the doubles the vectors of one real matrix have as workspace
// and the doubles their back-transformation needs for 2 n columns.  Host code only.
#include <stdio.h>

#include "skew_back.cuh"
#include "skew_internal.h"

int main() {
  for (int n = 3; n <= 2048; n++)
    printf("%d %zu %zu\n", n, skew::large_vectors_ws_doubles(n), skew::back_ws_doubles<false>(n, n - 2, 2 * n, 1));
  return 0;
}

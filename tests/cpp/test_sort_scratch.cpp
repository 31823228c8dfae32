// The sort scratch of worlds, the tick and the CK solver holds what the radix sort uses and nothing else;
// the estimate of its bytes (the server's budget) covers it.
#include <cstdio>
#include <cstdlib>

#include "../../ae-engine_b200/csrc/radix_sort.cuh"

static cudaError_t count(void* user, void** p, size_t bytes) {
  *static_cast<size_t*>(user) += bytes;
  return (*p = malloc(bytes)) ? cudaSuccess : cudaErrorMemoryAllocation;
}
static void release(void*, void* p) { free(p); }

int main() {
  for (const uint64_t n : {uint64_t(1), uint64_t(16384), uint64_t(16385), uint64_t(1000000)}) {
    const uint64_t tiles = aemp::sort_tiles(n);
    const size_t want = 4 * (2 * 256 * tiles + 4 * 256 + 3 * n);
    size_t got = 0;
    aemp::SortScratch s;
    if (aemp::sort_scratch_alloc(s, n, count, &got) != cudaSuccess) return 2;
    if (got != want || aemp::sort_scratch_bytes(n) < got || aemp::sort_scratch_bytes(n) > got + 7 * 256) {
      printf("n %zu: %zu bytes, %zu needed, %zu estimated\n", size_t(n), got, want, size_t(aemp::sort_scratch_bytes(n)));
      return 1;
    }
    aemp::sort_scratch_free(s, release, &got);
  }
  printf("ok\n");
  return 0;
}

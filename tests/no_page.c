/* Preloaded: aligned_alloc of a page fails while PD_TEST_NO_PAGE is set. */
#include <stdlib.h>

void* aligned_alloc(size_t alignment, size_t bytes) {
  void* p = NULL;
  if (alignment == 4096 && bytes == 4096 && getenv("PD_TEST_NO_PAGE")) return NULL;
  return posix_memalign(&p, alignment, bytes) ? NULL : p;
}

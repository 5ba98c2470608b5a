// operator new of the library's host code, which fails after a number of calls
#include <stdlib.h>

#include <new>

static long long left = -1;  // calls until it fails; < 0: it does not

extern "C" void fake_new_left(long long n) { left = n; }

void *operator new(size_t n) {
  if (left == 0) throw std::bad_alloc();
  if (left > 0) --left;
  if (void *p = malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }

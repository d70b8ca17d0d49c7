/* Preloaded ahead of the CUDA runtime: makes one of its host calls fail, as it
 * does when memory is short. FAIL_CALL names it; fail_calls_left(n) makes the
 * next n calls of it fail (none until then), fail_calls_after(k) the one after k. */
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdlib.h>
#include <string.h>

static int left = 0, skip = 0, failed = 0;
void fail_calls_left(int n) { left = n; }
void fail_calls_after(int k) { skip = k, left = 1; }
int fail_calls_failed(void) { return failed; }

static int fails(const char* name) {
  const char* want = getenv("FAIL_CALL");
  if (!want || strcmp(want, name) != 0 || left <= 0) return 0;
  if (skip > 0) return --skip, 0;
  --left;
  ++failed;
  return 1;
}

/* the runtime's own (it is loaded by then, and not into the global scope) */
static void* own(const char* name) {
  void* lib = dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD);
  return lib ? dlsym(lib, name) : 0;
}

/* cudaErrorMemoryAllocation */
enum { NO_MEMORY = 2 };

int cudaGraphInstantiate(void** exec, void* graph, unsigned long long flags) {
  static int (*real)(void**, void*, unsigned long long);
  if (fails("cudaGraphInstantiate")) return NO_MEMORY;
  if (!real) *(void**)&real = own("cudaGraphInstantiate");
  return !real ? NO_MEMORY : real(exec, graph, flags);
}

int cudaHostAlloc(void** p, size_t size, unsigned flags) {
  static int (*real)(void**, size_t, unsigned);
  if (fails("cudaHostAlloc")) return NO_MEMORY;
  if (!real) *(void**)&real = own("cudaHostAlloc");
  return !real ? NO_MEMORY : real(p, size, flags);
}

int cudaStreamWaitEvent(void* stream, void* event, unsigned flags) {
  static int (*real)(void*, void*, unsigned);
  if (fails("cudaStreamWaitEvent")) return NO_MEMORY;
  if (!real) *(void**)&real = own("cudaStreamWaitEvent");
  return !real ? NO_MEMORY : real(stream, event, flags);
}

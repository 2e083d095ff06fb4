/* Stand-in for a device with little memory: loaded with LD_PRELOAD before the CUDA
 * runtime, it refuses device allocations on the host and passes the others on.
 * alloc_refuse_from(n): after n more allocations, refuse every one (-1: none).
 * alloc_limit(bytes): refuse what would take the live total past the limit (0: none).
 * alloc_live(): bytes held now.  alloc_refused(): allocations refused so far. */
#define _GNU_SOURCE
#include <dlfcn.h>
#include <pthread.h>
#include <stddef.h>

enum { kOk = 0, kOutOfMemory = 2, kTable = 1 << 16 };
static pthread_mutex_t lock = PTHREAD_MUTEX_INITIALIZER;
static long granted = -1, refused = 0;
static size_t limit = 0, live = 0;
static struct { void* p; size_t n; } held[kTable];

void alloc_refuse_from(long n) { granted = n; }
void alloc_limit(size_t bytes) { limit = bytes; }
size_t alloc_live(void) { return live; }
long alloc_refused(void) { return refused; }

static int refuse(size_t n) {
  int r = 0;
  pthread_mutex_lock(&lock);
  if (granted == 0 || (limit && live + n > limit)) r = 1;
  if (granted > 0 && !r) --granted;
  refused += r;
  pthread_mutex_unlock(&lock);
  return r;
}

static int keep(int status, void* p, size_t n) {
  pthread_mutex_lock(&lock);
  for (int i = 0; status == kOk && i < kTable; ++i)
    if (!held[i].p) {
      held[i].p = p;
      held[i].n = n;
      live += n;
      break;
    }
  pthread_mutex_unlock(&lock);
  return status;
}

static void drop(void* p) {
  pthread_mutex_lock(&lock);
  for (int i = 0; p && i < kTable; ++i)
    if (held[i].p == p) {
      live -= held[i].n;
      held[i].p = NULL;
      break;
    }
  pthread_mutex_unlock(&lock);
}

/* the runtime's own function: the library that uses it has loaded it by now */
static void* real(const char* name) {
  return dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), name);
}

int cudaMalloc(void** p, size_t n) {
  if (refuse(n)) return kOutOfMemory;
  const int status = ((int (*)(void**, size_t))real("cudaMalloc"))(p, n);
  return keep(status, *p, n);
}

int cudaMallocFromPoolAsync(void** p, size_t n, void* pool, void* stream) {
  if (refuse(n)) return kOutOfMemory;
  const int status = ((int (*)(void**, size_t, void*, void*))real("cudaMallocFromPoolAsync"))(
      p, n, pool, stream);
  return keep(status, *p, n);
}

int cudaFree(void* p) {
  drop(p);
  return ((int (*)(void*))real("cudaFree"))(p);
}

int cudaFreeAsync(void* p, void* stream) {
  drop(p);
  return ((int (*)(void*, void*))real("cudaFreeAsync"))(p, stream);
}

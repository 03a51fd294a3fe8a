/* Loaded before the CUDA runtime (LD_PRELOAD): counts the pool allocations that are
 * out and fails the one asked for, for tests of what a call does without memory. */
#include <dlfcn.h>
#include <pthread.h>
#include <stddef.h>

#define MAX_OUT 65536

static pthread_mutex_t mu = PTHREAD_MUTEX_INITIALIZER;
static void* out[MAX_OUT];
static int n_out;
static long made, fail_at = -1;
static size_t failed_bytes;

/* The runtime is loaded later, with the library that needs it. */
static void* real_of(const char* name)
{
	void* h = dlopen("libcudart.so.13", RTLD_LAZY);
	return h ? dlsym(h, name) : NULL;
}

int cudaMallocFromPoolAsync(void** p, size_t bytes, void* pool, void* stream)
{
	static int (*real)(void**, size_t, void*, void*);
	int rc;
	pthread_mutex_lock(&mu);
	if (!real) real = (int (*)(void**, size_t, void*, void*)) real_of("cudaMallocFromPoolAsync");
	if (made++ == fail_at) {
		failed_bytes = bytes;
		rc = 2; /* cudaErrorMemoryAllocation */
	} else {
		rc = real(p, bytes, pool, stream);
		if (rc == 0 && n_out < MAX_OUT) out[n_out++] = *p;
	}
	pthread_mutex_unlock(&mu);
	return rc;
}

int cudaFreeAsync(void* p, void* stream)
{
	static int (*real)(void*, void*);
	int i;
	pthread_mutex_lock(&mu);
	if (!real) real = (int (*)(void*, void*)) real_of("cudaFreeAsync");
	for (i = n_out - 1; i >= 0; --i)
		if (out[i] == p) { out[i] = out[--n_out]; break; }
	pthread_mutex_unlock(&mu);
	return real(p, stream);
}

/* The k-th allocation from now fails (k < 0: none does). */
void failalloc_next(long k)
{
	pthread_mutex_lock(&mu);
	fail_at = k < 0 ? -1 : made + k;
	failed_bytes = 0;
	pthread_mutex_unlock(&mu);
}

int failalloc_out(void) { return n_out; }
long failalloc_failed_bytes(void) { return (long) failed_bytes; }

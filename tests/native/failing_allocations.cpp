/*
 * A preloaded stand-in for a machine with less memory: cudaMalloc fails where
 * the device memory in use would pass a budget, and operator new, called from
 * a named library, throws at a chosen call.  A test sets both through the
 * functions below (ctypes on the running process).
 */
#include <dlfcn.h>
#include <stdlib.h>
#include <string.h>

#include <map>
#include <mutex>
#include <new>

typedef int (*malloc_t)(void **, size_t);
typedef int (*free_t)(void *);

static std::mutex lock;
static size_t budget = ~(size_t)0, in_use, peak;
static long refused;
static char library[256];       /* whose calls of operator new count */
static long at, calls;          /* the call that throws (0: none); calls so far */

static std::map<void *, size_t> &blocks()
{
	static std::map<void *, size_t> *m = new std::map<void *, size_t>;
	return *m;
}

static void *runtime(const char *name)
{
	void *h = dlopen("libcudart.so.13", RTLD_NOLOAD | RTLD_LAZY);
	void *f = h ? dlsym(h, name) : NULL;
	if (!f) abort();
	return f;
}

extern "C" int cudaMalloc(void **p, size_t n)
{
	static malloc_t real = (malloc_t)runtime("cudaMalloc");
	{
		std::lock_guard<std::mutex> g(lock);
		if (in_use + n > budget) {
			refused++;
			*p = NULL;
			return 2;       /* cudaErrorMemoryAllocation */
		}
	}
	const int e = real(p, n);
	std::lock_guard<std::mutex> g(lock);
	if (e == 0) {
		blocks()[*p] = n;
		in_use += n;
		peak = in_use > peak ? in_use : peak;
	}
	return e;
}

extern "C" int cudaFree(void *p)
{
	static free_t real = (free_t)runtime("cudaFree");
	{
		std::lock_guard<std::mutex> g(lock);
		auto b = blocks().find(p);
		if (b != blocks().end()) {
			in_use -= b->second;
			blocks().erase(b);
		}
	}
	return real(p);
}

void *operator new(size_t n)
{
	Dl_info i;
	if (library[0] && dladdr(__builtin_return_address(0), &i) && i.dli_fname && strstr(i.dli_fname, library) && ++calls == at)
		throw std::bad_alloc();
	void *p = malloc(n ? n : 1);
	if (!p) throw std::bad_alloc();
	return p;
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }

extern "C" void fa_budget(size_t bytes) { budget = bytes; refused = 0; peak = in_use; }
extern "C" size_t fa_peak(void) { return peak; }
extern "C" long fa_refused(void) { return refused; }
extern "C" void fa_new(const char *lib, long call)
{
	strncpy(library, lib, sizeof library - 1);
	at = call;
	calls = 0;
}
extern "C" long fa_calls(void) { return calls; }

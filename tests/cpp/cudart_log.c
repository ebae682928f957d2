/* Preloaded in front of the CUDA runtime by tests that check what the library asks of it: writes a
 * line to the file named by CUDART_LOG for every shared-memory limit set ("smem <kernel> <bytes>") and
 * every page-locked block taken and given back ("lock <address> <bytes>", "unlock <address>"), and a
 * line of the test's own for every cudart_log_mark(text). */
#include <dlfcn.h>
#include <stdarg.h>
#include <stddef.h>
#include <stdio.h>
#include <stdlib.h>

static void line(const char * format, ...)
{
    FILE * f = fopen(getenv("CUDART_LOG"), "a");
    if (!f) return;
    va_list args;
    va_start(args, format);
    vfprintf(f, format, args);
    va_end(args);
    fclose(f);
}

/* the runtime's own function (the library that asks for it is loaded with its symbols kept local) */
static void * runtime(const char * name)
{
    void * f = dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), name);
    if (!f) abort();
    return f;
}

void cudart_log_mark(const char * text) { line("%s\n", text); }

int cudaFuncSetAttribute(const void * kernel, int attribute, int value)
{
    int (*next)(const void *, int, int) = (int (*)(const void *, int, int)) runtime("cudaFuncSetAttribute");
    if (attribute == 8) line("smem %p %d\n", kernel, value);       /* cudaFuncAttributeMaxDynamicSharedMemorySize */
    return next(kernel, attribute, value);
}

int cudaHostAlloc(void ** p, size_t bytes, unsigned flags)
{
    int (*next)(void **, size_t, unsigned) = (int (*)(void **, size_t, unsigned)) runtime("cudaHostAlloc");
    const int e = next(p, bytes, flags);
    if (e == 0) line("lock %p %zu\n", *p, bytes);
    return e;
}

int cudaFreeHost(void * p)
{
    int (*next)(void *) = (int (*)(void *)) runtime("cudaFreeHost");
    line("unlock %p\n", p);
    return next(p);
}

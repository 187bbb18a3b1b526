// Test-only: a process that cannot start threads. Its pthread_create lets the
// first argv[1] threads start and refuses the rest. What is printed must not
// depend on argv[1]: the spectral tables (akvisqol_b200/csrc/spectral_tables.cpp)
// as a checksum, the items that run_threads (akvisqol_b200/csrc/threads.h)
// worked through, and an exception out of a worker, caught by its caller.
#ifndef _GNU_SOURCE
#define _GNU_SOURCE
#endif
#include <dlfcn.h>
#include <pthread.h>

#include <atomic>
#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>

#include "../../akvisqol_b200/csrc/host_model.h"
#include "../../akvisqol_b200/csrc/spectral_tables.h"
#include "../../akvisqol_b200/csrc/threads.h"

static std::atomic<int> left{0};

extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg) {
    using Create = int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
    static const Create real = reinterpret_cast<Create>(dlsym(RTLD_NEXT, "pthread_create"));
    return left-- > 0 ? real(t, a, f, arg) : EAGAIN;
}

static void add(unsigned long long &h, const void *p, size_t n) {
    for (size_t i = 0; i < n; ++i) h = (h ^ static_cast<const unsigned char *>(p)[i]) * 1099511628211ull;
}

int main(int, char **argv) {
    using namespace vqb;
    left = std::atoi(argv[1]);
    const host::Filterbank fb = host::make_filterbank(32, 16000, 50.0, 8000.0);
    const auto t = spectral_tables(fb.run, 1280);
    unsigned long long h = 14695981039346656037ull;
    add(h, t->weights.data(), t->weights.size() * sizeof(double));
    add(h, t->tails.data(), t->tails.size() * sizeof(double));
    std::printf("%016llx\n", h);

    left = std::atoi(argv[1]);
    std::atomic<int> next{0}, sum{0};
    run_threads(6, [&](size_t) {
        for (int i = next++; i < 1000; i = next++) sum += i;
    });
    std::printf("%d\n", sum.load());

    left = std::atoi(argv[1]);
    try {
        run_threads(4, [&](size_t) { throw std::bad_alloc(); });
        std::printf("no exception\n");
    } catch (const std::bad_alloc &) {
        std::printf("caught\n");
    }
}

// The thread pool (host_pool.h) where the process may start only argv[1] more threads: every job is done all the same. Stands
// in front of pthread_create, so that no limit of the machine has to be touched. Exit code 0: everything was done.
// With "quota" and the paths of a list of control groups and of their root: prints the cpus they grant; with "workers", a number of
// cpus and a quota: the pool's threads.
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
#include <cstdio>
#include <cstdlib>
#include "../msnhnet_b200/csrc/host_pool.h"

static std::atomic<int> g_left{0};

extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*fn)(void *), void *arg) {
    static auto real = reinterpret_cast<int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *)>(dlsym(RTLD_NEXT, "pthread_create"));
    if (g_left.fetch_sub(1) <= 0) return EAGAIN;
    return real(t, a, fn, arg);
}

int main(int argc, char **argv) {
    if (argc > 3 && argv[1][0] == 'w') { std::printf("%d\n", msnh::HostPool::workers_for(std::atoi(argv[2]), std::atoi(argv[3]))); return 0; }   // workers <cpus> <quota>
    if (argc > 3) { std::printf("%d\n", msnh::cpu_quota(argv[2], argv[3])); return 0; }        // quota <groups> <root>
    const int may_start = argc > 1 ? std::atoi(argv[1]) : 0;
    g_left = may_start;
    std::vector<int> done(1000, 0);
    {
        msnh::HostPool pool(7);
        for (int n : {1, 3, 1000, 40}) {
            std::fill(done.begin(), done.end(), 0);
            pool.run(n, [&](int i) { ++done[i]; });
            for (int i = 0; i < 1000; ++i) if (done[i] != (i < n)) { std::printf("job of %d: item %d ran %d times\n", n, i, done[i]); return 1; }
        }
        if (pool.workers() != std::min(may_start, 7)) { std::printf("%d workers\n", pool.workers()); return 1; }
    }
    for (int threads : {1, 2, 16}) {
        g_left = may_start;
        std::fill(done.begin(), done.end(), 0);
        msnh::strided_rows(1000, threads, [&](int i) { ++done[i]; });
        for (int i = 0; i < 1000; ++i) if (done[i] != 1) { std::printf("%d threads: row %d ran %d times\n", threads, i, done[i]); return 1; }
    }
    return 0;
}

// operator new that fails when it is told to, for a process this library is preloaded into: fail_new_at(k) lets the k-th allocation of
// this thread from now on throw std::bad_alloc (k < 0: none); it returns how many there were since the last call.
#include <cstdlib>
#include <new>

static thread_local long g_at = -1, g_count = 0;

extern "C" long fail_new_at(long k) { const long n = g_count; g_count = 0; g_at = k; return n; }

void *operator new(std::size_t n) {
    if (g_count++ == g_at) throw std::bad_alloc();
    if (void *p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void *operator new[](std::size_t n) { return operator new(n); }
void operator delete(void *p) noexcept { std::free(p); }
void operator delete[](void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }
void operator delete[](void *p, std::size_t) noexcept { std::free(p); }

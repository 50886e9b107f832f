// Allocation that, while g_strict is set, fails on every thread but those that set t_first.
#include <cstdlib>
#include <new>

thread_local bool t_first = false;
bool g_strict = false;

void *operator new(std::size_t n) {
    if (g_strict && !t_first) throw std::bad_alloc();
    if (void *p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }

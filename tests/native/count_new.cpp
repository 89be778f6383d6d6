// Preloaded by tests/test_host_calls_alloc.py: counts operator new while armed.
#include <atomic>
#include <cstdlib>
#include <new>

static std::atomic<bool> armed{false};
static std::atomic<long> calls{0};

extern "C" void cn_arm() {
    calls = 0;
    armed = true;
}
extern "C" long cn_disarm() {
    armed = false;
    return calls;
}

void* operator new(std::size_t n) {
    if (armed.load(std::memory_order_relaxed)) calls.fetch_add(1, std::memory_order_relaxed);
    if (void* p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

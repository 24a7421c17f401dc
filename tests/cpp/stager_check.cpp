// The staging of host arrays when memory runs out while its threads are started: the constructor either
// reports it or carries on with the threads that run, and nothing ends the process.  Needs no device (without one the threads
// stop at once; with one they fill the ring and wait).  Prints "k threads" for the k-th allocation failing (-1: reported).
#include "host_pipeline.cu"
#include <cstdio>
#include <cstdlib>
#include <new>

namespace {
std::atomic<long> g_left{ 1000000 };
}

void* operator new(std::size_t n)
{
    if(--g_left == 0) throw std::bad_alloc();
    if(void* p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

int main()
{
    static char src[16], dst[16], ring[agb::RING * agb::PIECE];
    for(int k = 1; k <= 7; k++) {
        agb::StreamSet set;
        set.device = 0;
        set.ring = ring;
        std::vector<agb::Piece> pieces(20, agb::Piece{ src, dst, sizeof(src) });
        int running = -1;
        try {
            g_left = k;
            agb::Stager s(&set, std::move(pieces));
            g_left = 1000000;
            running = s.running();
        } catch(const std::bad_alloc&) {}
        g_left = 1000000;
        std::printf("%d %d\n", k, running);
    }
    return 0;
}

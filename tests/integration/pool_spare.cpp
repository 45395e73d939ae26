// Buffers that a call can do without: from the idle ones or from what the allocator has left, never from idle buffers that would have to go back to it, and
// without an error when there are none.  Prints what fails; 0 when nothing does.
#include "pool.hpp"

#include <cstdio>
#include <cstdlib>

static size_t room = 1 << 20;
static std::unordered_map<void *, size_t> sizes;
static cudaError_t last = cudaSuccess;
extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
    if (n > room) return last = cudaErrorMemoryAllocation;
    *p = std::malloc(n); sizes[*p] = n; room -= n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) { room += sizes[p]; sizes.erase(p); std::free(p); return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
}

static int bad = 0;
#define EXPECT(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); ++bad; } } while (0)

int main() {
    Pool pool;
    void *idle = pool.get(4096);
    pool.put(idle);
    EXPECT(pool.spare(1 << 20) == nullptr && last == cudaSuccess); // would only fit without the idle buffer
    EXPECT(sizes.count(idle) && pool.total == 4096 && pool.in_use == 0);
    EXPECT(pool.get(4096) == idle);
    pool.put(idle);
    void *p = pool.spare(4000); // an idle one of its size
    EXPECT(p == idle && pool.in_use == 4096 && pool.total == 4096);
    pool.put(p);
    Pool::Buffers graph;
    pool.recording = &graph;
    void *q = pool.spare(1 << 19);
    EXPECT(q && graph.count(q) && pool.total == 4096 + (1 << 19));
    pool.put(q);
    EXPECT(pool.spare(1 << 20) == nullptr && graph.size() == 1);
    pool.recording = nullptr;
    pool.unhold(graph);
    void *need = pool.get((1 << 20) - 8192); // what a call must have still takes the place of an idle buffer
    EXPECT(need && !sizes.count(q));
    pool.put(nullptr);
    return bad != 0;
}

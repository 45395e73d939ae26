// The context's pool over a stand-in for the CUDA allocator that knows what is allocated and can run out: buffers that a recorded graph
// addresses are never given back to the driver while the graph lives, whoever asks.  Prints what fails; 0 when nothing does.
#include "pool.hpp"

#include <cstdio>
#include <cstdlib>
#include <set>

static std::set<void *> allocated;
static size_t room = 1 << 20;
static std::unordered_map<void *, size_t> sizes;
static cudaError_t last = cudaSuccess;
extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
    if (n > room) return last = cudaErrorMemoryAllocation;
    *p = std::malloc(n); allocated.insert(*p); sizes[*p] = n; room -= n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    if (!allocated.erase(p)) { std::puts("freed twice"); std::exit(2); }
    room += sizes[p]; std::free(p);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
}

static int bad = 0;
#define EXPECT(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); ++bad; } } while (0)
static bool oom(Pool &p, size_t n, bool raw) {
    try { raw ? p.raw(n) : p.get(n); } catch (const ArgFail &e) { return e.code == HB_E_OOM && last == cudaSuccess; }
    return false;
}

int main() {
    {
        Pool pool;
        Pool::Buffers first, second;
        void *operand = pool.get(1000), *before = pool.get(2048);
        pool.put(before);
        pool.recording = &first; // a pass: a temporary that comes back, a result that stays, a buffer that was idle before
        void *tmp = pool.get(4096), *result = pool.get(8192);
        EXPECT(pool.get(2048) == before);
        pool.put(tmp); pool.put(before);
        EXPECT(pool.get(4096) == tmp);
        pool.put(tmp);
        void *idle_then = tmp;
        EXPECT(oom(pool, 2 << 20, false)); // the retry that empties the pool, in the middle of a recording
        EXPECT(allocated.count(idle_then) && allocated.count(before));
        pool.recording = &second;
        EXPECT(pool.get(4096) == tmp);
        pool.put(tmp);
        pool.recording = nullptr;
        EXPECT(first.size() == 3 && second.size() == 1);
        void *other = pool.get(16384);
        pool.put(other);
        pool.release_cached();
        EXPECT(!allocated.count(other));
        EXPECT(allocated.count(tmp) && allocated.count(before) && allocated.count(result) && allocated.count(operand));
        EXPECT(pool.get(4096) == tmp); // idle buffers of a graph still serve other calls
        pool.put(tmp);
        EXPECT(oom(pool, 2 << 20, false) && oom(pool, 2 << 20, true));
        EXPECT(allocated.count(tmp) && allocated.count(before));
        pool.unhold(first);
        pool.put(result);
        pool.release_cached();
        EXPECT(allocated.count(tmp) && !allocated.count(before) && !allocated.count(result)); // the second graph still has tmp
        pool.unhold(second);
        pool.release_cached();
        EXPECT(!allocated.count(tmp) && pool.held_.empty());
        EXPECT(pool.total == 1024 && pool.in_use == 1024 && allocated.size() == 1);
        void *big = pool.get(1 << 19);
        pool.put(big);
        void *p = pool.raw((1 << 20) - 4096); // only fits once the idle buffer went back
        EXPECT(allocated.count(p) && allocated.size() == 2 && pool.total == 1024 && last == cudaSuccess);
        cudaFree(p);
        pool.recording = &first;
        first.clear();
        pool.put(pool.get(512));
        pool.recording = nullptr;
    }
    EXPECT(allocated.empty()); // a pool that goes takes the buffers of its graphs with it
    return bad != 0;
}

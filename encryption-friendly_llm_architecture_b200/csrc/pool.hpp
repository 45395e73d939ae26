// Size-bucketed caching allocator of a context: the matmul schedules allocate and free the same few buffer sizes thousands of times;
// cudaMalloc is reached only the first time a size is seen.
#pragma once
#include "../../include/hemmer_b200.h"

#include <cuda_runtime_api.h>

#include <string>
#include <unordered_map>
#include <unordered_set>
#include <vector>

struct ArgFail { int code; std::string msg; };
[[noreturn]] inline void fail(int code, const std::string &m) { throw ArgFail{code, m}; }

struct Pool {
    using Buffers = std::unordered_set<void *>;
    std::unordered_map<size_t, std::vector<void *>> free_;
    std::unordered_map<void *, size_t> live_;
    std::unordered_map<void *, int> held_; // addresses in recorded graphs, with the number of those graphs: idle or not, they stay allocated
    Buffers *recording = nullptr;          // takes what is handed out while a graph records
    size_t total = 0, in_use = 0;

    // Device memory that does not come back to the pool: from the driver, if need be after the pool's idle buffers went back to it.
    void *raw(size_t bytes) {
        void *p = nullptr;
        cudaError_t e = cudaMalloc(&p, bytes);
        if (e != cudaSuccess) { cudaGetLastError(); release_cached(); e = cudaMalloc(&p, bytes); } // the first failure must not stay behind as the last error
        if (e != cudaSuccess) { cudaGetLastError(); fail(HB_E_OOM, "device allocation of " + std::to_string(bytes) + " bytes failed"); }
        return p;
    }
    void *get(size_t bytes) {
        bytes = (bytes + 255) & ~(size_t)255;
        void *p = idle(bytes);
        if (!p) { p = raw(bytes); total += bytes; }
        return hand_out(p, bytes);
    }
    // A buffer that the caller can do without: an idle one or what the driver has left; null otherwise, and no idle buffer goes back to the driver for it.
    void *spare(size_t bytes) {
        bytes = (bytes + 255) & ~(size_t)255;
        void *p = idle(bytes);
        if (!p) {
            if (cudaMalloc(&p, bytes) != cudaSuccess) { cudaGetLastError(); return nullptr; }
            total += bytes;
        }
        return hand_out(p, bytes);
    }
    void put(void *p) {
        if (!p) return;
        auto it = live_.find(p);
        if (it == live_.end()) return;
        free_[it->second].push_back(p); in_use -= it->second; live_.erase(it);
    }
    void unhold(const Buffers &graph) {
        for (void *p : graph) {
            auto it = held_.find(p);
            if (it != held_.end() && --it->second == 0) held_.erase(it);
        }
    }
    // A graph writes to the buffers that it was recorded with although they are idle between two replays, so those stay.
    void release_cached() {
        for (auto &kv : free_) {
            std::vector<void *> stay;
            for (void *p : kv.second) {
                if (held_.count(p)) { stay.push_back(p); continue; }
                cudaFree(p); total -= kv.first;
            }
            kv.second.swap(stay);
        }
    }
    ~Pool() { held_.clear(); release_cached(); for (auto &kv : live_) cudaFree(kv.first); }

private:
    void *idle(size_t bytes) {
        auto &v = free_[bytes];
        if (v.empty()) return nullptr;
        void *p = v.back();
        v.pop_back();
        return p;
    }
    void *hand_out(void *p, size_t bytes) {
        live_[p] = bytes; in_use += bytes;
        if (recording && recording->insert(p).second) ++held_[p];
        return p;
    }
};

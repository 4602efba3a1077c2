// Page-locked blocks for results that kernels write straight to the host: cudaMallocHost takes longer than a small
// proof, so freed blocks are kept (at most MAX_KEPT, the rest go back to the driver). Any thread may take or give one;
// the owner has synchronised with whatever wrote the block before it gives it back.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <mutex>
#include <vector>

namespace mbhost {

class PinnedPool {
public:
    static constexpr size_t WORDS = 8192;   // 64 KB
    static constexpr size_t MAX_KEPT = 32;
    static uint64_t* take() {
        PinnedPool& p = instance();
        {
            std::lock_guard<std::mutex> lk(p.mu_);
            if (!p.free_.empty()) {
                uint64_t* b = p.free_.back();
                p.free_.pop_back();
                return b;
            }
        }
        uint64_t* b = nullptr;
        return cudaHostAlloc(reinterpret_cast<void**>(&b), WORDS * sizeof(uint64_t), cudaHostAllocPortable) == cudaSuccess ? b : nullptr;
    }
    static void give(uint64_t* b) {
        if (!b) return;
        PinnedPool& p = instance();
        {
            std::lock_guard<std::mutex> lk(p.mu_);
            if (p.free_.size() < MAX_KEPT) {
                p.free_.push_back(b);
                return;
            }
        }
        cudaFreeHost(b);
    }

private:
    static PinnedPool& instance() {
        static PinnedPool* p = new PinnedPool;   // never destroyed: proofs may end during process exit
        return *p;
    }
    std::mutex mu_;
    std::vector<uint64_t*> free_;
};

}  // namespace mbhost

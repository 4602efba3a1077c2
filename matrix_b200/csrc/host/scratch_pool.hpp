// Scratch of a prover's passes: a page-locked block for results that kernels write straight to the host, and a device block
// for the sums over blocks, which is zero whenever no kernel is using it (a kernel's last block puts it back,
// pair_kernels.cuh). Allocating and clearing the two takes longer than a small proof, so freed pairs are kept (at most
// MAX_KEPT, the rest go back to the driver). Any thread may take or give one. When the owner gives a pair back, nothing
// may touch it any more: it has synchronised with whatever wrote the blocks, or has waited for a word whose store was the last access
// to either of them, behind a fence (reduce_tc_partials_kernel). It discards them if that went wrong.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <mutex>
#include <vector>

namespace mbhost {

struct ScratchBlock {
    uint64_t *host = nullptr, *dev = nullptr;
    int device = -1;
    explicit operator bool() const { return host != nullptr; }
};
class ScratchPool {
public:
    static constexpr size_t WORDS = 8192;       // host: 64 KB
    static constexpr size_t DEV_WORDS = 33280;  // device: 260 KB (64 instances of sixteen sums in eight copies)
    static constexpr size_t MAX_KEPT = 32;
    static ScratchBlock take() {
        ScratchBlock b;
        int device = 0;
        if (cudaGetDevice(&device) != cudaSuccess) return b;
        ScratchPool& p = instance();
        {
            std::lock_guard<std::mutex> lk(p.mu_);
            for (size_t i = p.free_.size(); i-- > 0;)
                if (p.free_[i].device == device) {
                    b = p.free_[i];
                    p.free_.erase(p.free_.begin() + i);
                    return b;
                }
        }
        b.device = device;
        if (cudaHostAlloc(reinterpret_cast<void**>(&b.host), WORDS * sizeof(uint64_t), cudaHostAllocPortable) != cudaSuccess ||
            cudaMalloc(reinterpret_cast<void**>(&b.dev), DEV_WORDS * sizeof(uint64_t)) != cudaSuccess ||
            cudaMemsetAsync(b.dev, 0, DEV_WORDS * sizeof(uint64_t), cudaStreamPerThread) != cudaSuccess ||
            cudaStreamSynchronize(cudaStreamPerThread) != cudaSuccess) {
            discard(b);
            b = ScratchBlock{};
        }
        return b;
    }
    // Once nothing touches it any more (above); clean: that went well, the device block is zero again.
    static void give(ScratchBlock b, bool clean) {
        if (!b) return;
        ScratchPool& p = instance();
        if (clean) {
            std::lock_guard<std::mutex> lk(p.mu_);
            if (p.free_.size() < MAX_KEPT) {
                p.free_.push_back(b);
                return;
            }
        }
        discard(b);
    }

private:
    static void discard(ScratchBlock b) {
        if (b.host) cudaFreeHost(b.host);
        if (b.dev) cudaFree(b.dev);
    }
    static ScratchPool& instance() {
        static ScratchPool* p = new ScratchPool;   // never destroyed: proofs may end during process exit
        return *p;
    }
    std::mutex mu_;
    std::vector<ScratchBlock> free_;
};

}  // namespace mbhost

// fl_blocks.h -- device blocks of a context's problems and workspaces.
//
// Mapping and unmapping device memory is what a short call on a fresh problem
// used to wait for: of 5.4 ms for a propagation at Nt = 2^12 with five save
// positions, 0.8 ms in cudaMalloc and 0.8 ms in cudaFree, beside 3.5 ms of
// kernels.  Released blocks are kept for the next object of the context: at
// most kKeep bytes and, where the context has a memory budget, no more than
// the blocks in use leave of it.  They are given back with the context and
// before an allocation fails, of this cache or of one that names it as its
// lender.  A block is reused only after the context's stream has run dry.
#pragma once
#include <algorithm>
#include <memory>
#include <mutex>
#include <vector>

#include <cuda_runtime_api.h>

namespace fl {

class BlockCache {
public:
    static constexpr size_t kKeep = size_t(256) << 20;

    explicit BlockCache(size_t budget_bytes = 0) : budget(budget_bytes) {}
    BlockCache(const BlockCache&) = delete;
    BlockCache& operator=(const BlockCache&) = delete;

    cudaError_t alloc(void** out, size_t bytes) {
        std::lock_guard<std::mutex> lk(mu);
        *out = nullptr;
        bytes = (std::max<size_t>(bytes, 1) + 511) & ~size_t(511);
        // the smallest spare block that wastes no more than half of itself
        size_t best = spare.size();
        for (size_t i = 0; i < spare.size(); i++)
            if (spare[i].bytes >= bytes && spare[i].bytes <= 2 * bytes &&
                (best == spare.size() || spare[i].bytes < spare[best].bytes))
                best = i;
        Block b{nullptr, bytes, true};
        if (best < spare.size() && settle(spare[best])) {
            b = spare[best];
            spare.erase(spare.begin() + best);
            kept -= b.bytes;
        } else {
            cudaError_t e = cudaMalloc(&b.p, bytes);
            if (e == cudaErrorMemoryAllocation && give_back()) {
                cudaGetLastError();
                e = cudaMalloc(&b.p, bytes);
            }
            if (e != cudaSuccess) return e;
        }
        live.push_back(b);
        used += b.bytes;
        trim(room());
        *out = b.p;
        return cudaSuccess;
    }
    // The stream is not touched here (its owner may have destroyed it since
    // the last call): a kept block waits for it when it is reused.
    void release(void* p) {
        if (!p) return;
        std::lock_guard<std::mutex> lk(mu);
        for (size_t i = 0; i < live.size(); i++) {
            if (live[i].p != p) continue;
            Block b = live[i];
            live.erase(live.begin() + i);
            used -= b.bytes;
            if (!open || b.bytes > kKeep / 2) {
                cudaFree(p);
                return;
            }
            b.settled = false;
            spare.push_back(b);
            kept += b.bytes;
            trim(room());
            return;
        }
    }
    // the context's next stream; the one before has run dry
    void set_stream(cudaStream_t s) {
        std::lock_guard<std::mutex> lk(mu);
        stream = s;
        for (auto& b : spare) b.settled = true;
    }
    // the cache whose spare blocks go before an allocation of this one fails
    void set_lender(std::shared_ptr<BlockCache> c) { lender = std::move(c); }
    // nothing is kept from here on
    void close() {
        std::lock_guard<std::mutex> lk(mu);
        open = false;
        trim(0);
    }

private:
    struct Block {
        void* p;
        size_t bytes;
        bool settled;  // no work on it is queued
    };
    std::mutex mu;
    bool open = true;                // the context is alive
    cudaStream_t stream = nullptr;   // its stream
    size_t budget, used = 0, kept = 0;
    std::vector<Block> live, spare;  // spare: oldest first
    std::shared_ptr<BlockCache> lender;

    size_t room() const {
        return budget ? std::min(kKeep, budget - std::min(budget, used)) : kKeep;
    }
    bool settle(const Block& b) {
        if (b.settled) return true;
        if (cudaStreamSynchronize(stream) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        for (auto& s : spare) s.settled = true;
        return true;
    }
    // all spare blocks, this cache's and the lender's; whether there were any
    bool give_back() {
        bool any = !spare.empty();
        trim(0);
        if (lender) {
            std::lock_guard<std::mutex> lk(lender->mu);
            any |= !lender->spare.empty();
            lender->trim(0);
        }
        return any;
    }
    void trim(size_t limit) {
        size_t n = 0;
        while (kept > limit && n < spare.size()) {
            kept -= spare[n].bytes;
            cudaFree(spare[n++].p);
        }
        spare.erase(spare.begin(), spare.begin() + n);
    }
};

}  // namespace fl

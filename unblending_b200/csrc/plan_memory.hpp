// Device memory of a batched pass's plan, handed on from plan to plan.
#pragma once
#include <algorithm>
#include <cstddef>
#include <memory>
#include <new>
#include <vector>

namespace unb {

// Cuts a plan's buffers from a few chunks, which the next plan takes over: some
// thirty allocations and frees per new job list, several hundred MB with the
// lanes' records, cost more than the solves at times (two lists of ten images
// in turn: 53-250 ms a call, up to 1,013; kept chunks: 46-48 ms). A Block owns
// one allocation: get<T>(count) makes it or throws std::bad_alloc; ptr, bytes.
template <class Block> class PlanMemory {
public:
    static constexpr size_t kChunk = size_t(32) << 20;
    size_t chunk = kChunk;   // the least size of a chunk; 0: every buffer its own

    template <class T> T* alloc(size_t count) {
        const size_t want = (std::max<size_t>(count * sizeof(T), 1) + 255) / 256 * 256;
        // The chunk with the least room that holds it: small tables stay out of the large chunks.
        size_t best = chunks_.size();
        for (size_t k = 0; k < chunks_.size(); ++k)
            if (room(k) >= want && (best == chunks_.size() || room(k) < room(best))) best = k;
        if (best == chunks_.size()) {
            auto fresh = std::make_unique<Block>();
            fresh->template get<unsigned char>(std::max(want, chunk));
            chunks_.push_back(std::move(fresh));
            used_.push_back(0);
        }
        T* p = reinterpret_cast<T*>(static_cast<unsigned char*>(chunks_[best]->ptr) + used_[best]);
        used_[best] += want;
        return p;
    }

    // The work on the old plan's memory must have ended.
    void take(PlanMemory& old) {
        chunks_ = std::move(old.chunks_);
        used_.assign(chunks_.size(), 0);
    }

    // Frees the chunks that this plan left empty, once they are more than half of what it holds.
    void give_back() {
        size_t held = 0, empty = 0;
        for (size_t k = 0; k < chunks_.size(); ++k) {
            held += chunks_[k]->bytes;
            if (!used_[k]) empty += chunks_[k]->bytes;
        }
        if (2 * empty <= held) return;
        for (size_t k = chunks_.size(); k-- > 0;)
            if (!used_[k]) {
                chunks_.erase(chunks_.begin() + k);
                used_.erase(used_.begin() + k);
            }
    }

private:
    size_t room(size_t k) const { return chunks_[k]->bytes - used_[k]; }

    std::vector<std::unique_ptr<Block>> chunks_;
    std::vector<size_t> used_;
};

// The plan that follows `last`: made by build(plan) on the memory of `last`,
// whose work has ended. Where that and what build adds to it do not fit on the
// device together, all of it is freed and build runs once more, each buffer an
// allocation of its size.
template <class Plan, class Build> std::unique_ptr<Plan> next_plan(std::unique_ptr<Plan>& last, Build&& build) {
    {
        auto plan = std::make_unique<Plan>();
        if (last) plan->memory.take(last->memory);
        last.reset();
        try {
            build(*plan);
            plan->memory.give_back();
            return plan;
        } catch (const std::bad_alloc&) {
        }
    }
    auto plan = std::make_unique<Plan>();
    plan->memory.chunk = 0;
    build(*plan);
    return plan;
}

}  // namespace unb

// unb::PlanMemory and unb::next_plan on a host "device" of a given capacity:
// what fits when the last plan is freed first has to fit.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <map>

#include "plan_memory.hpp"

static size_t capacity = 0, live = 0, calls = 0;

struct Block {
    void* ptr = nullptr;
    size_t bytes = 0;
    Block() = default;
    Block(const Block&) = delete;
    ~Block() { live -= bytes; std::free(ptr); }
    template <class T> T* get(size_t count) {
        const size_t want = count * sizeof(T);
        ++calls;
        if (live + want > capacity) throw std::bad_alloc();
        ptr = std::aligned_alloc(256, (want + 255) / 256 * 256);   // (never touched)
        bytes = want;
        live += want;
        return static_cast<T*>(ptr);
    }
};
struct Plan {
    unb::PlanMemory<Block> memory;
    std::map<uintptr_t, size_t> parts;
};

static int failures = 0;
static void expect(bool ok, const char* what) {
    if (!ok) { ++failures; std::printf("failed: %s\n", what); }
}

static constexpr size_t MB = size_t(1) << 20;

// Plans of the given sizes in turn; whether each could be made.
static bool follow(std::unique_ptr<Plan>& last, std::vector<size_t> sizes) {
    try {
        last = unb::next_plan(last, [&](Plan& p) {
            for (size_t n : sizes) {
                unsigned char* q = p.memory.alloc<unsigned char>(n);
                expect(reinterpret_cast<uintptr_t>(q) % 256 == 0, "aligned to 256 bytes");
                p.parts[reinterpret_cast<uintptr_t>(q)] = n;
            }
            uintptr_t end = 0;
            expect(p.parts.size() == sizes.size(), "parts are distinct");
            for (auto& [at, n] : p.parts) {
                expect(at >= end, "parts do not overlap");
                end = at + n;
            }
        });
        return true;
    } catch (const std::bad_alloc&) {
        return false;
    }
}

int main() {
    {   // A larger list after a middling one, each fitting alone.
        capacity = 100 * MB;
        std::unique_ptr<Plan> plan;
        expect(follow(plan, {40 * MB, 1000}), "first list");
        expect(follow(plan, {1000, 80 * MB - 1}), "a list that fits once the last one's memory is freed");
        expect(live <= capacity, "capacity");
    }
    expect(live == 0, "all freed");
    {   // Less than a chunk left.
        capacity = 10 * MB;
        std::unique_ptr<Plan> plan;
        expect(follow(plan, {1 * MB, 5, 2 * MB}), "a list smaller than a chunk");
    }
    {   // Small tables first: the large chunk stays free for the large buffer.
        capacity = 300 * MB;
        std::unique_ptr<Plan> plan;
        expect(follow(plan, {100 * MB, 3 * MB}), "first list");
        calls = 0;
        expect(follow(plan, {3 * MB, 2 * MB, 100 * MB}) && calls == 0, "the last plan's chunks hold it");
        expect(follow(plan, {100 * MB, 3 * MB}) && calls == 0, "and the first list again");
    }
    {   // Chunks left empty are freed once they are more than half.
        capacity = 1000 * MB;
        std::unique_ptr<Plan> plan;
        expect(follow(plan, {200 * MB, 300 * MB, 40 * MB}) && follow(plan, {40 * MB}), "a small list");
        expect(live == 40 * MB, "the large chunks are given back");
    }
    {   // A list that does not fit at all: refused, nothing held.
        capacity = 100 * MB;
        std::unique_ptr<Plan> plan;
        expect(follow(plan, {40 * MB}), "first list");
        expect(!follow(plan, {60 * MB, 50 * MB}), "too large a list is refused");
        expect(!plan && live == 0, "nothing is held after it");
        expect(follow(plan, {90 * MB}), "the next list");
    }
    return failures != 0;
}

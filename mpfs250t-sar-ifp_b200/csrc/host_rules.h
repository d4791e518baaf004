// Host-side decisions without CUDA: how a plan's buffers share device allocations, and which jobs the passes in runs take.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <vector>

namespace pfa {

// ------------------------------------------------------------------------------------------ allocations
// The driver maps device memory in steps of 2 MiB and serves small requests from what it has mapped (10 us or less); a new
// mapping takes 300 to 400 us, and as much again to give back.  So a plan of small buffers packs them into allocations of
// at most 1 MiB (a larger buffer by itself), which plans share the mapped memory with: 256 x 256 float plan 8 us, 360 in one
// allocation; 300 x 300 fixed 9 us, 360.  Every other plan takes a single allocation: 1000 x 1000 fixed 340 us, 1010 with one
// for each buffer.  The first `head` buffers stay together.
constexpr size_t kSmallAlloc = size_t(1) << 20, kSmallBuffer = size_t(5) << 18;
constexpr int kMaxBlocks = 12;

struct Packing {
    std::vector<size_t> block;       // bytes of each allocation
    std::vector<int> in;             // buffer -> allocation
    std::vector<size_t> offset;      // buffer -> offset in it
};

inline Packing pack_buffers(const std::vector<size_t> &bytes, size_t head) {
    auto pack = [&](size_t limit) {
        Packing p;
        size_t i = 0;
        while (i < bytes.size()) {
            const size_t end = i == 0 && head ? head : i + 1;        // the buffers that go in together
            size_t sum = 0;
            for (size_t k = i; k < end; ++k) sum += bytes[k];
            if (p.block.empty() || p.block.back() + sum > limit) p.block.push_back(0);
            for (; i < end; ++i) {
                p.in.push_back((int)p.block.size() - 1);
                p.offset.push_back(p.block.back());
                p.block.back() += bytes[i];
            }
        }
        return p;
    };
    const Packing small = pack(kSmallAlloc);
    const bool fits = std::all_of(small.block.begin(), small.block.end(), [](size_t b) { return b <= kSmallBuffer; });
    return fits && small.block.size() <= kMaxBlocks ? small : pack((size_t)-1);
}

// ------------------------------------------------------------------------------------------ routes
// Up to so many pulses the fused pass 2's one launch wins over the resample in a kernel of its own (float 256 x 240 frame: 28 us,
// 34 with the split, 400 x 380: 41, 37; fixed: 44, 50 and 69, 57).
constexpr int kFusedPulses = 256;

}  // namespace pfa

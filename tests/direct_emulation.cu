// Host run of the direct comparison of small ranking groups (sadcs_b200/csrc/segsort.cuh: directOrder,
// orderEqual, the kernel's own functions) for CPU tests. Test infrastructure only.
#include <cstdint>
#include <vector>

#include "../sadcs_b200/csrc/segsort.cuh"

using namespace sadcs;

// Sorts `size` (2 to kSegTiny) suffixes at position[] of a text of n codes of `bits` bits that share their
// first `depth` characters; number[i] gets the i-th one's group number, as segSortTiny<true> leaves it in the keys.
extern "C" void direct_sort(const uint8_t* codes, int64_t n, uint32_t bits, uint32_t depth, uint32_t size,
                            uint32_t* position, uint32_t* number) {
    std::vector<uint64_t> packed((static_cast<uint64_t>(n) + 64) * bits / 64 + 2, 0);
    for (int64_t q = 0; q < n; q++) {
        for (uint32_t k = 0; k < bits; k++) {
            const uint64_t bit = static_cast<uint64_t>(q) * bits + k;
            if ((codes[q] >> (bits - 1 - k)) & 1) packed[bit >> 6] |= uint64_t(1) << (63 - (bit & 63));
        }
    }
    uint32_t val[kSegTiny] = {};
    for (uint32_t i = 0; i < size; i++) val[i] = position[i];
    const uint32_t same = orderEqual(val, size, (1u << (size - 1)) - 1, [&](uint32_t x, uint32_t y) {
        return directOrder(packed.data(), bits, static_cast<uint32_t>(n), x, y, depth);
    });
    uint32_t group = 0;
    for (uint32_t i = 0; i < size; i++) {
        if (i > 0 && !((same >> (i - 1)) & 1)) group++;
        position[i] = val[i];
        number[i] = group;
    }
}

extern "C" uint32_t direct_words() { return SADCS_DIRECT_WORDS; }

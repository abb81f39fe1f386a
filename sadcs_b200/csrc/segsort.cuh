// segsort.cuh - sorting the ranking list by subkey inside each group (segment), in place.
//
// After the first ranking pass the list holds whole groups, each a contiguous segment, and a pass
// only has to order every segment by its subkey (no global sort by (group, subkey) is needed).
// Most segments are small (on genome-like text every segment left after the first pass has at most
// 4 members; on natural-language text 80-95% of the remaining suffixes are in segments of up to a
// few thousand), so:
//   - segments of up to kSegTiny elements are sorted by one thread each in registers, and finished
//     by comparing the suffixes directly where their keys agree;
//   - segments of up to kSegSmall elements are sorted entirely in shared memory: a block takes the
//     segments that start in one kSegChunk-wide range of list positions (at most kSegCap elements)
//     and radix-sorts them by (segment, subkey) with 8-bit digits, the keys travelling in registers
//     and through one shared buffer per pass;
//   - larger segments are sorted by onesweep passes over their own ranges only (segmented tiles,
//     per-segment digit bases), in place between the two list buffers.
// Order among equal subkeys is not kept (nothing downstream depends on it).
#pragma once

#include <utility>

#include "alphabet.cuh"
#include "primitives.cuh"

namespace sadcs {

#ifndef SADCS_SEGSORT_BLOCKS
#define SADCS_SEGSORT_BLOCKS 5  // resident blocks per SM the register budget is set for (tuning)
#endif

#ifndef SADCS_SEGSORT_SMALL
// Largest segment sorted in shared memory (tuning; 1024 with 4 blocks per SM: 1.4 ms less ranking at 256 MiB than
// 2048 with 2).
#define SADCS_SEGSORT_SMALL 1024
#endif

constexpr uint32_t kSegSmall = SADCS_SEGSORT_SMALL;  // largest segment sorted in one block
constexpr uint32_t kSegTiny = 8;  // largest segment one thread sorts in registers
constexpr uint32_t kSegChunk = SADCS_SEGSORT_SMALL;  // a block owns the segments starting in such a range
constexpr uint32_t kSegCap = kSegChunk + kSegSmall;  // elements a block can hold
constexpr int kSegThreads = 256;
constexpr int kSegWarps = kSegThreads / 32;
constexpr int kSegItems = kSegCap / kSegThreads;     // 8 at the default
constexpr uint32_t kSegMaxLocal = kSegChunk / (kSegTiny + 1) + 1;  // segments of kSegTiny + 1 on starting in a chunk
static_assert(kSegMaxLocal <= 256, "one digit for a block's segments");

// The segments' big-path tables (host-sized): begin, size and first tile of each big segment.
struct ListSegments {
    const uint32_t* __restrict__ tileStart;  // [segments + 1]
    const uint32_t* __restrict__ begin;      // [segments]
    const uint32_t* __restrict__ size;       // [segments]
    uint32_t segments;
    __device__ __forceinline__ void locate(uint32_t tile, uint32_t& segment, uint32_t& firstTile, uint32_t& b,
                                           uint32_t& n) const {
        uint32_t lo = 0, hi = segments;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (__ldg(tileStart + mid) <= tile) lo = mid; else hi = mid;
        }
        segment = lo;
        firstTile = __ldg(tileStart + lo);
        b = __ldg(begin + lo);
        n = __ldg(size + lo);
    }
};

// flags[i] = 1 where a segment (run of equal group ids) starts.
__global__ void segMarkHeads(const uint32_t* __restrict__ grp, uint32_t u, uint32_t* __restrict__ flags) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < u) flags[i] = i == 0 || grp[i] != grp[i - 1];
}

// heads[index[i]] = i for every segment start (index = exclusive scan of the flags); heads[S] = u.
__global__ void segCollectHeads(const uint32_t* __restrict__ grp, const uint32_t* __restrict__ index, uint32_t u,
                                uint32_t segments, uint32_t* __restrict__ heads) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < u && (i == 0 || grp[i] != grp[i - 1])) heads[index[i]] = i;
    if (i == 0) heads[segments] = u;
}

// The heads of a list of at most kSegOneBlock elements, in one block: heads[0 .. S] as segCollectHeads
// leaves them, counter[0..2] = S, the big segments and their tiles. A short list's pass is bound by its
// launches and the waits for its counts: one launch and one wait here, against nine and two.
constexpr uint32_t kSegOneBlock = 16384;
constexpr int kSegOneThreads = 1024;
__global__ void __launch_bounds__(kSegOneThreads) segHeadsOneBlock(const uint32_t* __restrict__ grp, uint32_t u,
                                                                   uint32_t* __restrict__ heads,
                                                                   uint32_t* __restrict__ counter) {
    __shared__ uint32_t warpTotals[32];
    __shared__ uint32_t sBig, sTiles;
    constexpr uint32_t kItems = kSegOneBlock / kSegOneThreads;
    if (threadIdx.x == 0) sBig = sTiles = 0;
    const uint32_t base = threadIdx.x * kItems;
    uint32_t starts = 0;  // bit k: a segment starts at base + k
    uint32_t before = base > 0 && base <= u ? grp[base - 1] : 0;
#pragma unroll
    for (uint32_t k = 0; k < kItems; k++) {
        const uint32_t i = base + k;
        if (i < u) {
            const uint32_t g = grp[i];
            if (i == 0 || g != before) starts |= 1u << k;
            before = g;
        }
    }
    uint32_t segments;
    uint32_t at = blockInclusiveScan<OpSum>(__popc(starts), warpTotals, segments) - __popc(starts);
#pragma unroll
    for (uint32_t k = 0; k < kItems; k++) {
        if ((starts >> k) & 1) heads[at++] = base + k;
    }
    if (threadIdx.x == 0) heads[segments] = u;
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < segments; k += kSegOneThreads) {
        const uint32_t size = heads[k + 1] - heads[k];
        if (size > kSegSmall) {
            atomicAdd(&sBig, 1u);
            atomicAdd(&sTiles, (size + kSortTile - 1) / kSortTile);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        counter[0] = segments;
        counter[1] = sBig;
        counter[2] = sTiles;
    }
}

// Per segment k: bigFlag[k] = size > kSegSmall, tiles[k] = its tiles if big (both scanned later).
__global__ void segClassify(const uint32_t* __restrict__ heads, uint32_t segments, uint32_t* __restrict__ bigFlag,
                            uint32_t* __restrict__ tiles) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= segments) return;
    const uint32_t size = heads[k + 1] - heads[k];
    const bool big = size > kSegSmall;
    bigFlag[k] = big;
    tiles[k] = big ? (size + kSortTile - 1) / kSortTile : 0;
}

// The big segments' tables, from the scanned flags and tile counts.
__global__ void segCollectBig(const uint32_t* __restrict__ heads, uint32_t segments,
                              const uint32_t* __restrict__ bigIndex, const uint32_t* __restrict__ tileBase,
                              uint32_t bigCount, uint32_t totalTiles, uint32_t* __restrict__ begin,
                              uint32_t* __restrict__ size, uint32_t* __restrict__ tileStart) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < segments) {
        const uint32_t s = heads[k + 1] - heads[k];
        if (s > kSegSmall) {
            const uint32_t j = bigIndex[k];
            begin[j] = heads[k];
            size[j] = s;
            tileStart[j] = tileBase[k];
        }
    }
    if (k == 0) tileStart[bigCount] = totalTiles;
}

// hist[(p * segments + s) * 256 + digit] of digit passes first .. first + passes - 1 (bits [8q, 8q + 8) of
// pass q) of every big segment s (zeroed by the caller), one tile per block. All passes are counted from one
// read of the keys where their tables fit the scratch: the 4096-text batch's first sort spent 6.5 ms
// of 45 on reading its keys once per pass. Runs of equal digits are counted in registers and added to
// the shared histogram when the digit changes, as in radixHistogramFrom. Four tiles per block, whose counts
// go out once per segment, gain the batch nothing (74.5 ms of ranking both ways) and leave smaller lists too
// few blocks (a run of 32 MiB of one character 13.9 ms, 13.5 with one).
__global__ void __launch_bounds__(256) segHistogram(const uint64_t* __restrict__ keys, ListSegments segs, int firstPass,
                                                    int passes, uint32_t* __restrict__ hist) {
    __shared__ uint32_t h[8][256];
    for (int p = 0; p < passes; p++) h[p][threadIdx.x] = 0;
    __syncthreads();
    uint32_t segment, segTile, begin, size;
    segs.locate(blockIdx.x, segment, segTile, begin, size);
    const uint32_t local = blockIdx.x - segTile;
    const uint32_t tileEnd = min((local + 1) * kSortTile, size);
    uint32_t run[8], digit[8];
#pragma unroll
    for (int p = 0; p < 8; p++) run[p] = digit[p] = 0;
    for (uint32_t k = local * kSortTile + threadIdx.x; k < tileEnd; k += blockDim.x) {
        const uint64_t key = keys[begin + k] >> (8 * firstPass);
#pragma unroll
        for (int p = 0; p < 8; p++) {
            if (p < passes) {
                const uint32_t d = static_cast<uint32_t>(key >> (8 * p)) & 0xFF;
                if (d != digit[p]) {
                    if (run[p]) atomicAdd(&h[p][digit[p]], run[p]);
                    digit[p] = d;
                    run[p] = 0;
                }
                run[p]++;
            }
        }
    }
#pragma unroll
    for (int p = 0; p < 8; p++) {
        if (p < passes && run[p]) atomicAdd(&h[p][digit[p]], run[p]);
    }
    __syncthreads();
    for (int p = 0; p < passes; p++) {
        const uint32_t c = h[p][threadIdx.x];
        if (c) atomicAdd(hist + (static_cast<size_t>(p) * segs.segments + segment) * 256 + threadIdx.x, c);
    }
}

// Row p * segments + s of hist becomes begin[s] + its exclusive prefix. One block per row.
__global__ void __launch_bounds__(256) segDigitBase(uint32_t* __restrict__ hist, const uint32_t* __restrict__ begin,
                                                    uint32_t segments) {
    __shared__ uint32_t warpTotals[32];
    uint32_t* row = hist + static_cast<size_t>(blockIdx.x) * 256;
    const uint32_t v = row[threadIdx.x];
    uint32_t total;
    const uint32_t inclusive = blockInclusiveScan<OpSum>(v, warpTotals, total);
    row[threadIdx.x] = begin[blockIdx.x % segments] + inclusive - v;
}

// Suffixes i and j of one text ending at `end`, compared from their characters at `from` on, up to
// SADCS_DIRECT_WORDS stream words: -1 or 1, or 0 if they agree so far and neither has ended. One that ends
// within the last word is decided too: left at 0 it would be equal to suffixes that differ from one another after its
// end, and no order of the group would be consistent with that.
#ifndef SADCS_DIRECT_WORDS
#define SADCS_DIRECT_WORDS 8
#endif
#ifndef SADCS_DIRECT_LIST
#define SADCS_DIRECT_LIST (8u << 20)
#endif
constexpr uint32_t kDirectList = SADCS_DIRECT_LIST;
// Direct where at least 1 of kDirectShare elements in the sample (one block in kDirectSample) was decided.
// Ranking of a text and one copy of it with point changes, without direct comparisons, with them in every pass, and
// by the rule: 192 MiB of 2-bit codes, changes at 0.2% (40% of the pairs decided) 44.2, 36.7, 36.5 ms, 0.8% 28.8,
// 17.9, 17.8; three copies of 96 MiB of bytes, 0.4% (23%) 42.3, 52.8, 42.4, 0.8% (40%) 36.6, 40.1, 36.7, 1.6%
// 30.8, 27.3, 25.3; exact copies of it 144.5, 148.3, 144.6. With 1 in 2 and 1 in 3 some of the gains are left, with
// 1 in 6 the next rate's are had too; none of them costs more than 0.3% anywhere.
#ifndef SADCS_DIRECT_SHARE
#define SADCS_DIRECT_SHARE 4
#endif
constexpr uint32_t kDirectShare = SADCS_DIRECT_SHARE;
constexpr uint32_t kDirectSample = 64;
__host__ __device__ __forceinline__ bool directWorthwhile(uint32_t compared, uint32_t decided) {
    return static_cast<uint64_t>(decided) * kDirectShare >= compared;
}
__host__ __device__ __noinline__ int directOrder(const uint64_t* __restrict__ packed, uint32_t b, uint32_t end,
                                                 uint32_t i, uint32_t j, uint32_t from) {
    const uint32_t perWord = 64 / b, shorter = end - (i > j ? i : j);  // characters of the shorter suffix
    uint64_t at = from;
    for (int w = 0; w < SADCS_DIRECT_WORDS; w++, at += perWord) {
        if (at >= shorter) return i > j ? -1 : 1;  // one ends: the shorter is the smaller
        const uint32_t bits = (shorter - at < perWord ? static_cast<uint32_t>(shorter - at) : perWord) * b;
        const uint64_t x = streamBits(packed, (i + at) * b) >> (64 - bits);
        const uint64_t y = streamBits(packed, (j + at) * b) >> (64 - bits);
        if (x != y) return x < y ? -1 : 1;
    }
    return at < shorter ? 0 : (i > j ? -1 : 1);
}

// The values of up to kSegTiny elements sorted by order (-1, 0 or 1) within the runs of equal keys, by
// exchanges of neighbours. equal, bit i: elements i and i + 1 have the same key. Returns it without the
// bits of neighbours that are now known to differ.
template <class Order>
__host__ __device__ __forceinline__ uint32_t orderEqual(uint32_t (&val)[kSegTiny], uint32_t size, uint32_t equal,
                                                        Order order) {
    uint32_t same = equal;
    for (uint32_t round = 1; round < size; round++) {  // until a round exchanges nothing
        bool exchanged = false;
        same = equal;
#pragma unroll
        for (uint32_t i = 0; i + 1 < kSegTiny; i++) {
            if ((equal >> i) & 1) {
                const int o = order(val[i], val[i + 1]);
                if (o) same &= ~(1u << i);
                if (o > 0) {
                    const uint32_t tv = val[i];
                    val[i] = val[i + 1];
                    val[i + 1] = tv;
                    exchanged = true;
                }
            }
        }
        if (!exchanged || size == 2) break;
        same = equal;  // known only after a round without an exchange
    }
    return same;
}

// Segments of 2 to kSegTiny elements, one thread each: keys and values into registers, sorted
// by compare-exchange at fixed register indices (an insertion sort unrolled for kSegTiny). With kDirect,
// elements whose keys agree (they share their first `depth` characters) are then compared directly, up to
// SADCS_DIRECT_WORDS words of the code stream further, instead of staying listed for more passes: on
// genome-like text most groups left after the first pass are a repeat and its copies (2-4 members),
// which agree for about a hundred characters. A sorted segment's keys are replaced by
// numbers that differ where the order is known, so members that still agree stay a group, which
// shares `depth` characters as every group of the pass does. Written back in place.
// Whole copies agree for far longer, and comparing them would only repeat itself in every pass. So one block
// in kDirectSample goes first (sampled) and counts what it compared and decided in direct[0] and [1]; the
// others compare if that share was worth it. direct[2] counts all elements decided this way.
template <bool kDirect>
__global__ void __launch_bounds__(256) segSortTiny(const uint32_t* __restrict__ heads, uint32_t segments, TextSet texts,
                                                   uint32_t depth, uint64_t* __restrict__ keys,
                                                   uint32_t* __restrict__ vals, uint32_t* __restrict__ direct,
                                                    bool sampled) {
    uint32_t block = blockIdx.x;
    bool compare = false;
    if constexpr (kDirect) {
        if (sampled) {
            block *= kDirectSample;
            compare = true;
        } else {
            if (block % kDirectSample == 0) return;
            compare = directWorthwhile(direct[0], direct[1]);
        }
    }
    const uint32_t k = block * blockDim.x + threadIdx.x;
    if (k >= segments) return;
    const uint32_t begin = heads[k], size = heads[k + 1] - begin;
    if (size < 2 || size > kSegTiny) return;
    uint64_t key[kSegTiny];
    uint32_t val[kSegTiny];
#pragma unroll
    for (uint32_t i = 0; i < kSegTiny; i++) {
        if (i < size) {
            key[i] = keys[begin + i];
            val[i] = vals[begin + i];
        }
    }
#pragma unroll
    for (uint32_t i = 1; i < kSegTiny; i++) {
        if (i < size) {
#pragma unroll
            for (uint32_t j = i; j > 0; j--) {
                if (key[j - 1] > key[j]) {
                    const uint64_t tk = key[j - 1];
                    key[j - 1] = key[j];
                    key[j] = tk;
                    const uint32_t tv = val[j - 1];
                    val[j - 1] = val[j];
                    val[j] = tv;
                }
            }
        }
    }
    if constexpr (kDirect) {
        uint32_t equal = 0;  // bit i: elements i and i + 1 have the same key
#pragma unroll
        for (uint32_t i = 0; i + 1 < kSegTiny; i++) {
            if (i + 1 < size && key[i] == key[i + 1]) equal |= 1u << i;
        }
        if (equal && compare) {
            const uint32_t end = texts.endOf(samplePosition(val[0]));  // a segment is of one text
            const uint32_t same = orderEqual(val, size, equal, [&](uint32_t x, uint32_t y) {
                return directOrder(texts.packed, texts.bits, end, samplePosition(x), samplePosition(y), depth);
            });
            const uint32_t compared = equal | (equal << 1), decided = compared & ~(same | (same << 1));
            if (sampled) {
                atomicAdd(direct, static_cast<uint32_t>(__popc(compared)));
                atomicAdd(direct + 1, static_cast<uint32_t>(__popc(decided)));
            }
            if (decided) atomicAdd(direct + 2, static_cast<uint32_t>(__popc(decided)));
            uint64_t number = 0;
#pragma unroll
            for (uint32_t i = 0; i < kSegTiny; i++) {
                if (i > 0 && !((same >> (i - 1)) & 1)) number++;
                key[i] = number;
            }
        }
    }
#pragma unroll
    for (uint32_t i = 0; i < kSegTiny; i++) {
        if (i < size) {
            keys[begin + i] = key[i];
            vals[begin + i] = val[i];
        }
    }
}

// Copies the big segments' ranges from one buffer pair to the other.
__global__ void segCopyBack(ListSegments segs, const uint64_t* __restrict__ kFrom, const uint32_t* __restrict__ vFrom,
                            uint64_t* __restrict__ kTo, uint32_t* __restrict__ vTo) {
    uint32_t segment, firstTile, begin, size;
    segs.locate(blockIdx.x, segment, firstTile, begin, size);
    const uint32_t local = blockIdx.x - firstTile;
    const uint32_t end = min((local + 1) * kSortTile, size);
    for (uint32_t k = local * kSortTile + threadIdx.x; k < end; k += blockDim.x) {
        kTo[begin + k] = kFrom[begin + k];
        vTo[begin + k] = vFrom[begin + k];
    }
}

// The segments of kSegTiny + 1 to kSegSmall elements starting in [blockIdx.x * kSegChunk, + kSegChunk):
// sorted by (segment, subkey) in shared memory, stable 8-bit passes, and written to out (which may
// be in). Bound by the passes' barriers and serial warp matches, so: digits on which every segment's
// keys agree have no pass (after a few doubling rounds the ranks of a group's members at p + h are close
// together: 1-2 of 3 digits differ), the segments need one pass (none for a single one), and the
// elements are spread evenly over the warps. The ranking of a 48 MiB text of versions of one document
// took 16.7 ms with every pass made over the block's first warps, 13.6 now (of it 1.5 by the direct
// rank writes of small arrays), of 256 MiB of natural-language-like text 17.8 and 16.9.
__global__ void __launch_bounds__(kSegThreads, SADCS_SEGSORT_BLOCKS)
    segSortSmall(const uint32_t* __restrict__ heads, uint32_t segments, const uint64_t* keyIn, const uint32_t* valIn,
                 uint64_t* keyOut, uint32_t* valOut, int keyBits) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t* sKey = reinterpret_cast<uint64_t*>(smem);                 // kSegCap
    uint32_t* sVal = reinterpret_cast<uint32_t*>(sKey + kSegCap);       // kSegCap
    uint32_t* segStart = sVal + kSegCap;                                // kSegMaxLocal + 1 (global start)
    uint32_t* segLocal = segStart + kSegMaxLocal + 1;                   // kSegMaxLocal + 1 (local start)
    uint32_t* warpCount = segLocal + kSegMaxLocal + 1;                  // kSegWarps * 256
    uint32_t* digitStart = warpCount + kSegWarps * 256;                 // 256
    uint8_t* sSeg = reinterpret_cast<uint8_t*>(digitStart + 256);       // kSegCap
    __shared__ uint32_t warpTotals[32];
    __shared__ uint32_t sFirst, sCount;
    __shared__ uint32_t sDiffer[2];  // key bits (low, high) in which some segment's keys differ

    if (threadIdx.x == 0) {
        const uint32_t lo = blockIdx.x * kSegChunk, hi = lo + kSegChunk;
        uint32_t a = 0, b = segments;  // first segment starting at or after lo
        while (a < b) {
            const uint32_t mid = (a + b) >> 1;
            if (heads[mid] < lo) a = mid + 1; else b = mid;
        }
        uint32_t c = a, d = segments;  // first segment starting at or after hi
        while (c < d) {
            const uint32_t mid = (c + d) >> 1;
            if (heads[mid] < hi) c = mid + 1; else d = mid;
        }
        sFirst = a;
        sCount = c - a;
        sDiffer[0] = sDiffer[1] = 0;
    }
    __syncthreads();
    const uint32_t first = sFirst, started = sCount;
    // The block's segments in order: their starts in the list and in the block (their number in the
    // high half of the scanned words, their elements in the low half: at most kSegCap).
    static_assert(kSegCap < 65536, "elements in the low half");
    uint32_t running = 0;
    for (uint32_t base = 0; base < started; base += kSegThreads) {
        const uint32_t s = base + threadIdx.x;
        uint32_t size = 0, start = 0;
        if (s < started) {
            start = heads[first + s];
            size = heads[first + s + 1] - start;
            if (size > kSegSmall || size <= kSegTiny) size = 0;  // larger: onesweep passes; smaller: segSortTiny
        }
        const uint32_t mine = size ? (1u << 16) | size : 0;
        uint32_t all;
        const uint32_t before = running + blockInclusiveScan<OpSum>(mine, warpTotals, all) - mine;
        if (size) {
            segStart[before >> 16] = start;
            segLocal[before >> 16] = before & 0xFFFF;
        }
        running += all;
    }
    const uint32_t count = running >> 16, total = running & 0xFFFF;
    if (total == 0) return;
    if (threadIdx.x == 0) segLocal[count] = total;
    __syncthreads();

    // Load: item j of warp w is element (w * per + j) * 32 + lane, in segment order.
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = static_cast<int>((total + kSegThreads - 1) / kSegThreads);  // at most kSegItems
    const uint32_t warpBase = warp * per * 32 + lane;
    uint64_t key[kSegItems];
    uint32_t val[kSegItems];
    uint32_t seg[kSegItems];
    uint64_t differ = 0;
#pragma unroll
    for (int j = 0; j < kSegItems; j++) {
        const uint32_t t = warpBase + j * 32;
        seg[j] = 0xFFFF;
        if (j < per && t < total) {
            uint32_t a = 0, b = count;  // last s with segLocal[s] <= t
            while (b - a > 1) {
                const uint32_t mid = (a + b) >> 1;
                if (segLocal[mid] <= t) a = mid; else b = mid;
            }
            const uint32_t g = segStart[a] + (t - segLocal[a]);
            key[j] = keyIn[g];
            val[j] = valIn[g];
            seg[j] = a;
            differ |= key[j] ^ keyIn[segStart[a]];
        }
    }
    const uint32_t low = __reduce_or_sync(0xffffffffu, static_cast<uint32_t>(differ));
    const uint32_t high = __reduce_or_sync(0xffffffffu, static_cast<uint32_t>(differ >> 32));
    if (lane == 0) {
        if (low) atomicOr(&sDiffer[0], low);
        if (high) atomicOr(&sDiffer[1], high);
    }
    __syncthreads();
    differ = (static_cast<uint64_t>(sDiffer[1]) << 32) | sDiffer[0];
    const uint32_t lt = (1u << lane) - 1;
    const int keyPasses = (keyBits + 7) / 8;
    for (int pass = 0; pass <= keyPasses; pass++) {  // the last one by segment
        if (pass < keyPasses ? ((differ >> (8 * pass)) & 0xFF) == 0 : count == 1) continue;
        for (int i = threadIdx.x; i < kSegWarps * 256; i += kSegThreads) warpCount[i] = 0;
        __syncthreads();
        uint32_t* myCount = warpCount + warp * 256;
        uint32_t rankDigit[kSegItems];
#pragma unroll
        for (int j = 0; j < kSegItems; j++) {
            if (j >= per) break;  // the same for the block
            uint32_t d = kNoDigit;
            if (seg[j] != 0xFFFF) d = pass < keyPasses ? static_cast<uint32_t>(key[j] >> (8 * pass)) & 0xFF : seg[j];
            const uint32_t peers = __match_any_sync(0xffffffffu, d);
            uint32_t before = 0;
            if (d != kNoDigit) before = myCount[d];
            __syncwarp();
            if (d != kNoDigit && (peers & lt) == 0) myCount[d] = before + __popc(peers);
            __syncwarp();
            rankDigit[j] = ((before + __popc(peers & lt)) << 9) | d;
        }
        __syncthreads();
        const uint32_t dd = threadIdx.x;
        uint32_t digitTotal = 0;
#pragma unroll
        for (int w = 0; w < kSegWarps; w++) {
            const uint32_t c = warpCount[w * 256 + dd];
            warpCount[w * 256 + dd] = digitTotal;
            digitTotal += c;
        }
        uint32_t all;
        const uint32_t inclusive = blockInclusiveScan<OpSum>(digitTotal, warpTotals, all);
        digitStart[dd] = inclusive - digitTotal;
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kSegItems; j++) {
            if (j >= per) break;
            const uint32_t d = rankDigit[j] & 0x1FF;
            if (d != kNoDigit) {
                const uint32_t pos = digitStart[d] + warpCount[warp * 256 + d] + (rankDigit[j] >> 9);
                sKey[pos] = key[j];
                sVal[pos] = val[j];
                sSeg[pos] = static_cast<uint8_t>(seg[j]);
            }
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kSegItems; j++) {
            if (j >= per) break;
            const uint32_t t = warpBase + j * 32;
            if (t < total) {
                key[j] = sKey[t];
                val[j] = sVal[t];
                seg[j] = sSeg[t];
            }
        }
        __syncthreads();
    }
    // Sorted by (segment, key): segment s occupies [segLocal[s], segLocal[s + 1]) again.
#pragma unroll
    for (int j = 0; j < kSegItems; j++) {
        const uint32_t t = warpBase + j * 32;
        if (j < per && t < total) {
            const uint32_t s = seg[j];
            const uint32_t g = segStart[s] + (t - segLocal[s]);
            keyOut[g] = key[j];
            valOut[g] = val[j];
        }
    }
}

constexpr size_t segSortSharedBytes() {
    return kSegCap * (8 + 4 + 1) + 2 * (kSegMaxLocal + 1) * 4 + (kSegWarps * 256 + 256) * 4 + 64;
}

// Scratch words of segmentedSort for a list of u elements (besides the list buffers and aux arrays).
inline size_t segScratchWords(uint64_t u) {
    const uint64_t big = u / (kSegSmall + 1) + 2;
    const uint64_t tiles = u / kSortTile + big + 2;
    return static_cast<size_t>(big * 256 + 3 * (big + 1) + tiles * 256 + 256);
}

struct SegBuffers {
    uint32_t* radixControl;  // [0] tile counter, [1] the error word the caller checks
    uint32_t* flags;    // u words (aux)
    uint32_t* heads;    // u + 1 words (aux)
    uint32_t* perSeg;   // 2 * u words (free key buffer): big flags and tile counts per segment
    uint32_t* scratch;  // scratchWords words, at least segScratchWords(u)
    size_t scratchWords;
    uint32_t* counter;  // device words [0..5]; [3..5]: segSortTiny<true>'s counts
    uint32_t* scanScratch;
    bool direct;        // (host) whether elements of equal keys may be compared directly
    bool* compared;     // (host) set when segSortTiny<true> ran: counter[3..5] hold its counts
};

// Sorts the list (keys, vals: u elements, compact sample indices, in segments of equal grp) by key inside
// each segment; elements of one segment with equal keys share their first `depth` characters.
// Big segments use the alternates as the other buffer of their passes; the result is left in
// keys/vals (pointers unchanged). hostWords: page-locked words for counts.
inline cudaError_t segmentedSort(const uint32_t* grp, uint32_t u, uint64_t* keys, uint32_t* vals, uint64_t* keysAlt,
                                 uint32_t* valsAlt, int keyBits, const TextSet& texts, uint32_t depth, SegBuffers b,
                                 uint32_t* hostWords, cudaStream_t stream) {
    if (u <= 1) return cudaSuccess;
    // A list of up to kSegOneBlock elements: one launch and one wait (the ranking of a 64 KiB text, with the
    // one-tile refinement, 0.67 -> 0.54 ms); its big segments' tables are made only if it has some.
    const bool oneBlock = u <= kSegOneBlock;
    if (oneBlock) {
        SADCS_TRY(launch(segHeadsOneBlock, 1, kSegOneThreads, 0, stream, grp, u, b.heads, b.counter));
        SADCS_TRY(cudaMemcpyAsync(hostWords, b.counter, 12, cudaMemcpyDeviceToHost, stream));
        SADCS_TRY(cudaStreamSynchronize(stream));
    } else {
        SADCS_TRY(launch(segMarkHeads, ceilDiv(u, 256), 256, 0, stream, grp, u, b.flags));
        SADCS_TRY((deviceScan<OpSum, false>(b.flags, b.flags, u, b.scanScratch, b.counter, stream)));
        SADCS_TRY(cudaMemcpyAsync(hostWords, b.counter, 4, cudaMemcpyDeviceToHost, stream));
        SADCS_TRY(cudaStreamSynchronize(stream));
        SADCS_TRY(launch(segCollectHeads, ceilDiv(u, 256), 256, 0, stream, grp, b.flags, u, hostWords[0], b.heads));
    }
    const uint32_t segments = hostWords[0];
    uint32_t* bigFlag = b.perSeg;
    uint32_t* tiles = b.perSeg + u;
    if (!oneBlock || hostWords[1]) {
        SADCS_TRY(launch(segClassify, ceilDiv(segments, 256), 256, 0, stream, b.heads, segments, bigFlag, tiles));
        SADCS_TRY((deviceScan<OpSum, false>(bigFlag, bigFlag, segments, b.scanScratch, b.counter + 1, stream)));
        SADCS_TRY((deviceScan<OpSum, false>(tiles, tiles, segments, b.scanScratch, b.counter + 2, stream)));
    }
    if (!oneBlock) {
        SADCS_TRY(cudaMemcpyAsync(hostWords + 1, b.counter + 1, 8, cudaMemcpyDeviceToHost, stream));
        SADCS_TRY(cudaStreamSynchronize(stream));
    }
    const uint32_t big = hostWords[1], bigTiles = hostWords[2];

    // Small segments, in place.
    static std::atomic<uint64_t> configured{0};
    SADCS_TRY(configureOnce(configured, [] {
        return cudaFuncSetAttribute(segSortSmall, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(segSortSharedBytes()));
    }));
    // Direct comparisons pay where the list is long (a pass over it costs DRAM traffic) and mostly pairs and
    // triples: 2 GiB of genome-like text (59M samples listed, groups of 2.2) ranks in 49.8 ms against
    // 58.2, five doubling rounds fewer; elsewhere they are made again in every pass for groups that
    // stay (48 MiB of versions of one document, groups of 48: 15.9 ms against 13.5) or come on top of the
    // passes that larger groups need anyway (256 MiB of natural-language-like text: 17.3 against 16.9). Whether
    // the pairs and triples agree for too long is found by a sample (kDirectShare). kDirectList is on the safe side:
    // a text of 64 MiB and a 2% changed copy, listed 10M, ranks in 4.7 ms against 6.0 (bytes) and 3.7 against 4.5 (5-bit
    // codes); half of it, listed 5M, would in 2.9 against 3.5 and 2.3 against 2.7.
    const bool direct = b.direct && u >= kDirectList && u <= 3 * static_cast<uint64_t>(segments);
    if (direct) {
        *b.compared = true;
        SADCS_TRY(cudaMemsetAsync(b.counter + 3, 0, 3 * sizeof(uint32_t), stream));
        const uint32_t blocks = ceilDiv(segments, 256);
        SADCS_TRY(launch(segSortTiny<true>, ceilDiv(blocks, kDirectSample), 256, 0, stream, b.heads, segments, texts, depth,
                         keys, vals, b.counter + 3, true));
        SADCS_TRY(launch(segSortTiny<true>, blocks, 256, 0, stream, b.heads, segments, texts, depth, keys, vals,
                         b.counter + 3, false));
    } else {
        SADCS_TRY(launch(segSortTiny<false>, ceilDiv(segments, 256), 256, 0, stream, b.heads, segments, texts, depth, keys,
                         vals, b.counter + 3, false));
    }
    SADCS_TRY(launch(segSortSmall, ceilDiv(u, kSegChunk), kSegThreads, segSortSharedBytes(), stream, b.heads,
                     segments, keys, vals, keys, vals, keyBits));
    if (big == 0) return cudaSuccess;

    // Big segments: onesweep passes over their own ranges, ping-ponging with the alternates.
    uint32_t* begin = b.scratch;
    uint32_t* size = begin + big + 1;
    uint32_t* tileStart = size + big + 1;
    uint32_t* hist = tileStart + big + 1;
    const int passes = (keyBits + 7) / 8;
    // every pass's digit bases at once where they fit beside the status words, else one pass's at a time
    const size_t table = static_cast<size_t>(big) * 256, status = static_cast<size_t>(bigTiles) * 256;
    const size_t tables = static_cast<size_t>(hist - b.scratch);
    const int together = tables + passes * table + status <= b.scratchWords ? passes : 1;
    uint32_t* statusWords = hist + together * table;
    const RadixScratch radix = RadixScratch::at(b.radixControl, statusWords);
    SADCS_TRY(launch(segCollectBig, ceilDiv(segments, 256), 256, 0, stream, b.heads, segments, bigFlag, tiles, big,
                     bigTiles, begin, size, tileStart));
    ListSegments segs{tileStart, begin, size, big};
    uint64_t* kIn = keys;
    uint64_t* kOut = keysAlt;
    uint32_t* vIn = vals;
    uint32_t* vOut = valsAlt;
    for (int p = 0; p < passes; p++) {
        if (p % together == 0) {
            SADCS_TRY(cudaMemsetAsync(hist, 0, together * table * 4, stream));
            SADCS_TRY(launch(segHistogram, bigTiles, 256, 0, stream, kIn, segs, p, together, hist));
            SADCS_TRY(launch(segDigitBase, big * together, 256, 0, stream, hist, begin, big));
        }
        SortLoader<uint64_t> ld{kIn, vIn, 8 * p};
        SortStorer<uint64_t> st{kOut, vOut, u};
        SADCS_TRY((radixOnesweepPass<uint64_t, SortLoader<uint64_t>, SortStorer<uint64_t>, ListSegments>(
            ld, st, segs, u, bigTiles, hist + (p % together) * table, radix, stream)));
        std::swap(kIn, kOut);
        std::swap(vIn, vOut);
    }
    if (kIn != keys) {
        // An odd number of passes left the big segments in the alternates: copy their ranges back.
        SADCS_TRY(launch(segCopyBack, bigTiles, 256, 0, stream, segs, kIn, vIn, keys, vals));
    }
    return cudaSuccess;
}

}  // namespace sadcs

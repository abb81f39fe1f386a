// merge_wide.cuh - the merge levels of texts with few long repeats (useWideMerge, merge_final.cuh):
// every tile of the 7 lists of a level merged in shared memory; the last level writes the suffix array
// and the BWT, an upper level the rows of the level below.
//
// A tile's window set (at most mergeCap(R) records, merge.cuh) is a short stretch of the final
// order, so its suffixes share their first characters: the tile's common prefix, in bits, is found
// from the first and last record of every window (all others lie between them) and left out of the
// records. What is left is held as
//   entry[cap]  48 key bits (the code stream after the common prefix) above the record's 16-bit
//               number in the window set; with several texts in the tile the key starts with the
//               text's number within the tile
//   tail[cap]   the next 64 bits of the stream
//   pos[cap]    p; prev[cap] the code of the character before p (the BWT byte)
// so most comparisons read one 8-byte word per side.
// The entries move through a 3-level tree of 2-way merges in place: (0,1) (2,3) (4,5) 6, then
// (01,23) (45,6), then (0123,456). A thread finds the start of its C outputs on the merge path by
// binary search, walks the two runs with both heads in registers, keeps its C outputs in registers,
// and writes them back once every thread has read. The tree compares entries and tails only: of
// records that agree in them the one of the earlier list comes first, which the record's number in
// the entry's low bits says by itself. So after the tree every group of records that agree is
// contiguous, list by list and in list order inside; only then are the groups put in suffix order,
// with the rest of the comparison (the code stream and the sample ranks): eight threads per tied
// record, one per list, find its place among that list's members of its group by binary search and
// add up. The searches read the sample ranks and the next stream bits from shared memory, staged there
// (in the tails' place) for the tile's tied records at once, so a comparison that leaves shared
// memory is not made by a lane or two of a warp at every step of the tree.
// The final order gives every record's rank within the window set, hence its place in the output
// (base + rank) for the records between the tile's two splitters.
#pragma once

#include "merge.cuh"

namespace sadcs {

// Shared-memory share of the unified L1/shared array preferred, in percent of the maximum: the rest is
// L1, which the record gathers go through.
#ifndef SADCS_WIDE_CARVEOUT
#define SADCS_WIDE_CARVEOUT 66
#endif

// Records of a thread whose stream words are in flight at once.
#ifndef SADCS_WIDE_BATCH
#define SADCS_WIDE_BATCH 2
#endif

template <bool kFinal>
struct WideTile {
    static constexpr uint32_t kCap = mergeCap(kWideR);
    // entry (one more: a run's end may be read as its next head), tail, pos, tied, prev (final) or rank
    static constexpr size_t sharedBytes() { return 8 * (kCap + 1) + 8 * kCap + 6 * kCap + (kFinal ? 1 : 2) * kCap + 4; }
    static constexpr uint32_t kStaged = 8 * kCap / (8 + 4 * kK);
    uint64_t* entry;
    uint64_t* tail;
    // The tails' memory once the groups are known: of the first kStaged tied records, the 64
    // stream bits after those the words hold, and the kK sample ranks.
    uint64_t* next;
    uint32_t* staged;
    uint32_t* pos;
    uint16_t* tied;  // tied record -> its place, by the words, then in suffix order
    uint8_t* prev;
    uint16_t* rank;
    __device__ __forceinline__ void carve(unsigned char* smem) {
        entry = reinterpret_cast<uint64_t*>(smem);
        tail = entry + kCap + 1;
        next = tail;
        staged = reinterpret_cast<uint32_t*>(next + kStaged);
        pos = reinterpret_cast<uint32_t*>(tail + kCap);
        tied = reinterpret_cast<uint16_t*>(pos + kCap);
        rank = tied + kCap;
        prev = reinterpret_cast<uint8_t*>(rank);
    }
};

__device__ __forceinline__ uint32_t recordOf(uint64_t entry) { return static_cast<uint32_t>(entry) & 0xFFFF; }

// Entry a (of an earlier list) before entry b, as far as their words tell, else by record number. A
// first difference in the words orders the suffixes whatever the tie offset: past its text's end a
// record's bits are 0, the smallest code, so the shorter suffix is the smaller there too, as it must be.
template <bool kFinal>
__device__ __forceinline__ bool entryLess(const WideTile<kFinal>& s, uint64_t a, uint64_t b) {
    if ((a ^ b) >> 16 == 0) {
        const uint64_t x = s.tail[recordOf(a)], y = s.tail[recordOf(b)];
        if (x != y) return x < y;
    }
    return a < b;
}

// One tree level, in place: merge m joins the runs [mb[3m], mb[3m + 1]) and [mb[3m + 1], mb[3m + 2])
// of the entries; mb is in shared memory. Every merge of two runs has its own threads, C outputs
// each; a merge with an empty run is done already.
template <bool kFinal>
__device__ __forceinline__ void treeLevel(const WideTile<kFinal>& s, const uint32_t* mb, int merges) {
    constexpr int C = SADCS_WIDE_ITEMS;
    uint32_t t = threadIdx.x, a0 = 0, lenA = 0, lenB = 0;
    bool active = false;
    for (int m = 0; m < merges; m++) {
        a0 = mb[3 * m];
        lenA = mb[3 * m + 1] - a0;
        lenB = mb[3 * m + 2] - mb[3 * m + 1];
        const uint32_t threads = lenA && lenB ? (lenA + lenB + C - 1) / C : 0;
        if (t < threads) {
            active = true;
            break;
        }
        t -= threads;
    }
    const uint32_t d = t * C;
    uint64_t out[C];
    if (active) {
        const uint64_t* A = s.entry + a0;
        const uint64_t* B = A + lenA;
        uint32_t lo = d > lenB ? d - lenB : 0, hi = min(d, lenA);
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (entryLess(s, A[mid], B[d - 1 - mid])) {
                lo = mid + 1;
            } else {
                hi = mid;
            }
        }
        uint32_t i = lo, j = d - lo;
        // A step takes one side and loads that side's next entry whichever it is (no divergence on
        // the side taken; the entry after a run's end is never compared).
        uint64_t ha = A[i], hb = B[j];
#pragma unroll
        for (int k = 0; k < C; k++) {
            bool takeA = false;
            if (i < lenA) takeA = j >= lenB || entryLess(s, ha, hb);
            out[k] = takeA ? ha : hb;
            i += takeA ? 1u : 0u;
            j += takeA ? 0u : 1u;
            if (k + 1 < C) {
                const uint64_t next = takeA ? A[i] : B[min(j, lenB)];
                if (takeA) {
                    ha = next;
                } else {
                    hb = next;
                }
            }
        }
    }
    __syncthreads();
    if (active) {
        const uint32_t len = lenA + lenB;
#pragma unroll
        for (int k = 0; k < C; k++) {
            if (d + k < len) s.entry[a0 + d + k] = out[k];
        }
    }
    __syncthreads();
}

// The group [begin, end) of place r. head: bit q set where the record at place q differs from the one
// before (place 0 is one).
__device__ __forceinline__ void groupOf(const uint32_t* head, uint32_t size, uint32_t r, uint32_t& begin,
                                        uint32_t& end) {
    uint32_t w = r >> 5;
    uint32_t m = head[w] & (0xFFFFFFFFu >> (31 - (r & 31)));
    while (m == 0) m = head[--w];
    begin = 32 * w + 31 - __clz(static_cast<int>(m));
    w = r >> 5;
    m = (r & 31) == 31 ? 0 : head[w] & (0xFFFFFFFFu << ((r & 31) + 1));
    while (m == 0 && 32 * (w + 1) < size) m = head[++w];
    end = m ? 32 * w + __ffs(static_cast<int>(m)) - 1 : size;
}

// The members of list b in the group [begin, end) that come before the record at place r of the
// group. The entries of tied records hold their index in s.tied above the record's number.
template <bool kFinal>
__device__ __forceinline__ uint32_t membersBefore(const WideTile<kFinal>& s, const MergeTileInfo& t, uint32_t r,
                                                  uint32_t begin, uint32_t end, uint32_t b, const MergeArgs& a,
                                                  uint32_t held) {
    const auto firstFrom = [&](uint32_t lo, uint32_t record) {  // the first place from lo on with a later record
        uint32_t hi = end;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (recordOf(s.entry[mid]) < record) lo = mid + 1; else hi = mid;
        }
        return lo;
    };
    const uint32_t from = firstFrom(begin, t.seg[b]), to = firstFrom(from, t.seg[b + 1]);
    if (r >= from && r < to) return r - from;
    const uint64_t mine = s.entry[r];
    const uint32_t i = s.pos[recordOf(mine)], rotI = coverRotation(i), number = static_cast<uint32_t>(mine >> 16);
    const bool stagedI = number < s.kStaged;
    const uint32_t n = a.texts.endOf(i), bits = a.texts.bits;
    uint32_t lo = from, up = to;  // members below lo are smaller, members from up on are not
    while (lo < up) {
        const uint32_t mid = (lo + up) >> 1;
        const uint64_t e = s.entry[mid];
        const uint32_t j = s.pos[recordOf(e)], other = static_cast<uint32_t>(e >> 16);
        bool less;  // j < i
        if (stagedI && other < s.kStaged) {
            const uint32_t rotJ = coverRotation(j), k = tieOffset(rotI, rotJ);
            const uint32_t shorter = n - max(i, j), stop = min(k, shorter) * bits;
            const uint64_t mask = stop > held ? topMask(stop - held) : 0;
            const uint64_t x = s.next[other] & mask, y = s.next[number] & mask;
            const int order = x == y && stop > held + 64 ? streamOrder(a.texts, j, i, held + 64, min(k, shorter)) : 0;
            if (x != y) {
                less = x < y;
            } else if (order) {
                less = order < 0;
            } else if (k >= shorter) {  // one is a prefix of the other
                less = j > i;
            } else {
                less = s.staged[other * kK + sampleSlot(rotJ, k)] < s.staged[number * kK + sampleSlot(rotI, k)];
            }
        } else {
            less = suffixLess(a.ranks, a.texts, n, j, i, held);
        }
        if (less) lo = mid + 1; else up = mid;
    }
    return lo - from;
}

// The tile's common prefix, by a whole warp (every warp computes the same): lanes 2b and 2b + 1 take
// the first and the last record of list b's window. Returns the common leading bits of the 14
// suffixes (at most 64 * kWords; a tile inside a long repeat shares many words) and, with several
// texts, the first text and the key bits that hold the text's number within the tile (0 when all 14
// are in one text; otherwise no prefix is left out). load(b, e, text): called once per lane, the
// suffix of the e-th element of list b; wordOf(w): its w-th stream word (0 past its text's end).
struct TilePrefix {
    uint32_t bits;       // left out of every record
    uint32_t textBits;   // key bits taken by the text's number
    uint32_t firstText;
};

template <bool kMulti, uint32_t kWords, class Load, class WordOf>
__device__ __forceinline__ TilePrefix tilePrefix(const MergeTileInfo& t, Load load, WordOf wordOf) {
    const uint32_t lane = threadIdx.x & 31, b = lane >> 1;
    uint32_t text = 0;
    const bool mine = b < kClasses && t.seg[b + 1] > t.seg[b];
    if (mine) load(b, t.win[b] + ((lane & 1) ? t.seg[b + 1] - t.seg[b] - 1 : 0), text);
    const uint32_t valid = __ballot_sync(0xffffffffu, mine);
    TilePrefix p{0, 0, 0};
    if constexpr (kMulti) {
        p.firstText = __reduce_min_sync(0xffffffffu, mine ? text : 0xFFFFFFFFu);
        const uint32_t range = __reduce_max_sync(0xffffffffu, mine ? text : 0u) - p.firstText;
        if (valid && range) {
            p.textBits = 32 - __clz(static_cast<int>(range));  // at most 20 (kMaxTexts)
            return p;
        }
    }
    const int src = valid ? __ffs(static_cast<int>(valid)) - 1 : 0;
    for (uint32_t w = 0; w < kWords; w++) {  // warp-uniform
        const uint64_t word = mine ? wordOf(w) : 0;
        const uint64_t first = __shfl_sync(0xffffffffu, word, src);
        const uint64_t diff = mine ? word ^ first : 0;
        const uint32_t high = __reduce_or_sync(0xffffffffu, static_cast<uint32_t>(diff >> 32));
        const uint32_t low = __reduce_or_sync(0xffffffffu, static_cast<uint32_t>(diff));
        if (high | low) {
            p.bits += high ? __clz(static_cast<int>(high)) : 32 + __clz(static_cast<int>(low));
            break;
        }
        p.bits += 64;
    }
    return p;
}

// kFinal: the last level, writing the SA and the BWT; otherwise an upper level, writing the rows
// (every R-th element of the merged order with its per-list counts) that bound the tiles below.
//
// Bound: instruction issue and shared-memory latency (integer compares on 8-byte entries).
template <bool kMulti, bool kFinal>
__global__ void __launch_bounds__(SADCS_WIDE_THREADS, SADCS_WIDE_TILES) mergeWide(MergeArgs a) {
    constexpr uint32_t kThreads = SADCS_WIDE_THREADS;
    constexpr uint32_t kR = kWideR;
    constexpr uint32_t kCap = WideTile<kFinal>::kCap;
    extern __shared__ __align__(16) unsigned char smem[];
    WideTile<kFinal> s;
    s.carve(smem);
    uint32_t held;  // stream bits from a suffix's start that the records' words hold or share
    __shared__ MergeTileInfo t;
    __shared__ uint32_t sLo, sHi, sTies;
    __shared__ uint32_t head[(kCap + 31) / 32];  // places whose record differs from the one before
    __shared__ uint32_t bounds[3 * 6];  // the tree's merges: 3 + 2 + 1 triples of window offsets
    if (threadIdx.x < 32) {
        planTileWindows(a, kCap, t);
        __syncwarp();
        // (0,1) (2,3) (4,5), then (01,23) (45,6), then (0123,456): indices into t.seg, 3 bits
        // each (a register constant: a table indexed by the lane would live in local memory)
        constexpr uint8_t kTree[18] = {0, 1, 2, 2, 3, 4, 4, 5, 6, 0, 2, 4, 4, 6, 7, 0, 4, 7};
        constexpr uint64_t kTreePacked = [] {
            uint64_t v = 0;
            for (int i = 0; i < 18; i++) v |= static_cast<uint64_t>(kTree[i]) << (3 * i);
            return v;
        }();
        if (threadIdx.x < 18) bounds[threadIdx.x] = t.seg[(kTreePacked >> (3 * threadIdx.x)) & 7];
        if (threadIdx.x == 0) {
            sLo = 0;
            sHi = t.size;
            sTies = 0;
            if (t.bad && a.error) atomicExch(a.error, 1u);
        }
    }
    __syncthreads();
    if (t.bad) return;
    const uint32_t size = t.size;
    const uint32_t* st = a.level.start;
    const TextSet& texts = a.texts;
    const uint32_t bits = texts.bits;

    // Gather: the positions of all records of a thread from the lists (coalesced, all in flight), then
    // each record's stream bits from the common prefix on.
    constexpr int kItems = (kCap + kThreads - 1) / kThreads;
    const auto slotOf = [&](uint32_t e) { return t.slot[listOfElement(t.seg, e)] + e; };
    uint32_t p[kItems];
#pragma unroll
    for (int j = 0; j < kItems; j++) {
        const uint32_t e = j * kThreads + threadIdx.x;
        p[j] = e < size ? a.level.lists[slotOf(e)] : 0;
    }
    uint32_t q = 0, qEnd = 0;
    const TilePrefix prefix = tilePrefix<kMulti, 8>(
        t,
        [&](uint32_t b, uint32_t e, uint32_t& text) {
            q = a.level.lists[st[b] + e];
            if (q >= a.span) q = 0;  // reported below
            if constexpr (kMulti) text = texts.textOf(q);
            qEnd = texts.endOfText(text);
        },
        [&](uint32_t w) {
            const uint32_t left = q < qEnd ? min(qEnd - q, 1024u) * bits : 0;  // the suffix's own bits
            if (left <= 64 * w) return uint64_t(0);
            return streamBits(texts.packed, static_cast<uint64_t>(q) * bits + 64 * w) & topMask(left - 64 * w);
        });
    // Past the last text's end the stream is 0: reads beyond it are moved there.
    const uint64_t endUnit = (static_cast<uint64_t>(a.span) * bits + 127) >> 7;
    const uint32_t keyBits = 48 - prefix.textBits;  // of the stream
    held = prefix.bits + keyBits + 64;
    constexpr int kBatch = SADCS_WIDE_BATCH;
#pragma unroll
    for (int first = 0; first < kItems; first += kBatch) {
        // Two 16-byte loads hold any 112 bits that begin in the first of them.
        ulonglong2 w0[kBatch], w1[kBatch];
        uint32_t c[kFinal ? kBatch : 1], text[kMulti ? kBatch : 1], end[kMulti ? kBatch : 1];
#pragma unroll
        for (int j = 0; j < kBatch && first + j < kItems; j++) {
            if (p[first + j] >= a.span) {  // cannot happen for valid class lists; never read out of range
                atomicExch(a.error, 3u);
                p[first + j] = 0;
            }
            const uint32_t x = p[first + j];
            const uint64_t bit = static_cast<uint64_t>(x) * bits;
            const uint64_t unit = min((bit + prefix.bits) >> 7, endUnit);
            const ulonglong2* src = reinterpret_cast<const ulonglong2*>(texts.packed) + unit;
            w0[j] = __ldg(src);
            w1[j] = __ldg(src + 1);
            if constexpr (kFinal) c[j] = x ? charCode(texts, x - 1) : 0;
            if constexpr (kMulti) {
                text[j] = texts.textOf(x);
                end[j] = texts.endOfText(text[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < kBatch && first + j < kItems; j++) {
            const uint32_t e = (first + j) * kThreads + threadIdx.x, pos = p[first + j];
            if (e >= size) continue;
            const uint64_t bit = static_cast<uint64_t>(pos) * bits + prefix.bits;
            const uint32_t o = static_cast<uint32_t>(bit & 63);
            const bool odd = (bit >> 6) & 1;
            const uint64_t v0 = odd ? w0[j].y : w0[j].x, v1 = odd ? w1[j].x : w0[j].y, v2 = odd ? w1[j].y : w1[j].x;
            uint64_t x = o ? (v0 << o) | (v1 >> (64 - o)) : v0;
            uint64_t y = o ? (v1 << o) | (v2 >> (64 - o)) : v1;
            if constexpr (kMulti) {  // the stream goes on into the next text: keep the suffix's own bits
                const uint32_t left = pos < end[j] ? min(end[j] - pos, 1024u) * bits : 0;
                const uint32_t own = left > prefix.bits ? left - prefix.bits : 0;
                x &= topMask(own);
                y &= topMask(own > 64 ? own - 64 : 0);
            }
            s.pos[e] = pos;
            uint64_t key = x >> (64 - keyBits);
            if constexpr (kMulti) {
                if (prefix.textBits) key |= static_cast<uint64_t>(text[j] - prefix.firstText) << keyBits;
            }
            s.entry[e] = (key << 16) | e;
            s.tail[e] = (x << keyBits) | (y >> (64 - keyBits));
            if constexpr (kFinal) s.prev[e] = static_cast<uint8_t>(c[j]);
        }
    }
    __syncthreads();

    // The merge tree.
    treeLevel(s, bounds, 3);
    treeLevel(s, bounds + 9, 2);
    treeLevel(s, bounds + 15, 1);

    // The groups of records that agree in their words.
#pragma unroll
    for (int j = 0; j < kItems; j++) {
        const uint32_t r = j * kThreads + threadIdx.x;
        bool differs = false;
        if (r < size) {
            const uint64_t x = s.entry[r], y = s.entry[r ? r - 1 : 0];
            differs = r == 0 || (x ^ y) >> 16 != 0 || s.tail[recordOf(x)] != s.tail[recordOf(y)];
        }
        const uint32_t word = __ballot_sync(0xffffffffu, differs);
        if ((threadIdx.x & 31) == 0 && r < size) head[r >> 5] = word;
    }
    __syncthreads();
    // Ranks of the tile's splitters in the window set bound the outputs this tile owns.
    const auto settle = [&](uint32_t x, uint32_t place) {
        if (x == t.loIdx) sLo = place;
        if (x == t.hiIdx) sHi = place;
        if constexpr (!kFinal) s.rank[x] = static_cast<uint16_t>(place);
    };
    const auto alone = [&](uint32_t r) {
        const uint32_t next = r + 1;
        return (head[r >> 5] >> (r & 31)) & (next < size ? head[next >> 5] >> (next & 31) : 1u) & 1u;
    };
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < kItems; j++) {
        const uint32_t r = j * kThreads + threadIdx.x;
        const bool tied = r < size && !alone(r);
        if (r < size && !tied) settle(recordOf(s.entry[r]), r);
        const uint32_t votes = __ballot_sync(0xffffffffu, tied);
        if (votes) {
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(&sTies, __popc(votes));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(votes & ((1u << lane) - 1));
            if (tied) {
                s.tied[at] = static_cast<uint16_t>(r);
                s.entry[r] = (static_cast<uint64_t>(at) << 16) | recordOf(s.entry[r]);  // the keys are done with
            }
        }
    }
    __syncthreads();
    const uint32_t ties = sTies;
    if (ties) {  // the same for every thread
        // Their ranks and next stream bits (a record's samples are consecutive in the rank array: the
        // kK from its first on), kStage loads of a thread in flight.
        constexpr uint32_t kStage = 4;
        const uint32_t words = min(ties, s.kStaged) * (kK + 1);
        for (uint32_t first = 0; first < words; first += kStage * kThreads) {
            uint64_t v[kStage];
#pragma unroll
            for (uint32_t j = 0; j < kStage; j++) {
                const uint32_t k = first + j * kThreads + threadIdx.x, x = k / (kK + 1), q = k % (kK + 1);
                v[j] = 0;
                if (k < words) {
                    const uint32_t pos = s.pos[recordOf(s.entry[s.tied[x]])];
                    if (q < kK) {
                        v[j] = __ldg(a.ranks + pack(pos) + q);
                    } else if (31 * bits > held) {
                        v[j] = streamBits(texts.packed, static_cast<uint64_t>(pos) * bits + held);
                    }
                }
            }
#pragma unroll
            for (uint32_t j = 0; j < kStage; j++) {
                const uint32_t k = first + j * kThreads + threadIdx.x, x = k / (kK + 1), q = k % (kK + 1);
                if (k < words) {
                    if (q < kK) s.staged[x * kK + q] = static_cast<uint32_t>(v[j]); else s.next[x] = v[j];
                }
            }
        }
        __syncthreads();
        static_assert(kClasses <= 8, "eight threads per record");
        for (uint32_t first = 0; first < 8 * ties; first += kThreads) {
            const uint32_t k = (first + threadIdx.x) >> 3, b = threadIdx.x & 7;
            uint32_t r = 0, begin = 0, end = 0, before = 0;
            if (k < ties) {
                r = s.tied[k];
                groupOf(head, size, r, begin, end);
                if (b < kClasses) before = membersBefore(s, t, r, begin, end, b, a, held);
            }
#pragma unroll
            for (int d = 1; d < 8; d <<= 1) before += __shfl_xor_sync(0xffffffffu, before, d);
            if (k < ties && b == 0) {
                settle(recordOf(s.entry[r]), begin + before);
                s.tied[k] = static_cast<uint16_t>(begin + before);
            }
        }
        __syncthreads();
    }
    const uint32_t lo = sLo, hi = sHi;
    if constexpr (kFinal) {
        for (uint32_t k = threadIdx.x; k < size; k += kThreads) {
            const uint64_t entry = s.entry[k];
            const uint32_t x = recordOf(entry);
            const uint32_t r = alone(k) ? k : s.tied[entry >> 16];
            if (r < lo || r >= hi) continue;
            const uint32_t q = s.pos[x];
            const uint32_t gIdx = t.base + r;
            if (gIdx >= a.level.start[kClasses]) {  // cannot happen for a correct tiling; never write out of range
                atomicExch(a.error, 2u);
                continue;
            }
            const uint32_t tj = kMulti ? texts.textOf(q) : 0;
            const uint32_t first = kMulti ? texts.startOf(tj) : 0;
            const uint32_t base = kMulti ? __ldg(a.outBase + tj) : 0;
            if (kMulti && a.saTexts) {
                a.saTexts[tj][gIdx - base] = q - first;
            } else if (a.sa) {
                a.sa[gIdx] = q - first;
            }
            if ((a.bwt || (kMulti && a.bwtTexts)) && q != first) {
                const uint32_t row = gIdx - base, zero = __ldg(a.rowZero + tj);
                const uint32_t local = row < zero ? row + 1 : row;
                const uint8_t c = __ldg(texts.decode + s.prev[x]);
                if (kMulti && a.bwtTexts) {
                    a.bwtTexts[tj][local] = c;
                } else {
                    a.bwt[base + local] = c;
                }
            }
        }
    } else {
        // The rows: for a sampled element, the elements of each other list before it are those of its
        // window with a smaller rank (a binary search: each window is in list order, hence in rank
        // order).
        for (uint32_t k = threadIdx.x; k < size; k += kThreads) {
            const uint64_t entry = s.entry[k];
            const uint32_t x = recordOf(entry);
            const uint32_t r = alone(k) ? k : s.tied[entry >> 16];
            const uint32_t g = t.base + r;
            if (r < lo || r >= hi || g % kR != 0) continue;
            if (g >= a.level.start[kClasses]) {  // cannot happen for a correct tiling; never write out of range
                atomicExch(a.error, 2u);
                continue;
            }
            const uint32_t l = listOfElement(t.seg, x);
            MergeRow row;
            row.list = l;
#pragma unroll
            for (uint32_t b = 0; b < kClasses; b++) {
                if (b == l) {
                    row.c[b] = t.win[l] + (x - t.seg[l]);
                    continue;
                }
                uint32_t from = t.seg[b], to = t.seg[b + 1];  // first record of list b ranked at or after r
                while (from < to) {
                    const uint32_t mid = (from + to) >> 1;
                    if (s.rank[mid] < r) from = mid + 1; else to = mid;
                }
                row.c[b] = t.win[b] + (from - t.seg[b]);
            }
            a.rowsOut[g / kR] = row;
        }
    }
}

// Launches a level (kFinal: the last).
template <bool kMulti, bool kFinal>
inline cudaError_t launchWide(const MergeArgs& args, uint32_t tiles, cudaStream_t stream) {
    constexpr size_t shared = WideTile<kFinal>::sharedBytes();
    static std::atomic<uint64_t> configured{0};
    SADCS_TRY(configureOnce(configured, [] {
        SADCS_TRY(cudaFuncSetAttribute(mergeWide<kMulti, kFinal>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(shared)));
        return cudaFuncSetAttribute(mergeWide<kMulti, kFinal>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                    SADCS_WIDE_CARVEOUT);
    }));
    return launch(mergeWide<kMulti, kFinal>, tiles, SADCS_WIDE_THREADS, shared, stream, args);
}

}  // namespace sadcs

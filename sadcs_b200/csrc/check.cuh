// check.cuh - suffix array and BWT checks on the device (the reference's checker,
// src/common/checker.cpp:53-109 and :196-245, restated as data-parallel kernels).
//
// Suffix array (Burkhardt-Karkkainen): SA is a permutation (every entry in range, inverse SA
// written by scatter, each slot owned by exactly one entry), and every neighbour pair is in order
// by (T[SA[i]], ISA[SA[i] + 1]) with the empty suffix's rank -1.
//
// BWT: the inverse of the LF mapping (a stable counting pass on the BWT's bytes), followed from the
// sentinel's row, must reach row 0 after n steps; it then spells the text. The walk is sequential in
// the reference; here it is cut at one row in kInverseStride, the pieces are walked side by side,
// and their order along the walk is found by pointer jumping over the pieces.
#pragma once

#include <algorithm>

#include "common.cuh"
#include "primitives.cuh"

namespace sadcs {

constexpr uint64_t kNoFailure = ~uint64_t(0);

// isa[p] = the largest i with sa[i] = p (isa zeroed by the caller), so that of equal entries the
// last one owns the slot whatever the order of the writes, as in a sequential scatter: the first
// duplicate reported is then the smallest index of any repeated entry, on every run.
__global__ void checkScatter(const uint32_t* __restrict__ sa, uint32_t n, uint32_t* __restrict__ isa,
                             unsigned long long* __restrict__ firstBad) {
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t p = sa[i];
    if (p >= n) {
        atomicMin(firstBad, static_cast<unsigned long long>(i));
    } else {
        atomicMax(isa + p, static_cast<uint32_t>(i));
    }
}

__global__ void checkDuplicates(const uint32_t* __restrict__ sa, uint32_t n, const uint32_t* __restrict__ isa,
                                unsigned long long* __restrict__ firstBad) {
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (isa[sa[i]] != i) atomicMin(firstBad, static_cast<unsigned long long>(i));
}

__global__ void checkOrder(const uint8_t* __restrict__ text, const uint32_t* __restrict__ sa, uint32_t n,
                           const uint32_t* __restrict__ isa, unsigned long long* __restrict__ firstBad) {
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i + 1 >= n) return;
    const uint32_t l = sa[i], r = sa[i + 1];
    bool ok = text[l] < text[r];
    if (text[l] == text[r]) {
        const int64_t ln = l + 1 < n ? static_cast<int64_t>(isa[l + 1]) : -1;
        const int64_t rn = r + 1 < n ? static_cast<int64_t>(isa[r + 1]) : -1;
        ok = ln < rn;
    }
    if (!ok) atomicMin(firstBad, static_cast<unsigned long long>(i));
}

// ---- the check of a correct suffix array ---------------------------------------------------------
//
// The same conditions, for the common case that they hold: no failing index is kept, so the inverse
// suffix array needs no order among equal entries and is written slice by slice (scatterBySlices), and
// two passes check the conditions: the first characters in text order, then the permutation
// and the order of neighbours from one read of each entry's inverse. A suffix array that fails goes to the
// kernels above, which find the first failing index. isa starts as all ones, which no entry is.
struct InversePairs {
    const uint32_t* __restrict__ sa;
    uint32_t n;
    __device__ __forceinline__ uint64_t operator()(uint32_t i) const {
        const uint32_t p = __ldcs(sa + i);
        return p < n ? (static_cast<uint64_t>(p) << 32) | i : kNoPair;
    }
};

// failed != 0 unless the suffix at every inverse rank starts with the character of that rank: rank i
// belongs to the byte c whose range [starts[c], starts[c + 1]) of the text's sorted bytes holds it. In
// text order, so nothing is read at random.
constexpr int kVerifyThreads = 256;
__global__ void __launch_bounds__(kVerifyThreads) checkFirst(const uint8_t* __restrict__ text, uint32_t n,
                                                             const uint32_t* __restrict__ isa,
                                                             const uint32_t* __restrict__ starts,
                                                             uint32_t* __restrict__ failed) {
    __shared__ uint32_t first[257];
    first[threadIdx.x] = starts[threadIdx.x];
    if (threadIdx.x == 0) first[256] = n;
    __syncthreads();
    bool ok = true;
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * kVerifyThreads;
    for (uint64_t p = static_cast<uint64_t>(blockIdx.x) * kVerifyThreads + threadIdx.x; p < n; p += stride) {
        const uint32_t r = __ldcs(isa + p), c = text[p];
        ok = ok && r >= first[c] && r < first[c + 1];
    }
    if (!ok) *failed = 1;
}

// failed != 0 unless every i has sa[i] < n, isa[sa[i]] = i (so sa is a permutation: n distinct slots are
// owned), and neighbours of the same first character (by starts; checkFirst says that they have it) in
// order by the inverse of the suffix after it. Bound by its one random read per entry, isa[sa[i]] with
// the entry after it (usually the same sector): read once and handed to the entry before by the warp,
// the last lane's by memory. 2.4 ms at 128 MiB; with the characters read here too, instead of by checkFirst (0.26 ms),
// check and gather took 8.2 ms a call against 6.6.
__global__ void __launch_bounds__(kVerifyThreads) checkVerify(const uint32_t* __restrict__ sa, uint32_t n,
                                                              const uint32_t* __restrict__ isa,
                                                              const uint32_t* __restrict__ starts,
                                                              uint32_t* __restrict__ failed) {
    __shared__ uint32_t boundary[kVerifyThreads / 32];  // bit: a byte's range starts at the place after this one
    const uint64_t base = static_cast<uint64_t>(blockIdx.x) * kVerifyThreads, i = base + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31;
    if (threadIdx.x < kVerifyThreads / 32) boundary[threadIdx.x] = 0;
    __syncthreads();
    static_assert(kVerifyThreads == 256, "one thread per byte value");
    const uint64_t at = starts[threadIdx.x];
    if (at > base && at <= base + kVerifyThreads) {
        const uint32_t k = static_cast<uint32_t>(at - 1 - base);
        atomicOr(&boundary[k >> 5], 1u << (k & 31));
    }
    // 1 + the inverse of the suffix after entry e's first character, 0 for the empty one
    const auto look = [&](uint64_t e, uint32_t& after) {
        const uint32_t p = sa[e];
        after = 0;
        if (p >= n) return false;
        after = p + 1 < n ? isa[p + 1] + 1 : 0;
        return isa[p] == e;
    };
    uint32_t after = 0;
    bool ok = true;
    if (i < n) ok = look(i, after);
    uint32_t after2 = __shfl_down_sync(0xffffffffu, after, 1);
    __syncthreads();
    if (i + 1 < n) {
        if (lane == 31) look(i + 1, after2);
        ok = ok && (after < after2 || ((boundary[threadIdx.x >> 5] >> lane) & 1));
    }
    if (!ok) *failed = 1;
}

}  // namespace sadcs

namespace sadcs {

// ---- BWT inversion ------------------------------------------------------------------------------
//
// Rows of the BWT matrix with the sentinel: n + 1; row r < primary holds bwt[r], row primary the
// sentinel, row r > primary bwt[r - 1]; bwt[u] is in row u + (u >= primary). The s-th position u in a
// stable sort of the BWT bytes says that row s + 1 starts with the byte bwt[u] and that the suffix after
// that byte is row(u). So psi(r) = row(sorted[r - 1]) leads from a suffix's row to the row of the suffix one
// character later, and row r's first character is the byte whose range of the sorted bytes holds
// r - 1. psi maps rows 1..n one to one to all rows but the primary, so following it from the primary row
// (suffix 0) ends in row 0 (the empty suffix); the BWT is valid if that takes n steps, and the first
// characters on the way are the text (checker.cpp:196-245 walks LF the other way).
//
// One random read per character is what the walk costs, so it is done once and by as many threads as
// the device holds: the walk is cut at the splitter rows (one at a hashed place in every kInverseStride
// rows, so that no period of the text lines up with them), a thread walks piece after piece, and the
// characters go to a buffer in chunks of 16 as they come (a chunk's piece and index beside it), because
// a piece's place in the text is known only when all lengths are. Pointer jumping over the pieces
// (n / kInverseStride of them) then gives the characters from each piece to the end, and a last pass
// moves the chunks to their places. At 64 MiB of natural-language-like text the walk takes 2.0 of 2.8 ms
// on the device: 34 G random 4-byte reads a second, against 62 ms for pointer jumping over every row
// (27 rounds). A splitter in 64 or 256 rows costs 0.3-0.4 ms more than one in 128: more pieces to
// order, or longer last pieces.
constexpr uint32_t kInverseStride = 128;
constexpr uint32_t kChunkChars = 16;
constexpr uint32_t kChunkRun = 8;            // chunks a thread reserves at a time
constexpr int kWalkThreads = 256;
constexpr uint32_t kWalkBlocks = 148 * 8;    // resident at once: 2048 threads per SM
constexpr uint32_t kCoarse = 2048;           // entries of the walk's table of first characters
constexpr uint32_t kNoPiece = 0xFFFFFFFFu;

// The splitter row of rows [128q, 128q + 128).
__host__ __device__ __forceinline__ uint32_t splitterRow(uint32_t q) {
    uint32_t h = q * 0x9E3779B1u;
    h ^= h >> 15;
    h *= 0x85EBCA77u;
    return q * kInverseStride + (h >> 25);
}
static_assert(kInverseStride == 128, "seven hash bits");

// Pieces: one per splitter row (piece q starts at splitterRow(q)), piece count from the primary row,
// piece count + 1 is the end (row 0).
inline uint32_t inversePieces(uint64_t n) { return static_cast<uint32_t>(n / kInverseStride + 1); }
inline uint32_t inverseBlocks(uint64_t n) {
    return std::min<uint32_t>(kWalkBlocks, ceilDiv(static_cast<uint64_t>(inversePieces(n)) + 1, kWalkThreads));
}
inline uint64_t inverseChunks(uint64_t n) {
    return n / kChunkChars + inversePieces(n) + 1 + static_cast<uint64_t>(inverseBlocks(n)) * kWalkThreads * kChunkRun;
}

// Walks every piece. sorted: BWT positions in sorted order; starts[c]: the first sorted place of byte c
// (256 entries). control[0]: pieces handed out, control[1]: chunks reserved (both zeroed by the
// caller). jump[q] = the piece after piece q in the high word and q's length in the low one. gaveUp: the
// sort's error word; where it is set, sorted is no permutation and a walk along it may never come to a
// splitter, so every piece is left empty.
__global__ void __launch_bounds__(kWalkThreads) inverseWalk(const uint32_t* __restrict__ sorted, uint32_t n,
                                                            uint32_t primary, const uint32_t* __restrict__ starts,
                                                            uint32_t pieces, uint32_t* __restrict__ control,
                                                            uint32_t maxChunks, uint4* __restrict__ chunks,
                                                            uint2* __restrict__ owner, uint64_t* __restrict__ jump,
                                                            const uint32_t* __restrict__ gaveUp) {
    __shared__ uint32_t first[257];
    __shared__ uint8_t coarse[kCoarse];
    first[threadIdx.x] = starts[threadIdx.x];
    if (threadIdx.x == 0) first[256] = n;
    __syncthreads();
    const uint32_t shift = max(0, 32 - __clz(static_cast<int>(n)) - 11);  // n >> shift < kCoarse
    for (uint32_t i = threadIdx.x; i < kCoarse; i += kWalkThreads) {
        const uint64_t at = static_cast<uint64_t>(i) << shift;  // the last byte starting at or before it
        uint32_t lo = 0, hi = 256;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (first[mid] <= at) lo = mid; else hi = mid;
        }
        coarse[i] = static_cast<uint8_t>(lo);
    }
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x == 0) jump[pieces + 1] = static_cast<uint64_t>(pieces + 1) << 32;
    uint32_t piece = kNoPiece, row = 0, length = 0;
    uint32_t chunk = 0, chunksLeft = 0;
    uint64_t word[2] = {0, 0};
    const auto flush = [&] {  // the characters since the last chunk
        if (chunksLeft == 0) {
            chunk = atomicAdd(control + 1, kChunkRun);
            chunksLeft = kChunkRun;
        }
        if (chunk < maxChunks) {  // always, by the bound on the chunks
            chunks[chunk] = make_uint4(static_cast<uint32_t>(word[0]), static_cast<uint32_t>(word[0] >> 32),
                                       static_cast<uint32_t>(word[1]), static_cast<uint32_t>(word[1] >> 32));
            owner[chunk] = make_uint2(piece, length);
        }
        chunk++;
        chunksLeft--;
        word[0] = word[1] = 0;
    };
    for (;;) {
        if (piece == kNoPiece) {
            piece = atomicAdd(control, 1u);
            if (piece > pieces) break;
            row = piece < pieces ? splitterRow(piece) : primary;
            length = 0;
            if (row == 0 || row > n || *gaveUp || (piece == pieces && row == splitterRow(row / kInverseStride))) {
                // no such row, no order to follow, or the primary row is a splitter itself
                jump[piece] = static_cast<uint64_t>(piece == pieces ? row / kInverseStride : pieces + 1) << 32;
                piece = kNoPiece;
                continue;
            }
        }
        const uint32_t place = row - 1;
        const uint32_t u = __ldg(sorted + place);
        uint32_t c = coarse[place >> shift];
        while (first[c + 1] <= place) c++;
        const uint64_t bits = static_cast<uint64_t>(c) << (8 * (length & 7));
        if (length & 8) word[1] |= bits; else word[0] |= bits;
        length++;
        row = u + (u >= primary ? 1u : 0u);
        const bool end = row == 0 || row > n || row == splitterRow(row / kInverseStride) || length > n;
        if (end || (length & (kChunkChars - 1)) == 0) flush();
        if (end) {
            const uint32_t next = row == 0 || row > n ? pieces + 1 : row / kInverseStride;
            jump[piece] = (static_cast<uint64_t>(next) << 32) | length;
            piece = kNoPiece;
        }
    }
    for (; chunksLeft; chunksLeft--, chunk++) {
        if (chunk < maxChunks) owner[chunk] = make_uint2(kNoPiece, 0);
    }
}

// One round of pointer jumping for one piece: where the piece after it leads, the lengths added (mod 2^32).
__host__ __device__ __forceinline__ uint64_t jumpOver(uint64_t mine, uint64_t next) {
    const uint32_t length = static_cast<uint32_t>(mine) + static_cast<uint32_t>(next);
    return (next & 0xFFFFFFFF00000000ull) | length;
}

// One round of pointer jumping over the pieces and the end.
__global__ void inverseJump(const uint64_t* __restrict__ in, uint64_t* __restrict__ out, uint32_t pieces) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q > pieces + 1) return;
    const uint64_t mine = in[q];
    out[q] = jumpOver(mine, in[mine >> 32]);
}

// The first place in the text of a chunk of `length` characters that follow `before` characters of its
// piece; false if it has none. toEnd: the piece's entry after the jumps. Only a BWT that does not
// invert has pieces that never reach the end (they lie on cycles of psi, and the lengths added up over their
// laps mean nothing); the characters of those that do reach it are on one way, so their sum is exact.
__host__ __device__ __forceinline__ bool chunkPlace(uint64_t toEnd, uint32_t pieces, uint32_t n, uint32_t before,
                                                    uint32_t length, uint64_t& at) {
    const uint32_t left = static_cast<uint32_t>(toEnd);  // characters from the piece's start to the end
    if (toEnd >> 32 != pieces + 1 || left > n || before > left || length > left - before) return false;
    at = n - left + before;
    return true;
}

// Every chunk to its place: the characters from its piece to the end of the text are known now. control[1]
// chunks were reserved; owner: piece and the piece's length once the chunk was full. Whole words of
// the text are written as words.
__global__ void __launch_bounds__(256) inverseSpell(const uint4* __restrict__ chunks, const uint2* __restrict__ owner,
                                                    const uint32_t* __restrict__ control, uint32_t maxChunks,
                                                    const uint64_t* __restrict__ toEnd, uint32_t pieces,
                                                    uint32_t n, uint8_t* __restrict__ text) {
    const uint32_t count = min(control[1], maxChunks);
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const uint2 o = owner[k];
    if (o.x == kNoPiece) return;
    const uint32_t length = (o.y - 1) % kChunkChars + 1, before = o.y - length;
    uint64_t at;
    if (!chunkPlace(toEnd[o.x], pieces, n, before, length, at)) return;
    const uint4 v = chunks[k];
    const uint32_t words[5] = {v.x, v.y, v.z, v.w, 0};
    uint8_t* to = text + at;
    const uint32_t head = min(length, static_cast<uint32_t>((4 - (reinterpret_cast<uintptr_t>(to) & 3)) & 3));
    const uint32_t whole = (length - head) / 4;
#pragma unroll
    for (uint32_t i = 0; i < 3; i++) {
        if (i < head) to[i] = static_cast<uint8_t>(words[0] >> (8 * i));
    }
#pragma unroll
    for (uint32_t i = 0; i < 4; i++) {
        const uint32_t w = __funnelshift_r(words[i], words[i + 1], 8 * head);
        if (i < whole) {
            reinterpret_cast<uint32_t*>(to + head)[i] = w;
        } else if (i == whole) {
            for (uint32_t b = head + 4 * i; b < length; b++) to[b] = static_cast<uint8_t>(w >> (8 * (b - head - 4 * i)));
        }
    }
}

// First text position where the inverse differs from the text.
__global__ void lfCompare(const uint8_t* __restrict__ a, const uint8_t* __restrict__ b, uint32_t n,
                          unsigned long long* __restrict__ firstBad) {
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n && a[i] != b[i]) atomicMin(firstBad, static_cast<unsigned long long>(i));
}

struct ByteLoader {
    const uint8_t* __restrict__ bytes;
    __device__ __forceinline__ bool load(uint32_t, uint32_t i, uint32_t, uint8_t& k, uint32_t& d) const {
        k = bytes[i];
        d = k;
        return true;
    }
    __device__ __forceinline__ uint32_t value(uint32_t, uint32_t i, uint32_t) const { return i; }
};

struct ValueStorer {
    static constexpr bool kKeys = false;
    uint32_t* __restrict__ out;
    uint32_t limit;
    __device__ __forceinline__ void storeKey(uint32_t, uint32_t, uint8_t) const {}
    __device__ __forceinline__ void storeValue(uint32_t, uint32_t pos, uint32_t v) const {
        if (pos < limit) out[pos] = v;
    }
};

// Byte histogram (256 words, zeroed by the caller) of bytes[0, n).
__global__ void __launch_bounds__(256) byteHistogram(const uint8_t* __restrict__ bytes, uint32_t n,
                                                     uint32_t* __restrict__ counts) {
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t lt = (1u << (threadIdx.x & 31)) - 1;
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t base = static_cast<uint64_t>(blockIdx.x) * blockDim.x; base < n; base += stride) {
        const uint64_t i = base + threadIdx.x;
        const uint32_t c = i < n ? bytes[i] : kNoDigit;
        const uint32_t peers = __match_any_sync(0xffffffffu, c);
        if (c != kNoDigit && (peers & lt) == 0) atomicAdd(&h[c], static_cast<uint32_t>(__popc(peers)));
    }
    __syncthreads();
    if (h[threadIdx.x]) atomicAdd(counts + threadIdx.x, h[threadIdx.x]);
}

// The stable pass by byte runs over chunks of kInverseChunk positions, each a segment with its own
// digit bases (the digit's start plus its count in the chunks before), so that no segment reaches the
// 2^30 counts a look-back word holds; one chunk below that size.
constexpr uint32_t kInverseChunk = 1u << 29;
constexpr uint32_t kInverseMaxChunks = 8;  // n < 2^32

// elementStart[s] / tileStart[s] of the chunks (s = 0..chunks). One thread per entry.
__global__ void inverseChunkTables(uint32_t n, uint32_t chunks, uint32_t* __restrict__ elementStart,
                                   uint32_t* __restrict__ tileStart) {
    const uint32_t s = threadIdx.x;
    if (s > chunks) return;
    const uint64_t e = min(static_cast<uint64_t>(s) * kInverseChunk, static_cast<uint64_t>(n));
    elementStart[s] = static_cast<uint32_t>(e);
    tileStart[s] = static_cast<uint32_t>((e + kSortTile - 1) / kSortTile);
}

// hist[s][d] (byte counts of chunk s) becomes the first output slot of byte d in chunk s: every
// smaller byte, then byte d in the chunks before. One block of 256 threads.
__global__ void __launch_bounds__(256) inverseChunkBases(uint32_t* __restrict__ hist, uint32_t chunks) {
    __shared__ uint32_t warpTotals[32];
    const uint32_t d = threadIdx.x;
    uint32_t total = 0;
    for (uint32_t s = 0; s < chunks; s++) total += hist[s * 256 + d];
    uint32_t all;
    const uint32_t inclusive = blockInclusiveScan<OpSum>(total, warpTotals, all);
    uint32_t base = inclusive - total;
    for (uint32_t s = 0; s < chunks; s++) {
        const uint32_t c = hist[s * 256 + d];
        hist[s * 256 + d] = base;
        base += c;
    }
}

// Inverts bwt (n bytes, primary) into text (n bytes) on the device. scratch: inverseScratchWords(n)
// words, 16-byte aligned; hostWords: four words (page-locked or not). valid = false if the BWT is not
// a valid one (the way from the primary row misses rows).
inline size_t inverseScratchWords(uint64_t n) {
    const uint64_t sort = n + 64 + radixScratchWords(n) + 2 * kInverseMaxChunks * 256 + 64;
    const uint64_t walk = 6 * inverseChunks(n) + 4 * (static_cast<uint64_t>(inversePieces(n)) + 2) + 16;
    return static_cast<size_t>(sort + walk + 64);
}

inline cudaError_t inverseBwt(const uint8_t* bwt, uint32_t n, uint32_t primary, uint8_t* text, uint32_t* scratch,
                              uint32_t* hostWords, cudaStream_t stream, bool& valid) {
    valid = true;
    if (n == 0) return cudaSuccess;
    const uint32_t pieces = inversePieces(n);
    const uint32_t maxChunks = static_cast<uint32_t>(std::min<uint64_t>(inverseChunks(n), 0xFFFFFFFFu));
    uint4* chunkData = reinterpret_cast<uint4*>(scratch);                            // 16-byte words first
    uint2* owner = reinterpret_cast<uint2*>(chunkData + inverseChunks(n));
    uint64_t* jump[2];
    jump[0] = reinterpret_cast<uint64_t*>(owner + inverseChunks(n));
    jump[1] = jump[0] + pieces + 2;
    uint32_t* control = reinterpret_cast<uint32_t*>(jump[1] + pieces + 2);           // 16 words
    uint32_t* sorted = control + 16;                                                 // n
    uint32_t* radixWords = sorted + n;
    uint32_t* hist = radixWords + radixScratchWords(n);  // [chunks][256], then the chunk tables
    uint32_t* starts = hist + kInverseMaxChunks * 256;   // [256] first sorted place of every byte
    uint32_t* elementStart = starts + kInverseMaxChunks * 256;  // 16 words, then tileStart (16)
    uint32_t* tileStart = elementStart + 16;
    const uint32_t segments = ceilDiv(n, kInverseChunk);
    const RadixScratch radix(radixWords, n);
    SADCS_TRY(cudaMemsetAsync(control, 0, 16 * 4, stream));
    SADCS_TRY(cudaMemsetAsync(radix.control, 0, 8, stream));
    SADCS_TRY(cudaMemsetAsync(hist, 0, static_cast<size_t>(segments) * 256 * 4, stream));
    for (uint32_t c = 0; c < segments; c++) {
        const uint32_t count = std::min<uint32_t>(kInverseChunk, n - c * kInverseChunk);
        const uint32_t histBlocks = std::min<uint32_t>(ceilDiv(count, 256 * 16), 148 * 8);
        SADCS_TRY(launch(byteHistogram, histBlocks, 256, 0, stream, bwt + static_cast<size_t>(c) * kInverseChunk,
                         count, hist + static_cast<size_t>(c) * 256));
    }
    SADCS_TRY(launch(inverseChunkBases, 1, 256, 0, stream, hist, segments));
    // the first segment's bases are the bytes' first places
    SADCS_TRY(cudaMemcpyAsync(starts, hist, 256 * 4, cudaMemcpyDeviceToDevice, stream));
    SADCS_TRY(launch(inverseChunkTables, 1, 32, 0, stream, n, segments, elementStart, tileStart));
    SADCS_TRY((radixOnesweepPass<uint8_t, ByteLoader, ValueStorer, ManySegments>(
        ByteLoader{bwt}, ValueStorer{sorted, n}, ManySegments{tileStart, elementStart, segments}, n, ceilDiv(n, kSortTile),
        hist, radix, stream)));
    SADCS_TRY(launch(inverseWalk, inverseBlocks(n), kWalkThreads, 0, stream, sorted, n, primary, starts, pieces, control,
                     maxChunks, chunkData, owner, jump[0], radix.control + 1));
    int cur = 0;
    for (uint64_t reach = 1; reach < static_cast<uint64_t>(pieces) + 2; reach *= 2, cur ^= 1) {
        SADCS_TRY(launch(inverseJump, ceilDiv(static_cast<uint64_t>(pieces) + 2, 256), 256, 0, stream, jump[cur],
                         jump[cur ^ 1], pieces));
    }
    SADCS_TRY(launch(inverseSpell, ceilDiv(inverseChunks(n), 256), 256, 0, stream, chunkData, owner, control, maxChunks,
                     jump[cur], pieces, n, text));
    SADCS_TRY(cudaMemcpyAsync(hostWords, jump[cur] + pieces, 8, cudaMemcpyDeviceToHost, stream));
    SADCS_TRY(cudaMemcpyAsync(hostWords + 2, radix.control + 1, 4, cudaMemcpyDeviceToHost, stream));
    SADCS_TRY(cudaStreamSynchronize(stream));
    if (hostWords[2]) return cudaErrorLaunchTimeout;
    valid = hostWords[1] == pieces + 1 && hostWords[0] == n;
    return cudaSuccess;
}

}  // namespace sadcs

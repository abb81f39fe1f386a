// Host run of the inverse BWT's walk (sadcs_b200/csrc/check.cuh) for CPU tests: the splitter rows, the
// jumps over the pieces and the chunks' places are the kernels' own functions; the walk is followed
// here piece by piece, and every chunk's characters are written only where they lie inside the text, with
// the places outside it counted. Test infrastructure only.
#include <cstdint>
#include <vector>

#include "../sadcs_b200/csrc/check.cuh"

using namespace sadcs;

// Inverts bwt (n bytes, 1 <= primary <= n) into text (n bytes). Returns whether the BWT is a valid one;
// *outside gets the number of characters whose place is outside [0, n).
extern "C" int inverse_emulate(const uint8_t* bwt, int64_t n64, int64_t primary64, uint8_t* text, int64_t* outside) {
    const uint32_t n = static_cast<uint32_t>(n64), primary = static_cast<uint32_t>(primary64);
    std::vector<uint32_t> sorted(n), start(257, 0);
    for (uint32_t u = 0; u < n; u++) start[bwt[u] + 1]++;
    for (int c = 0; c < 256; c++) start[c + 1] += start[c];
    for (uint32_t u = 0; u < n; u++) sorted[start[bwt[u]]++] = u;
    const uint32_t pieces = inversePieces(n);
    std::vector<uint64_t> jump(pieces + 2), out(pieces + 2);
    std::vector<std::vector<uint8_t>> spelled(pieces + 1);
    jump[pieces + 1] = static_cast<uint64_t>(pieces + 1) << 32;
    for (uint32_t piece = 0; piece <= pieces; piece++) {
        uint32_t row = piece < pieces ? splitterRow(piece) : primary;
        if (row == 0 || row > n || (piece == pieces && row == splitterRow(row / kInverseStride))) {
            jump[piece] = static_cast<uint64_t>(piece == pieces ? row / kInverseStride : pieces + 1) << 32;
            continue;
        }
        do {
            const uint32_t u = sorted[row - 1];
            spelled[piece].push_back(bwt[u]);
            row = u + (u >= primary ? 1u : 0u);
        } while (row != 0 && row != splitterRow(row / kInverseStride));
        jump[piece] = (static_cast<uint64_t>(row == 0 ? pieces + 1 : row / kInverseStride) << 32) | spelled[piece].size();
    }
    for (uint64_t reach = 1; reach < static_cast<uint64_t>(pieces) + 2; reach *= 2) {
        for (uint32_t q = 0; q <= pieces + 1; q++) out[q] = jumpOver(jump[q], jump[jump[q] >> 32]);
        jump.swap(out);
    }
    *outside = 0;
    for (uint32_t piece = 0; piece <= pieces; piece++) {
        const uint32_t length = static_cast<uint32_t>(spelled[piece].size());
        for (uint32_t before = 0; before < length; before += kChunkChars) {
            const uint32_t chunk = std::min(kChunkChars, length - before);
            uint64_t at;
            if (!chunkPlace(jump[piece], pieces, n, before, chunk, at)) continue;
            for (uint32_t i = 0; i < chunk; i++) {
                if (at + i < n) text[at + i] = spelled[piece][before + i]; else ++*outside;
            }
        }
    }
    return jump[pieces] >> 32 == pieces + 1 && static_cast<uint32_t>(jump[pieces]) == n;
}

// On the GPU: the walk after a sort that gave up (its error word set). order: what the sort left (n
// entries). Returns the characters walked, or -1 if a CUDA call failed; *chunks gets the chunks reserved.
extern "C" int64_t inverse_walk_after_time_out(const uint32_t* order, int64_t n64, int64_t primary, int64_t* chunks) {
    const uint32_t n = static_cast<uint32_t>(n64), pieces = inversePieces(n);
    const uint64_t most = inverseChunks(n);
    uint32_t *sorted = nullptr, *starts = nullptr, *control = nullptr;  // control[0..1], then the error word
    uint4* data = nullptr;
    uint2* owner = nullptr;
    uint64_t* jump = nullptr;
    std::vector<uint64_t> lengths(pieces + 2, 0);
    const uint32_t words[4] = {0, 0, 1, 0};
    uint32_t after[2] = {0, 0};
    const bool ok = cudaMalloc(&sorted, 4 * static_cast<size_t>(n)) == cudaSuccess && cudaMalloc(&starts, 1024) == cudaSuccess &&
                    cudaMalloc(&control, sizeof words) == cudaSuccess && cudaMalloc(&data, 16 * most) == cudaSuccess &&
                    cudaMalloc(&owner, 8 * most) == cudaSuccess && cudaMalloc(&jump, 8 * lengths.size()) == cudaSuccess &&
                    cudaMemcpy(sorted, order, 4 * static_cast<size_t>(n), cudaMemcpyHostToDevice) == cudaSuccess &&
                    cudaMemset(starts, 0, 1024) == cudaSuccess &&
                    cudaMemcpy(control, words, sizeof words, cudaMemcpyHostToDevice) == cudaSuccess &&
                    launch(inverseWalk, inverseBlocks(n), kWalkThreads, 0, nullptr, sorted, n, static_cast<uint32_t>(primary),
                           starts, pieces, control, static_cast<uint32_t>(most), data, owner, jump, control + 2) == cudaSuccess &&
                    cudaDeviceSynchronize() == cudaSuccess &&
                    cudaMemcpy(lengths.data(), jump, 8 * lengths.size(), cudaMemcpyDeviceToHost) == cudaSuccess &&
                    cudaMemcpy(after, control, sizeof after, cudaMemcpyDeviceToHost) == cudaSuccess;
    for (void* p : {static_cast<void*>(sorted), static_cast<void*>(starts), static_cast<void*>(control),
                    static_cast<void*>(data), static_cast<void*>(owner), static_cast<void*>(jump)}) {
        if (p) cudaFree(p);
    }
    if (!ok) return -1;
    *chunks = after[1];
    int64_t walked = 0;
    for (uint64_t v : lengths) {
        walked += static_cast<uint32_t>(v);
        if (v >> 32 > pieces + 1) return -1;  // an entry that the jumps could not follow
    }
    return walked;
}

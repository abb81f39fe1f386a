// The calls without a context before and after cudaDeviceReset (sadcs_b200/csrc/sadcs_gpu.cu included whole,
// so that the reset is of the library's own runtime). Run in a process of its own. Test infrastructure only.
#include "../sadcs_b200/csrc/sadcs_gpu.cu"

namespace {

// Checks sa and computes the LCP array of text and its BWT; 0 if all calls succeed.
int once(const uint8_t* text, int64_t n, const uint32_t* sa, uint32_t* lcp, uint8_t* bwt) {
    uint8_t *dText = nullptr, *dBwt = nullptr;
    uint32_t *dSa = nullptr, *dLcp = nullptr;
    int64_t bad = 0, primary = 0;
    const size_t words = 4 * static_cast<size_t>(n);
    if (cudaMalloc(&dText, n) != cudaSuccess || cudaMalloc(&dBwt, n) != cudaSuccess || cudaMalloc(&dSa, words) != cudaSuccess ||
        cudaMalloc(&dLcp, words) != cudaSuccess || cudaMemcpy(dText, text, n, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(dSa, sa, words, cudaMemcpyHostToDevice) != cudaSuccess) {
        return 1;
    }
    if (sadcs_gpu_check_suffix_array(dText, n, dSa, &bad, nullptr, nullptr) != SADCS_OK || bad != -1) return 2;
    if (sadcs_gpu_lcp(dText, n, dSa, dLcp, nullptr) != SADCS_OK) return 3;
    if (sadcs_gpu_bwt_from_sa(dText, n, dSa, dBwt, &primary, nullptr) != SADCS_OK) return 4;
    if (cudaMemcpy(lcp, dLcp, words, cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(bwt, dBwt, n, cudaMemcpyDeviceToHost) != cudaSuccess) {
        return 5;
    }
    cudaFree(dText);
    cudaFree(dBwt);
    cudaFree(dSa);
    cudaFree(dLcp);
    return 0;
}

int64_t freeBytes() {
    size_t available = 0, total = 0;
    return cudaMemGetInfo(&available, &total) == cudaSuccess ? static_cast<int64_t>(available) : -1;
}

}  // namespace

// The calls, then cudaDeviceReset and the calls again, `resets` times; lcp and bwt are the last ones'. left[k]:
// the free memory after the k-th round, left[resets + 1]: after sadcs_gpu_query_device has given back what is kept.
extern "C" int reset_rounds(const uint8_t* text, int64_t n, const uint32_t* sa, uint32_t* lcp, uint8_t* bwt, int resets,
                            int64_t* left) {
    for (int k = 0; k <= resets; k++) {
        if (k > 0 && cudaDeviceReset() != cudaSuccess) return 10;
        if (const int failedAt = once(text, n, sa, lcp, bwt); failedAt) return 100 * k + failedAt;
        left[k] = freeBytes();
    }
    sadcs_gpu_device device;
    if (sadcs_gpu_query_device(&device) != SADCS_OK) return 11;
    left[resets + 1] = freeBytes();
    return 0;
}

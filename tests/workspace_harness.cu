// The calls without a context and their memory pool (sadcs_b200/csrc/sadcs_gpu.cu included whole: the pool is the
// library's own, and a device reset is of the library's own runtime). Test infrastructure only.
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
// the free memory after the k-th round, left[resets + 1]: after sadcs_gpu_query_device has given back what is kept. Run in a process of its own.
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

// The most bytes in use at a time from the pool while the check that allocates runs (high[0]) and
// while the one without allocation runs twice (high[1]), on device buffers.
extern "C" int pool_use_of_checks(const uint8_t* dText, int64_t n, const uint32_t* dSa, uint64_t* high) {
    const auto used = [&](uint64_t* out) {
        return withWorkspacePool(true, [&](cudaMemPool_t pool) {
            const cudaError_t error = cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemHigh, out);
            uint64_t zero = 0;
            return error == cudaSuccess ? cudaMemPoolSetAttribute(pool, cudaMemPoolAttrUsedMemHigh, &zero) : error;
        });
    };
    uint64_t before = 0;
    if (used(&before) != cudaSuccess) return 1;
    if (sadcs_gpu_check_suffix_array(dText, n, dSa, nullptr, nullptr, nullptr) != SADCS_OK) return 2;
    if (used(&high[0]) != cudaSuccess) return 3;
    for (int k = 0; k < 2; k++) {
        if (sadcs_gpu_check_suffix_array_static(dText, n, dSa, nullptr, nullptr, nullptr) != SADCS_OK) return 4;
    }
    return used(&high[1]) == cudaSuccess ? 0 : 5;
}

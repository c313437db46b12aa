#include "fu_kernels.h"
#include "host_util.h"

#include <mutex>
#include <set>
#include <utility>

namespace fu {
char* error_buffer()
{
    static thread_local char buf[512] = {0};
    return buf;
}

int raise_smem_limit(const void* kernel, int bytes)
{
    static std::mutex                            lock;
    static std::set<std::pair<int, const void*>> raised;
    int                                          dev = 0;
    FU_CUDA_OK(cudaGetDevice(&dev));
    const std::lock_guard<std::mutex> guard(lock);
    if (raised.count({dev, kernel}) == 0) {
        FU_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        raised.insert({dev, kernel});
    }
    return FU_OK;
}
}  // namespace fu

// The word lies in the library's image, zero from the moment it is loaded: nothing is allocated, filled or waited
// for when it is first asked for, which may be inside a stream capture.
static __device__ uint32_t g_error_word;

extern "C" int fu_error_word(void** word)
{
    if (!word) {
        return fu::fail(FU_E_ARG, "fu_error_word: null argument");
    }
    FU_CUDA_OK(cudaGetSymbolAddress(word, g_error_word));
    return FU_OK;
}

#define FU_STR2(x) #x
#define FU_STR(x) FU_STR2(x)

extern "C" const char* fu_last_error(void)
{
    return fu::error_buffer();
}

extern "C" const char* fu_build_info(void)
{
    return "sm_100a;nvcc " FU_STR(__CUDACC_VER_MAJOR__) "." FU_STR(__CUDACC_VER_MINOR__) "." FU_STR(
        __CUDACC_VER_BUILD__) ";fast_ulysses_b200 0.1.0";
}

// The kNN filter's approximate distances, behind a C entry for the test that compares them with FP64.
#include "../../masterthesislucas_gb300/csrc/knn_gram.cuh"

void tc_set_error(const char*, ...) {}
int tc_cuda_fail(cudaError_t, const char*) { return TC_ERR_CUDA; }
namespace tc {
int sm_count() { return 152; }
}  // namespace tc

// a: [column block of 256][row block of 128][column][row], norms s (npad = n rounded up to 256), stat: 4 words.
// hi and lo hold npad * dim (rounded up to 16) BF16 numbers, gmin a quarter of a.  Device pointers.
extern "C" int gram(const float* x, long long n, int dim, uint8_t* hi, uint8_t* lo, float* s, float* a, float* gmin,
                    void* stat)
{
    using namespace tc;
    const int dimp = (dim + 15) & ~15;
    const int64_t npad = (n + kGramCols - 1) / kGramCols * kGramCols, rblocks = (n + kGramRows - 1) / kGramRows;
    const int64_t tiles = rblocks * (npad / kGramCols);
    GramStat* st = static_cast<GramStat*>(stat);
    TC_CUDA_TRY(cudaFuncSetAttribute(k_gram, cudaFuncAttributeMaxDynamicSharedMemorySize, kGramSmem));
    TC_CUDA_TRY(cudaMemset(st, 0, sizeof(GramStat)));
    k_gram_split<<<(unsigned)(npad / 8), 256>>>(x, n, dim, dimp, hi, lo, s, st);
    k_gram<<<(unsigned)(tiles < sm_count() ? tiles : sm_count()), kGramThreads, kGramSmem>>>(
        hi, lo, s, n, npad, dimp, 0, (int)rblocks, a, gmin, st);
    TC_CUDA_TRY(cudaDeviceSynchronize());
    return TC_OK;
}

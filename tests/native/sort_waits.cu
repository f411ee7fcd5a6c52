// The radix sort with waits that run out at once (TC_SORT_POLLS 0), behind a C entry for the test that loads it.
#include "../../masterthesislucas_gb300/csrc/scan.cu"
#include "../../masterthesislucas_gb300/csrc/sort.cu"

void tc_set_error(const char*, ...) {}
int tc_cuda_fail(cudaError_t, const char*) { return TC_ERR_CUDA; }
namespace tc {
int sm_count() { return 152; }
}  // namespace tc

extern "C" long long sort_tmp_words(long long n) { return tc::radix_tmp_words(n); }
// keys (or alt_keys, for an odd number of passes) in, sorted keys and their input positions out; device pointers
extern "C" int sort_u32(uint32_t* keys, uint32_t* vals, uint32_t* alt_keys, uint32_t* alt_vals, long long n,
                        uint32_t* tmp, int lo_bit, void* stream)
{
    return tc::radix_sort_u32(keys, vals, alt_keys, alt_vals, n, tmp, (cudaStream_t)stream, nullptr, lo_bit);
}

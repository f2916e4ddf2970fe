/*
 * index.cu -- what an index holds in device memory (gs_index.cu), on the fake
 * runtime.  Its tables stay empty; the text structures' kernel reports every
 * row as reached.
 */
#include "../../gpuseed_gb300/csrc/gs_index.cu"

#include "fake_cuda.h"

void gs_set_error(const char *, ...) {}
int gs_cuda_fail(cudaError_t e, const char *) { return e == cudaErrorMemoryAllocation ? GS_ENOMEM : GS_ECUDA; }
int gs_build_kmer_table(const GsDevIndex &, uint2 *, cudaStream_t) { return GS_OK; }
int gs_build_kmerx_table(const GsDevIndex &, uint4 *, int, cudaStream_t) { return GS_OK; }

static void fake_kernel(const std::string &name, void **args)
{
    if (name.find("gs_text_chain_kernel") == std::string::npos) return;
    unsigned long long *stat = *(unsigned long long **)args[4];
    stat[0] = ((const GsDevIndex *)args[0])->seq_len + 1ull;
}

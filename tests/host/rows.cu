/*
 * rows.cu -- device rules that are plain functions of row numbers, on the host.
 */
#include "../../gpuseed_gb300/csrc/gs_internal.h"

#include "fake_cuda.h"

static void fake_kernel(const std::string &, void **) {}

extern "C" {
int rows_text_mode(int32_t text_min, uint32_t jl) { return gs_text_mode(text_min, jl); }
int rows_clear_in_kernel(uint32_t n_reads, uint32_t tile, uint64_t words)
{
    return gs_clear_in_kernel(n_reads, tile, words);
}
/* entry `idx` of a buffer of four, of which the first three are a warp's, after
 * a walker of a read of iL bases was put there */
int rows_put_walker(uint64_t idx, int iL, GsWalker *w)
{
    GsWalker four[4];
    memset(four, 0x55, sizeof(four));
    const bool there = gs_put_walker(four, idx, 3, 7, true, 5, 1, 2, 3, 4, true, iL);
    *w = four[idx];
    return there;
}
}

/*
 * rows.cu -- device rules that are plain functions of row numbers, on the host.
 */
#include "../../gpuseed_gb300/csrc/gs_internal.h"

#include "fake_cuda.h"

static void fake_kernel(const std::string &, void **) {}

extern "C" {
int rows_text_mode(int32_t text_min, uint32_t jl) { return gs_text_mode(text_min, jl); }
}

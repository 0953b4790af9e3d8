// GEMM for operands the TMA kernels cannot take as they lie in memory: fp32 matrices, rows that
// do not start on 16-byte boundaries, problems of a few tiles.  See gemm_direct.cu.
#pragma once
#include "gemm.h"

namespace lt {

// Launches the direct kernel (tensor cores) for `a`; every size, stride and alignment.
cudaError_t gemm_direct(const GemmArgs& a, cudaStream_t stream);
// Estimated time (s) of gemm_direct for `a`.
double gemm_direct_cost(const GemmArgs& a);
// Packing operands for the TMA kernels: bytes of workspace, and the launch that fills it and
// rewrites `a` to the packed product.
size_t gemm_pack_bytes(const GemmArgs& a);
bool gemm_pack_fits(const GemmArgs& a);   // one launch holds all of its blocks
cudaError_t gemm_pack(GemmArgs& a, void* workspace, cudaStream_t stream);
// Error word of its bounded waits (0 = ok).  Reading synchronises.
int gemm_direct_last_error();
void gemm_direct_clear_error();

}  // namespace lt

// Batched matrix product Y[rows, n_out] = X[rows, k] * W^T with fused de-quantisation (see gemm.cu).
#pragma once
#include <cuda.h>

#include "../../include/albatross_b200.h"
#include "common.cuh"

namespace ab {

// Tensor maps of a weight matrix and, for NVFP4 where the pitch allows it, of its block scales. They depend on the matrix
// only, so a model encodes them once and its launches take them from there.
struct WeightMaps {
    CUtensorMap w, s;
    int valid;       // 0: not encoded (a shape or address the products do not take; the launch names the reason)
    int scale_map;   // s is there
};
int encode_weight_maps(const ab_mat& m, WeightMaps* out);

// One product of a grouped launch: Y[rows, n_out] = epilogue(X[rows, k] * W^T).
struct GemmOp {
    ab_mat w;
    const __half* x;
    __half* y;
    const __half* resid;
    int epi;
    const WeightMaps* maps;   // of `w` (null: encoded for this launch)
};
// Scratch: split-K arrival counters and fp32 partial tiles. It must be zero when first used; the kernels
// leave the counters at zero again. What a launch needs is not monotonic in `rows` (few rows are split along K where many
// fill the GPU), so a caller with several launches takes the largest; a launch whose partial sums do not fit into
// `scratch_bytes` runs without the split.
size_t gemm_group_scratch_bytes(const GemmOp* ops, int n, int rows);
// pdl: launch with programmatic stream serialisation (the kernel waits for the preceding grid itself, after it has
// started its weight stream).
int gemm_group_launch(const GemmOp* ops, int n, int rows, void* scratch, size_t scratch_bytes, cudaStream_t stream, bool pdl = false);
// The same for few rows (stream.cu): *taken tells whether it took the launch.
int stream_group_launch(const GemmOp* ops, int n, int rows, cudaStream_t stream, bool pdl, bool* taken);
size_t gemm_scratch_bytes(const ab_mat& m, int rows);
int static_scratch_reset(cudaStream_t stream);   // built-in scratch of ab_gemm_static: counters back to zero
int gemm_launch(const ab_mat& m, int rows, const __half* x, __half* y, int epi, const __half* resid, void* scratch,
                size_t scratch_bytes, cudaStream_t stream, bool pdl = false, const WeightMaps* maps = nullptr);
int dequant_launch(const ab_mat& m, float* out, cudaStream_t stream);
int check_mat(const ab_mat& m, const char* what);

}  // namespace ab

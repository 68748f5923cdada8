// igemm_unit.cuh -- the one-wave form of the contraction (see igemm_unit.cu).
#pragma once
#include "igemm.cuh"

namespace one {

// What a launch of the unit kernel needs beside IgemmParams (M, N, num_kb, slab, A addressing, epilogue fields; split_k,
// tma_store, res_mma, nchw_hw and lut_smem are not read).
struct UnitParams {
    int splits;           // CTAs of a cluster that share a tile along K: 1, 2, 4 or 8
    int b_const;          // B holds a prepared operator's weights and bias its own copy: no earlier kernel of the stream writes
                          // them, so their loads start before the wait
    int nchw_hw;          // > 0: out is fp32 [M / hw][N][hw] (the reference layout of a convolution's output)
    // fp32 operands read as the caller left them (tf32 launches with `raw`): rounded to tf32 on their way through
    // shared memory.  0: by TMA, K-major; 1: by plain loads, K-major rows of `pitch` floats; 2: by plain loads,
    // [K][rows] (the second operand of a MatMul).  K: row length.
    int raw, a_ld, b_ld, K;
    const float *a, *b;
    long long a_pitch, b_pitch, a_bstride, b_bstride;
};
constexpr int UNIT_BN = 64;          // output columns of a tile
constexpr int UNIT_MAX_STAGES = 4;
// Which epilogue a launch takes, or -1 when the unit kernel does not have it (the persistent kernel does).
int unit_epilogue(int kind, const IgemmParams &p, const UnitParams &u);
// tmB's box holds UNIT_BN rows.  tmA / tmB may be unset maps for operands that are not loaded by TMA.
cudaError_t launch_unit(int kind, const CUtensorMap &tmA, const CUtensorMap &tmB, const IgemmParams &p, const UnitParams &u, cudaStream_t stream);

}  // namespace one

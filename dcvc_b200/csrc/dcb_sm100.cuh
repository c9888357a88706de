// Tail of a DepthConvBlock for sm_100a in one kernel: dc.3 (1x1 + residual), ffn.0 (quad GEMM) and
// ffn.2 (1x1 + residual), the two intermediate activations kept on chip; see dcb_sm100.cu.
#pragma once

#include "common.cuh"

namespace dcvc {

struct DcbTailParams {
    int M;                // pixels
    int C;                // block channels
    int cdc;              // dc.3 input channels; 0: the block starts at ffn.0 (ConvFFN alone)
    int cffn;             // quad outputs: ffn.0 has 4 cffn output channels, ffn.2 cffn input channels
    const void* a;        // [M, cdc] depthwise output, pitch lda (cdc > 0)
    int lda;
    const void* x;        // [M, C] residual of dc.3, or the ConvFFN's input when cdc = 0; pitch ldx
    int ldx;
    const void* w0;       // [C, cdc] dense
    const void* w1;       // [4 cffn, C] dense
    const void* w2;       // [C, cffn] dense
    const float* b0;      // [C]
    const float* b1;      // [4 cffn]
    const float* b2;      // [C]
    const void* qscale;   // [C] multiplier of the output (activation dtype) or null
    int q_rows;           // > 0: one row of C factors per image of q_rows rows
    void* out;            // [M, C], pitch ldo
    int ldo;
    int* err;             // device error word
    // Test hook (gemm_inject_stall; 0 in production): the MMA warp issues nothing, so every wait behind it runs out
    // after wait_limit cycles (0: the kernel's own limit, ~1 s) and the drains find copies that have landed.
    int stall_test;
    long long wait_limit;
};

// Whether dcb_tail_sm100 has a form for these channel counts (n1 = ffn.0 output channels, cdc = 0:
// ConvFFN alone), and whether it is the faster choice at M pixels.
bool dcb_tail_supported(int C, int cdc, int cffn, int n1);
bool dcb_tail_preferred(int M, int C, int cdc, int cffn, int n1);

// dtype 0 = FP16, 1 = BF16.  Bitwise the outputs of the separate launches.
cudaError_t dcb_tail_sm100(int dtype, const DcbTailParams& p, cudaStream_t stream);

}  // namespace dcvc

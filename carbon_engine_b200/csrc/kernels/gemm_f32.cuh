// What the float32 product (gemm_f32.cu) and the plain product (gemm_plain.cu) share: the epilogues.
#pragma once
#include "common.cuh"

enum { GP_STORE = 0, GP_STORE_F32 = 1, GP_ACCUM_F32 = 2, GP_SWIGLU = 3, GP_RELUGLU = 4, GP_RELU2 = 5, GP_CLAMPGLU = 6 };     // 4: relu(gate) * up; 5: relu(v)^2; 6: ce_clamp_glu(gate + bias, up + bias)
#define GP_GATED(mode) ((mode) == GP_SWIGLU || (mode) == GP_RELUGLU || (mode) == GP_CLAMPGLU)

struct GpGate {
    const float* bias;           // float32 [2N] or null: gate rows, then up rows (mode 6)
    float limit, alpha;
};

// The product in float32 (sizes and pointers checked by the caller).  weights_ready: no kernel on the stream may still be writing W,
// so its first rows are read while the kernels in front run.
int ce_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldc, int mode, const GpGate& gate,
                bool weights_ready, cudaStream_t stream);

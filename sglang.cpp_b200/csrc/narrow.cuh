// Epilogue of the products of a handful of rows (gemm_narrow.cu, gemm_ring.cu): a thread has two features of a token.
#pragma once

#include "common.cuh"
#include "kernels.h"

namespace b200 {

// From this K on a warp walks much of its share of K behind the wait, and CTAs of the next kernels, let in early, only take
// bandwidth from it (2048 x 6144 in a decode step of 16 requests: 568 us per step without, 585 with; 1024 x 3072, most of which
// is requested ahead, the other way round: 723 us per step with, 770 without).
constexpr int kWalkedK = 4096;
constexpr int kTokenPitch = 20;  // floats: 16 features of a token, padded so that a warp's stores hit 32 banks

struct NarrowOut {
    __nv_bfloat16* y;            // [M, y_pitch]
    int n_out, epilogue;
    int64_t y_pitch;
    float act_limit;
};

__device__ __forceinline__ float activate_pair(int epilogue, float g, float u, float limit) {
    switch (epilogue) {
        case B200_EPILOGUE_SWIGLU: return __fdividef(g, 1.0f + __expf(-g)) * u;
        case B200_EPILOGUE_GEGLU_ERF: return 0.5f * g * (1.0f + erff(g * 0.70710678118654752f)) * u;
        case B200_EPILOGUE_CLAMPED_SWIGLU: return clamped_swiglu<false>(g, u, limit);
        default: return 0.5f * g * (1.0f + tanhf(0.7978845608f * (g + 0.044715f * g * g * g))) * u;
    }
}

// Activation and store of a row's features n0 and n1 (gated: of the one feature that they are the gate and up part of).
__device__ __forceinline__ void store_plain(const NarrowOut& p, bool gated, int64_t row, int n0, int n1, float v0, float v1) {
    const int64_t at = row * p.y_pitch + n0;
    if (gated) {
        p.y[at] = __float2bfloat16_rn(activate_pair(p.epilogue, round_bf16(v0), round_bf16(v1), p.act_limit));
        return;
    }
    if (p.epilogue == B200_EPILOGUE_RELU2) {
        v0 = fmaxf(v0, 0.f) * fmaxf(v0, 0.f);
        v1 = fmaxf(v1, 0.f) * fmaxf(v1, 0.f);
    } else if (p.epilogue == B200_EPILOGUE_GELU_ERF) {
        v0 = 0.5f * v0 * (1.0f + erff(v0 * 0.70710678118654752f));
        v1 = 0.5f * v1 * (1.0f + erff(v1 * 0.70710678118654752f));
    }
    if (p.epilogue == B200_EPILOGUE_F32) {
        float* y = reinterpret_cast<float*>(p.y) + at;
        y[0] = v0;
        if (n1 < p.n_out) y[8] = v1;
        return;
    }
    p.y[at] = __float2bfloat16_rn(v0);
    if (n1 < p.n_out) p.y[at + 8] = __float2bfloat16_rn(v1);
}
}  // namespace b200

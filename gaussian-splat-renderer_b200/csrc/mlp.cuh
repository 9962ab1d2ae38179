// The learned colour stage (no reference counterpart): a per-gaussian 8-dim fp16 latent, encoded
// from the gaussian's 48 SH coefficients, and one small MLP that decodes (latent, view direction)
// to RGB in place of the SH evaluation.
//
//   encoder  48 -> 64 (ReLU) -> 8                      (training and latent encoding only)
//   decoder  (8 latent + 3 direction) -> 32 (ReLU) -> 32 (ReLU) -> 3 (sigmoid)
//
// The decoder runs inside the preprocess on the tensor cores: one warp decodes the colours of
// its 32 gaussians as three chained mma.sync.m16n8k16 BF16 products with FP32 accumulation (the
// accumulator fragment of one layer is, after ReLU and BF16 rounding, the A fragment of the
// next). The matrices are tiny (K <= 32, N <= 32), so the stage is bound by the latent reads,
// not by tensor throughput. A gaussian whose decoded colour is more than the gate away from its
// SH colour on the training directions keeps the SH path: its latent's last half is NaN.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstdint>

#include "kernels.cuh"

namespace gsr {

constexpr int kMlpIn = 11, kMlpHidden = 32, kMlpOut = 3, kMlpLatent = 8;
constexpr int kEncIn = 48, kEncHidden = 64;

// Parameter offsets (floats) in the fp32 master array (row-major W[in][out]).
struct MlpLayout {
    static constexpr int kEncW1 = 0;                                 // [48][64]
    static constexpr int kEncB1 = kEncW1 + kEncIn * kEncHidden;      // [64]
    static constexpr int kEncW2 = kEncB1 + kEncHidden;               // [64][8]
    static constexpr int kEncB2 = kEncW2 + kEncHidden * kMlpLatent;  // [8]
    static constexpr int kDecW1 = kEncB2 + kMlpLatent;               // [11][32]
    static constexpr int kDecB1 = kDecW1 + kMlpIn * kMlpHidden;      // [32]
    static constexpr int kDecW2 = kDecB1 + kMlpHidden;               // [32][32]
    static constexpr int kDecB2 = kDecW2 + kMlpHidden * kMlpHidden;  // [32]
    static constexpr int kDecW3 = kDecB2 + kMlpHidden;               // [32][3]
    static constexpr int kDecB3 = kDecW3 + kMlpHidden * kMlpOut;     // [3]
    static constexpr int kCount = kDecB3 + kMlpOut;                  // 5195
};

// The decoder for the tensor cores: each weight matrix transposed to [n][k] BF16 (k padded to a
// multiple of 16, n to a multiple of 8) so that a B fragment register is two consecutive k of
// one column; biases fp32, padded. Rows carry 8 more BF16, so that the eight rows (g) x four words (tig)
// of a fragment lie in 32 banks; see mlpDecodeWarp.
constexpr int kMlpPad = 8;
struct alignas(16) DecoderWeights {
    __nv_bfloat16 w1[32][16 + kMlpPad];  // [n][k], k = 0..10 used
    __nv_bfloat16 w2[32][32 + kMlpPad];
    __nv_bfloat16 w3[8][32 + kMlpPad];   // n = 0..2 used
    float b1[32], b2[32], b3[8];
};

static_assert(sizeof(DecoderWeights) == kDecoderWeightsBytes, "the host allocates kDecoderWeightsBytes");
static_assert(MlpLayout::kCount == int(kColorModelParams), "the host's parameter count");

__device__ __forceinline__ float bf16Round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

__device__ __forceinline__ uint32_t packBf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);  // .x = lo (low half), .y = hi
    return *reinterpret_cast<const uint32_t*>(&v);
}

__device__ __forceinline__ void mmaBf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ float sigmoidF(float x) { return 1.0f / (1.0f + __expf(-x)); }

// A staged row of 16 BF16 inputs; 48 bytes, so that the rows' 16-byte stores and the fragments' reads
// (eight rows, four words) meet every bank once.
struct alignas(16) MlpRow {
    union {
        uint4 q[3];
        uint32_t w[12];
    };
};

// Decodes the colours of the warp's 32 rows; all 32 lanes call it. feat = the lane's row
// (latent 8, direction 3), stage = this warp's 32 staged rows and out4 its 32 results in shared
// memory. Rows of lanes that need no colour may hold anything.
// Bound by shared memory where it is called back to back: unpadded rows, staged 16 bits at a time, took some
// 400 wavefronts a call, twice what they take now (the gate over 64 directions of 559,000 gaussians
// 1.5 -> 1.0 ms, the learned preprocess of 1.24 M at 1080p 152 -> 143 us). A weight fragment is read once for both
// halves of the warp's rows: 142 -> 136 us.
__device__ __forceinline__ void mlpDecodeWarp(const DecoderWeights& W, const float (&feat)[kMlpIn],
                                              MlpRow* stage, float4* out4, float (&rgb)[3]) {
    const uint32_t lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    uint32_t in[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
        in[k] = packBf16(2 * k < kMlpIn ? feat[2 * k < kMlpIn ? 2 * k : 0] : 0.0f,
                         2 * k + 1 < kMlpIn ? feat[2 * k + 1 < kMlpIn ? 2 * k + 1 : 0] : 0.0f);
    stage[lane].q[0] = make_uint4(in[0], in[1], in[2], in[3]);
    stage[lane].q[1] = make_uint4(in[4], in[5], in[6], in[7]);
    __syncwarp();
    uint32_t a[2][4];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
        const MlpRow &r0 = stage[mt * 16 + g], &r1 = stage[mt * 16 + g + 8];
        a[mt][0] = r0.w[tig];
        a[mt][1] = r1.w[tig];
        a[mt][2] = r0.w[tig + 4];
        a[mt][3] = r1.w[tig + 4];
    }
    // the next layer's A fragments from this one's accumulators
    auto activate = [](const float (&c)[2][4][4], uint32_t (&o)[2][2][4]) {
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int kb = 0; kb < 2; ++kb) {
                o[mt][kb][0] = packBf16(fmaxf(c[mt][2 * kb][0], 0.0f), fmaxf(c[mt][2 * kb][1], 0.0f));
                o[mt][kb][1] = packBf16(fmaxf(c[mt][2 * kb][2], 0.0f), fmaxf(c[mt][2 * kb][3], 0.0f));
                o[mt][kb][2] = packBf16(fmaxf(c[mt][2 * kb + 1][0], 0.0f), fmaxf(c[mt][2 * kb + 1][1], 0.0f));
                o[mt][kb][3] = packBf16(fmaxf(c[mt][2 * kb + 1][2], 0.0f), fmaxf(c[mt][2 * kb + 1][3], 0.0f));
            }
    };
    // layer 1: 16 -> 32 (a weight fragment serves both halves of the warp's rows)
    float c[2][4][4];
    uint32_t h[2][2][4];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
        const float2 b = *reinterpret_cast<const float2*>(&W.b1[nt * 8 + tig * 2]);
        const int n = nt * 8 + g;
        const uint32_t w0 = *reinterpret_cast<const uint32_t*>(&W.w1[n][tig * 2]);
        const uint32_t w1 = *reinterpret_cast<const uint32_t*>(&W.w1[n][tig * 2 + 8]);
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            c[mt][nt][0] = b.x; c[mt][nt][1] = b.y; c[mt][nt][2] = b.x; c[mt][nt][3] = b.y;
            mmaBf16(c[mt][nt], a[mt], w0, w1);
        }
    }
    activate(c, h);
    // layer 2: 32 -> 32
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
        const float2 b = *reinterpret_cast<const float2*>(&W.b2[nt * 8 + tig * 2]);
        const int n = nt * 8 + g;
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            c[mt][nt][0] = b.x; c[mt][nt][1] = b.y; c[mt][nt][2] = b.x; c[mt][nt][3] = b.y;
        }
#pragma unroll
        for (int kb = 0; kb < 2; ++kb) {
            const uint32_t w0 = *reinterpret_cast<const uint32_t*>(&W.w2[n][kb * 16 + tig * 2]);
            const uint32_t w1 = *reinterpret_cast<const uint32_t*>(&W.w2[n][kb * 16 + tig * 2 + 8]);
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) mmaBf16(c[mt][nt], h[mt][kb], w0, w1);
        }
    }
    activate(c, h);
    // layer 3: 32 -> 8 (3 used)
    const float2 b3 = *reinterpret_cast<const float2*>(&W.b3[tig * 2]);
    float c3[2][4] = {{b3.x, b3.y, b3.x, b3.y}, {b3.x, b3.y, b3.x, b3.y}};
#pragma unroll
    for (int kb = 0; kb < 2; ++kb) {
        const uint32_t w0 = *reinterpret_cast<const uint32_t*>(&W.w3[g][kb * 16 + tig * 2]);
        const uint32_t w1 = *reinterpret_cast<const uint32_t*>(&W.w3[g][kb * 16 + tig * 2 + 8]);
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) mmaBf16(c3[mt], h[mt][kb], w0, w1);
    }
    if (tig < 2) {
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            reinterpret_cast<float2*>(&out4[mt * 16 + g])[tig] = make_float2(c3[mt][0], c3[mt][1]);
            reinterpret_cast<float2*>(&out4[mt * 16 + g + 8])[tig] = make_float2(c3[mt][2], c3[mt][3]);
        }
    }
    __syncwarp();
    const float4 o = out4[lane];
    rgb[0] = sigmoidF(o.x);
    rgb[1] = sigmoidF(o.y);
    rgb[2] = sigmoidF(o.z);
    __syncwarp();  // the staging areas may be reused by the caller's next decode
}

// The fallback marker: a latent whose last half is NaN keeps the SH colour.
__device__ __forceinline__ bool latentIsFallback(const uint4& q) { return __hisnan(__ushort_as_half(uint16_t(q.w >> 16))); }

}  // namespace gsr

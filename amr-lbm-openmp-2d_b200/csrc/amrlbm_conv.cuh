// amrlbm_conv.cuh - the refine-flag forecaster's forward pass in shared
// memory, one CTA per sample: the fused forecast of the learned regrid
// (amrlbm_forecast.cu) and the network's own forward and gradient
// (amrlbm_net.cu) share it, so that their logits agree bit for bit. Device
// helpers with internal linkage: each translation unit gets its own copy.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "amrlbm_launch.h"

namespace {

constexpr int CH = 32, CIN = 4, TILE = 18, PIX = TILE * TILE;
constexpr int MTILES = (PIX + 15) / 16;  // 21 row tiles of 16 pixels
constexpr int K1P = 48, K2 = 9 * CH;     // layer 1 (36 padded to 48), layers 2 and 3
// shared row lengths (BF16) of the transposed weights W^T[n][k] and of the
// activations [pixel][channel]: chosen so that the 32 lanes of one fragment
// load hit 32 different banks
constexpr int KW1 = 72, KW2 = 328, AROW = 40;
constexpr int NT = 256, NWARP = NT / 32;

// weights, sample and activations of one CTA
struct ConvSmem {
    __nv_bfloat16 w1[CH][KW1];
    __nv_bfloat16 w2[CH][KW2];
    __nv_bfloat16 w3[CH][KW2];
    __nv_bfloat16 x0[PIX][CIN];  // the samples, channels last
    __nv_bfloat16 act[2][PIX][AROW];
    float b[3][CH], wd[CH], bd;
    float pmax[NWARP][CH];
    __align__(16) unsigned zero[4];  // the operand row outside the tile
};

__device__ __forceinline__ unsigned pack2(float lo, float hi) {
    return (unsigned)__bfloat16_as_ushort(__float2bfloat16(lo)) |
           ((unsigned)__bfloat16_as_ushort(__float2bfloat16(hi)) << 16);
}

// the im2col pair (k, k+1) of row `row` (k even, tap-major k = o*CI + ci):
// one 32-bit word of the activation (AW words per pixel), 0 outside
template <int CI, int AW>
__device__ __forceinline__ unsigned a_pair(const unsigned* act, int row, int k) {
    const int o = k / CI, ci = k % CI;
    if (o >= 9 || row >= PIX) return 0u;
    const int y = row / TILE + o / 3 - 1, x = row % TILE + o % 3 - 1;
    if (x < 0 || x >= TILE || y < 0 || y >= TILE) return 0u;
    return act[(y * TILE + x) * AW + (ci >> 1)];
}

// one row tile mt of a layer's product: acc[j][.] = columns 8j + 2q, +1 of
// rows 16mt + g (acc[j][0..1]) and 16mt + g + 8 (acc[j][2..3])
template <int CI, int AW, int K, int KW>
__device__ __forceinline__ void tile_product(const unsigned* act, const __nv_bfloat16 (*wt)[KW],
                                             int mt, int g, int q, float acc[4][4]) {
    const unsigned* w32 = reinterpret_cast<const unsigned*>(wt);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[j][i] = 0.f;
    const int r0 = 16 * mt + g, r1 = r0 + 8;
#pragma unroll 2
    for (int k0 = 0; k0 < K; k0 += 16) {
        const unsigned a0 = a_pair<CI, AW>(act, r0, k0 + 2 * q);
        const unsigned a1 = a_pair<CI, AW>(act, r1, k0 + 2 * q);
        const unsigned a2 = a_pair<CI, AW>(act, r0, k0 + 2 * q + 8);
        const unsigned a3 = a_pair<CI, AW>(act, r1, k0 + 2 * q + 8);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int nrow = (8 * j + g) * (KW / 2);
            const unsigned b0 = w32[nrow + ((k0 + 2 * q) >> 1)];
            const unsigned b1 = w32[nrow + ((k0 + 2 * q + 8) >> 1)];
            asm volatile(
                "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
                "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                : "+f"(acc[j][0]), "+f"(acc[j][1]), "+f"(acc[j][2]), "+f"(acc[j][3])
                : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
        }
    }
}

// ReLU(acc + bias) of one row tile as BF16 into an activation
__device__ __forceinline__ void store_tile(const float acc[4][4], const float* bias, unsigned* o32,
                                           int mt, int g, int q) {
    const int r0 = 16 * mt + g, r1 = r0 + 8;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int n = 8 * j + 2 * q;
        if (r0 < PIX)
            o32[r0 * (AROW / 2) + (n >> 1)] =
                pack2(fmaxf(acc[j][0] + bias[n], 0.f), fmaxf(acc[j][1] + bias[n + 1], 0.f));
        if (r1 < PIX)
            o32[r1 * (AROW / 2) + (n >> 1)] =
                pack2(fmaxf(acc[j][2] + bias[n], 0.f), fmaxf(acc[j][3] + bias[n + 1], 0.f));
    }
}

// the first layer (4 input channels: one 16-column step spans four taps):
// operands gathered pair by pair
__device__ __forceinline__ void first_layer(const unsigned* x0, const __nv_bfloat16 (*wt)[KW1],
                                            const float* bias, __nv_bfloat16 (*out)[AROW], int warp,
                                            int g, int q) {
    unsigned* o32 = reinterpret_cast<unsigned*>(out);
    for (int mt = warp; mt < MTILES; mt += NWARP) {
        float acc[4][4];
        tile_product<CIN, CIN / 2, K1P, KW1>(x0, wt, mt, g, q, acc);
        store_tile(acc, bias, o32, mt, g, q);
    }
}

__device__ __forceinline__ unsigned smem_addr(const void* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void ldsm4(unsigned addr, unsigned& r0, unsigned& r1, unsigned& r2,
                                      unsigned& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}

// a 32-channel layer: each 16-column step is one tap of 16 adjacent
// channels, so the operand fragments come by ldmatrix: A rows are the
// activation rows of the shifted pixels (a zero row outside the tile), B the
// transposed weights. The warp's row tiles mt = warp, warp + 8, warp + 16
// share each step's B fragments. Accumulated along K from the first column on,
// 16 at a time.
template <int KW>
__device__ __forceinline__ void conv32(const __nv_bfloat16 (*act)[AROW], const __nv_bfloat16 (*wt)[KW],
                                       unsigned zero_row, int warp, int lane, float acc[3][4][4]) {
    const int lr = lane & 15;
    int pix[3];
    unsigned vmask[3];  // bit o: tap o of this lane's row lies in the tile
#pragma unroll
    for (int u = 0; u < 3; ++u) {
        const int r = 16 * (warp + NWARP * u) + lr;
        pix[u] = r;
        vmask[u] = 0u;
        if (r < PIX) {
            const int y = r / TILE, x = r % TILE;
#pragma unroll
            for (int o = 0; o < 9; ++o) {
                const int yy = y + o / 3 - 1, xx = x + o % 3 - 1;
                if (yy >= 0 && yy < TILE && xx >= 0 && xx < TILE) vmask[u] |= 1u << o;
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[u][j][i] = 0.f;
    }
    const unsigned abase = smem_addr(&act[0][0]) + (unsigned)((lane >> 4) * 8 * 2);
    const unsigned bbase = smem_addr(&wt[(lane & 7) + ((lane >> 4) << 3)][((lane >> 3) & 1) * 8]);
    const bool third = warp + 2 * NWARP < MTILES;
#pragma unroll
    for (int c = 0; c < K2 / 16; ++c) {
        const int o = c >> 1, c0 = (c & 1) * 16;
        const int shift = (o / 3 - 1) * TILE + (o % 3 - 1);
        unsigned b[8];
        ldsm4(bbase + (unsigned)(c * 32), b[0], b[1], b[2], b[3]);                    // n 0..15
        ldsm4(bbase + (unsigned)(16 * KW * 2 + c * 32), b[4], b[5], b[6], b[7]);      // n 16..31
#pragma unroll
        for (int u = 0; u < 3; ++u) {
            if (u == 2 && !third) break;
            const unsigned addr = ((vmask[u] >> o) & 1u)
                                      ? abase + (unsigned)(((pix[u] + shift) * AROW + c0) * 2)
                                      : zero_row;
            unsigned a0, a1, a2, a3;
            ldsm4(addr, a0, a1, a2, a3);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                asm volatile(
                    "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
                    "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                    : "+f"(acc[u][j][0]), "+f"(acc[u][j][1]), "+f"(acc[u][j][2]), "+f"(acc[u][j][3])
                    : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b[2 * j]), "r"(b[2 * j + 1]));
        }
    }
}

// the weights, transposed (W^T[n][k]), and the biases into shared memory
__device__ __forceinline__ void load_weights(const ForecastNet& net, ConvSmem& S, int t) {
    auto put = [&](const void* w, auto& dst, int rows) {  // 8 columns of a row of W at a time
        const uint4* src = static_cast<const uint4*>(w);
        for (int i = t; i < rows * CH / 8; i += NT) {
            const uint4 v = __ldg(src + i);
            const unsigned u[4] = {v.x, v.y, v.z, v.w};
            const int k = i / (CH / 8), n = i % (CH / 8) * 8;
#pragma unroll
            for (int m = 0; m < 8; ++m)
                dst[n + m][k] = __ushort_as_bfloat16((unsigned short)(u[m / 2] >> (16 * (m & 1))));
        }
    };
    put(net.w1, S.w1, K1P);
    put(net.w2, S.w2, K2);
    put(net.w3, S.w3, K2);
    if (t < CH) {
        S.b[0][t] = net.b1[t];
        S.b[1][t] = net.b2[t];
        S.b[2][t] = net.b3[t];
        S.wd[t] = net.wd[t];
    }
    if (t == 0) S.bd = net.bd[0];
    if (t < 4) S.zero[t] = 0u;
}

// layers 1 and 2 of the sample in S.x0: activations in S.act[0] and S.act[1].
// Ends with a barrier.
__device__ __forceinline__ void two_layers(ConvSmem& S, unsigned zero_row, int warp, int lane) {
    const int g = lane >> 2, q = lane & 3;
    first_layer(reinterpret_cast<const unsigned*>(S.x0), S.w1, S.b[0], S.act[0], warp, g, q);
    __syncthreads();
    float acc[3][4][4];
    conv32<KW2>(S.act[0], S.w2, zero_row, warp, lane, acc);
#pragma unroll
    for (int u = 0; u < 3; ++u)
        if (warp + NWARP * u < MTILES)
            store_tile(acc[u], S.b[1], reinterpret_cast<unsigned*>(S.act[1]), warp + NWARP * u, g, q);
    __syncthreads();
}

}  // namespace

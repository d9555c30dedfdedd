// amrlbm_net.cu - the refine-flag forecaster of the learned regrid: a small
// convolutional network over one block with its ghost ring (4 channels on
// 18 x 18 cells for 16 x 16 blocks: C, |grad C| against the refine tolerance,
// Ux and Uy as cells moved over the forecast horizon), three 3x3 convolutions
// of 32 channels with ReLU, a global max pool and a dense output: the logit
// of "this block is flagged for refinement k steps from now". No counterpart
// in the reference, which flags blocks from the current field only
// (Err_Interface, Refine_Derefine.f90:327-351).
//
// Forward pass and gradient run one CTA per sample with everything of a
// sample in shared memory (k_net): the convolutions as implicit products on
// the tensor cores (mma.sync m16n8k16, BF16 operands, FP32 accumulation); the
// weight gradients are products over the rows it leaves in memory (k_dw).
// Weights are kept in FP32 (Adam) and rounded to BF16 for every product.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "amrlbm.h"
#include "amrlbm_conv.cuh"
#include "amrlbm_dev.cuh"
#include "amrlbm_launch.h"

namespace {

static_assert(CIN == AMRLBM_NET_CHANNELS && TILE == AMRLBM_NET_TILE, "sample layout");
constexpr int K1 = CIN * 9;
// FP32 parameter vector: W1 [K1][CH], b1, W2 [K2][CH], b2, W3 [K2][CH], b3, wd [CH], bd
constexpr int O_W1 = 0, O_B1 = O_W1 + K1 * CH, O_W2 = O_B1 + CH, O_B2 = O_W2 + K2 * CH,
              O_W3 = O_B2 + CH, O_B3 = O_W3 + K2 * CH, O_WD = O_B3 + CH, O_BD = O_WD + CH,
              NPARAM = O_BD + 1;

// ---- the plain tensor-core product, for amrlbm_net_selftest_gemm alone ---------
// (the network's own products are those of k_net and k_dw)
// C[M][N] (FP32, row stride ldc) = sum_k A(m, k) B(k, n), A(m, k) = A[m*sam + k*sak],
// B(k, n) = B[k*sbk + n*sbn], BF16. CTA: 4 warps, a 64 x 32 tile of C; each
// warp 16 rows x 4 n-tiles of 8. Operands go through shared memory with zero
// padding outside M, N, K.
constexpr int GM = 64, GN = 32, GK = 16;

__device__ __forceinline__ unsigned pack_bf16(__nv_bfloat16 lo, __nv_bfloat16 hi) {
    return (unsigned)__bfloat16_as_ushort(lo) | ((unsigned)__bfloat16_as_ushort(hi) << 16);
}

__global__ void __launch_bounds__(128) k_gemm(int M, int N, int K, const __nv_bfloat16* A,
                                              long long sam, long long sak,
                                              const __nv_bfloat16* B, long long sbk,
                                              long long sbn, float* C, long long ldc) {
    __shared__ __nv_bfloat16 sA[GM][GK + 2];
    __shared__ __nv_bfloat16 sB[GK][GN + 2];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5, g = lane >> 2, q = lane & 3;
    const int m0 = blockIdx.x * GM, n0 = blockIdx.y * GN;
    float acc[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[j][i] = 0.f;
    const __nv_bfloat16 zero = __float2bfloat16(0.f);
    for (int k0 = 0; k0 < K; k0 += GK) {
        for (int i = t; i < GM * GK; i += 128) {
            const int r = i / GK, c = i % GK, m = m0 + r, k = k0 + c;
            sA[r][c] = (m < M && k < K) ? A[(long long)m * sam + (long long)k * sak] : zero;
        }
        for (int i = t; i < GK * GN; i += 128) {
            const int r = i / GN, c = i % GN, k = k0 + r, n = n0 + c;
            sB[r][c] = (k < K && n < N) ? B[(long long)k * sbk + (long long)n * sbn] : zero;
        }
        __syncthreads();
        const int r = 16 * w;
        const unsigned a0 = pack_bf16(sA[r + g][2 * q], sA[r + g][2 * q + 1]);
        const unsigned a1 = pack_bf16(sA[r + g + 8][2 * q], sA[r + g + 8][2 * q + 1]);
        const unsigned a2 = pack_bf16(sA[r + g][2 * q + 8], sA[r + g][2 * q + 9]);
        const unsigned a3 = pack_bf16(sA[r + g + 8][2 * q + 8], sA[r + g + 8][2 * q + 9]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const unsigned b0 = pack_bf16(sB[2 * q][8 * j + g], sB[2 * q + 1][8 * j + g]);
            const unsigned b1 = pack_bf16(sB[2 * q + 8][8 * j + g], sB[2 * q + 9][8 * j + g]);
            asm volatile(
                "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
                "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                : "+f"(acc[j][0]), "+f"(acc[j][1]), "+f"(acc[j][2]), "+f"(acc[j][3])
                : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
        }
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int n = n0 + 8 * j + 2 * q;
        const int m = m0 + 16 * w + g;
        if (m < M) {
            if (n < N) C[(long long)m * ldc + n] = acc[j][0];
            if (n + 1 < N) C[(long long)m * ldc + n + 1] = acc[j][1];
        }
        if (m + 8 < M) {
            if (n < N) C[(long long)(m + 8) * ldc + n] = acc[j][2];
            if (n + 1 < N) C[(long long)(m + 8) * ldc + n + 1] = acc[j][3];
        }
    }
}

void gemm(cudaStream_t st, int M, int N, int K, const __nv_bfloat16* A, long long sam,
          long long sak, const __nv_bfloat16* B, long long sbk, long long sbn, float* C,
          long long ldc) {
    dim3 grid((M + GM - 1) / GM, (N + GN - 1) / GN);
    k_gemm<<<grid, 128, 0, st>>>(M, N, K, A, sam, sak, B, sbk, sbn, C, ldc);
    count_launches(1);
}

// ---- elementwise parts -------------------------------------------------------
inline int blocks_for(long long n) { return (int)std::min<long long>((n + 255) / 256, 8192); }
#define GRID_STRIDE(i, n) for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < (n); i += (long long)gridDim.x * blockDim.x)

// ---- forward pass and gradient, one CTA per sample ------------------------------
struct GradSmem {
    ConvSmem c;
    __nv_bfloat16 wb[2][CH][KW2];  // [layer 2 | 3][ci][o * CH + co] = W[o * CH + ci][co]
    __nv_bfloat16 dz[PIX][AROW];   // gradient of layer 3's pre-activations
    int parg[NWARP][CH], arg[CH];
    float dz3[CH];
};
// what a batch's weight gradients are formed from, BF16, rows = pixels of all
// samples: the inputs of the three layers and the gradients of their
// pre-activations
struct GradRows {
    __nv_bfloat16 *x0, *a1, *a2;        // [rows][CIN], [rows][CH] x 2
    __nv_bfloat16* dz[3];               // [rows][CH]
    float* df[3];                       // the same in FP32, for the bias gradients
    float *pooled, *dlogit;             // [samples][CH], [samples]
};

__device__ __forceinline__ void ldsm4t(unsigned addr, unsigned* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void mma16816(float* d, const unsigned* a, unsigned b0, unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
        "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// bit o: tap o of pixel p lies in the tile (0 for p outside it)
__device__ __forceinline__ unsigned tap_mask(int p) {
    if (p >= PIX) return 0u;
    const int y = p / TILE, x = p % TILE;
    const unsigned rows = (y > 0 ? 7u : 0u) | 7u << 3 | (y < TILE - 1 ? 7u << 6 : 0u);
    const unsigned cols = (x > 0 ? 0111u : 0u) | 0222u | (x < TILE - 1 ? 0444u : 0u);
    return rows & cols;
}
__device__ __forceinline__ int tap_shift(int o) { return (o / 3 - 1) * TILE + (o % 3 - 1); }

// The transposed convolution of dz with W (wb[ci][o * CH + co]): the product of
// each tap on its own, then their sum in tap order (acc), as a product with
// all of W^T followed by the sum over the taps forms it. Operands as conv32's.
__device__ __forceinline__ void conv32_back(const __nv_bfloat16 (*dz)[AROW], const __nv_bfloat16 (*wb)[KW2],
                                            unsigned zero_row, int warp, int lane, float acc[3][4][4]) {
    int pix[3];
    unsigned vmask[3];
#pragma unroll
    for (int u = 0; u < 3; ++u) {
        pix[u] = 16 * (warp + NWARP * u) + (lane & 15);
        vmask[u] = tap_mask(pix[u]);
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[u][j][i] = 0.f;
    }
    const unsigned abase = smem_addr(&dz[0][0]) + (unsigned)((lane >> 4) * 8 * 2);
    const unsigned bbase = smem_addr(&wb[(lane & 7) + ((lane >> 4) << 3)][((lane >> 3) & 1) * 8]);
    const bool third = warp + 2 * NWARP < MTILES;
#pragma unroll 1
    for (int o = 0; o < 9; ++o) {
        unsigned b[2][8];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const unsigned at = bbase + (unsigned)((o * CH + 16 * c) * 2);
            ldsm4(at, b[c][0], b[c][1], b[c][2], b[c][3]);
            ldsm4(at + (unsigned)(16 * KW2 * 2), b[c][4], b[c][5], b[c][6], b[c][7]);
        }
        const int shift = tap_shift(8 - o);  // pixel p - tap o
#pragma unroll
        for (int u = 0; u < 3; ++u) {
            if (u == 2 && !third) break;
            const bool in = (vmask[u] >> (8 - o)) & 1u;
            float s[4][4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) s[j][i] = 0.f;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                unsigned a[4];
                ldsm4(in ? abase + (unsigned)(((pix[u] + shift) * AROW + 16 * c) * 2) : zero_row, a[0], a[1],
                      a[2], a[3]);
#pragma unroll
                for (int j = 0; j < 4; ++j) mma16816(s[j], a, b[c][2 * j], b[c][2 * j + 1]);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[u][j][i] = acc[u][j][i] + s[j][i];
        }
    }
}

// Logits of samples x [n][CIN][TILE][TILE]; with GRAD also the loss terms and
// the rows that the gradients are summed from (k_dw, k_head_back).
// The gradients equal, bit for bit, those of the plain sequence of products and
// elementwise kernels that this replaced (im2col, product, bias and ReLU;
// backwards product, col2im): the same operands in the same order.
// What bounds it: the mma.sync of a sample (3,276 forward, 6,300 with the
// gradient) and the ldmatrix that feed them, 8 warps per CTA; one CTA per SM
// for the gradient (175 KB of shared memory), two for the forward pass. The
// im2col matrices of that sequence, 191 MB per layer for 512 samples, took
// 1.7 ms per gradient.
template <bool GRAD>
__global__ void __launch_bounds__(NT, GRAD ? 1 : 2)
    k_net(const ForecastNet net, int n, const float* x, const float* y, float posw, float* logits,
          float* lterm, GradRows rows) {
    extern __shared__ __align__(16) unsigned char smraw[];
    GradSmem& B = *reinterpret_cast<GradSmem*>(smraw);
    ConvSmem& S = B.c;  // the forward pass has no more than this
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, g = lane >> 2, q = lane & 3;
    load_weights(net, S, t);
    __syncthreads();
    if (GRAD)
        for (int i = t; i < K2 * CH; i += NT) {
            const int ci = i / K2, k = i % K2, o = k / CH, co = k % CH;
            B.wb[0][ci][k] = S.w2[co][o * CH + ci];
            B.wb[1][ci][k] = S.w3[co][o * CH + ci];
        }
    const unsigned zero_row = smem_addr(S.zero);
    // rows of an activation to memory
    auto put_rows = [&](const __nv_bfloat16 (*src)[AROW], __nv_bfloat16* dst) {
        for (int i = t; i < PIX * (CH / 8); i += NT)
            reinterpret_cast<uint4*>(dst)[i] =
                *reinterpret_cast<const uint4*>(&src[i / (CH / 8)][i % (CH / 8) * 8]);
    };
    for (int b = blockIdx.x; b < n; b += gridDim.x) {
        __syncthreads();  // the previous sample's buffers have been read
        const float* xb = x + (size_t)b * CIN * PIX;
        for (int p = t; p < PIX; p += NT) {
            unsigned* x32 = reinterpret_cast<unsigned*>(&S.x0[p][0]);
            x32[0] = pack2(__ldg(xb + p), __ldg(xb + PIX + p));
            x32[1] = pack2(__ldg(xb + 2 * PIX + p), __ldg(xb + 3 * PIX + p));
        }
        __syncthreads();
        two_layers(S, zero_row, warp, lane);
        // layer 3 reduced to the channel maxima and the first pixel of each
        float mx[4][2];
        int am[4][2];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                mx[j][h] = -1.f;
                am[j][h] = 0;
            }
        {
            float acc[3][4][4];
            conv32<KW2>(S.act[1], S.w3, zero_row, warp, lane, acc);
#pragma unroll
            for (int u = 0; u < 3; ++u) {
                const int mt = warp + NWARP * u;
                if (mt >= MTILES) continue;
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int p = 16 * mt + g + 8 * r;
                    if (p >= PIX) continue;
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const float v = fmaxf(acc[u][j][2 * r + h] + S.b[2][8 * j + 2 * q + h], 0.f);
                            if (v > mx[j][h]) {
                                mx[j][h] = v;
                                am[j][h] = p;
                            }
                        }
                }
            }
        }
        // across the lanes of a column, then the warps: ties to the lower pixel
        auto take = [](float& m, int& a, float m2, int a2) {
            if (m2 > m || (m2 == m && a2 < a)) {
                m = m2;
                a = a2;
            }
        };
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) {
                    const float m2 = __shfl_xor_sync(0xffffffffu, mx[j][h], o);
                    const int a2 = __shfl_xor_sync(0xffffffffu, am[j][h], o);
                    take(mx[j][h], am[j][h], m2, a2);
                }
        if (g == 0)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    S.pmax[warp][8 * j + 2 * q + h] = mx[j][h];
                    if (GRAD) B.parg[warp][8 * j + 2 * q + h] = am[j][h];
                }
        __syncthreads();
        if (warp == 0) {
            float p = S.pmax[0][lane];
            int a = GRAD ? B.parg[0][lane] : 0;
            for (int w = 1; w < NWARP; ++w) {
                if (GRAD)
                    take(p, a, S.pmax[w][lane], B.parg[w][lane]);
                else
                    p = fmaxf(p, S.pmax[w][lane]);
            }
            // the dense output, in channel order
            float z = S.bd;
            for (int c = 0; c < CH; ++c) z += S.wd[c] * __shfl_sync(0xffffffffu, p, c);
            if (lane == 0) logits[b] = z;
            if (GRAD) {
                // weighted binary cross-entropy on the logit:
                // log(1 + exp(-|z|)) + max(z, 0) - z y
                const float yy = y[b], wt = yy > 0.5f ? posw : 1.f;
                const float dl = wt * (1.f / (1.f + expf(-z)) - yy) / (float)n;
                if (lane == 0) lterm[b] = wt * (log1pf(expf(-fabsf(z))) + fmaxf(z, 0.f) - z * yy);
                const float d3 = p > 0.f ? dl * S.wd[lane] : 0.f;  // at the maximum alone
                rows.pooled[(size_t)b * CH + lane] = p;
                if (lane == 0) rows.dlogit[b] = dl;
                B.dz3[lane] = d3;
                B.arg[lane] = a;
            }
        }
        if constexpr (GRAD) {
        const size_t row0 = (size_t)b * PIX;
        put_rows(S.act[0], rows.a1 + row0 * CH);
        put_rows(S.act[1], rows.a2 + row0 * CH);
        for (int i = t; i < PIX; i += NT)
            reinterpret_cast<uint2*>(rows.x0 + row0 * CIN)[i] = *reinterpret_cast<const uint2*>(&S.x0[i][0]);
        __syncthreads();
        // layer 3: the maxima's pixels alone
        for (int p = warp; p < PIX; p += NWARP) {
            const float v = B.arg[lane] == p ? B.dz3[lane] : 0.f;
            B.dz[p][lane] = __float2bfloat16(v);
            rows.df[2][(row0 + p) * CH + lane] = v;
        }
        __syncthreads();
        put_rows(B.dz, rows.dz[2] + row0 * CH);
        // layer 2, then layer 1: the transposed convolution of the layer
        // above, through the ReLU, in FP32 to memory and as BF16 over the
        // activation (each value read by its writer alone)
        auto back = [&](const __nv_bfloat16 (*dz)[AROW], const __nv_bfloat16 (*wb)[KW2],
                        __nv_bfloat16 (*act)[AROW], float* df) {
            float acc[3][4][4];
            conv32_back(dz, wb, zero_row, warp, lane, acc);
#pragma unroll
            for (int u = 0; u < 3; ++u) {
                const int mt = warp + NWARP * u;
                if (mt >= MTILES) continue;
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int p = 16 * mt + g + 8 * r;
                    if (p >= PIX) continue;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int c = 8 * j + 2 * q;
                        unsigned* a32 = reinterpret_cast<unsigned*>(&act[p][c]);
                        const unsigned w = *a32;
                        float2 v;
                        v.x = __uint_as_float(w << 16) > 0.f ? acc[u][j][2 * r] : 0.f;
                        v.y = __uint_as_float(w & 0xffff0000u) > 0.f ? acc[u][j][2 * r + 1] : 0.f;
                        *a32 = pack2(v.x, v.y);
                        *reinterpret_cast<float2*>(df + (row0 + p) * CH + c) = v;
                    }
                }
            }
            __syncthreads();
        };
        back(B.dz, B.wb[1], S.act[1], rows.df[1]);
        put_rows(S.act[1], rows.dz[1] + row0 * CH);
        back(S.act[1], B.wb[0], S.act[0], rows.df[0]);
        put_rows(S.act[0], rows.dz[0] + row0 * CH);
        }
    }
}

// Bias gradients: column sums of df [rows][CH]. 256 partial sums per column, of
// the rows t, t + 256, ..., then a binary tree over them. colsum forms 4 of
// the partial sums of one layer, coalesced, in CTAs of k_dw's launch beside the
// products, which leave half of the SMs idle; k_head_back forms the trees.
constexpr int NPART = 256;
__device__ __forceinline__ void colsum(unsigned rows, const GradRows& R, int job, float* part) {
    const int c = threadIdx.x % CH, l = job / (NPART / 4), t = job % (NPART / 4) * 4 + threadIdx.x / CH;
    if (threadIdx.x >= 4 * CH) return;
    const float* dz = l == 0 ? R.df[0] : l == 1 ? R.df[1] : R.df[2];
    float s = 0.f;
#pragma unroll 16
    for (unsigned r = t; r < rows; r += NPART) s += dz[(size_t)r * CH + c];
    part[((size_t)l * CH + c) * NPART + t] = s;
}
// CTAs 0..95: the tree of one layer's channel; CTA 96: the dense layer's
// gradient, the samples in order
__global__ void __launch_bounds__(NPART) k_head_back(int n, const GradRows R, const float* part, float* grad) {
    __shared__ float sh[NPART * (CH + 1)];
    const int t = threadIdx.x, col = blockIdx.x;
    if (col < 3 * CH) {
        sh[t] = part[(size_t)col * NPART + t];
        __syncthreads();
        for (int o = NPART / 2; o > 0; o >>= 1) {
            if (t < o) sh[t] += sh[t + o];
            __syncthreads();
        }
        const int off[3] = {O_B1, O_B2, O_B3};
        if (t == 0) grad[off[col / CH] + col % CH] = sh[0];
        return;
    }
    float s = 0.f;
    for (int b0 = 0; b0 < n; b0 += NPART) {
        const int cnt = min(NPART, n - b0);
        for (int i = t; i < cnt * CH; i += NPART) sh[i / CH * (CH + 1) + i % CH] = R.pooled[(size_t)b0 * CH + i];
        for (int i = t; i < cnt; i += NPART) sh[i * (CH + 1) + CH] = R.dlogit[b0 + i];
        __syncthreads();
        if (t <= CH)
            for (int b = 0; b < cnt; ++b)
                s += sh[b * (CH + 1) + CH] * (t < CH ? sh[b * (CH + 1) + t] : 1.f);
        __syncthreads();
    }
    if (t <= CH) grad[O_WD + t] = s;
}

// ---- weight gradients -------------------------------------------------------------
// dW[o * cin + ci][co] = sum over the rows r (pixels of all samples, in order)
// of in[r + tap o][ci] dz[r][co]: 16 rows per mma.sync, one accumulation chain
// per output over all rows, as the plain product of the two matrices forms it
// (the chain's order is kept: the tensor core truncates as it accumulates, and
// training multiplies a change of the sum some hundredfold over ten steps).
// A job is 16 x 16 outputs (two warps, a chain each); 36 jobs each for layers 3
// and 2 (tap, half of the inputs, half of the outputs) and 6 for layer 1 (four
// taps of the 4 inputs), one CTA each: warps 2-4 copy rows with cp.async into
// a ring of stages, warps 0-1 multiply. Bound by the chain, 10,368 dependent
// mma.sync for 512 samples. The generic product kernel loaded its operands
// element by element between the steps of the chain: 30.8 ms per layer; all
// three take 0.37 ms together.
constexpr int DW_ROWS = 192, DW_STAGES = 6, DW_PITCH = 24;  // row pitch 48 bytes: no bank conflicts
constexpr int DW_JOBS = 78, DW_THREADS = 160;
struct DwSmem {
    __nv_bfloat16 a[DW_STAGES][DW_ROWS][DW_PITCH], b[DW_STAGES][DW_ROWS][DW_PITCH];
};
// BYTES from src, or zeros
template <int BYTES>
__device__ __forceinline__ void cp_async_or_zero(void* dst, const void* src, bool ok) {
    if (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src),
                     "r"(ok ? 16 : 0)
                     : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_addr(dst)), "l"(src),
                     "r"(ok ? 8 : 0)
                     : "memory");
}
__global__ void __launch_bounds__(DW_THREADS) k_dw(int n, const GradRows R, float* g, float* part) {
    extern __shared__ __align__(16) unsigned char smraw[];
    DwSmem& S = *reinterpret_cast<DwSmem*>(smraw);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const unsigned rows = (unsigned)n * PIX;
    if (blockIdx.x >= DW_JOBS) return colsum(rows, R, blockIdx.x - DW_JOBS, part);
    const int job = blockIdx.x, layer = job < 36 ? 3 : (job < 72 ? 2 : 1);
    const int jj = layer == 3 ? job : (layer == 2 ? job - 36 : job - 72);
    const int nh = jj & 1, ch = (jj >> 1) & 1, o = layer == 1 ? jj >> 1 : jj >> 2;  // o: tap, or row tile
    const __nv_bfloat16* in = layer == 3 ? R.a2 : R.a1;
    const __nv_bfloat16* dz = (layer == 3 ? R.dz[2] : layer == 2 ? R.dz[1] : R.dz[0]) + 16 * nh;
    const int stages = (int)((rows + DW_ROWS - 1) / DW_ROWS);
    auto load = [&](int s) {  // warps 2-4: rows of stage s
        const int buf = s % DW_STAGES;
#pragma unroll
        for (int i = t - 64; i < DW_ROWS; i += 96) {
            const unsigned r = (unsigned)(s * DW_ROWS + i);
            const bool ok = r < rows;
            const unsigned taps = ok ? tap_mask((int)(r % PIX)) : 0u;
            const __nv_bfloat16* bs = dz + (size_t)(ok ? r : 0u) * CH;
            cp_async_or_zero<16>(&S.b[buf][i][0], bs, ok);
            cp_async_or_zero<16>(&S.b[buf][i][8], bs + 8, ok);
            if (layer > 1) {
                const bool in_tile = (taps >> o) & 1u;
                const __nv_bfloat16* as = in + (size_t)(in_tile ? r + tap_shift(o) : 0u) * CH + 16 * ch;
                cp_async_or_zero<16>(&S.a[buf][i][0], as, in_tile);
                cp_async_or_zero<16>(&S.a[buf][i][8], as + 8, in_tile);
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int oo = 4 * o + k;
                    const bool in_tile = oo < 9 && ((taps >> oo) & 1u);
                    cp_async_or_zero<8>(&S.a[buf][i][4 * k],
                                        R.x0 + (size_t)(in_tile ? r + tap_shift(oo) : 0u) * CIN, in_tile);
                }
            }
        }
    };
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    if (warp > 1)
        for (int s = 0; s < DW_STAGES - 1; ++s) {
            if (s < stages) load(s);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
    // the lane's row and column of a warp's operand tiles (ldmatrix.trans):
    // 16 rows of 16 inputs, 32 rows (two steps) of 8 outputs
    const unsigned arow = (unsigned)(((lane & 7) + ((lane >> 4) << 3)) * DW_PITCH + ((lane >> 3) & 1) * 8) * 2u;
    const unsigned brow = (unsigned)(lane * DW_PITCH + (warp & 1) * 8) * 2u;
    for (int s = 0; s < stages; ++s) {
        if (warp > 1) asm volatile("cp.async.wait_group %0;" ::"n"(DW_STAGES - 2) : "memory");
        __syncthreads();  // stage s has landed, stage s - 1 has been read
        if (warp > 1) {
            if (s + DW_STAGES - 1 < stages) load(s + DW_STAGES - 1);
            asm volatile("cp.async.commit_group;" ::: "memory");
            continue;
        }
        const unsigned abase = smem_addr(&S.a[s % DW_STAGES][0][0]) + arow;
        const unsigned bbase = smem_addr(&S.b[s % DW_STAGES][0][0]) + brow;
        // the operands of two steps ahead of the products, whose chain then
        // waits for itself alone
        unsigned a[2][2][4], b[2][4];
        auto fetch = [&](int k) {  // steps k, k + 1
            const int m = (k / 2) % 2;
            ldsm4t(abase + (unsigned)(k * 16 * DW_PITCH * 2), a[m][0]);
            ldsm4t(abase + (unsigned)((k + 1) * 16 * DW_PITCH * 2), a[m][1]);
            ldsm4t(bbase + (unsigned)(k * 16 * DW_PITCH * 2), b[m]);
        };
        fetch(0);
#pragma unroll
        for (int k = 0; k < DW_ROWS / 16; k += 2) {
            const int m = (k / 2) % 2;
            if (k + 2 < DW_ROWS / 16) fetch(k + 2);
            mma16816(acc, a[m][0], b[m][0], b[m][1]);
            mma16816(acc, a[m][1], b[m][2], b[m][3]);
        }
    }
    if (warp > 1) return;
    const int k0 = layer == 1 ? 16 * o : o * CH + 16 * ch, kk = layer == 1 ? K1 : K2;
    float* out = g + (layer == 3 ? O_W3 : layer == 2 ? O_W2 : O_W1) + 16 * nh + 8 * warp;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int k = k0 + (lane >> 2) + 8 * (i >> 1);
        if (k < kk) out[k * CH + 2 * (lane & 3) + (i & 1)] = acc[i];
    }
}
// Adam on the FP32 parameters
__global__ void k_adam(int np, float* p, const float* g, float* m1, float* m2, float lr, float b1,
                       float b2, float eps, float c1, float c2) {
    GRID_STRIDE(i, np) {
        const float gi = g[i];
        m1[i] = b1 * m1[i] + (1.f - b1) * gi;
        m2[i] = b2 * m2[i] + (1.f - b2) * gi * gi;
        p[i] -= lr * (m1[i] / c1) / (sqrtf(m2[i] / c2) + eps);
    }
}
// BF16 weight matrices for the products: W1 padded to K1P rows
__global__ void k_pack(const float* p, __nv_bfloat16* w1, __nv_bfloat16* w2, __nv_bfloat16* w3) {
    GRID_STRIDE(i, (long long)K1P * CH) {
        const int k = (int)(i / CH);
        w1[i] = __float2bfloat16(k < K1 ? p[O_W1 + i] : 0.f);
    }
    GRID_STRIDE(i, (long long)K2 * CH) {
        w2[i] = __float2bfloat16(p[O_W2 + i]);
        w3[i] = __float2bfloat16(p[O_W3 + i]);
    }
}

// deterministic normal draws for the initial weights (splitmix64 + Box-Muller)
struct Rng {
    uint64_t s;
    uint64_t next() {
        uint64_t z = (s += 0x9e3779b97f4a7c15ull);
        z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
        z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
        return z ^ (z >> 31);
    }
    double uniform() { return ((next() >> 11) + 0.5) * (1.0 / 9007199254740992.0); }
    double normal() { return std::sqrt(-2.0 * std::log(uniform())) * std::cos(6.283185307179586 * uniform()); }
};

}  // namespace

struct amrlbm_net {
    int max_n = 0;
    cudaStream_t st = nullptr;
    std::vector<void*> allocs;
    float *p = nullptr, *g = nullptr, *m1 = nullptr, *m2 = nullptr;  // [NPARAM]
    __nv_bfloat16 *w1 = nullptr, *w2 = nullptr, *w3 = nullptr;
    // a batch's samples and labels, logits and loss terms; partial bias sums
    float *x = nullptr, *y = nullptr, *logits = nullptr, *lterm = nullptr, *part = nullptr;
    GradRows rows{};
    int num_sms = 0;
    int steps = 0;
    std::string err;
};

namespace {

template <class T>
T* nalloc(amrlbm_net* net, size_t n, cudaError_t* e) {
    void* q = nullptr;
    if (*e == cudaSuccess) *e = cudaMalloc(&q, n * sizeof(T));
    if (*e == cudaSuccess) {
        cudaMemset(q, 0, n * sizeof(T));
        net->allocs.push_back(q);
    }
    return (T*)q;
}

void repack(amrlbm_net* net) {
    k_pack<<<blocks_for((long long)K2 * CH), 256, 0, net->st>>>(net->p, net->w1, net->w2, net->w3);
    count_launches(1);
}

ForecastNet weights_of(const amrlbm_net* net) {
    ForecastNet f;
    f.w1 = net->w1;
    f.w2 = net->w2;
    f.w3 = net->w3;
    f.b1 = net->p + O_B1;
    f.b2 = net->p + O_B2;
    f.b3 = net->p + O_B3;
    f.wd = net->p + O_WD;
    f.bd = net->p + O_BD;
    return f;
}

// logits of n samples x (device memory)
void forward(amrlbm_net* net, int n, const float* x) {
    const int grid = std::min(n, 2 * net->num_sms);
    k_net<false><<<grid, NT, sizeof(ConvSmem), net->st>>>(weights_of(net), n, x, nullptr, 1.f,
                                                           net->logits, nullptr, net->rows);
    count_launches(1);
}

// logits, loss terms and gradient (net->g) of the n samples of the batch
void gradient(amrlbm_net* net, int n, float pos_weight) {
    const int grid = std::min(n, net->num_sms);
    k_net<true><<<grid, NT, sizeof(GradSmem), net->st>>>(weights_of(net), n, net->x, net->y, pos_weight,
                                                          net->logits, net->lterm, net->rows);
    k_dw<<<DW_JOBS + 3 * NPART / 4, DW_THREADS, sizeof(DwSmem), net->st>>>(n, net->rows, net->g, net->part);
    k_head_back<<<3 * CH + 1, NPART, 0, net->st>>>(n, net->rows, net->part, net->g);
    count_launches(3);
}

int net_fail(amrlbm_net* net, int code, const std::string& m) {
    if (net) net->err = m;
    return code;
}
#define NCK(call)                                                                    \
    do {                                                                             \
        cudaError_t e_ = (call);                                                     \
        if (e_ != cudaSuccess) return net_fail(net, AMRLBM_ERR_CUDA, cudaGetErrorString(e_)); \
    } while (0)

int load_batch(amrlbm_net* net, int n, const float* x, const float* y) {
    if (n < 1 || n > net->max_n || !x) return AMRLBM_ERR_ARG;
    NCK(cudaMemcpyAsync(net->x, x, sizeof(float) * (size_t)n * CIN * PIX, cudaMemcpyHostToDevice, net->st));
    if (y) NCK(cudaMemcpyAsync(net->y, y, sizeof(float) * (size_t)n, cudaMemcpyHostToDevice, net->st));
    return AMRLBM_OK;
}

}  // namespace

ForecastNet net_forecast_params(const amrlbm_net* net) { return weights_of(net); }

extern "C" {

int amrlbm_net_create(uint64_t seed, int32_t max_batch, amrlbm_net** out) {
    if (!out || max_batch < 1) return AMRLBM_ERR_ARG;
    *out = nullptr;
    int dev = 0, cc = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return AMRLBM_ERR_CUDA;
    cudaDeviceGetAttribute(&cc, cudaDevAttrComputeCapabilityMajor, dev);
    if (cc != 10) return AMRLBM_ERR_CUDA;
    amrlbm_net* net = new amrlbm_net();
    net->max_n = max_batch;
    cudaError_t e = cudaStreamCreateWithFlags(&net->st, cudaStreamNonBlocking);
    const size_t n = (size_t)max_batch;
    cudaDeviceGetAttribute(&net->num_sms, cudaDevAttrMultiProcessorCount, dev);
    net->p = nalloc<float>(net, NPARAM, &e);
    net->g = nalloc<float>(net, NPARAM, &e);
    net->m1 = nalloc<float>(net, NPARAM, &e);
    net->m2 = nalloc<float>(net, NPARAM, &e);
    net->w1 = nalloc<__nv_bfloat16>(net, (size_t)K1P * CH, &e);
    net->w2 = nalloc<__nv_bfloat16>(net, (size_t)K2 * CH, &e);
    net->w3 = nalloc<__nv_bfloat16>(net, (size_t)K2 * CH, &e);
    net->x = nalloc<float>(net, n * CIN * PIX, &e);
    net->y = nalloc<float>(net, n, &e);
    net->logits = nalloc<float>(net, n, &e);
    net->lterm = nalloc<float>(net, n, &e);
    net->part = nalloc<float>(net, 3 * CH * (size_t)NPART, &e);
    net->rows.x0 = nalloc<__nv_bfloat16>(net, n * PIX * CIN, &e);
    net->rows.a1 = nalloc<__nv_bfloat16>(net, n * PIX * CH, &e);
    net->rows.a2 = nalloc<__nv_bfloat16>(net, n * PIX * CH, &e);
    for (int l = 0; l < 3; ++l) {
        net->rows.dz[l] = nalloc<__nv_bfloat16>(net, n * PIX * CH, &e);
        net->rows.df[l] = nalloc<float>(net, n * PIX * CH, &e);
    }
    net->rows.pooled = nalloc<float>(net, n * CH, &e);
    net->rows.dlogit = nalloc<float>(net, n, &e);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_net<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(ConvSmem));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_net<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(GradSmem));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_dw, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DwSmem));
    if (e != cudaSuccess) {
        amrlbm_net_destroy(net);
        return AMRLBM_ERR_CUDA;
    }
    // He-normal weights, zero biases
    std::vector<float> p(NPARAM, 0.f);
    Rng r{seed};
    auto fill = [&](int off, int count, int fan_in) {
        const double s = std::sqrt(2.0 / fan_in);
        for (int i = 0; i < count; ++i) p[off + i] = (float)(s * r.normal());
    };
    fill(O_W1, K1 * CH, K1);
    fill(O_W2, K2 * CH, K2);
    fill(O_W3, K2 * CH, K2);
    fill(O_WD, CH, CH);
    *out = net;
    return amrlbm_net_set(net, p.data());
}

int amrlbm_net_destroy(amrlbm_net* net) {
    if (!net) return AMRLBM_OK;
    if (net->st) cudaStreamSynchronize(net->st);
    for (void* q : net->allocs) cudaFree(q);
    if (net->st) cudaStreamDestroy(net->st);
    delete net;
    return AMRLBM_OK;
}

int32_t amrlbm_net_param_count(void) { return NPARAM; }

const char* amrlbm_net_last_error(const amrlbm_net* net) { return net ? net->err.c_str() : "no net"; }

int amrlbm_net_get(amrlbm_net* net, float* params) {
    if (!net || !params) return AMRLBM_ERR_ARG;
    NCK(cudaMemcpyAsync(params, net->p, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost, net->st));
    NCK(cudaStreamSynchronize(net->st));
    return AMRLBM_OK;
}

int amrlbm_net_set(amrlbm_net* net, const float* params) {
    if (!net || !params) return AMRLBM_ERR_ARG;
    NCK(cudaMemcpyAsync(net->p, params, sizeof(float) * NPARAM, cudaMemcpyHostToDevice, net->st));
    NCK(cudaMemsetAsync(net->m1, 0, sizeof(float) * NPARAM, net->st));
    NCK(cudaMemsetAsync(net->m2, 0, sizeof(float) * NPARAM, net->st));
    net->steps = 0;
    repack(net);
    NCK(cudaStreamSynchronize(net->st));
    return AMRLBM_OK;
}

int amrlbm_net_forward(amrlbm_net* net, int32_t n, const float* x, float* logits) {
    if (!net || !logits) return AMRLBM_ERR_ARG;
    if (int r = load_batch(net, n, x, nullptr)) return r;
    forward(net, n, net->x);
    NCK(cudaMemcpyAsync(logits, net->logits, sizeof(float) * n, cudaMemcpyDeviceToHost, net->st));
    NCK(cudaStreamSynchronize(net->st));
    return AMRLBM_OK;
}

// forward of samples already in device memory (the learned regrid's
// features), logits to the host; n may exceed the batch capacity
int amrlbm_net_forward_device(amrlbm_net* net, int32_t n, const float* x_dev, float* logits) {
    if (!net || !logits || n < 0 || (n > 0 && !x_dev)) return AMRLBM_ERR_ARG;
    const size_t per = (size_t)CIN * PIX;
    for (int i0 = 0; i0 < n; i0 += net->max_n) {
        const int b = std::min(net->max_n, n - i0);
        forward(net, b, x_dev + per * i0);
        NCK(cudaMemcpyAsync(logits + i0, net->logits, sizeof(float) * b, cudaMemcpyDeviceToHost, net->st));
    }
    NCK(cudaStreamSynchronize(net->st));
    return AMRLBM_OK;
}

int amrlbm_net_gradient(amrlbm_net* net, int32_t n, const float* x, const float* y,
                        float pos_weight, float* loss, float* grad) {
    if (!net || !y || !loss) return AMRLBM_ERR_ARG;
    if (int r = load_batch(net, n, x, y)) return r;
    gradient(net, n, pos_weight);
    std::vector<float> lt(n);
    NCK(cudaMemcpyAsync(lt.data(), net->lterm, sizeof(float) * n, cudaMemcpyDeviceToHost, net->st));
    if (grad) NCK(cudaMemcpyAsync(grad, net->g, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost, net->st));
    NCK(cudaStreamSynchronize(net->st));
    double s = 0.0;
    for (float v : lt) s += v;
    *loss = (float)(s / n);
    return AMRLBM_OK;
}

int amrlbm_net_train_step(amrlbm_net* net, int32_t n, const float* x, const float* y,
                          float pos_weight, float lr, float* loss) {
    if (int r = amrlbm_net_gradient(net, n, x, y, pos_weight, loss, nullptr)) return r;
    net->steps += 1;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)net->steps), c2 = 1.f - std::pow(b2, (float)net->steps);
    k_adam<<<blocks_for(NPARAM), 256, 0, net->st>>>(NPARAM, net->p, net->g, net->m1, net->m2, lr, b1,
                                                    b2, 1e-8f, c1, c2);
    count_launches(1);
    repack(net);
    NCK(cudaStreamSynchronize(net->st));
    return AMRLBM_OK;
}

// the tensor-core product on its own, for its test: C = A B, A [M][K], B [K][N]
// (BF16 row-major on the host), C [M][N] FP32
int amrlbm_net_selftest_gemm(int32_t M, int32_t N, int32_t K, const uint16_t* A, const uint16_t* B,
                             float* C) {
    if (M < 1 || N < 1 || K < 1 || !A || !B || !C) return AMRLBM_ERR_ARG;
    __nv_bfloat16 *dA = nullptr, *dB = nullptr;
    float* dC = nullptr;
    cudaError_t e = cudaMalloc(&dA, sizeof(uint16_t) * (size_t)M * K);
    if (e == cudaSuccess) e = cudaMalloc(&dB, sizeof(uint16_t) * (size_t)K * N);
    if (e == cudaSuccess) e = cudaMalloc(&dC, sizeof(float) * (size_t)M * N);
    if (e == cudaSuccess) e = cudaMemcpy(dA, A, sizeof(uint16_t) * (size_t)M * K, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(dB, B, sizeof(uint16_t) * (size_t)K * N, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        gemm(nullptr, M, N, K, dA, K, 1, dB, N, 1, dC, N);
        e = cudaDeviceSynchronize();
    }
    if (e == cudaSuccess) e = cudaMemcpy(C, dC, sizeof(float) * (size_t)M * N, cudaMemcpyDeviceToHost);
    cudaFree(dA);
    cudaFree(dB);
    cudaFree(dC);
    return e == cudaSuccess ? AMRLBM_OK : AMRLBM_ERR_CUDA;
}

}  // extern "C"

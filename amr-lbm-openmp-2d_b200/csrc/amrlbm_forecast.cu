// amrlbm_forecast.cu - the learned regrid's forecast inside the time step:
// one fused kernel evaluates the refine-flag forecaster (amrlbm_net.cu) on
// every leaf that may still refine, between the error indicator of the
// regrid step (Err_Interface, Refine_Derefine.f90:327-351) and the refine
// flags (Refine_Derefine.f90:18-54), and raises the error of each leaf it
// forecasts to twice the refine tolerance. No counterpart in the reference,
// which flags blocks from the current field only.
//
// One CTA per leaf item, persistent over the leaf list. The item's samples
// (the four channels of amrlbm_block_features) are formed from the pool in
// shared memory, the three convolutions run as implicit products on the
// tensor cores (mma.sync m16n8k16, BF16 operands gathered straight from the
// channels-last activations, FP32 accumulation), bias and ReLU in the
// epilogue, the last layer reduced to its channel maxima in registers, and
// the dense output by one thread. The operands, their order along K and the
// rounding steps are those of the network's own forward pass (amrlbm_net.cu;
// both use amrlbm_conv.cuh), so the logits are bit for bit the same.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "amrlbm_conv.cuh"
#include "amrlbm_dev.cuh"
#include "amrlbm_launch.h"

namespace {

template <bool MP>
__global__ void __launch_bounds__(NT, 2)
    k_forecast(const __grid_constant__ DevState s, ForecastNet net, int n_ids, const int* ids,
               float* logits, float horizon, double tol, float thr) {
    extern __shared__ __align__(16) unsigned char smraw[];
    ConvSmem& S = *reinterpret_cast<ConvSmem*>(smraw);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, g = lane >> 2, q = lane & 3;
    load_weights(net, S, t);
    grid_wait();
    grid_release();
    const unsigned zero_row = smem_addr(S.zero);
    const bool explicit_ids = ids != nullptr;
    const int total = explicit_ids ? n_ids : s.cnt->nleaf;
    const int lmin = s.cnt->level_min, lmax = s.cnt->level_max;
    unsigned long long st_pred = 0, st_crit = 0, st_miss = 0, st_extra = 0;
    const int W = s.nx + 2;
    for (int i = blockIdx.x; i < total; i += gridDim.x) {
        const int n = explicit_ids ? ids[i] : s.leaf[i];
        if (!explicit_ids) {
            const int L = s.level[n];
            if (!(L < maxlv_of(s, n) && L >= lmin && L <= lmax)) continue;  // uniform in the CTA
        }
        __syncthreads();  // the previous item's reads of x0 and pmax are done
        // the samples (amrlbm_block_features): C, log(1 + e/tol), U horizon/dx
        const double dx = (double)s.dx[n];
        for (int c = t; c < PIX; c += NT) {
            const int x = c % W, y = c / W;
            double cc, cxp, cxm, cyp, cym, ux = 0.0, uy = 0.0;
            if (MP) {
                cc = s.mp.C[c_idx(s, n, x, y)];
                cxp = s.mp.C[c_idx(s, n, x + 1, y)];
                cxm = s.mp.C[c_idx(s, n, x - 1, y)];
                cyp = s.mp.C[c_idx(s, n, x, y + 1)];
                cym = s.mp.C[c_idx(s, n, x, y - 1)];
            } else {
                cc = s.C[c_idx(s, n, x, y)];
                cxp = s.C[c_idx(s, n, x + 1, y)];
                cxm = s.C[c_idx(s, n, x - 1, y)];
                cyp = s.C[c_idx(s, n, x, y + 1)];
                cym = s.C[c_idx(s, n, x, y - 1)];
            }
            const bool in = x >= 1 && x <= s.nx && y >= 1 && y <= s.ny;
            if (in) {
                ux = MP ? (double)s.mp.Ux[p_idx(s, n, x, y)] : s.Ux[p_idx(s, n, x, y)];
                uy = MP ? (double)s.mp.Uy[p_idx(s, n, x, y)] : s.Uy[p_idx(s, n, x, y)];
            }
            const double gx = cxp - cxm, gy = cyp - cym;
            const float f0 = (float)cc;
            const float f1 = (float)log1p(sqrt(gx * gx + gy * gy) / (2.0 * dx) / tol);
            const float f2 = in ? (float)(ux * horizon / dx) : 0.f;
            const float f3 = in ? (float)(uy * horizon / dx) : 0.f;
            unsigned* x32 = reinterpret_cast<unsigned*>(&S.x0[c][0]);
            x32[0] = pack2(f0, f1);
            x32[1] = pack2(f2, f3);
        }
        __syncthreads();
        two_layers(S, zero_row, warp, lane);
        // layer 3 reduced to the channel maxima (global max pool)
        float mx[4][2];
#pragma unroll
        for (int j = 0; j < 4; ++j) mx[j][0] = mx[j][1] = -1.f;
        {
            float acc[3][4][4];
            conv32<KW2>(S.act[1], S.w3, zero_row, warp, lane, acc);
#pragma unroll
            for (int u = 0; u < 3; ++u) {
                const int mt = warp + NWARP * u;
                if (mt >= MTILES) continue;
                const int r0 = 16 * mt + g, r1 = r0 + 8;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int n2 = 8 * j + 2 * q;
                    if (r0 < PIX) {
                        mx[j][0] = fmaxf(mx[j][0], fmaxf(acc[u][j][0] + S.b[2][n2], 0.f));
                        mx[j][1] = fmaxf(mx[j][1], fmaxf(acc[u][j][1] + S.b[2][n2 + 1], 0.f));
                    }
                    if (r1 < PIX) {
                        mx[j][0] = fmaxf(mx[j][0], fmaxf(acc[u][j][2] + S.b[2][n2], 0.f));
                        mx[j][1] = fmaxf(mx[j][1], fmaxf(acc[u][j][3] + S.b[2][n2 + 1], 0.f));
                    }
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int o = 4; o < 32; o <<= 1)
                    mx[j][h] = fmaxf(mx[j][h], __shfl_xor_sync(0xffffffffu, mx[j][h], o));
        if (g == 0)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                S.pmax[warp][8 * j + 2 * q] = mx[j][0];
                S.pmax[warp][8 * j + 2 * q + 1] = mx[j][1];
            }
        __syncthreads();
        if (t == 0) {  // the dense output, in channel order
            float z = S.bd;
            for (int c = 0; c < CH; ++c) {
                float p = S.pmax[0][c];
                for (int w = 1; w < NWARP; ++w) p = fmaxf(p, S.pmax[w][c]);
                z += S.wd[c] * p;
            }
            if (explicit_ids) {
                logits[i] = z;
            } else {
                const bool pr = z > thr, cr = s.err[n] > tol;
                st_pred += pr;
                st_crit += cr;
                st_miss += cr && !pr;
                st_extra += pr && !cr;
                if (pr && !cr) s.err[n] = 2.0 * tol;
            }
        }
    }
    if (!explicit_ids && t == 0 && (st_pred | st_crit)) {
        atomicAdd(&s.cnt->rstat[1], st_pred);
        atomicAdd(&s.cnt->rstat[2], st_crit);
        atomicAdd(&s.cnt->rstat[3], st_miss);
        atomicAdd(&s.cnt->rstat[4], st_extra);
    }
}

template <bool MP>
void forecast_launch(const DevState& s, const LaunchCfg& lc, cudaStream_t st, const ForecastNet& net,
                     int n_ids, const int* ids, float* logits, float horizon, double tol, float thr) {
    const size_t sm = sizeof(ConvSmem);
    cudaFuncSetAttribute(k_forecast<MP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    int grid = 2 * lc.num_sms;
    if (ids && n_ids < grid) grid = n_ids > 0 ? n_ids : 1;
    launch_dep(k_forecast<MP>, grid, NT, sm, st, s, net, n_ids, ids, logits, horizon, tol, thr);
}

}  // namespace

void launch_forecast(const DevState& s, const LaunchCfg& lc, cudaStream_t st, const ForecastNet& net,
                     int n_ids, const int* ids, float* logits, float horizon, double tol, float thr) {
    if (s.mp.fmt)
        forecast_launch<true>(s, lc, st, net, n_ids, ids, logits, horizon, tol, thr);
    else
        forecast_launch<false>(s, lc, st, net, n_ids, ids, logits, horizon, tol, thr);
    count_launches(1);
}

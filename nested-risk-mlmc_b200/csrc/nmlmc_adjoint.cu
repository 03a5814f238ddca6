// Path-simulated portfolio loss with its adjoint, for a batch of portfolios in one launch.
//
// Per portfolio p and outer sample m (stream key (seed, ell<<56 | p<<32 | m), so a single
// portfolio at p = 0 draws exactly the outer samples of the OUTER layout):
//   R_tau,j  = S0_j exp(sigma_j W_j + (mu_j - sigma_j^2/2) tau),  W_j = rho W_sys + sqrt(1-rho^2) W_ind,j
//              (portfolio_sampler.cpp:293-311, normal 0 systemic, 1 + j per stock)
//   C_i(m)   = e^{-r (T_i - tau)} (1/N) sum_n (pay(S+_n) + pay(S-_n)) / 2, S+- an antithetic pair of
//              Milstein paths (gbm_approx.hpp:18-57, risk-neutral drift r) on 2^ell steps from
//              (tau, R_tau,s(i)) to T_i; pay(S) = max(type (S - K_i), 0)
//   L_m      = sum_i w_i (V_i(0) - e^{-r tau} C_i(m))
// Pass 1 sums L_m over the options; the weight kernel forms E[L], the sigmoid-smoothed
// P_delta = E[s((L - K)/delta)], the plain exceedance frequency and the adjoint weights
// dF/dL_m (1/M for E[L], s'(x)/(delta M) for P_delta).  Pass 1 carries dS/dsigma along each path
// (one scalar parameter per path, so the tangent costs what a reverse sweep would and needs no
// tape) and keeps the two derivatives dl_im/dw_i and dl_im/dsigma of every option and outer sample;
// pass 2 pulls the weights back through them to every option position w_i and stock volatility
// sigma_j.  Outer samples whose derivatives do not fit the kept buffer (AdjLaunch::m_store) have
// their inner draws recomputed from the counter RNG in pass 2; the draws themselves are never
// stored.
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>

#include "nmlmc_common.cuh"
#include "nmlmc_internal.h"

namespace nmlmc {

namespace {

constexpr int kAdjThreads = 128;

__device__ __forceinline__ uint64_t adj_stream_id(uint32_t ell, uint32_t p, uint64_t m) {
    return ((uint64_t)ell << 56) | ((uint64_t)p << 32) | (m & 0xffffffffull);
}

// Four normals of one Threefry block: Box-Muller on the words (v0 lo, v0 hi) and (v1 lo, v1 hi);
// SFU Box-Muller for float, the double one for double.
template <class RT>
__device__ __forceinline__ void normals4(uint64_t v0, uint64_t v1, RT* z) {
    if constexpr (sizeof(RT) == 4) {
        boxmuller32_f4(v0, v1, z);
    } else {
        boxmuller32_d((uint32_t)v0, (uint32_t)(v0 >> 32), z[0], z[1]);
        boxmuller32_d((uint32_t)v1, (uint32_t)(v1 >> 32), z[2], z[3]);
    }
}

// Portfolio p with off[p] <= k < off[p + 1] (offsets strictly increasing).
__device__ __forceinline__ uint32_t segment_of(const uint32_t* off, uint32_t n, uint32_t k) {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (off[mid] <= k) lo = mid; else hi = mid;
    }
    return lo;
}

template <class RT>
__device__ __forceinline__ RT rexp(RT x) {
    if constexpr (sizeof(RT) == 4) return expf(x); else return exp(x);
}

// ---- outer draws: R_tau and dR_tau/dsigma per (portfolio, outer sample, stock) ----------------
template <class RT>
__global__ void __launch_bounds__(256) k_adj_outer(AdjLaunch<RT> A) {
    const uint64_t total = (uint64_t)A.n * A.M;
    for (uint64_t id = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; id < total;
         id += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t p = (uint32_t)(id / A.M);
        const uint64_t m = id % A.M;
        const TfKey key = tf_key(A.seed, adj_stream_id(A.ell, p, m));
        const uint32_t s0 = A.stock_off[p], Q = A.stock_off[p + 1] - s0;
        RT* Rrow = A.R + (size_t)s0 * A.M + (size_t)m * Q;
        RT* Drow = A.dR + (size_t)s0 * A.M + (size_t)m * Q;
        const uint32_t nnorm = Q == 1 ? 1 : Q + 1;
        RT dW_sys = 0;
        for (uint32_t b = 0; 4 * b < nnorm; b++) {
            uint64_t v0, v1;
            threefry2x64(b, PH_OUTER, key, v0, v1);
            RT z[4];
            normals4<RT>(v0, v1, z);
            for (uint32_t q = 0; q < 4; q++) {
                const uint32_t k = 4 * b + q;
                if (k >= nnorm) break;
                if (k == 0) {
                    dW_sys = A.stau * z[0];
                    if (Q > 1) continue;
                }
                const uint32_t j = Q == 1 ? 0 : k - 1;
                const RT W = Q == 1 ? dW_sys : A.rho * dW_sys + A.s1_rho2 * (A.stau * z[q]);
                const RT sg = A.sigma[s0 + j];
                const RT R = A.S0[s0 + j] * rexp<RT>(sg * W + (A.mu[s0 + j] - (RT)0.5 * sg * sg) * A.tau);
                Rrow[j] = R;
                Drow[j] = R * (W - sg * A.tau);
            }
        }
    }
}

// A CTA's gradient sums into the global ones: one atomic per option, and per stock through the
// shared sums gs_sh [2][Q] (zeroed by the caller).
template <class RT>
__device__ __forceinline__ void adj_flush(const AdjLaunch<RT>& A, bool valid, uint32_t i, uint32_t s, uint32_t s0, uint32_t Q,
                                          double gwE, double gwP, double gsE, double gsP, double* gs_sh) {
    if (valid) {
        atomicAdd(&A.gw_E[i], gwE);
        atomicAdd(&A.gw_P[i], gwP);
        atomicAdd(&gs_sh[s], gsE);
        atomicAdd(&gs_sh[Q + s], gsP);
    }
    __syncthreads();
    for (uint32_t t = threadIdx.x; t < Q; t += blockDim.x) {
        if (gs_sh[t] != 0) atomicAdd(&A.gs_E[s0 + t], gs_sh[t]);
        if (gs_sh[Q + t] != 0) atomicAdd(&A.gs_P[s0 + t], gs_sh[Q + t]);
    }
}

// ---- per-option constants from the caller's double arrays ------------------------------------
// V_i(0) (Black-Scholes, portfolio_sampler.cpp:140-150) and vega_i = dV_i(0)/dsigma =
// S0 phi(d1) sqrt(T), in double and rounded once, with the narrowed inputs of the path kernels.
template <class RT>
__global__ void __launch_bounds__(256) k_adj_setup(AdjLaunch<RT> A, AdjInputs in) {
    const uint32_t NS = A.stock_off[A.n], NO = A.option_off[A.n];
    const uint32_t id = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    for (uint32_t j = id; j < NS; j += stride) {
        A.S0[j] = (RT)in.S0[j];
        A.mu[j] = (RT)in.mu[j];
        A.sigma[j] = (RT)in.sigma[j];
    }
    for (uint32_t i = id; i < NO; i += stride) {
        const uint32_t s = A.stock_off[segment_of(A.option_off, A.n, i)] + A.stock_ind[i];
        const double S = in.S0[s], sg = in.sigma[s], K = in.strike[i], T = in.maturity[i];
        const int type = in.type[i];
        const double d1 = bs_d1_ref<double>(S, K, in.r, T, sg);
        A.strike[i] = (RT)K;
        A.maturity[i] = (RT)T;
        A.w[i] = (RT)in.w[i];
        A.type[i] = (int8_t)type;
        A.V0[i] = (RT)calc_bs_ref<double>(type, S, K, in.r, T, sg);
        A.vega[i] = (RT)(S * exp(-0.5 * d1 * d1) * 0.39894228040143268 * sqrt(T));
    }
}

// ---- inner paths -------------------------------------------------------------------------------
// The sums over the antithetic path pairs of one (option, outer sample): the payoffs, and with TAN
// their pathwise derivatives by sigma (dS/dsigma carried along each path).
template <class RT>
struct PairSums { RT C, dC; };

// Products that a sum follows are rounded on their own (no contraction), whatever MIL is.
__device__ __forceinline__ float rmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }

// MIL: Milstein steps, else Euler.
template <class RT, bool TAN, bool MIL>
struct AntitheticPaths {
    RT Sp, Sm, Dp, Dm;
    __device__ __forceinline__ void start(RT R, RT dR) { Sp = Sm = R; Dp = Dm = dR; }
    // one step of both paths on the normal z (gbm_approx.hpp:18-57)
    __device__ __forceinline__ void step(RT z, RT sh, RT h, RT rh1, RT sg, RT hs2) {
        const RT dW = sh * z;
        const RT q = dW * dW - h, corr = MIL ? rmul(hs2, q) : (RT)0, dc = MIL ? rmul(sg, q) : (RT)0;
        const RT gp = rh1 + sg * dW + corr, gm = rh1 - sg * dW + corr;
        if (TAN) {
            Dp = Dp * gp + Sp * (dW + dc);
            Dm = Dm * gm + Sm * (dc - dW);
        }
        Sp *= gp;
        Sm *= gm;
    }
    __device__ __forceinline__ void payoff(RT type, RT K, PairSums<RT>& a) const {
        const RT xp = type * (Sp - K), xm = type * (Sm - K);
        a.C += (RT)0.5 * ((xp > 0 ? xp : (RT)0) + (xm > 0 ? xm : (RT)0));
        if (TAN) a.dC += (RT)0.5 * ((xp > 0 ? type * Dp : (RT)0) + (xm > 0 ? type * Dm : (RT)0));
    }
};

// What k_adj_paths does with the value l_im = w_i (V_i(0) - e^{-r tau} C_i(m)) of its options:
//   ADJ_LOSS   adds it to L_m
//   ADJ_STORE  the same, and keeps dl/dw_i and dl/dsigma for k_adj_pull
//   ADJ_PULL   pulls the weights back at once (outer samples past the kept ones: the draws again)
enum AdjMode { ADJ_LOSS, ADJ_STORE, ADJ_PULL };

// A thread per option, a tile of outer samples [A.m0 + blockIdx.y tile, ...) per CTA.  Bound by
// the integer (ALU) pipe of the counter generator (139 warp instructions per four normals, half
// rate).  Each pair-step is drawn once: the derivatives by w_i and sigma_j that the weights of
// k_adj_weights multiply are kept (two RT per option and outer sample, 8 bytes in FP32: 205 MB
// written and read once for 1e5 options x 256 outer samples, 0.06 ms of HBM time) instead of
// drawing and stepping every path a second time (4.4 ms).
template <class RT, int MODE, bool MIL>
__global__ void __launch_bounds__(kAdjThreads) k_adj_paths(AdjLaunch<RT> A) {
    constexpr bool TAN = MODE != ADJ_LOSS;
    extern __shared__ double adj_sh[];                  // [tile][warps] | 2 * Qmax (ADJ_PULL)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int warps = kAdjThreads / 32;
    const uint32_t chunk = blockIdx.x, p = segment_of(A.chunk_off, A.n, chunk);
    const uint32_t o0 = A.option_off[p], P = A.option_off[p + 1] - o0;
    const uint32_t s0 = A.stock_off[p], Q = A.stock_off[p + 1] - s0;
    const uint32_t il = (chunk - A.chunk_off[p]) * kAdjThreads + threadIdx.x;
    const bool valid = il < P;
    const uint32_t i = o0 + (valid ? il : 0);
    const uint64_t m0 = A.m0 + (uint64_t)blockIdx.y * A.tile;
    const uint64_t m1 = m0 + A.tile < A.m1 ? m0 + A.tile : A.m1;

    double* gs_sh = adj_sh;                              // ADJ_PULL: [2][Q]
    if (MODE == ADJ_PULL) {
        for (uint32_t t = threadIdx.x; t < 2 * Q; t += blockDim.x) gs_sh[t] = 0;
        __syncthreads();
    }

    const uint32_t s = A.stock_ind[i];
    const RT K = A.strike[i], T = A.maturity[i], w = A.w[i];
    const RT type = (RT)A.type[i];
    const RT sg = A.sigma[s0 + s];
    const uint32_t steps = 1u << A.ell;
    const RT Tr = T - A.tau;
    const RT h = Tr / (RT)steps;
    const RT sh = sqrt(h);
    const RT rh1 = (RT)1 + A.r * h;
    const RT hs2 = (RT)0.5 * sg * sg;
    const RT disc_in = rexp<RT>(-A.r * Tr);
    const RT V0 = A.V0[i], vega = A.vega[i];
    const RT invN = (RT)1 / (RT)A.pairs;
    const uint64_t ctr1 = ((uint64_t)il << 32) | PH_ADJOINT;

    double gwE = 0, gwP = 0, gsE = 0, gsP = 0;
    for (uint64_t m = m0; m < m1; m++) {
        const TfKey key = tf_key(A.seed, adj_stream_id(A.ell, p, m));
        const size_t ridx = (size_t)s0 * A.M + (size_t)m * Q + s;
        const RT Rt = A.R[ridx];
        const RT Dt = TAN ? A.dR[ridx] : (RT)0;
        PairSums<RT> sum{(RT)0, (RT)0};
        AntitheticPaths<RT, TAN, MIL> S;
        RT z[4];
        if (steps >= 4) {                                // a path takes whole blocks of four normals
            uint64_t blk = 0;
            for (uint32_t n = 0; n < A.pairs; n++) {
                S.start(Rt, Dt);
#pragma unroll 1
                for (uint32_t k = 0; k < steps; k += 4, blk++) {
                    uint64_t v0, v1;
                    threefry2x64(blk, ctr1, key, v0, v1);
                    normals4<RT>(v0, v1, z);
#pragma unroll
                    for (int e = 0; e < 4; e++) S.step(z[e], sh, h, rh1, sg, hs2);
                }
                S.payoff(type, K, sum);
            }
        } else {                                         // one or two steps: several pairs share a block
            uint64_t q = 0;
            for (uint32_t n = 0; n < A.pairs; n++) {
                S.start(Rt, Dt);
                for (uint32_t k = 0; k < steps; k++, q++) {
                    const uint32_t e = (uint32_t)(q & 3);
                    if (e == 0) {
                        uint64_t v0, v1;
                        threefry2x64(q >> 2, ctr1, key, v0, v1);
                        normals4<RT>(v0, v1, z);
                    }
                    S.step(e == 0 ? z[0] : (e == 1 ? z[1] : (e == 2 ? z[2] : z[3])), sh, h, rh1, sg, hs2);
                }
                S.payoff(type, K, sum);
            }
        }
        const RT C = disc_in * sum.C * invN;
        const RT dl_dw = V0 - A.disc_tau * C;
        RT dl_ds = (RT)0;
        if (TAN) dl_ds = w * (vega - A.disc_tau * disc_in * sum.dC * invN);
        if (MODE == ADJ_PULL) {
            if (valid) {
                const double wE = A.wE[p], wP = A.omega[(size_t)p * A.M + m];
                gwE += wE * (double)dl_dw;
                gwP += wP * (double)dl_dw;
                gsE += wE * (double)dl_ds;
                gsP += wP * (double)dl_ds;
            }
        } else {
            if (MODE == ADJ_STORE && valid) A.store[(size_t)m * A.n_options + i] = typename Pair2<RT>::type{dl_dw, dl_ds};
            double v = valid ? (double)(w * dl_dw) : 0.0;
            v = warp_sum(v);
            if (lane == 0) adj_sh[(m - m0) * warps + warp] = v;
        }
    }
    if (MODE != ADJ_PULL) {
        __syncthreads();
        for (uint64_t t = threadIdx.x; t < m1 - m0; t += blockDim.x) {
            double v = 0;
            for (int k = 0; k < warps; k++) v += adj_sh[t * warps + k];
            atomicAdd(&A.L[(size_t)p * A.M + m0 + t], v);
        }
        return;
    }
    adj_flush<RT>(A, valid, i, s, s0, Q, gwE, gwP, gsE, gsP, gs_sh);
}

// Pull-back of the weights through the kept derivatives: gradients by w_i (a thread per option) and
// by sigma_j (summed per stock in shared memory).  One coalesced pass over the kept values, bound
// by HBM; a CTA walks a tile of outer samples so few sums per stock reach the global atomics.
template <class RT>
__global__ void __launch_bounds__(kAdjThreads) k_adj_pull(AdjLaunch<RT> A) {
    extern __shared__ double adj_sh[];                  // [2][Q]
    const uint32_t chunk = blockIdx.x, p = segment_of(A.chunk_off, A.n, chunk);
    const uint32_t o0 = A.option_off[p], P = A.option_off[p + 1] - o0;
    const uint32_t s0 = A.stock_off[p], Q = A.stock_off[p + 1] - s0;
    const uint32_t il = (chunk - A.chunk_off[p]) * kAdjThreads + threadIdx.x;
    const bool valid = il < P;
    const uint32_t i = o0 + (valid ? il : 0);
    const uint64_t m0 = A.m0 + (uint64_t)blockIdx.y * A.tile;
    const uint64_t m1 = m0 + A.tile < A.m1 ? m0 + A.tile : A.m1;
    for (uint32_t t = threadIdx.x; t < 2 * Q; t += blockDim.x) adj_sh[t] = 0;
    __syncthreads();
    double gwE = 0, gwP = 0, gsE = 0, gsP = 0;
    if (valid) {
        const double wE = A.wE[p];
        const double* om = A.omega + (size_t)p * A.M;
#pragma unroll 8
        for (uint64_t m = m0; m < m1; m++) {
            const typename Pair2<RT>::type d = A.store[(size_t)m * A.n_options + i];
            const double wP = om[m];
            gwE += wE * (double)d.x;
            gwP += wP * (double)d.x;
            gsE += wE * (double)d.y;
            gsP += wP * (double)d.y;
        }
    }
    adj_flush<RT>(A, valid, i, A.stock_ind[i], s0, Q, gwE, gwP, gsE, gsP, adj_sh);
}

// ---- estimates and adjoint weights per portfolio (one block per portfolio) -------------------
template <class RT>
__global__ void __launch_bounds__(256) k_adj_weights(AdjLaunch<RT> A) {
    const uint32_t p = blockIdx.x;
    const double K = A.K[p], delta = A.delta[p];
    const double invM = 1.0 / (double)A.M;
    double sL = 0, sS = 0, sH = 0;
    for (uint64_t m = threadIdx.x; m < A.M; m += blockDim.x) {
        const double L = A.L[(size_t)p * A.M + m];
        const double x = (L - K) / delta;
        const double sgm = 1.0 / (1.0 + exp(-x));
        A.omega[(size_t)p * A.M + m] = sgm * (1.0 - sgm) / delta * invM;
        sL += L;
        sS += sgm;
        sH += L > K ? 1.0 : 0.0;
    }
    __shared__ double red[3][8];
    sL = warp_sum(sL);
    sS = warp_sum(sS);
    sH = warp_sum(sH);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { red[0][warp] = sL; red[1][warp] = sS; red[2][warp] = sH; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0, b = 0, c = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) { a += red[0][k]; b += red[1][k]; c += red[2][k]; }
        A.est[3 * p + 0] = a * invM;
        A.est[3 * p + 1] = b * invM;
        A.est[3 * p + 2] = c * invM;
        A.wE[p] = invM;
    }
}

// Outer samples per CTA: at most `cap`, and small enough for about 64 CTAs per SM (several waves,
// so the last one costs little) when the option chunks alone are too few.
template <class RT>
uint32_t adj_tile(const AdjLaunch<RT>& A, uint64_t rows_m, uint64_t ctas, uint64_t cap) {
    const uint64_t rows = (ctas + A.n_chunks - 1) / A.n_chunks;
    const uint64_t t = (rows_m + rows - 1) / rows;
    return (uint32_t)(t < 1 ? 1 : (t < cap ? t : cap));
}

template <class RT, int MODE, bool MIL>
cudaError_t launch_paths_m(AdjLaunch<RT> A, uint64_t m0, uint64_t m1, cudaStream_t stream) {
    if (m0 >= m1) return cudaSuccess;
    A.m0 = m0;
    A.m1 = m1;
    A.tile = adj_tile(A, m1 - m0, 148ull * 64, kAdjMaxTile);
    const uint64_t per = A.tile;
    const size_t sh = MODE == ADJ_PULL ? (size_t)2 * A.q_max * sizeof(double) : per * (kAdjThreads / 32) * sizeof(double);
    if (sh > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_adj_paths<RT, MODE, MIL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh);
        if (e != cudaSuccess) return e;
    }
    for (uint64_t a = m0; a < m1; a += per * 65535) {     // at most 65,535 rows of tiles per launch
        A.m0 = a;
        A.m1 = m1 - a < per * 65535 ? m1 : a + per * 65535;
        const dim3 grid(A.n_chunks, (uint32_t)((A.m1 - a + per - 1) / per));
        k_adj_paths<RT, MODE, MIL><<<grid, kAdjThreads, sh, stream>>>(A);
        count_launch();
    }
    return cudaGetLastError();
}

template <class RT, int MODE>
cudaError_t launch_paths(const AdjLaunch<RT>& A, uint64_t m0, uint64_t m1, cudaStream_t stream) {
    return A.milstein ? launch_paths_m<RT, MODE, true>(A, m0, m1, stream) : launch_paths_m<RT, MODE, false>(A, m0, m1, stream);
}

template <class RT>
cudaError_t launch_pull(AdjLaunch<RT> A, uint64_t m1, cudaStream_t stream) {
    if (m1 == 0) return cudaSuccess;
    A.m0 = 0;
    A.m1 = m1;
    const size_t sh = (size_t)2 * A.q_max * sizeof(double);
    if (sh > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_adj_pull<RT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh);
        if (e != cudaSuccess) return e;
    }
    A.tile = adj_tile(A, m1, 148ull * 4, 1u << 20);
    const uint64_t rows = (m1 + A.tile - 1) / A.tile;
    if (rows > 65535) A.tile = (uint32_t)((m1 + 65534) / 65535);
    k_adj_pull<RT><<<dim3(A.n_chunks, (uint32_t)((m1 + A.tile - 1) / A.tile)), kAdjThreads, sh, stream>>>(A);
    count_launch();
    return cudaGetLastError();
}

template <class RT>
cudaError_t launch_adjoint_t(const AdjLaunch<RT>& A, const AdjInputs& in, bool grad, cudaStream_t stream) {
    if (A.m_store > A.M) return cudaErrorInvalidValue;
    const uint32_t sb = (A.n_options + 255) / 256;
    k_adj_setup<RT><<<sb < 148 * 8 ? sb : 148 * 8, 256, 0, stream>>>(A, in);
    const uint64_t ob = ((uint64_t)A.n * A.M + 255) / 256;
    k_adj_outer<RT><<<(uint32_t)(ob < 148 * 8 ? ob : 148 * 8), 256, 0, stream>>>(A);
    count_launch(2);
    const uint64_t ms = grad ? A.m_store : 0;
    cudaError_t e = launch_paths<RT, ADJ_STORE>(A, 0, ms, stream);
    if (e == cudaSuccess) e = launch_paths<RT, ADJ_LOSS>(A, ms, A.M, stream);
    if (e != cudaSuccess) return e;
    k_adj_weights<RT><<<A.n, 256, 0, stream>>>(A);
    count_launch();
    if (grad) {
        e = launch_pull<RT>(A, ms, stream);
        if (e == cudaSuccess) e = launch_paths<RT, ADJ_PULL>(A, ms, A.M, stream);
        if (e != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_adjoint(const AdjLaunch<float>& A, const AdjInputs& in, bool grad, cudaStream_t stream) {
    return launch_adjoint_t<float>(A, in, grad, stream);
}
cudaError_t launch_adjoint(const AdjLaunch<double>& A, const AdjInputs& in, bool grad, cudaStream_t stream) {
    return launch_adjoint_t<double>(A, in, grad, stream);
}

}  // namespace nmlmc

// OUTER-layout (batched) level sampler: the precision/kind dispatch of a level call, the
// full-portfolio loss sweep, device timestamps, launch counting and the utility kernels.  The
// kernels and the launch sequence of a level are in nmlmc_outer_impl.cuh; their instantiations per
// sampler kind are compiled from nmlmc_outer_kind.cu.
#include <atomic>

#include "nmlmc_outer_impl.cuh"

namespace nmlmc {

// ---- host orchestration ----------------------------------------------------------------------
static std::atomic<uint64_t> g_launches{0};
void count_launch(uint64_t n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
uint64_t launches_total() { return g_launches.load(std::memory_order_relaxed); }

cudaError_t outer_level_begin(OuterBuffers& B, cudaStream_t stream) {
    return cudaMemsetAsync(B.level_acc, 0, 16 * sizeof(double), stream);
}

// Level sequences instantiated per kind in nmlmc_outer_kind.cu.
#define NMLMC_SLT(RT, KIND, PREC) \
    extern template cudaError_t sample_level_t<RT, KIND, PREC>(const OuterLevel<RT>&, OuterBuffers&, TraceRec*, cudaStream_t);
NMLMC_SLT(float, KIND_REF_MODEL, PREC_FP32) NMLMC_SLT(float, KIND_SHIFT_MODEL, PREC_FP32) NMLMC_SLT(float, KIND_PORTFOLIO, PREC_FP32)
NMLMC_SLT(float, KIND_REF_MODEL, PREC_REF32) NMLMC_SLT(float, KIND_SHIFT_MODEL, PREC_REF32) NMLMC_SLT(float, KIND_PORTFOLIO, PREC_REF32)
NMLMC_SLT(double, KIND_REF_MODEL, PREC_FP64) NMLMC_SLT(double, KIND_SHIFT_MODEL, PREC_FP64) NMLMC_SLT(double, KIND_PORTFOLIO, PREC_FP64)
NMLMC_SLT(float, KIND_PF_PATHS, PREC_FP32) NMLMC_SLT(float, KIND_PF_PATHS, PREC_REF32) NMLMC_SLT(double, KIND_PF_PATHS, PREC_FP64)
#undef NMLMC_SLT

template <class RT>
cudaError_t outer_sample_level(const OuterLevel<RT>& L, int kind, int prec, OuterBuffers& B,
                               TraceRec* trace, cudaStream_t stream) {
    if (prec == PREC_FP64) {
        if constexpr (sizeof(RT) == 8) {
            if (kind == KIND_REF_MODEL) return sample_level_t<RT, KIND_REF_MODEL, PREC_FP64>(L, B, trace, stream);
            if (kind == KIND_SHIFT_MODEL) return sample_level_t<RT, KIND_SHIFT_MODEL, PREC_FP64>(L, B, trace, stream);
            if (L.ot.mixed) return sample_level_t<RT, KIND_PF_PATHS, PREC_FP64>(L, B, trace, stream);
            return sample_level_t<RT, KIND_PORTFOLIO, PREC_FP64>(L, B, trace, stream);
        }
        return cudaErrorInvalidValue;
    }
    if constexpr (sizeof(RT) == 4) {
        if (prec == PREC_FP32) {
            if (kind == KIND_REF_MODEL) return sample_level_t<RT, KIND_REF_MODEL, PREC_FP32>(L, B, trace, stream);
            if (kind == KIND_SHIFT_MODEL) return sample_level_t<RT, KIND_SHIFT_MODEL, PREC_FP32>(L, B, trace, stream);
            if (L.ot.mixed) return sample_level_t<RT, KIND_PF_PATHS, PREC_FP32>(L, B, trace, stream);
            return sample_level_t<RT, KIND_PORTFOLIO, PREC_FP32>(L, B, trace, stream);
        }
        if (kind == KIND_REF_MODEL) return sample_level_t<RT, KIND_REF_MODEL, PREC_REF32>(L, B, trace, stream);
        if (kind == KIND_SHIFT_MODEL) return sample_level_t<RT, KIND_SHIFT_MODEL, PREC_REF32>(L, B, trace, stream);
        if (L.ot.mixed) return sample_level_t<RT, KIND_PF_PATHS, PREC_REF32>(L, B, trace, stream);
        return sample_level_t<RT, KIND_PORTFOLIO, PREC_REF32>(L, B, trace, stream);
    }
    return cudaErrorInvalidValue;
}

template cudaError_t outer_sample_level<float>(const OuterLevel<float>&, int, int, OuterBuffers&, TraceRec*, cudaStream_t);
template cudaError_t outer_sample_level<double>(const OuterLevel<double>&, int, int, OuterBuffers&, TraceRec*, cudaStream_t);

// ---- full portfolio loss sweep ---------------------------------------------------------------
// L(Y) over every option: init_inner_sampler without sub-sampling and sample_inner_all_options
// (portfolio_sampler.cpp:312-324, 336-344), one warp per outer sample, for the K quantile.
template <class RT, int PREC>
__global__ void k_full_loss(DevLevel<RT> D, uint32_t nb, double* loss) {
    // one warp per outer sample: lanes stride the option table, double accumulation
    const int lane = threadIdx.x & 31;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const OptionTable<RT>& ot = D.L.ot;
    for (uint32_t i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < nb; i += warps) {
        constexpr uint32_t RS = RStride<PREC>::v;
        const RT* Rrow = reinterpret_cast<const RT*>(D.B.Rt) + (size_t)i * ot.Q * RS;
        double s = 0;
        for (uint32_t j = lane; j < ot.P; j += 32) {
            const RefOption<RT> o = ot.ref[j];
            s += (double)ref_option_value<RT>(o, Rrow[o.stock * RS], false);
        }
        s = warp_sum(s);
        if (lane == 0) loss[i] = s;
    }
}

// FP32 sweep of the packed option table: a CTA takes a tile of TILE outer samples and streams the
// table once per tile, so every 32-byte record fetched from L2/HBM feeds TILE Black-Scholes
// evaluations.  Two outer samples share each instruction (f32x2); their R and ln R sit in shared
// memory as one 16-byte entry per stock (R_o, R_o+1, ln R_o, ln R_o+1), rows one entry longer than
// the tile so that the lanes' random stocks spread over the banks.  Per-thread partial sums are
// float (each thread adds P/256 options in table order), combined in double across the CTA, so the
// tile's length changes no result.  Bound by the FMA pipe (75 % busy at 10^5 outer samples of 10^4
// options) with the four SFU operations of an evaluation close behind (68 %).
template <int TILE>
__global__ void __launch_bounds__(kTile) k_full_loss_fast(DevLevel<float> D, uint32_t nb, double* loss) {
    constexpr int H = TILE / 2;
    extern __shared__ float4 sm_rows[];  // [Q][H + 1]
    __shared__ double red[kWarps][TILE];
    const OptionTable<float>& ot = D.L.ot;
    const uint32_t Q = ot.Q, P = ot.P;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const float2* Rt = reinterpret_cast<const float2*>(D.B.Rt);     // (R, ln R) per stock
    const uint32_t ntiles = (nb + TILE - 1) / TILE;
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const uint32_t o0 = tile * TILE;
        const uint32_t n_here = (nb - o0) < (uint32_t)TILE ? (nb - o0) : (uint32_t)TILE;
        for (uint32_t k = t; k < (uint32_t)H * Q; k += blockDim.x) {
            const uint32_t o = k / Q, q = k - o * Q;
            const float2 a = 2 * o < n_here ? Rt[(size_t)(o0 + 2 * o) * Q + q] : make_float2(1.0f, 0.0f);
            const float2 b = 2 * o + 1 < n_here ? Rt[(size_t)(o0 + 2 * o + 1) * Q + q] : make_float2(1.0f, 0.0f);
            sm_rows[(size_t)q * (H + 1) + o] = make_float4(a.x, b.x, a.y, b.y);
        }
        __syncthreads();
        F2 acc[H];
#pragma unroll
        for (int o = 0; o < H; o++) acc[o] = f2(0.f, 0.f);
        for (uint32_t j = t; j < P; j += blockDim.x) {
            const FastOption op = load_record_l1(ot.fast + j);     // full-loss records: no control variate
            const float4* row = sm_rows + (size_t)op.stock * (H + 1);
#pragma unroll
            for (int o = 0; o < H; o++) {
                const float4 r = row[o];
                acc[o] = f2_add(acc[o], option_loss_fast2(op, f2(r.x, r.y), f2(r.z, r.w)));
            }
        }
#pragma unroll
        for (int o = 0; o < TILE; o++) {
            double v = (double)((o & 1) ? f2_hi(acc[o / 2]) : f2_lo(acc[o / 2]));
            for (int m = 16; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
            if (lane == 0) red[warp][o] = v;
        }
        __syncthreads();
        if (t < (int)n_here) {
            double s = 0;
            for (int w = 0; w < kWarps; w++) s += red[w][t];
            loss[o0 + t] = s;
        }
        __syncthreads();
    }
}

template <int TILE>
static cudaError_t launch_full_loss_fast(const DevLevel<float>& D, uint32_t nb, double* loss, cudaStream_t stream) {
    const size_t smem = (size_t)D.L.ot.Q * (TILE / 2 + 1) * sizeof(float4);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_full_loss_fast<TILE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    const uint32_t tiles = (nb + TILE - 1) / TILE;
    k_full_loss_fast<TILE><<<tiles < (uint32_t)D.B.grid * 2 ? tiles : D.B.grid * 2, kTile, smem, stream>>>(D, nb, loss);
    count_launch();
    return cudaGetLastError();
}

// Losses of outer samples L.first_index .. + L.M - 1 into the host's array.  A batch's losses sit in
// the item lists, which the sweep does not use (two doubles per outer sample), so a call allocates
// nothing (a device allocation and its release took up to 0.8 ms of a call).
template <class RT>
cudaError_t outer_full_loss(const OuterLevel<RT>& L, int prec, OuterBuffers& B, double* host_loss, cudaStream_t stream) {
    DevLevel<RT> D;
    D.L = L;
    D.B = B;
    double* loss = reinterpret_cast<double*>(B.lists);
    for (uint64_t done = 0; done < L.M;) {
        const uint64_t nb = (L.M - done) < B.cap ? (L.M - done) : B.cap;
        D.L.first_index = L.first_index + done;
        int og = (int)((nb + kTile - 1) / kTile);
        if (og > B.grid) og = B.grid;
        if (og < 1) og = 1;
        const uint32_t n = (uint32_t)nb;
        cudaError_t e = cudaSuccess;
        if (prec == PREC_FP64) {
            if constexpr (sizeof(RT) == 8) {
                k_outer<RT, KIND_PORTFOLIO, PREC_FP64><<<og, kTile, 0, stream>>>(D, n, 0);
                k_full_loss<RT, PREC_FP64><<<B.grid, kTile, 0, stream>>>(D, n, loss);
                count_launch(2);
            }
        } else {
            if constexpr (sizeof(RT) == 4) {
                if (prec == PREC_FP32) k_outer<RT, KIND_PORTFOLIO, PREC_FP32><<<og, kTile, 0, stream>>>(D, n, 0);
                else k_outer<RT, KIND_PORTFOLIO, PREC_REF32><<<og, kTile, 0, stream>>>(D, n, 0);
                count_launch();
                if (prec == PREC_FP32 && L.ot.fast) {
                    if (L.ot.Q > 800) return cudaErrorInvalidValue;      // rows beyond the shared memory
                    // Tiles: long ones read the table less often, short ones fill the chip at few outer
                    // samples.  10^5 / 3 10^4 / 1.2 10^4 / 5000 / 1000 outer samples (10^4 to 10^5
                    // options), us: tile 16 1535 / 492 / 991 / 1085 / 520, tile 8 1578 / 518 / 931 / 948 / 378,
                    // tile 4 1647 / 530 / 969 / 865 / 306
                    if (n >= 20000) e = launch_full_loss_fast<16>(D, n, loss, stream);
                    else if (n >= 8000) e = launch_full_loss_fast<8>(D, n, loss, stream);
                    else e = launch_full_loss_fast<4>(D, n, loss, stream);
                } else {
                    if (prec == PREC_FP32) k_full_loss<RT, PREC_FP32><<<B.grid, kTile, 0, stream>>>(D, n, loss);
                    else k_full_loss<RT, PREC_REF32><<<B.grid, kTile, 0, stream>>>(D, n, loss);
                    count_launch();
                }
            }
        }
        if (e == cudaSuccess) e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(host_loss + done, loss, nb * sizeof(double), cudaMemcpyDeviceToHost, stream);
        if (e != cudaSuccess) return e;
        done += nb;
    }
    return cudaSuccess;
}

template cudaError_t outer_full_loss<float>(const OuterLevel<float>&, int, OuterBuffers&, double*, cudaStream_t);
template cudaError_t outer_full_loss<double>(const OuterLevel<double>&, int, OuterBuffers&, double*, cudaStream_t);

}  // namespace nmlmc

// ---- utility kernels: raw Threefry blocks and OUTER-layout normals ---------------------------
namespace nmlmc {

__global__ void k_threefry_blocks(const uint64_t* ctr, const uint64_t* key, uint64_t* out, uint64_t n) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t o0, o1;
        threefry2x64(ctr[2 * i], ctr[2 * i + 1], tf_key(key[2 * i], key[2 * i + 1]), o0, o1);
        out[2 * i] = o0;
        out[2 * i + 1] = o1;
    }
}

template <int PREC>
__global__ void k_outer_normals(uint64_t seed, uint64_t stream, uint32_t tag, uint64_t n, double* out) {
    const TfKey key = tf_key(seed, stream);
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < n; k += (uint64_t)gridDim.x * blockDim.x) {
        if (PREC == PREC_FP32) out[k] = (double)outer_normal_at<PREC_FP32, float>(key, tag, k);
        else out[k] = outer_normal_at<PREC_FP64, double>(key, tag, k);
    }
}

cudaError_t launch_threefry_blocks(const uint64_t* ctr, const uint64_t* key, uint64_t* out, uint64_t n,
                                   cudaStream_t s) {
    k_threefry_blocks<<<256, 256, 0, s>>>(ctr, key, out, n);
    return cudaGetLastError();
}

// Phi(x) of the FP32 Black-Scholes path (norm_cdf_fast, nmlmc_bs.cuh) on n points.
__global__ void k_norm_cdf_fast(const float* x, float* out, uint64_t n) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = norm_cdf_fast(x[i]);
}

cudaError_t launch_norm_cdf_fast(const float* x, float* out, uint64_t n, cudaStream_t s) {
    k_norm_cdf_fast<<<256, 256, 0, s>>>(x, out, n);
    return cudaGetLastError();
}

cudaError_t launch_outer_normals(int prec, uint64_t seed, uint64_t stream, uint32_t tag, uint64_t n,
                                 double* out, cudaStream_t s) {
    if (prec == PREC_FP32) k_outer_normals<PREC_FP32><<<256, 256, 0, s>>>(seed, stream, tag, n, out);
    else k_outer_normals<PREC_FP64><<<256, 256, 0, s>>>(seed, stream, tag, n, out);
    return cudaGetLastError();
}

}  // namespace nmlmc

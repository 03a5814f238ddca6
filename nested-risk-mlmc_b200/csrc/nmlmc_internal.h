// Host/device interface between the C-ABI layer (nmlmc_api.cu) and the kernels.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "nmlmc_common.cuh"

namespace nmlmc {

// One random_state of the CORE layout: 64-bit word position and the cached second normal.
struct CoreStream {
    uint64_t wpos;
    uint32_t saved, pad;
    double sval;
};
static_assert(sizeof(CoreStream) == 24, "CoreStream layout");

template <class RT>
struct CoreLaunch {
    uint32_t cores, ell;
    uint32_t subs;            // warps per core (set by launch_core)
    uint64_t outer_normals;   // inner normals per outer sample of a level with fixed counts (likewise)
    uint64_t M;
    uint64_t seed;
    bool fine_only, antithetic;
    double adaptive_r;
    CountParams cf, cc;
    ModelParams<RT> mp;
    OptionTable<RT> ot;
};

// `states`: the cores' stream states, `states_out`: those after the call (another buffer: a core's
// warps may start after its last one has ended).  `part`: core_part_words(cores) words, `counts`: core_counts(cores) zeroed counters (left zero),
// `out`: the level's 16 words (10 sums: phi_f moments, difference moments, work, path-limit flag; 6
// counts), in device or pinned host memory.
size_t core_part_words(uint32_t cores);
size_t core_counts(uint32_t cores);
cudaError_t launch_core(const CoreLaunch<float>& L, int kind, const CoreStream* states, CoreStream* states_out, uint64_t* part, uint32_t* counts,
                        uint64_t* out, TraceRec* trace, cudaStream_t stream);
cudaError_t launch_core(const CoreLaunch<double>& L, int kind, const CoreStream* states, CoreStream* states_out, uint64_t* part, uint32_t* counts,
                        uint64_t* out, TraceRec* trace, cudaStream_t stream);
// Per-option constants of the reference-arithmetic tables (RefOption), P records, and the Unbiased
// levels' weights, kPathLevels each.
cudaError_t launch_ref_records(const OptionTable<float>& t, RefOption<float>* out, float* lvl_w, float* lvl_wf,
                               cudaStream_t stream);
cudaError_t launch_ref_records(const OptionTable<double>& t, RefOption<double>* out, double* lvl_w, float* lvl_wf,
                               cudaStream_t stream);

// ---- OUTER layout (batched) ----------------------------------------------------------------
enum Prec : int { PREC_REF32 = 0, PREC_FP64 = 1, PREC_FP32 = 2 };

// Per-level launch description of the batched path.
template <class RT>
struct OuterLevel {
    uint32_t ell;
    uint64_t M;             // outer samples of this call
    uint64_t first_index;   // stream index of the first outer sample (OUTER layout key)
    uint64_t seed;
    bool fine_only, antithetic, adaptive_f, adaptive_c;
    uint32_t N0, chunk;     // chunk = inner samples per thread (phase_chunk: a power of two of them in each count)
    uint32_t variant;       // phase-kernel register/occupancy variant (FP32 path: 0, 1, 2)
    bool no_small;          // not as one kernel for few outer samples, whatever their number (level_is_small)
    bool no_fixed;          // nor as one for fixed counts (level_is_fixed)
    RT adaptive_r;
    CountParams cf, cc;
    ModelParams<RT> mp;
    OptionTable<RT> ot;
};

// Device work buffers of the batched path, sized for `cap` outer samples per batch.
struct OuterBuffers {
    uint64_t cap;
    uint32_t Q;
    void* Yv;                // RT[cap]       model Y / portfolio constant
    void* Rt;                // cap * Q slots of 8 bytes: portfolio R_tau rows (RT R, or the
                             // float pair (R, ln R) on the FP32 path)
    uint32_t* cnt_f;         // final fine count / chunk size (0 = undecided)
    uint32_t* cnt_c;
    uint32_t* lists;         // 4 * cap: fine/coarse round lists, ping-pong
    uint32_t* class_items;   // cap: items sorted by final class
    uint32_t* counters;      // device counters (see nmlmc_outer.cu)
    double* block_sums;      // per-CTA partial moments [grid][16]
    double* level_acc;       // the level's result [16] (device or pinned host memory), written by its last
                             // kernel: the sums of block_sums, entry 12 the path-limit flag
                             // (path-simulated portfolios, 0 otherwise)
    int grid;                // CTA slots of block_sums
    int slots;               // slots the current level uses (set per level)
    uint64_t* stamps;        // optional: %globaltimer at the level's begin and end [2] (as level_acc)
    // KIND_USER only (caller-written SAMPLER classes): the SAMPLER object of every outer sample
    // (its outer state, state_bytes each) and its workspace (ws_bytes each)
    void* user_state;
    void* user_ws;
    uint32_t state_bytes, ws_bytes;
    // optional CUDA-event timing of the phase kernel: called around each k_phase launch
    void (*prof_mark)(void* user, int end, cudaStream_t stream);
    void* prof_user;
};

// Inner samples per thread of the batched phases for a chosen chunk length (a power of two from 4
// dividing N0).  A tile of threads holds a power of two of chunks per outer sample, so the odd factor
// of an N0 that is no power of two goes into the chunk, about as long as the chosen one: N0 = 96 takes
// 4 chunks of 24 for 32.
inline uint32_t phase_chunk(uint32_t N0, uint32_t chunk) {
    uint32_t odd = N0;
    while (odd && !(odd & 1)) odd >>= 1;
    if (odd <= 1) return chunk;
    for (uint32_t f = 1; f < odd && chunk > 4; f <<= 1) chunk >>= 1;
    return chunk * odd;
}

// Whether a level call runs as one kernel, a warp per outer sample (k_small): while its warps'
// work, in units of one FP32 normal with 96 per phase for the sums and the decision (a phase of 32
// samples keeps 8 of 32 lanes busy), stays below what the launch sequence costs whatever its size —
// about 50 us for one phase, 105 to 200 us with pilots.  Measured on both sides of the lines (one
// kernel, sequence; the models' level 0 has since become k_fixed): model level 0, 6200 samples 47.8
// and 46.4 us; level 5, 12,500: 102 and 121 us; reference model level 3, 2600: 76 and 117 us; FP64
// level 3, 6200: 90 and 89 us; importance portfolio level 3, 10,400: 143 and 224 us.  Larger counts
// than 4096 (one phase: 2048) leave a single warp too long alone: model level 8, 12,000: 212 and
// 184 us.  An N0 that is no power of two stays with the sequence: its chunks are none either.
constexpr uint32_t kSmallMaxChunk = 32, kSmallMaxStocks = 256;
template <class RT>
bool level_is_small(const OuterLevel<RT>& L, int kind, int prec, const OuterBuffers& B) {
    if (kind == KIND_USER || (is_portfolio_kind(kind) && (L.ot.mixed || L.ot.Q > kSmallMaxStocks))) return false;
    if (B.prof_mark || L.chunk < 4 || L.chunk > kSmallMaxChunk || L.M > B.cap || (L.N0 & (L.N0 - 1))) return false;
    const uint64_t maxc = (L.fine_only || L.cf.max_count >= L.cc.max_count) ? L.cf.max_count : L.cc.max_count;
    const bool pilots = L.adaptive_f || L.adaptive_c;
    if (maxc > (pilots ? 4096u : 2048u)) return false;
    const uint64_t per = pilots ? 4 * 96 + 3 * L.cf.base_count : 96 + maxc;
    const uint64_t unit = (kind == KIND_REF_MODEL ? 2 : 1) * (prec == PREC_FP32 ? 1 : 2);
    return L.M * per * unit <= (pilots ? 6000000ull : is_portfolio_kind(kind) ? 1300000ull : 800000ull);
}

// Whether a level runs as k_fixed, a thread per outer sample: a model without pilots at up to
// kFixedChunks chunks per outer sample.  One chunk is one thread's work in the launch sequence too;
// more of them a thread takes one after another, so few outer samples leave the chip idle: at four
// chunks k_fixed and the sequence take, in us, FP32 reference model 5000 outer samples 32 and 29, 8000
// 32 and 29 to 34, 33,000 34 and 54; FP64 X = Y + Z 5000 42 and 29, 20,000 42 and 43, 300,000 202 and 212;
// FP64 reference model 5000 71 and 41, 33,000 73 and 67, 120,000 199 and 173, 300,000 386 and 388.
constexpr uint32_t kFixedChunks = 4;
template <class RT>
bool level_is_fixed(const OuterLevel<RT>& L, int kind, int prec) {
    if (kind != KIND_REF_MODEL && kind != KIND_SHIFT_MODEL) return false;
    if (L.no_fixed || L.adaptive_f || L.adaptive_c || (L.N0 & (L.N0 - 1))) return false;
    const uint64_t maxc = (L.fine_only || L.cf.max_count >= L.cc.max_count) ? L.cf.max_count : L.cc.max_count;
    const uint64_t nch = maxc / L.chunk;
    if (nch > kFixedChunks) return false;
    const uint64_t serial = nch * (kind == KIND_REF_MODEL ? 2 : 1);       // chunks of normals per thread
    if (nch <= 1) return true;
    if (prec == PREC_FP32) return serial <= 4 || L.M >= 8192;
    return L.M >= (serial <= 4 ? 16384u : 262144u);
}

// Device counter slot (OuterBuffers::counters) that the batched kernels set when a
// path-simulated inner sample would exceed kMaxPathSteps (the call then fails with
// NMLMC_ERR_LIMIT); k_outer clears it on a level's first batch.
constexpr uint32_t kCounterPathLimit = 240;

// Records a failed status for nmlmc_last_error() (this thread) and returns it.
int set_last_error(int e);

// Kernel launches issued by the library (incremented at every launch site).
void count_launch(uint64_t n = 1);
uint64_t launches_total();

template <class RT>
cudaError_t outer_sample_level(const OuterLevel<RT>& L, int kind, int prec, OuterBuffers& B,
                               TraceRec* trace, cudaStream_t stream);
// Zeroes the level's result: for levels without outer samples, which launch nothing.
cudaError_t outer_level_begin(OuterBuffers& B, cudaStream_t stream);

// Portfolio loss sweep L(Y) over all options (K-quantile precompute) into a host array; the copies
// are queued on the stream.
template <class RT>
cudaError_t outer_full_loss(const OuterLevel<RT>& L, int prec, OuterBuffers& B, double* host_loss, cudaStream_t stream);

// ---- path-simulated loss and its adjoint (nmlmc_adjoint.cu) --------------------------------
constexpr uint32_t kAdjMaxTile = 64;     // outer samples per CTA of the path kernels

template <class RT> struct Pair2;
template <> struct Pair2<float> { using type = float2; };
template <> struct Pair2<double> { using type = double2; };

// The caller's arrays on the device, as given (nmlmc_portfolio_batch).
struct AdjInputs {
    const double *S0, *mu, *sigma;                         // [stocks]
    const double *strike, *maturity, *w;                   // [options]
    const int32_t* type;                                   // [options]
    double r;
};

template <class RT>
struct AdjLaunch {
    uint32_t n, n_chunks, q_max;          // portfolios, option chunks of 128, max stocks per portfolio
    uint32_t n_options;
    uint32_t ell, pairs, tile;            // 2^ell steps, antithetic pairs, outer samples per CTA
    uint64_t M, seed;
    uint64_t m0, m1;                      // outer samples of a launch
    uint64_t m_store;                     // outer samples [0, m_store) whose derivatives are kept
    int milstein;
    RT r, rho, s1_rho2, tau, stau, disc_tau;
    const uint32_t *stock_off, *option_off, *chunk_off;   // [n + 1]
    RT *S0, *mu, *sigma;                                   // [stocks] (k_adj_setup)
    RT *strike, *maturity, *w, *V0, *vega;                 // [options] (k_adj_setup)
    const uint32_t* stock_ind;                             // [options], within the portfolio
    int8_t* type;                                          // [options] (k_adj_setup)
    typename Pair2<RT>::type* store;                       // [m_store][n_options] (dl/dw_i, dl/dsigma)
    const double *K, *delta;                               // [n]
    RT *R, *dR;                                            // [stocks * M], row (p, m) of Q_p values
    double *L, *omega, *est, *wE;                          // [n * M], [n * M], [3 n], [n]
    double *gw_E, *gw_P, *gs_E, *gs_P;                     // [options], [stocks]
};
cudaError_t launch_adjoint(const AdjLaunch<float>& A, const AdjInputs& in, bool grad, cudaStream_t stream);
cudaError_t launch_adjoint(const AdjLaunch<double>& A, const AdjInputs& in, bool grad, cudaStream_t stream);

cudaError_t launch_threefry_blocks(const uint64_t* ctr, const uint64_t* key, uint64_t* out, uint64_t n,
                                   cudaStream_t s);
cudaError_t launch_norm_cdf_fast(const float* x, float* out, uint64_t n, cudaStream_t s);
cudaError_t launch_outer_normals(int prec, uint64_t seed, uint64_t stream, uint32_t tag, uint64_t n,
                                 double* out, cudaStream_t s);

}  // namespace nmlmc

// The readout row (token 320) of the SISA block and the classifier head, fp32 in every mode, in two kernels around
// the attention kernel:
//
//   readout_qc    xl = rmsnorm(h[320]) * w;  [Q | C] = xl . W_qc^T                                 (before sisa_attn)
//   readout_tail  x1 = h[320] + Y . W_O^T;  x2 = x1 + down(silu(gate(n)) * up(n)), n = rmsnorm(x1) * w;
//                 z = rmsnorm(x2) * w;  logit = w2 . silu(W0 z + b0) + b2                           (after sisa_attn)
//
// Only row 320 leaves the SISA block, so this work is B rows, not 321 B (engine/cuda/engine.cu:451-469;
// engine/model/isa_impl.hpp:1092-1133).  A CTA takes TB clips (16 when the batch is large enough to give every SM a
// CTA that way, else 4, 2 or 1; up to about 120 clips eight CTAs share a batch's clips, see below) and walks the small
// matrix products one after the other with all activations of its clips in shared memory: a thread owns one or two output
// columns for all TB clips (TB or 2 TB accumulators), reads its weights coalesced from a [K][N] (transposed) copy that
// stays in L2, several steps of k in flight at a time, and the activations as 128-bit broadcast loads.  Every output is one fp32 FMA chain over k in ascending order, whatever the
// batch and whatever TB, so a clip's logit does not depend on its neighbours (engine/include/shv_cuda.h:31-34).
//
// Replaces two launch_rmsnorm, five gemm<float> and launch_head of the reference's run_classify
// (engine/cuda/engine.cu:451-469, engine/cuda/seq.cu:309-336).
#include "device_utils.cuh"
#include "shv_seq_kernels.h"

namespace sb {
namespace {

constexpr int XP = kD + 4, HP = kDFF + 4;     // row pitches (floats) of the shared-memory activation tiles

// acc[c][e] = sum_k X[c][k] * Wt[k][n0 + e], e < NC, for the TB clips of the tile; k ascending, one FMA chain per output.
template <int K, int NC, int TB>
__device__ __forceinline__ void dot_columns(const float* __restrict__ X, int xp, const float* __restrict__ Wt, int ldw, int n0,
                                            float (&acc)[TB][NC]) {
#pragma unroll
    for (int c = 0; c < TB; ++c)
#pragma unroll
        for (int e = 0; e < NC; ++e) acc[c][e] = 0.0f;
    const float* wp = Wt + n0;
    // The weights of D steps of four k are loaded before the first of them is used, so that D x 4 loads are in flight per
    // thread (with few clips per CTA the kernel is bound by the latency of exactly these loads).  This needs the registers
    // for them: the kernels are declared with a minimum number of CTAs per SM, because without one they get 32 to 37
    // registers (-Xptxas -v) and the steps run one L2 round trip after the other (B = 512: 0.27 ms for the tail kernel against
    // 0.14 ms).
    constexpr int D = TB >= 8 ? 4 : 8;
    static_assert(K % (4 * D) == 0, "the k loop walks whole groups of steps");
#pragma unroll 1
    for (int k0 = 0; k0 < K; k0 += 4 * D) {
        float w[D][4][NC];
#pragma unroll
        for (int d = 0; d < D; ++d)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if constexpr (NC == 2) {
                    const float2 v = __ldg(reinterpret_cast<const float2*>(wp + (long long)(k0 + 4 * d + i) * ldw));
                    w[d][i][0] = v.x; w[d][i][1] = v.y;
                } else {
                    w[d][i][0] = __ldg(wp + (long long)(k0 + 4 * d + i) * ldw);
                }
            }
#pragma unroll
        for (int d = 0; d < D; ++d)
#pragma unroll
            for (int c = 0; c < TB; ++c) {
                const float4 x = *reinterpret_cast<const float4*>(X + c * xp + k0 + 4 * d);
#pragma unroll
                for (int e = 0; e < NC; ++e) {
                    acc[c][e] = fmaf(x.x, w[d][0][e], acc[c][e]);
                    acc[c][e] = fmaf(x.y, w[d][1][e], acc[c][e]);
                    acc[c][e] = fmaf(x.z, w[d][2][e], acc[c][e]);
                    acc[c][e] = fmaf(x.w, w[d][3][e], acc[c][e]);
                }
            }
    }
}

// out[c] = (in[c] * (1 / sqrt(mean(in[c]^2) + 1e-6))) * w over rows of 384 in shared memory; warp w takes clips w, w + 8.
// A row is read into registers before it is written, so out may be in.
template <int TB, int NT>
__device__ __forceinline__ void norm_rows(const float* in, float* out, const float* __restrict__ w, int warp, int lane) {
    for (int c = warp; c < TB; c += NT / 32) {
        float v[kD / 32];
        float ss = 0.0f;
#pragma unroll
        for (int i = 0; i < kD / 32; ++i) {
            v[i] = in[c * XP + lane + 32 * i];
            ss = fmaf(v[i], v[i], ss);
        }
        ss = warp_sum(ss);
        const float r = 1.0f / sqrtf(ss / float(kD) + 1e-6f);
#pragma unroll
        for (int i = 0; i < kD / 32; ++i) out[c * XP + lane + 32 * i] = (v[i] * r) * __ldg(w + lane + 32 * i);
    }
}

template <int TB, int NT>
__global__ void __launch_bounds__(NT, NT <= 256 ? 2 : 1)
readout_qc_kernel(const float* __restrict__ h_last, long long ldh, const float* __restrict__ norm_w, const float* __restrict__ wqc_t,
                  float* __restrict__ QC, int B) {
    __shared__ __align__(16) float xs[TB * XP];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int clip0 = blockIdx.x * TB;
    for (int i = tid; i < TB * kD; i += NT) {
        const int c = i / kD, k = i - c * kD;
        xs[c * XP + k] = clip0 + c < B ? h_last[(long long)(clip0 + c) * ldh + k] : 0.0f;
    }
    __syncthreads();
    norm_rows<TB, NT>(xs, xs, norm_w, warp, lane);
    __syncthreads();
    for (int n0 = 2 * tid; n0 < kSQN; n0 += 2 * NT) {          // 576 columns = 288 pairs
        float acc[TB][2];
        dot_columns<kD, 2, TB>(xs, XP, wqc_t, kSQN, n0, acc);
#pragma unroll
        for (int c = 0; c < TB; ++c)
            if (clip0 + c < B) *reinterpret_cast<float2*>(QC + (long long)(clip0 + c) * kSQN + n0) = make_float2(acc[c][0], acc[c][1]);
    }
}

struct TailWeights {
    const float *wo_t;          // [384][384]   W_O transposed
    const float *ffn_norm_w;    // [384]
    const float *up_t;          // [384][1920]  gate / up rows interleaved (2j, 2j + 1), transposed
    const float *down_t;        // [960][384]   down projection transposed
    const float *final_norm_w;  // [384]
    const float *head_w0_t;     // [384][128]   head.0 transposed
    const float *head_b0;       // [128]
    const float *head_w2;       // [128]
    const float *head_b2;       // [1]
};

template <int TB, int NT>
__global__ void __launch_bounds__(NT, NT <= 256 ? 2 : 1)
readout_tail_kernel(const float* __restrict__ Y, const float* __restrict__ h_last, long long ldh, const TailWeights tw,
                    float* __restrict__ x2_out, float* __restrict__ logits, int B) {
    extern __shared__ __align__(16) float tail_smem[];
    float* x1 = tail_smem;                  // [TB][XP]  residual stream of the row
    float* xa = x1 + TB * XP;               // [TB][XP]  attention output, then normalised rows
    float* hid = xa + TB * XP;              // [TB][HP]  SwiGLU product; later the head's hidden layer [TB][128]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int clip0 = blockIdx.x * TB;
    for (int i = tid; i < TB * kD; i += NT) {
        const int c = i / kD, k = i - c * kD;
        const bool live = clip0 + c < B;
        xa[c * XP + k] = live ? Y[(long long)(clip0 + c) * kD + k] : 0.0f;
        x1[c * XP + k] = live ? h_last[(long long)(clip0 + c) * ldh + k] : 0.0f;
    }
    __syncthreads();
    // x1 = h + Y . W_O^T: 192 column pairs
    float keep[TB][2];
    if (tid < kD / 2) {
        dot_columns<kD, 2, TB>(xa, XP, tw.wo_t, kD, 2 * tid, keep);
#pragma unroll
        for (int c = 0; c < TB; ++c) {
            float2* p = reinterpret_cast<float2*>(x1 + c * XP + 2 * tid);
            const float2 r = *p;
            *p = make_float2(r.x + keep[c][0], r.y + keep[c][1]);
        }
    }
    __syncthreads();
    norm_rows<TB, NT>(x1, xa, tw.ffn_norm_w, warp, lane);
    __syncthreads();
    // hid[j] = silu(gate_j) * up_j: 960 (gate, up) column pairs
    for (int j = tid; j < kDFF; j += NT) {
        float acc[TB][2];
        dot_columns<kD, 2, TB>(xa, XP, tw.up_t, 2 * kDFF, 2 * j, acc);
#pragma unroll
        for (int c = 0; c < TB; ++c) hid[c * HP + j] = silu_f(acc[c][0]) * acc[c][1];
    }
    __syncthreads();
    // x2 = x1 + hid . W_down^T
    if (tid < kD / 2) {
        dot_columns<kDFF, 2, TB>(hid, HP, tw.down_t, kD, 2 * tid, keep);
#pragma unroll
        for (int c = 0; c < TB; ++c) {
            float2* p = reinterpret_cast<float2*>(x1 + c * XP + 2 * tid);
            const float2 r = *p;
            const float2 v = make_float2(r.x + keep[c][0], r.y + keep[c][1]);
            *p = v;
            if (x2_out && clip0 + c < B) *reinterpret_cast<float2*>(x2_out + (long long)(clip0 + c) * kD + 2 * tid) = v;
        }
    }
    __syncthreads();
    norm_rows<TB, NT>(x1, xa, tw.final_norm_w, warp, lane);
    __syncthreads();
    // head: 128 hidden units (one column per thread of the first four warps), then their weighted sum per clip
    float* hh = hid;                         // [TB][128]; the SwiGLU product is consumed
    if (tid < 128) {
        float acc[TB][1];
        dot_columns<kD, 1, TB>(xa, XP, tw.head_w0_t, 128, tid, acc);
        const float b0 = __ldg(tw.head_b0 + tid), w2 = __ldg(tw.head_w2 + tid);
#pragma unroll
        for (int c = 0; c < TB; ++c) hh[c * 128 + tid] = w2 * silu_f(acc[c][0] + b0);
    }
    __syncthreads();
    for (int c = warp; c < TB; c += NT / 32) {
        const float s = warp_sum((hh[c * 128 + lane] + hh[c * 128 + lane + 32]) + (hh[c * 128 + lane + 64] + hh[c * 128 + lane + 96]));
        if (lane == 0 && clip0 + c < B) logits[clip0 + c] = s + __ldg(tw.head_b2);
    }
}

// ---------------------------------------------------------------------------------------------------- small batches
// The two kernels above keep a clip's whole row on one SM, which then reads all 5.2 MB (0.9 MB) of the matrices, and with one
// clip per SM waits for most of those loads: 81 us (23 us) whether the batch has 45 clips or 128.  Here eight SMs share TB
// clips: each takes an eighth of the columns of every product for all of them.  Its slices of the matrices stream through
// a ring of shared-memory chunks (cp.async, up to three chunks of 23 to 30 KB ahead, across the products: nothing of them
// depends on the data), and the eight hand each other their outputs through distributed shared memory, a buffer per
// hand-over, so that a cluster barrier between products is all they need.  An output is the same FMA chain over k.
constexpr int CL = 8, NTC = 256, RING = 4, CHUNK_BYTES = 30720;
constexpr int WO_C = kD / CL, UP_C = 2 * kDFF / CL, HEAD_C = 128 / CL, QC_C = kSQN / CL;         // columns of one SM: 48, 240, 16, 72
constexpr int WO_K = 128, UP_K = 32, DN_K = 120, HEAD_K = kD, QC_K = 96;                           // k rows of a chunk
constexpr int G_UP = kD / WO_K, G_DN = G_UP + kD / UP_K, G_HEAD = G_DN + kDFF / DN_K, G_END = G_HEAD + 1;   // first chunk of a product
static_assert(WO_K * WO_C * 4 <= CHUNK_BYTES && UP_K * UP_C * 4 <= CHUNK_BYTES && DN_K * WO_C * 4 <= CHUNK_BYTES &&
              HEAD_K * HEAD_C * 4 <= CHUNK_BYTES && QC_K * QC_C * 4 <= CHUNK_BYTES, "chunks");
static_assert(kD % WO_K == 0 && kD % UP_K == 0 && kDFF % DN_K == 0 && kD % QC_K == 0, "chunks");

__device__ __forceinline__ uint32_t smem_of(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void cp16(uint32_t dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// a float (pair) into the same place of every block of the cluster
__device__ __forceinline__ uint32_t peer_of(uint32_t local, int rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
    return remote;
}
__device__ __forceinline__ void share2(float* p, float a, float b) {
#pragma unroll
    for (int r = 0; r < CL; ++r)
        asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(peer_of(smem_of(p), r)), "f"(a), "f"(b) : "memory");
}
__device__ __forceinline__ void share1(float* p, float a) {
#pragma unroll
    for (int r = 0; r < CL; ++r) asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(peer_of(smem_of(p), r)), "f"(a) : "memory");
}

// rows [KC][COLS] of a [K][ldw] matrix into a chunk
template <int COLS, int KC> __device__ __forceinline__ void fetch_chunk(uint32_t dst, const float* src, int ldw, int tid) {
    constexpr int V = COLS / 4;
    for (int i = tid; i < KC * V; i += NTC) cp16(dst + uint32_t(i) * 16u, src + (long long)(i / V) * ldw + i % V * 4);
}
// One product's share of a thread: TPC clips of a column pair.  A block's pairs are dealt to the threads first, the clips to
// as many groups of threads as there are.
template <int COLS, int TB> struct Share {
    static constexpr int PAIRS = COLS / 2, MAXG = NTC / PAIRS, GROUPS = TB <= 4 && TB < MAXG ? TB : MAXG >= 4 ? 4 : MAXG >= 2 ? 2 : 1;
    static constexpr int TPC = TB / GROUPS;
    static_assert(TB % GROUPS == 0 && PAIRS * GROUPS <= NTC, "clips per thread");
    int pair, clip;
    bool active;
    __device__ explicit Share(int tid) : pair(tid % PAIRS), clip(tid / PAIRS * TPC), active(tid < PAIRS * GROUPS) {}
};
// acc[c][e] += sum over a chunk's k of X[c][k] W[k][pair]; k ascending
template <int COLS, int KC, int TPC>
__device__ __forceinline__ void chunk_product(const float* w, const float* x, int xp, float (&acc)[TPC][2]) {
    // 32 (40) k in flight, a chunk in whole groups: with 16 a classify of one window takes 211 us instead of 209; with the next
    // group's operands asked for ahead, through a second set of registers, 215
    constexpr int UNROLL = KC % 120 ? 8 : 10;
#pragma unroll UNROLL
    for (int k = 0; k < KC; k += 4) {
        float2 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = *reinterpret_cast<const float2*>(w + (k + i) * COLS);
#pragma unroll
        for (int c = 0; c < TPC; ++c) {
            const float4 q = *reinterpret_cast<const float4*>(x + c * xp + k);
            acc[c][0] = fmaf(q.x, v[0].x, acc[c][0]); acc[c][1] = fmaf(q.x, v[0].y, acc[c][1]);
            acc[c][0] = fmaf(q.y, v[1].x, acc[c][0]); acc[c][1] = fmaf(q.y, v[1].y, acc[c][1]);
            acc[c][0] = fmaf(q.z, v[2].x, acc[c][0]); acc[c][1] = fmaf(q.z, v[2].y, acc[c][1]);
            acc[c][0] = fmaf(q.w, v[3].x, acc[c][0]); acc[c][1] = fmaf(q.w, v[3].y, acc[c][1]);
        }
    }
}
template <int K, int COLS, int KC, int TB, typename Fetch>
__device__ __forceinline__ void stream_product(const Share<COLS, TB>& sh, int g0, const Fetch& fetch, const float* ring, const float* x, int xp,
                                               float (&acc)[Share<COLS, TB>::TPC][2]) {
    constexpr int TPC = Share<COLS, TB>::TPC;
#pragma unroll
    for (int c = 0; c < TPC; ++c) { acc[c][0] = 0.0f; acc[c][1] = 0.0f; }
    for (int c = 0; c < K / KC; ++c) {
        const int g = g0 + c;
        cp_wait<RING - 2>();                              // this thread's part of chunk g has landed
        __syncthreads();                                  // everyone's has, and chunk g - 1 is consumed
        fetch(g + RING - 1);
        if (sh.active) chunk_product<COLS, KC, TPC>(ring + (g % RING) * (CHUNK_BYTES / 4) + 2 * sh.pair, x + sh.clip * xp + c * KC, xp, acc);
    }
}

template <int TB>
__global__ void __launch_bounds__(NTC, 1)
readout_qc_split_kernel(const float* __restrict__ h_last, long long ldh, const float* __restrict__ norm_w, const float* __restrict__ wqc_t,
                        float* __restrict__ QC, int B) {
    extern __shared__ __align__(16) float split_smem[];
    float* ring = split_smem;
    float* xs = ring + RING * CHUNK_BYTES / 4;                // [TB][XP]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = blockIdx.x % CL;
    const int clip0 = int(blockIdx.x / CL) * TB;
    auto fetch = [&](int g) {
        if (g < kD / QC_K)
            fetch_chunk<QC_C, QC_K>(smem_of(ring) + uint32_t(g % RING) * CHUNK_BYTES, wqc_t + (long long)g * QC_K * kSQN + rank * QC_C, kSQN, tid);
        cp_commit();
    };
    for (int g = 0; g < RING - 1; ++g) fetch(g);
    for (int i = tid; i < TB * kD; i += NTC) {
        const int c = i / kD, k = i - c * kD;
        xs[c * XP + k] = clip0 + c < B ? h_last[(long long)(clip0 + c) * ldh + k] : 0.0f;
    }
    __syncthreads();
    norm_rows<TB, NTC>(xs, xs, norm_w, warp, lane);
    const Share<QC_C, TB> sh(tid);
    float acc[Share<QC_C, TB>::TPC][2];
    stream_product<kD, QC_C, QC_K, TB>(sh, 0, fetch, ring, xs, XP, acc);
    if (sh.active)
#pragma unroll
        for (int c = 0; c < Share<QC_C, TB>::TPC; ++c)
            if (clip0 + sh.clip + c < B)
                *reinterpret_cast<float2*>(QC + (long long)(clip0 + sh.clip + c) * kSQN + rank * QC_C + 2 * sh.pair) = make_float2(acc[c][0], acc[c][1]);
}

template <int TB>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(NTC, 1)
readout_tail_split_kernel(const float* __restrict__ Y, const float* __restrict__ h_last, long long ldh, const TailWeights tw,
                          float* __restrict__ x2_out, float* __restrict__ logits, int B) {
    extern __shared__ __align__(16) float split_smem[];
    float* ring = split_smem;
    float* ya = ring + RING * CHUNK_BYTES / 4;                // [TB][XP]  attention output
    float* xb = ya + TB * XP;                                 // [TB][XP]  x1, then normalised
    float* xc = xb + TB * XP;                                 // [TB][XP]  x2, then normalised
    float* hid = xc + TB * XP;                                // [TB][HP]  SwiGLU product
    float* hh = hid + TB * HP;                                // [TB][128] head's hidden layer (block 0 of the cluster)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = blockIdx.x % CL;
    const int clip0 = int(blockIdx.x / CL) * TB;
    auto fetch = [&](int g) {
        const uint32_t dst = smem_of(ring) + uint32_t(g % RING) * CHUNK_BYTES;
        if (g < G_UP) fetch_chunk<WO_C, WO_K>(dst, tw.wo_t + (long long)g * WO_K * kD + rank * WO_C, kD, tid);
        else if (g < G_DN) fetch_chunk<UP_C, UP_K>(dst, tw.up_t + (long long)(g - G_UP) * UP_K * (2 * kDFF) + rank * UP_C, 2 * kDFF, tid);
        else if (g < G_HEAD) fetch_chunk<WO_C, DN_K>(dst, tw.down_t + (long long)(g - G_DN) * DN_K * kD + rank * WO_C, kD, tid);
        else if (g < G_END) fetch_chunk<HEAD_C, HEAD_K>(dst, tw.head_w0_t + rank * HEAD_C, 128, tid);
        cp_commit();
    };
    for (int g = 0; g < RING - 1; ++g) fetch(g);
    for (int i = tid; i < TB * kD; i += NTC) {
        const int c = i / kD, k = i - c * kD;
        ya[c * XP + k] = clip0 + c < B ? Y[(long long)(clip0 + c) * kD + k] : 0.0f;
    }
    const Share<WO_C, TB> so(tid);
    float x1[Share<WO_C, TB>::TPC][2], acc[Share<WO_C, TB>::TPC][2];   // this thread's columns of the residual row
#pragma unroll
    for (int c = 0; c < Share<WO_C, TB>::TPC; ++c) {
        const int clip = clip0 + so.clip + c;
        const float2 r = so.active && clip < B ? *reinterpret_cast<const float2*>(h_last + (long long)clip * ldh + rank * WO_C + 2 * so.pair)
                                               : make_float2(0.0f, 0.0f);
        x1[c][0] = r.x; x1[c][1] = r.y;
    }
    cluster_sync();                                           // every block of the cluster runs: its shared memory may be written
    // x1 = h + Y . W_O^T
    stream_product<kD, WO_C, WO_K, TB>(so, 0, fetch, ring, ya, XP, acc);
    if (so.active)
#pragma unroll
        for (int c = 0; c < Share<WO_C, TB>::TPC; ++c) {
            x1[c][0] += acc[c][0]; x1[c][1] += acc[c][1];
            share2(xb + (so.clip + c) * XP + rank * WO_C + 2 * so.pair, x1[c][0], x1[c][1]);
        }
    cluster_sync();
    norm_rows<TB, NTC>(xb, xb, tw.ffn_norm_w, warp, lane);
    // hid[j] = silu(gate_j) * up_j  (the product's first barrier orders it behind the norm)
    {
        const Share<UP_C, TB> su(tid);
        float u[Share<UP_C, TB>::TPC][2];
        stream_product<kD, UP_C, UP_K, TB>(su, G_UP, fetch, ring, xb, XP, u);
        if (su.active)
#pragma unroll
            for (int c = 0; c < Share<UP_C, TB>::TPC; ++c) share1(hid + (su.clip + c) * HP + rank * (UP_C / 2) + su.pair, silu_f(u[c][0]) * u[c][1]);
    }
    cluster_sync();
    // x2 = x1 + hid . W_down^T
    stream_product<kDFF, WO_C, DN_K, TB>(so, G_DN, fetch, ring, hid, HP, acc);
    if (so.active)
#pragma unroll
        for (int c = 0; c < Share<WO_C, TB>::TPC; ++c) {
            const float a = x1[c][0] + acc[c][0], b = x1[c][1] + acc[c][1];
            share2(xc + (so.clip + c) * XP + rank * WO_C + 2 * so.pair, a, b);
            const int clip = clip0 + so.clip + c;
            if (x2_out && clip < B) *reinterpret_cast<float2*>(x2_out + (long long)clip * kD + rank * WO_C + 2 * so.pair) = make_float2(a, b);
        }
    cluster_sync();
    norm_rows<TB, NTC>(xc, xc, tw.final_norm_w, warp, lane);
    // head: 128 hidden units, then their weighted sum per clip on the cluster's first block
    {
        const Share<HEAD_C, TB> sh(tid);
        float u[Share<HEAD_C, TB>::TPC][2];
        stream_product<kD, HEAD_C, HEAD_K, TB>(sh, G_HEAD, fetch, ring, xc, XP, u);
        const int o = rank * HEAD_C + 2 * sh.pair;
        if (sh.active)
#pragma unroll
            for (int c = 0; c < Share<HEAD_C, TB>::TPC; ++c) {
                const float a = __ldg(tw.head_w2 + o) * silu_f(u[c][0] + __ldg(tw.head_b0 + o));
                const float b = __ldg(tw.head_w2 + o + 1) * silu_f(u[c][1] + __ldg(tw.head_b0 + o + 1));
                asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};"
                             ::"r"(peer_of(smem_of(hh + (sh.clip + c) * 128 + o), 0)), "f"(a), "f"(b) : "memory");
            }
    }
    cluster_sync();
    if (rank == 0)
        for (int c = warp; c < TB; c += NTC / 32) {
            const float s = warp_sum((hh[c * 128 + lane] + hh[c * 128 + lane + 32]) + (hh[c * 128 + lane + 64] + hh[c * 128 + lane + 96]));
            if (lane == 0 && clip0 + c < B) logits[clip0 + c] = s + __ldg(tw.head_b2);
        }
}
constexpr int qc_split_smem(int tb) { return RING * CHUNK_BYTES + tb * XP * 4; }
constexpr int tail_split_smem(int tb) { return RING * CHUNK_BYTES + tb * (3 * XP + HP + 128) * 4; }
static_assert(tail_split_smem(8) <= 232448, "shared memory");

constexpr int tail_smem_bytes(int tb) { return (2 * tb * XP + tb * HP) * int(sizeof(float)); }

// How the clips of a batch of B are dealt out: `tb` to a cluster of eight blocks (split) or to one block.  As long as one
// wave of clusters holds the batch (about 15 of them on a B200: 120 clips) it is split, with as few clips to a cluster as that
// allows; tail kernel in us, split / one block: 1 clip 28 / 43, 45 clips 36 / 82, 96 clips 43 / 82, but 128 clips (two
// waves) 83 / 81.  Above, a block takes 16 clips once that still gives every SM one, else 4, 2 (the few hundred clips of a
// pipeline batch: at 512 two clips per block 87 us, one 144, four 108) or 1.
// The split form copies the matrices 16 bytes at a time and reads the residual row in pairs (`may_split`: they are aligned for
// that); the one-block form wants 8 bytes of the matrices and nothing of the row.  Both give the same bits.
struct ReadoutShape { int tb; bool split; };
inline bool aligned_to(const void* p, uintptr_t bytes) { return (reinterpret_cast<uintptr_t>(p) & (bytes - 1)) == 0; }
ReadoutShape readout_shape(int B, bool may_split) {
    const int sms = device_sms();
    if ((B + 7) / 8 > sms / CL) may_split = false;     // no more clusters than that fit, whatever the answer below
    int clusters = 0;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(sms / CL) * CL);
    cfg.blockDim = dim3(NTC);
    cfg.dynamicSmemBytes = tail_split_smem(8);
    if (may_split && (cudaFuncSetAttribute(readout_tail_split_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, tail_split_smem(8)) != cudaSuccess ||
                      cudaOccupancyMaxActiveClusters(&clusters, readout_tail_split_kernel<8>, &cfg) != cudaSuccess)) {
        cudaGetLastError();
        clusters = 0;
    }
    for (int tb = 1; may_split && tb <= 8; tb *= 2)
        if ((B + tb - 1) / tb <= clusters) return {tb, true};
    return {B >= 16 * sms ? 16 : B >= 4 * sms ? 4 : B >= 2 * sms ? 2 : 1, false};
}

template <int TB, bool SPLIT>
int launch_qc(const float* h_last, long long ldh, const float* norm_w, const float* wqc_t, float* QC, int B, cudaStream_t s) {
    const unsigned groups = unsigned((B + TB - 1) / TB);
    if constexpr (SPLIT) {
        const cudaError_t e = cudaFuncSetAttribute(readout_qc_split_kernel<TB>, cudaFuncAttributeMaxDynamicSharedMemorySize, qc_split_smem(TB));
        if (e != cudaSuccess) return int(e);
        readout_qc_split_kernel<TB><<<groups * CL, NTC, qc_split_smem(TB), s>>>(h_last, ldh, norm_w, wqc_t, QC, B);
    } else {
        readout_qc_kernel<TB, 256><<<groups, 256, 0, s>>>(h_last, ldh, norm_w, wqc_t, QC, B);
    }
    return int(cudaGetLastError());
}
template <int TB, bool SPLIT>
int launch_tail(const float* Y, const float* h_last, long long ldh, const TailWeights& tw, float* x2_out, float* logits, int B,
                cudaStream_t s) {
    const unsigned groups = unsigned((B + TB - 1) / TB);
    if constexpr (SPLIT) {
        const cudaError_t e = cudaFuncSetAttribute(readout_tail_split_kernel<TB>, cudaFuncAttributeMaxDynamicSharedMemorySize, tail_split_smem(TB));
        if (e != cudaSuccess) return int(e);
        readout_tail_split_kernel<TB><<<groups * CL, NTC, tail_split_smem(TB), s>>>(Y, h_last, ldh, tw, x2_out, logits, B);
    } else {
        const cudaError_t e = cudaFuncSetAttribute(readout_tail_kernel<TB, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize, tail_smem_bytes(TB));
        if (e != cudaSuccess) return int(e);
        readout_tail_kernel<TB, 256><<<groups, 256, tail_smem_bytes(TB), s>>>(Y, h_last, ldh, tw, x2_out, logits, B);
    }
    return int(cudaGetLastError());
}

// the shapes that are compiled
#define SHVK_READOUT_SHAPES(X) X(16, false) X(4, false) X(2, false) X(1, false) X(8, true) X(4, true) X(2, true) X(1, true)

}  // namespace
}  // namespace sb

extern "C" int shvk_readout_qc(const float* h_last, long long ldh, const float* norm_w, const float* wqc_t, float* QC, int B,
                               void* stream) {
    if (B <= 0) return 0;
    if (!h_last || !norm_w || !wqc_t || !QC) return int(cudaErrorInvalidValue);
    cudaStream_t s = cudaStream_t(stream);
    const sb::ReadoutShape sh = sb::readout_shape(B, sb::aligned_to(wqc_t, 16));
    switch (2 * sh.tb + sh.split) {
#define X(TB, SPLIT) case 2 * TB + SPLIT: return sb::launch_qc<TB, SPLIT>(h_last, ldh, norm_w, wqc_t, QC, B, s);
        SHVK_READOUT_SHAPES(X)
#undef X
        default: return int(cudaErrorInvalidValue);
    }
}

extern "C" int shvk_readout_tail(const float* Y, const float* h_last, long long ldh, const shvk_readout_weights* w, float* x2_out,
                                 float* logits, int B, void* stream) {
    if (B <= 0) return 0;
    if (!Y || !h_last || !w || !logits) return int(cudaErrorInvalidValue);
    const sb::TailWeights tw{w->wo_t, w->ffn_norm_w, w->up_t, w->down_t, w->final_norm_w, w->head_w0_t, w->head_b0, w->head_w2, w->head_b2};
    cudaStream_t s = cudaStream_t(stream);
    const bool may_split = sb::aligned_to(w->wo_t, 16) && sb::aligned_to(w->up_t, 16) && sb::aligned_to(w->down_t, 16) &&
                           sb::aligned_to(w->head_w0_t, 16) && sb::aligned_to(h_last, 8) && (ldh & 1) == 0;
    const sb::ReadoutShape sh = sb::readout_shape(B, may_split);
    switch (2 * sh.tb + sh.split) {
#define X(TB, SPLIT) case 2 * TB + SPLIT: return sb::launch_tail<TB, SPLIT>(Y, h_last, ldh, tw, x2_out, logits, B, s);
        SHVK_READOUT_SHAPES(X)
#undef X
        default: return int(cudaErrorInvalidValue);
    }
}

// Long-sequence gated delta rule in chunked (WY / UT-transform) form on the tensor cores.
//
//   S_t = exp(g_t) S_{t-1} + k_t u_t^T,  u_t = beta_t (v_t - exp(g_t) S_{t-1}^T k_t),  o_t = S_t^T (scale q_t),  S_0 = 0
// for q, k [B,T,H,DK] (already L2-normalised, bf16), v [B,T,H,128] (bf16), log decay g and beta [B,T,H] (fp32): the
// recurrence of the reference's oracle (oracle/shieldv_ref.py:121-139, gated_delta_rule_recurrent), which the reference
// engines only evaluate token by token at T = 321 (engine/cuda/seq.cu:107-195).  This entry point is the long-T form.
//
// Per block of 16 tokens, with inclusive cumulative log decay c_i, e_i = exp(c_i), state S0 entering the block:
//     L_ij = beta_i exp(c_i - c_j) (k_i . k_j)  (j < i),  T2 = (I + L)^-1 diag(beta),  M_ij = scale exp(c_i - c_j) (q_i . k_j)  (j <= i)
//     R = K S0,  U = T2 (V - diag(e) R),  O = M U + diag(scale e) Q S0,  S' = e_16 S0 + K^T diag(exp(c_16 - c_j)) U.
// T2 and M do not depend on the state, only R, U, O and S' do.  Two kernels, chunk-parallel where the algebra allows:
//
//   prep   one warp per two blocks (per block while that is a single wave of warps), all B x H x T/16 blocks at once: the two
//          Gram products on mma.sync, the decay masks, the 16 x 16 triangular inverse (forward substitution over 16 lanes, both
//          blocks at once), T2 and M as bf16 tiles and the decays' exponentials into a workspace of 1,152 bytes per block
//   scan   one CTA per (batch, head), or two or four with a share of the value columns each where sequences are few (with warps of
//          their own for the state and for the outputs: gdn_chunked_chain_kernel), walks the blocks with the state
//          resident: per block only the chain R -> U -> O and the state update remain, every operand fragment read straight
//          out of the staged K, Q, V, T2, M tiles with ldmatrix (tiles arrive by cp.async into a ring of three or four slots,
//          two or three blocks ahead, XOR-swizzled so the fragment reads are conflict-free), one CTA barrier per block, the
//          previous block's output rows written while the next block's products run
//
// The value dimension (128) is the MMA row dimension and is split over the warps of the scan CTA: four warps of 32
// columns for DK = 64, eight warps of 16 columns for DK = 128, so that a warp's slice of S^T is 64 fp32 registers per lane
// in both cases (a sequence shared by two CTAs: four warps of 16 columns each); the hand-over between the products of a block stays in registers (the accumulator layout of one is the
// A-operand layout of the next).  Operands are bf16, the state and all accumulation fp32.  A caller's chunk size (e.g.
// 64) only groups these 16-token blocks: the result does not depend on it.
//
// Why not tcgen05 here: the chain of a block is three dependent products on 16-token tiles; tcgen05 wants M >= 64 rows
// per instruction and an asynchronous issue / commit / tensor-memory round trip per link.  With the state-independent
// half of the work moved into the chunk-parallel kernel, the sequential kernel is bound by the latency of that chain,
// not by the tensor pipe, and the whole computation by HBM (141 to 177 flop per byte, below the machine's ridge).
#include "device_utils.cuh"
#include "shv_seq_kernels.h"

namespace sb {
namespace {

constexpr int CB = 16;                       // tokens per block
constexpr int CDV = 128;
// workspace block: T2 | M (bf16 16 x 16) | exp(c_i) | exp(c_16 - c_i) (fp32 16 each)
constexpr int WS_T2 = 0, WS_M = 512, WS_EG = 1024, WS_DJ = 1088, WS_BLOCK = 1152;
constexpr int OT_PITCH = CDV + 4;            // floats per token row of the o tile (fragment stores fall into 32 banks)

__device__ __forceinline__ uint32_t cpack(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ void cmma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }
// 16-byte asynchronous copy global -> shared; `bytes` = 16, or 0 to fill the destination with zeros (tokens past T)
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A tile of 16 token rows of ROWB bytes in shared memory: the 16-byte chunk c of row r sits at chunk c ^ (r & 7), so the
// eight rows of one ldmatrix read (same chunk column) fall into eight different bank groups.
template <int ROWB> __device__ __forceinline__ uint32_t tile_off(int row, int chunk) {
    return uint32_t(row * ROWB + ((chunk ^ (row & 7)) << 4));
}

// ---------------------------------------------------------------------------------------------------- prep kernel
// A warp takes two blocks: their Gram products and masks one after the other on all 32 lanes (the second block's rows are
// fetched meanwhile), then both triangular inverses at once, a half-warp each, rows of L read 128 bits at a time.  The
// kernel is bound by issue and shared-memory latency, not by its 250 MB (64 x 2,048 tokens, 6 heads); with one block a warp
// everywhere both kernels take 259 us there against 248.
// (declared with a minimum of CTAs per SM: without one the kernel gets 40-48 registers)
constexpr int LF_PITCH = CB + 4, LF_SLOT = CB * LF_PITCH + 16;    // floats; the two slots start 16 banks apart
template <int DK> struct PrepWarp {
    __align__(16) uint8_t k[CB * DK * 2], q[CB * DK * 2];
    __align__(16) float lf[2 * LF_SLOT];
    float cum[CB], beta[2][CB];
    __align__(16) uint8_t out[2][WS_BLOCK];
};
template <int DK>
__global__ void __launch_bounds__(128, 4)
gdn_chunked_prep_kernel(const __nv_bfloat16* __restrict__ Q, const __nv_bfloat16* __restrict__ K, const float* __restrict__ G,
                        const float* __restrict__ Beta, uint8_t* __restrict__ ws, int T, int H, int NB, long long blocks,
                        int per, float scale) {
    constexpr int ROWB = DK * 2, VPR = DK / 8, KSTEP = DK / 16, VEC = CB * VPR / 32;     // bytes and 16-byte vectors per tile row
    extern __shared__ __align__(16) uint8_t prep_smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    PrepWarp<DK>& sm = reinterpret_cast<PrepWarp<DK>*>(prep_smem_raw)[warp];
    const long long blk0 = ((long long)blockIdx.x * 4 + warp) * per;
    if (blk0 >= blocks) return;
    const int nslot = blk0 + per <= blocks ? per : 1;
    const int g = lane >> 2, t = lane & 3, lm = lane >> 3, lr = lane & 7;
    const long long tok_stride = (long long)H * DK;

    // K and Q rows of a block, 16-byte vectors, eight (DK = 64) or sixteen lanes per 128 / 256-byte row; decay and beta of
    // its tokens; tokens past T are inert
    uint4 kv[VEC], qv[VEC];
    float dec, bt;
    auto fetch = [&](long long blk) {
        const long long bh = blk / NB;
        const int t0 = int(blk - bh * NB) * CB, bidx = int(bh / H), head = int(bh - (long long)bidx * H);
        const __nv_bfloat16* Ks = K + ((long long)bidx * T * H + head) * DK;
        const __nv_bfloat16* Qs = Q + ((long long)bidx * T * H + head) * DK;
        const uint4 z = make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
            const int v = lane + 32 * i, row = v / VPR, c8 = v % VPR;
            const bool ok = t0 + row < T;
            kv[i] = ok ? *reinterpret_cast<const uint4*>(Ks + (long long)(t0 + row) * tok_stride + c8 * 8) : z;
            qv[i] = ok ? *reinterpret_cast<const uint4*>(Qs + (long long)(t0 + row) * tok_stride + c8 * 8) : z;
        }
        const int tok = lane & (CB - 1);
        const bool ok = t0 + tok < T;
        dec = ok ? G[((long long)bidx * T + t0 + tok) * H + head] : 0.0f;
        bt = ok ? Beta[((long long)bidx * T + t0 + tok) * H + head] : 0.0f;
    };
    auto land = [&](int slot) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
            const int v = lane + 32 * i, row = v / VPR, c8 = v % VPR;
            *reinterpret_cast<uint4*>(sm.k + tile_off<ROWB>(row, c8)) = kv[i];
            *reinterpret_cast<uint4*>(sm.q + tile_off<ROWB>(row, c8)) = qv[i];
        }
        // inclusive prefix sum of the decays over the 16 tokens (both half-warps compute it)
        float cs = dec;
#pragma unroll
        for (int o = 1; o < CB; o <<= 1) {
            const float up = __shfl_up_sync(0xffffffffu, cs, o);
            if ((lane & (CB - 1)) >= o) cs += up;
        }
        const float last = __shfl_sync(0xffffffffu, cs, CB - 1);
        if (lane < CB) {
            sm.cum[lane] = cs;
            sm.beta[slot][lane] = bt;
            reinterpret_cast<float*>(sm.out[slot] + WS_EG)[lane] = __expf(cs);
            reinterpret_cast<float*>(sm.out[slot] + WS_DJ)[lane] = __expf(last - cs);
        }
        __syncwarp();
    };
    fetch(blk0);
#pragma unroll 1
    for (int slot = 0; slot < nslot; ++slot) {
        land(slot);
        if (slot + 1 < nslot) fetch(blk0 + 1);
        // Gram products over the keys: A = K K^T, Bm = Q K^T (16 x 16 each)
        float acc[2][4], accq[2][4];
#pragma unroll
        for (int ni = 0; ni < 2; ++ni)
#pragma unroll
            for (int e = 0; e < 4; ++e) { acc[ni][e] = 0.0f; accq[ni][e] = 0.0f; }
        const uint32_t k_s = smem_u32(sm.k), q_s = smem_u32(sm.q);
#pragma unroll
        for (int p = 0; p < KSTEP; ++p) {
            // matrices (tokens 0-7, keys lo), (tokens 8-15, keys lo), (tokens 0-7, keys hi), (tokens 8-15, keys hi) of k-step
            // p: the A fragment of [token][key]; as B fragments of the transposed product: (r[ni], r[ni + 2])
            const uint32_t off = tile_off<ROWB>((lm & 1) * 8 + lr, 2 * p + (lm >> 1));
            uint32_t kf[4], qf[4];
            ldsm4(k_s + off, kf);
            ldsm4(q_s + off, qf);
#pragma unroll
            for (int ni = 0; ni < 2; ++ni) {
                cmma(acc[ni], kf, kf[ni], kf[ni + 2]);
                cmma(accq[ni], qf, kf[ni], kf[ni + 2]);
            }
        }
        // acc[ni][0,1]: row i = g, columns j = 8 ni + 2t, + 1;  acc[ni][2,3]: row i = g + 8
        uint32_t* mw = reinterpret_cast<uint32_t*>(sm.out[slot] + WS_M);           // 8 words per row
        float* lf = sm.lf + slot * LF_SLOT;
#pragma unroll
        for (int ni = 0; ni < 2; ++ni) {
            float l[4], m[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = g + (e >> 1) * 8, j = 8 * ni + 2 * t + (e & 1);
                const float dcy = __expf(j <= i ? sm.cum[i] - sm.cum[j] : 0.0f);
                l[e] = j < i ? sm.beta[slot][i] * dcy * acc[ni][e] : 0.0f;
                m[e] = j <= i ? scale * dcy * accq[ni][e] : 0.0f;
            }
            *reinterpret_cast<float2*>(lf + g * LF_PITCH + 8 * ni + 2 * t) = make_float2(l[0], l[1]);
            *reinterpret_cast<float2*>(lf + (g + 8) * LF_PITCH + 8 * ni + 2 * t) = make_float2(l[2], l[3]);
            mw[g * 8 + 4 * ni + t] = cpack(m[0], m[1]);
            mw[(g + 8) * 8 + 4 * ni + t] = cpack(m[2], m[3]);
        }
        __syncwarp();                                     // L is complete; the tiles and cum may be overwritten
    }
    {                                                     // column `col` of (I + L)^-1 of the half-warp's block by forward substitution
        const int half = lane >> 4, col = lane & (CB - 1), slot = half < nslot ? half : 0;
        const float* lf = sm.lf + slot * LF_SLOT;
        float x[CB];
#pragma unroll
        for (int i = 0; i < CB; ++i) {
            // four partial sums: the dependent chain per row is i / 4 long instead of i
            float s0 = i == col ? 1.0f : 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;
#pragma unroll
            for (int j = 0; j < i; j += 4) {
                const float4 l = *reinterpret_cast<const float4*>(lf + i * LF_PITCH + j);
                s0 = fmaf(-l.x, x[j], s0);
                if (j + 1 < i) s1 = fmaf(-l.y, x[j + 1], s1);
                if (j + 2 < i) s2 = fmaf(-l.z, x[j + 2], s2);
                if (j + 3 < i) s3 = fmaf(-l.w, x[j + 3], s3);
            }
            x[i] = (s0 + s1) + (s2 + s3);
        }
        const float bc = sm.beta[slot][col];
        __nv_bfloat16* t2 = reinterpret_cast<__nv_bfloat16*>(sm.out[slot] + WS_T2);
        if (half < nslot)
#pragma unroll
            for (int i = 0; i < CB; ++i) t2[i * CB + col] = __float2bfloat16_rn(x[i] * bc);
    }
    __syncwarp();
    uint4* dst = reinterpret_cast<uint4*>(ws + blk0 * WS_BLOCK);
    const uint4* src = reinterpret_cast<const uint4*>(sm.out[0]);
    for (int i = lane; i < nslot * (WS_BLOCK / 16); i += 32) dst[i] = src[i];
}

// ---------------------------------------------------------------------------------------------------- scan kernel
template <int DK> struct ScanStage {                      // one block's operands as they lie in shared memory
    __align__(16) uint8_t k[CB * DK * 2], q[CB * DK * 2];  // [token][key] bf16, swizzled rows of DK * 2 bytes
    __align__(16) uint8_t v[2][CB * 128];                  // [token][value] bf16 as two halves of 64 values (128-byte rows)
    __align__(16) uint8_t w[WS_BLOCK];                     // the block's workspace: T2 | M | exp(c_i) | exp(c_16 - c_i)
};

// MI row tiles of 16 values per warp, NWARP warps: NWARP * 16 * MI values per CTA, blockIdx.y says which of the 128.
template <int DK, typename TO, int MI, int NWARP, int NSLOT>
__global__ void __launch_bounds__(NWARP * 32, NWARP * MI < 8 ? 0 : DK == 64 ? 3 : 2)
gdn_chunked_scan_kernel(const __nv_bfloat16* __restrict__ Q, const __nv_bfloat16* __restrict__ K, const __nv_bfloat16* __restrict__ V,
                        const uint8_t* __restrict__ ws, TO* __restrict__ O, int T, int H, int NB, float scale) {
    constexpr int NTHR = NWARP * 32, V8 = NWARP * 2 * MI;                  // V8: 16-byte vectors of a token's values here
    constexpr int KSTEP = DK / 16, NJ = DK / 8, ROWB = DK * 2, VPR = DK / 8, KI = CB * VPR / NTHR, VI = CB * V8 / NTHR;
    static_assert(CB * VPR % NTHR == 0 && CB * V8 % NTHR == 0, "whole rounds of copies");
    struct Smem {
        ScanStage<DK> st[NSLOT];
        float ot[2][CB][OT_PITCH];
    };
    extern __shared__ __align__(128) uint8_t cscan_smem_raw[];
    Smem& sm = *reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(cscan_smem_raw) + 127) & ~uintptr_t(127));
    const int bh = blockIdx.x, bidx = bh / H, head = bh % H;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3, lm = lane >> 3, lr = lane & 7;
    const int v0 = blockIdx.y * V8, dvb = v0 * 8 + warp * 16 * MI;
    const long long tok_stride_k = (long long)H * DK, tok_stride_v = (long long)H * CDV;
    const __nv_bfloat16* Qs = Q + ((long long)bidx * T * H + head) * DK;
    const __nv_bfloat16* Ks = K + ((long long)bidx * T * H + head) * DK;
    const __nv_bfloat16* Vs = V + ((long long)bidx * T * H + head) * CDV;
    const uint8_t* Ws = ws + (long long)bh * NB * WS_BLOCK;
    TO* Os = O + ((long long)bidx * T * H + head) * CDV;

    float S[MI][NJ][4];
#pragma unroll
    for (int mi = 0; mi < MI; ++mi)
#pragma unroll
        for (int nj = 0; nj < NJ; ++nj)
#pragma unroll
            for (int e = 0; e < 4; ++e) S[mi][nj][e] = 0.0f;

    // the thread's first element of the next block to fetch, and of the next block of output rows; its i-th copy is KROWS (VROWS)
    // token rows further on
    constexpr int KROWS = NTHR / VPR, VROWS = NTHR / V8;
    const __nv_bfloat16* kp = Ks + (tid / VPR) * tok_stride_k + tid % VPR * 8;
    const __nv_bfloat16* qp = Qs + (tid / VPR) * tok_stride_k + tid % VPR * 8;
    const __nv_bfloat16* vp = Vs + (tid / V8) * tok_stride_v + (v0 + tid % V8) * 8;
    TO* op = Os + (tid / V8) * tok_stride_v + (v0 + tid % V8) * 8;
    const uint8_t* wp = Ws;
    // a split sequence has registers to keep its destinations; a whole one computes them again
    constexpr bool KEEP = NWARP * MI < 8;
    auto k_dst = [&](int i) { return tile_off<ROWB>(tid / VPR + i * KROWS, tid % VPR); };
    auto v_dst = [&](int i) {
        const int c16 = v0 + tid % V8;
        return uint32_t(c16 >> 3) * (CB * 128) + tile_off<128>(tid / V8 + i * VROWS, c16 & 7);
    };
    uint32_t kdst[KEEP ? KI : 1], vdst[KEEP ? VI : 1];
    if constexpr (KEEP) {
#pragma unroll
        for (int i = 0; i < KI; ++i) { kdst[i] = k_dst(i); asm volatile("" : "+r"(kdst[i])); }
#pragma unroll
        for (int i = 0; i < VI; ++i) { vdst[i] = v_dst(i); asm volatile("" : "+r"(vdst[i])); }
    }
    const long long kstep = KROWS * tok_stride_k;
    // asynchronous copies of block `c` into ring slot c % NSLOT; every thread issues its share and commits one group
    auto issue = [&](int c) {
        if (c < NB) {
            ScanStage<DK>& st = sm.st[c % NSLOT];
            const int left = T - c * CB;                  // tokens from this block on: rows past them are filled with zeros
            const uint32_t sk = smem_u32(st.k), sq = smem_u32(st.q), sv = smem_u32(st.v[0]);
#pragma unroll
            for (int i = 0; i < KI; ++i) {
                const int row = tid / VPR + i * KROWS, n = row < left ? 16 : 0;
                const uint32_t dst = KEEP ? kdst[KEEP ? i : 0] : k_dst(i);
                cp_async16(sk + dst, n ? static_cast<const void*>(kp + i * kstep) : wp, n);
                cp_async16(sq + dst, n ? static_cast<const void*>(qp + i * kstep) : wp, n);
            }
#pragma unroll
            for (int i = 0; i < VI; ++i) {
                const int row = tid / V8 + i * VROWS, n = row < left ? 16 : 0;
                cp_async16(sv + (KEEP ? vdst[KEEP ? i : 0] : v_dst(i)), n ? static_cast<const void*>(vp + i * VROWS * tok_stride_v) : wp, n);
            }
            for (int v = tid; v < WS_BLOCK / 16; v += NTHR) cp_async16(smem_u32(st.w) + v * 16, wp + v * 16, 16);
            kp += CB * tok_stride_k;
            qp += CB * tok_stride_k;
            vp += CB * tok_stride_v;
            wp += WS_BLOCK;
        }
        cp_commit();                                      // an empty group past the end keeps the group count in step
    };
    // rows of a finished block from its o tile to global memory: 16 tokens, eight values per thread and pass
    auto store_rows = [&](int c) {
        const float* ot = &sm.ot[c & 1][0][0];
        const int left = T - c * CB;
#pragma unroll
        for (int i = 0; i < VI; ++i) {
            const int row = tid / V8 + i * VROWS, c8 = v0 + tid % V8;
            if (row < left) {
                const float4 a = *reinterpret_cast<const float4*>(ot + row * OT_PITCH + c8 * 8);
                const float4 b = *reinterpret_cast<const float4*>(ot + row * OT_PITCH + c8 * 8 + 4);
                TO* dst = op + i * VROWS * tok_stride_v;
                if constexpr (sizeof(TO) == 2) {
                    *reinterpret_cast<uint4*>(dst) = make_uint4(cpack(a.x, a.y), cpack(a.z, a.w), cpack(b.x, b.y), cpack(b.z, b.w));
                } else {
                    store_quad<TO>(dst, a.x, a.y, a.z, a.w);
                    store_quad<TO>(dst + 4, b.x, b.y, b.z, b.w);
                }
            }
        }
        op += CB * tok_stride_v;
    };

#pragma unroll
    for (int c = 0; c < NSLOT - 1; ++c) issue(c);
    for (int c = 0; c < NB; ++c) {
        cp_wait<NSLOT - 2>();                             // this thread's copies of block c have landed (later ones may still fly)
        __syncthreads();                                  // everyone's have; the o tile of block c - 1 is complete; the slot of block c - 1 is free
        issue(c + NSLOT - 1);
        if (c > 0) store_rows(c - 1);
        ScanStage<DK>& st = sm.st[c % NSLOT];
        const uint32_t k_s = smem_u32(st.k), q_s = smem_u32(st.q);
        const float* eg = reinterpret_cast<const float*>(st.w + WS_EG);
        const float* dj = reinterpret_cast<const float*>(st.w + WS_DJ);
        // ---------------------------------------------------------------- R^T = S0^T K^T and (Q S0)^T
        float R[MI][2][4], QS[MI][2][4];
#pragma unroll
        for (int mi = 0; mi < MI; ++mi)
#pragma unroll
            for (int ni = 0; ni < 2; ++ni)
#pragma unroll
                for (int e = 0; e < 4; ++e) { R[mi][ni][e] = 0.0f; QS[mi][ni][e] = 0.0f; }
#pragma unroll
        for (int p = 0; p < KSTEP; ++p) {
            // B fragments [key][token]: matrices (tokens 0-7, keys lo), (tokens 0-7, keys hi), (tokens 8-15, keys lo),
            // (tokens 8-15, keys hi) -> (b0, b1) of token block 0, then of token block 1
            const uint32_t off = tile_off<ROWB>((lm >> 1) * 8 + lr, 2 * p + (lm & 1));
            uint32_t bk[4], bq[4];
            ldsm4(k_s + off, bk);
            ldsm4(q_s + off, bq);
#pragma unroll
            for (int mi = 0; mi < MI; ++mi) {
                const uint32_t sa[4] = {cpack(S[mi][2 * p][0], S[mi][2 * p][1]), cpack(S[mi][2 * p][2], S[mi][2 * p][3]),
                                        cpack(S[mi][2 * p + 1][0], S[mi][2 * p + 1][1]), cpack(S[mi][2 * p + 1][2], S[mi][2 * p + 1][3])};
#pragma unroll
                for (int ni = 0; ni < 2; ++ni) {
                    cmma(R[mi][ni], sa, bk[2 * ni], bk[2 * ni + 1]);
                    cmma(QS[mi][ni], sa, bq[2 * ni], bq[2 * ni + 1]);
                }
            }
        }
        // per-token scalars of this lane's tokens 8 ni + 2t, + 1
        float2 ner[2], eq[2], dj2[2];
#pragma unroll
        for (int ni = 0; ni < 2; ++ni) {
            const float2 e = *reinterpret_cast<const float2*>(eg + 8 * ni + 2 * t);
            ner[ni] = make_float2(-e.x, -e.y);
            eq[ni] = make_float2(e.x * scale, e.y * scale);
            dj2[ni] = *reinterpret_cast<const float2*>(dj + 8 * ni + 2 * t);
        }
        // B fragments of T2 and M (row-major 16 x 16, 32-byte rows): matrices (rows 0-7, cols lo), (rows 0-7, cols hi),
        // (rows 8-15, cols lo), (rows 8-15, cols hi)
        uint32_t bt[4], bm[4];
        {
            const uint32_t off = uint32_t(((lm >> 1) * 8 + lr) * 32 + (lm & 1) * 16);
            ldsm4(smem_u32(st.w + WS_T2) + off, bt);
            ldsm4(smem_u32(st.w + WS_M) + off, bm);
        }
        // K^T fragments of the state update, B[token][key]: transposed reads; kf[q][2 h + c]: keys 16 q + 8 h + g, tokens 8 c + 2t, + 1
        // (eight warps of the wider keys have no registers to hold them that early)
        constexpr bool LATE_K = DK == 128 && NWARP == 8;
        uint32_t kf[KSTEP][4];
#pragma unroll
        for (int q = 0; q < KSTEP && !LATE_K; ++q) ldsm4t(k_s + tile_off<ROWB>((lm & 1) * 8 + lr, 2 * q + (lm >> 1)), kf[q]);
        float* otile = &sm.ot[c & 1][0][0];
        uint32_t da[MI][4];
#pragma unroll
        for (int mi = 0; mi < MI; ++mi) {
            const int r0 = dvb + 16 * mi + g, r1 = r0 + 8;
            // V^T fragment A[value][token] of value rows dvb + 16 mi .. + 15: transposed reads of [token][value]; matrices
            // (tokens 0-7, values lo), (tokens 0-7, values hi), (tokens 8-15, values lo), (tokens 8-15, values hi)
            uint32_t vv[4];
            {
                const int val0 = dvb + 16 * mi;                      // multiple of 16: both 8-value chunks lie in one 64-value half
                ldsm4t(smem_u32(st.v[val0 >> 6]) + tile_off<128>((lm >> 1) * 8 + lr, ((val0 & 63) >> 3) + (lm & 1)), vv);
            }
            // vv[0]: value g, tokens 2t, +1 | vv[1]: value g + 8, same tokens | vv[2]: value g, tokens 8 + 2t | vv[3]: value g + 8
            uint32_t va[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {                 // tokens 8 (h / 2) + 2t, + 1 of value row g + 8 (h % 2)
                const float2 r = make_float2(R[mi][h >> 1][2 * (h & 1)], R[mi][h >> 1][2 * (h & 1) + 1]);
                const float2 d = fma2(ner[h >> 1], r, make_float2(bf_lo(vv[h]), bf_hi(vv[h])));
                va[h] = cpack(d.x, d.y);
            }
            float U[2][4];
#pragma unroll
            for (int ni = 0; ni < 2; ++ni) {
#pragma unroll
                for (int e = 0; e < 4; ++e) U[ni][e] = 0.0f;
                cmma(U[ni], va, bt[2 * ni], bt[2 * ni + 1]);
            }
            uint32_t ua[4];
#pragma unroll
            for (int ni = 0; ni < 2; ++ni) {
                ua[2 * ni] = cpack(U[ni][0], U[ni][1]);
                ua[2 * ni + 1] = cpack(U[ni][2], U[ni][3]);
                const float2 d0 = mul2(make_float2(U[ni][0], U[ni][1]), dj2[ni]), d1 = mul2(make_float2(U[ni][2], U[ni][3]), dj2[ni]);
                da[mi][2 * ni] = cpack(d0.x, d0.y);
                da[mi][2 * ni + 1] = cpack(d1.x, d1.y);
            }
#pragma unroll
            for (int ni = 0; ni < 2; ++ni) {
                float Oa[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                cmma(Oa, ua, bm[2 * ni], bm[2 * ni + 1]);
                const int tok = 8 * ni + 2 * t;
                const float2 o0 = fma2(eq[ni], make_float2(QS[mi][ni][0], QS[mi][ni][1]), make_float2(Oa[0], Oa[1]));
                const float2 o1 = fma2(eq[ni], make_float2(QS[mi][ni][2], QS[mi][ni][3]), make_float2(Oa[2], Oa[3]));
                otile[tok * OT_PITCH + r0] = o0.x;
                otile[(tok + 1) * OT_PITCH + r0] = o0.y;
                otile[tok * OT_PITCH + r1] = o1.x;
                otile[(tok + 1) * OT_PITCH + r1] = o1.y;
            }
        }
        // ---------------------------------------------------------------- S^T <- e_last S^T + (diag(d) U)^T K
        {
            const float2 elast = make_float2(eg[CB - 1], eg[CB - 1]);
#pragma unroll
            for (int nj = 0; nj < NJ; ++nj) {
                if (LATE_K && nj % 2 == 0) ldsm4t(k_s + tile_off<ROWB>((lm & 1) * 8 + lr, nj + (lm >> 1)), kf[nj >> 1]);
                const uint32_t b0 = kf[nj >> 1][2 * (nj & 1)], b1 = kf[nj >> 1][2 * (nj & 1) + 1];
#pragma unroll
                for (int mi = 0; mi < MI; ++mi) {
#pragma unroll
                    for (int e = 0; e < 4; e += 2) {
                        const float2 v = mul2(make_float2(S[mi][nj][e], S[mi][nj][e + 1]), elast);
                        S[mi][nj][e] = v.x; S[mi][nj][e + 1] = v.y;
                    }
                    cmma(S[mi][nj], da[mi], b0, b1);
                }
            }
        }
    }
    cp_wait<0>();
    __syncthreads();
    store_rows(NB - 1);
}

// ---------------------------------------------------------------------------------------------------- scan of few sequences
// Few sequences leave the GPU to the latency of one: then a block's time is what one warp does for it, one instruction after the
// other.  So each 16 value columns get two warps.  The chain warp holds the state and runs R -> U -> state update alone; it hands the
// state and U, as the 16-bit fragments its own products used, through shared memory to the output warp, which computes Q S0 and M U a
// block behind, writes the rows, and brings in the blocks to come.  The same products and roundings as in the whole form, in the same
// order: the same bits.  NP pairs of warps per CTA, 16 NP of the 128 value columns (blockIdx.y says which).
//
// The hand-overs are named barriers (arrive on one side, sync on the other), two of each kind by the parity of the block:
//   FULL   the block's operands have landed (output warps -> chain warps)
//   HAND   state and U of the block are in shared memory, its operands are read (chain warps -> output warps)
//   TAKEN  the output warps have them in registers (-> chain warps, which write that buffer again two blocks later)
// and OUT among the output warps alone: all are through with a block, its ring slot may be filled again.
template <int DK, int NP> struct ChainSmem {
    static constexpr int NSLOT = 4;
    ScanStage<DK> st[NSLOT];
    uint4 sa[2][NP][DK / 16][32];                          // [parity][pair][k step][lane]: state, A fragments
    uint4 ua[2][NP][32];                                   // U
};
enum { BAR_OUT = 1, BAR_FULL = 2, BAR_HAND = 4, BAR_TAKEN = 6 };   // the latter three + parity; 0 is __syncthreads
template <int N> __device__ __forceinline__ void bar_arrive(int id) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(N) : "memory"); }
template <int N> __device__ __forceinline__ void bar_wait(int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(N) : "memory"); }

template <int DK, typename TO, int NP>
__global__ void __launch_bounds__(NP * 64, 2)
gdn_chunked_chain_kernel(const __nv_bfloat16* __restrict__ Q, const __nv_bfloat16* __restrict__ K, const __nv_bfloat16* __restrict__ V,
                         const uint8_t* __restrict__ ws, TO* __restrict__ O, int T, int H, int NB, float scale) {
    constexpr int NTHR = NP * 64, NOUT = NP * 32, KSTEP = DK / 16, NJ = DK / 8, ROWB = DK * 2, NSLOT = ChainSmem<DK, NP>::NSLOT;
    extern __shared__ __align__(128) uint8_t chain_smem_raw[];
    ChainSmem<DK, NP>& sm = *reinterpret_cast<ChainSmem<DK, NP>*>((reinterpret_cast<uintptr_t>(chain_smem_raw) + 127) & ~uintptr_t(127));
    const int bh = blockIdx.x, bidx = bh / H, head = bh % H;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3, lm = lane >> 3, lr = lane & 7;
    const int pair = warp % NP, dvb = (blockIdx.y * NP + pair) * 16;       // the pair's first value column
    if (warp < NP) {
        // ------------------------------------------------------------------------------------------- chain
        float S[NJ][4];
#pragma unroll
        for (int nj = 0; nj < NJ; ++nj)
#pragma unroll
            for (int e = 0; e < 4; ++e) S[nj][e] = 0.0f;
        for (int c = 0; c < NB; ++c) {
            const ScanStage<DK>& st = sm.st[c % NSLOT];
            uint32_t sa[KSTEP][4];
            if (c >= 2) bar_wait<NTHR>(BAR_TAKEN + (c & 1));
#pragma unroll
            for (int p = 0; p < KSTEP; ++p) {
                sa[p][0] = cpack(S[2 * p][0], S[2 * p][1]);
                sa[p][1] = cpack(S[2 * p][2], S[2 * p][3]);
                sa[p][2] = cpack(S[2 * p + 1][0], S[2 * p + 1][1]);
                sa[p][3] = cpack(S[2 * p + 1][2], S[2 * p + 1][3]);
                sm.sa[c & 1][pair][p][lane] = make_uint4(sa[p][0], sa[p][1], sa[p][2], sa[p][3]);
            }
            bar_wait<NTHR>(BAR_FULL + (c & 1));
            const uint32_t k_s = smem_u32(st.k);
            const float* eg = reinterpret_cast<const float*>(st.w + WS_EG);
            const float* dj = reinterpret_cast<const float*>(st.w + WS_DJ);
            float R[2][4];
#pragma unroll
            for (int ni = 0; ni < 2; ++ni)
#pragma unroll
                for (int e = 0; e < 4; ++e) R[ni][e] = 0.0f;
#pragma unroll
            for (int p = 0; p < KSTEP; ++p) {
                uint32_t bk[4];
                ldsm4(k_s + tile_off<ROWB>((lm >> 1) * 8 + lr, 2 * p + (lm & 1)), bk);
#pragma unroll
                for (int ni = 0; ni < 2; ++ni) cmma(R[ni], sa[p], bk[2 * ni], bk[2 * ni + 1]);
            }
            uint32_t vv[4], bt[4], kf[KSTEP][4];
            ldsm4t(smem_u32(st.v[dvb >> 6]) + tile_off<128>((lm >> 1) * 8 + lr, ((dvb & 63) >> 3) + (lm & 1)), vv);
            ldsm4(smem_u32(st.w + WS_T2) + uint32_t(((lm >> 1) * 8 + lr) * 32 + (lm & 1) * 16), bt);
#pragma unroll
            for (int q = 0; q < KSTEP; ++q) ldsm4t(k_s + tile_off<ROWB>((lm & 1) * 8 + lr, 2 * q + (lm >> 1)), kf[q]);
            float2 ner[2], dj2[2];
#pragma unroll
            for (int ni = 0; ni < 2; ++ni) {
                const float2 e = *reinterpret_cast<const float2*>(eg + 8 * ni + 2 * t);
                ner[ni] = make_float2(-e.x, -e.y);
                dj2[ni] = *reinterpret_cast<const float2*>(dj + 8 * ni + 2 * t);
            }
            const float2 elast = make_float2(eg[CB - 1], eg[CB - 1]);
#pragma unroll
            for (int nj = 0; nj < NJ; ++nj)
#pragma unroll
                for (int e = 0; e < 4; e += 2) {
                    const float2 v = mul2(make_float2(S[nj][e], S[nj][e + 1]), elast);
                    S[nj][e] = v.x; S[nj][e + 1] = v.y;
                }
            uint32_t va[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const float2 d = fma2(ner[h >> 1], make_float2(R[h >> 1][2 * (h & 1)], R[h >> 1][2 * (h & 1) + 1]), make_float2(bf_lo(vv[h]), bf_hi(vv[h])));
                va[h] = cpack(d.x, d.y);
            }
            float U[2][4];
#pragma unroll
            for (int ni = 0; ni < 2; ++ni) {
#pragma unroll
                for (int e = 0; e < 4; ++e) U[ni][e] = 0.0f;
                cmma(U[ni], va, bt[2 * ni], bt[2 * ni + 1]);
            }
            uint32_t da[4];
#pragma unroll
            for (int ni = 0; ni < 2; ++ni) {
                const float2 d0 = mul2(make_float2(U[ni][0], U[ni][1]), dj2[ni]), d1 = mul2(make_float2(U[ni][2], U[ni][3]), dj2[ni]);
                da[2 * ni] = cpack(d0.x, d0.y);
                da[2 * ni + 1] = cpack(d1.x, d1.y);
            }
#pragma unroll
            for (int nj = 0; nj < NJ; ++nj) cmma(S[nj], da, kf[nj >> 1][2 * (nj & 1)], kf[nj >> 1][2 * (nj & 1) + 1]);
            sm.ua[c & 1][pair][lane] = make_uint4(cpack(U[0][0], U[0][1]), cpack(U[0][2], U[0][3]), cpack(U[1][0], U[1][1]), cpack(U[1][2], U[1][3]));
            bar_arrive<NTHR>(BAR_HAND + (c & 1));
        }
        return;
    }
    // ----------------------------------------------------------------------------------------------- output
    constexpr int VPR = DK / 8, V8 = NP * 2, KI = CB * VPR / NOUT, KROWS = NOUT / VPR, VROWS = NOUT / V8;
    static_assert(CB * VPR % NOUT == 0 && VROWS == CB, "whole rounds of copies, one vector of V a thread");
    const int tid = threadIdx.x - NP * 32, v16 = blockIdx.y * V8 + tid % V8;
    const long long tok_stride_k = (long long)H * DK, tok_stride_v = (long long)H * CDV;
    const __nv_bfloat16* kp = K + ((long long)bidx * T * H + head) * DK + (tid / VPR) * tok_stride_k + tid % VPR * 8;
    const __nv_bfloat16* qp = Q + ((long long)bidx * T * H + head) * DK + (tid / VPR) * tok_stride_k + tid % VPR * 8;
    const __nv_bfloat16* vp = V + ((long long)bidx * T * H + head) * CDV + (tid / V8) * tok_stride_v + v16 * 8;
    const uint8_t* wp = ws + (long long)bh * NB * WS_BLOCK;
    TO* op = O + ((long long)bidx * T * H + head) * CDV + dvb;
    uint32_t kdst[KI];
#pragma unroll
    for (int i = 0; i < KI; ++i) kdst[i] = tile_off<ROWB>(tid / VPR + i * KROWS, tid % VPR);
    const uint32_t vdst = uint32_t(v16 >> 3) * (CB * 128) + tile_off<128>(tid / V8, v16 & 7);
    auto issue = [&](int c) {
        if (c < NB) {
            ScanStage<DK>& st = sm.st[c % NSLOT];
            const int left = T - c * CB;
            const uint32_t sk = smem_u32(st.k), sq = smem_u32(st.q);
#pragma unroll
            for (int i = 0; i < KI; ++i) {
                const int n = tid / VPR + i * KROWS < left ? 16 : 0;
                cp_async16(sk + kdst[i], n ? static_cast<const void*>(kp + i * KROWS * tok_stride_k) : wp, n);
                cp_async16(sq + kdst[i], n ? static_cast<const void*>(qp + i * KROWS * tok_stride_k) : wp, n);
            }
            const int n = tid / V8 < left ? 16 : 0;
            cp_async16(smem_u32(st.v[0]) + vdst, n ? static_cast<const void*>(vp) : wp, n);
            for (int v = tid; v < WS_BLOCK / 16; v += NOUT) cp_async16(smem_u32(st.w) + v * 16, wp + v * 16, 16);
            kp += CB * tok_stride_k;
            qp += CB * tok_stride_k;
            vp += CB * tok_stride_v;
            wp += WS_BLOCK;
        }
        cp_commit();                                       // an empty group past the end keeps the group count in step
    };
#pragma unroll
    for (int c = 0; c < NSLOT; ++c) issue(c);
    cp_wait<NSLOT - 1>();
    bar_arrive<NTHR>(BAR_FULL);
    for (int c = 0; c < NB; ++c) {
        if (c + 1 < NB) {
            cp_wait<NSLOT - 2>();                          // blocks up to c + 1
            bar_arrive<NTHR>(BAR_FULL + ((c + 1) & 1));
        }
        bar_wait<NTHR>(BAR_HAND + (c & 1));
        uint4 sa[KSTEP];
#pragma unroll
        for (int p = 0; p < KSTEP; ++p) sa[p] = sm.sa[c & 1][pair][p][lane];
        const uint4 ua = sm.ua[c & 1][pair][lane];
        const ScanStage<DK>& st = sm.st[c % NSLOT];
        const uint32_t q_s = smem_u32(st.q);
        uint32_t am[4];
        ldsm4(smem_u32(st.w + WS_M) + uint32_t(((lm & 1) * 8 + lr) * 32 + (lm >> 1) * 16), am);
        const float* eg = reinterpret_cast<const float*>(st.w + WS_EG);
        const float eqs[2] = {eg[g] * scale, eg[g + 8] * scale};
        float QS[2][4], Oa[2][4];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) { QS[nt][e] = 0.0f; Oa[nt][e] = 0.0f; }
        // Q as the operand A [token][key]; the state's registers are B fragments [key][value] of values 0-7 (0, 2) and 8-15 (1, 3)
#pragma unroll
        for (int p = 0; p < KSTEP; ++p) {
            uint32_t qf[4];
            ldsm4(q_s + tile_off<ROWB>((lm & 1) * 8 + lr, 2 * p + (lm >> 1)), qf);
            cmma(QS[0], qf, sa[p].x, sa[p].z);
            cmma(QS[1], qf, sa[p].y, sa[p].w);
        }
        cmma(Oa[0], am, ua.x, ua.z);
        cmma(Oa[1], am, ua.y, ua.w);
        if (c + 2 < NB) bar_arrive<NTHR>(BAR_TAKEN + (c & 1));
        bar_wait<NOUT>(BAR_OUT);
        issue(c + NSLOT);
        // rows straight from the accumulators [token][value].  float32: 8 bytes a lane, a whole 32-byte sector per token and n tile;
        // bf16: the lanes of a pair trade halves, so that a token's 32 bytes leave in one instruction
        const int left = T - c * CB;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float2 e2 = make_float2(eqs[h], eqs[h]);
            float2 o[2];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) o[nt] = fma2(e2, make_float2(QS[nt][2 * h], QS[nt][2 * h + 1]), make_float2(Oa[nt][2 * h], Oa[nt][2 * h + 1]));
            TO* const row = op + (g + 8 * h) * tok_stride_v;
            if constexpr (sizeof(TO) == 2) {
                const uint32_t w0 = cpack(o[0].x, o[0].y), w1 = cpack(o[1].x, o[1].y);
                const bool odd = (t & 1) != 0;
                const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? w0 : w1, 1);
                if (g + 8 * h < left) *reinterpret_cast<uint2*>(row + (odd ? 6 + 2 * t : 2 * t)) = odd ? make_uint2(got, w1) : make_uint2(w0, got);
            } else if (g + 8 * h < left) {
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) *reinterpret_cast<float2*>(row + 8 * nt + 2 * t) = o[nt];
            }
        }
        op += CB * tok_stride_v;
    }
    cp_wait<0>();
}

template <int DK, typename TO, int MI, int NWARP, int NSLOT>
int launch_scan(const void* q, const void* k, const void* v, const void* ws, void* o, int B, int T, int H, int NB, float scale, cudaStream_t s) {
    const int smem = NSLOT * int(sizeof(ScanStage<DK>)) + 2 * CB * OT_PITCH * 4 + 128;
    const cudaError_t e = cudaFuncSetAttribute(gdn_chunked_scan_kernel<DK, TO, MI, NWARP, NSLOT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return int(e);
    gdn_chunked_scan_kernel<DK, TO, MI, NWARP, NSLOT><<<dim3(unsigned(B) * unsigned(H), CDV / (16 * MI * NWARP)), NWARP * 32, smem, s>>>(
        static_cast<const __nv_bfloat16*>(q), static_cast<const __nv_bfloat16*>(k), static_cast<const __nv_bfloat16*>(v),
        static_cast<const uint8_t*>(ws), static_cast<TO*>(o), T, H, NB, scale);
    return int(cudaGetLastError());
}

template <int DK, typename TO, int NP>
int launch_chain(const void* q, const void* k, const void* v, const void* ws, void* o, int B, int T, int H, int NB, float scale, cudaStream_t s) {
    const int smem = int(sizeof(ChainSmem<DK, NP>)) + 128;
    const cudaError_t e = cudaFuncSetAttribute(gdn_chunked_chain_kernel<DK, TO, NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return int(e);
    gdn_chunked_chain_kernel<DK, TO, NP><<<dim3(unsigned(B) * unsigned(H), CDV / (16 * NP)), NP * 64, smem, s>>>(
        static_cast<const __nv_bfloat16*>(q), static_cast<const __nv_bfloat16*>(k), static_cast<const __nv_bfloat16*>(v),
        static_cast<const uint8_t*>(ws), static_cast<TO*>(o), T, H, NB, scale);
    return int(cudaGetLastError());
}

template <int DK, typename TO>
int launch_chunked(const void* q, const void* k, const void* v, const float* g, const float* beta, void* o, void* ws, int B, int T,
                   int H, float scale, cudaStream_t s) {
    const int NB = (T + CB - 1) / CB;
    const long long blocks = (long long)B * H * NB, seqs = (long long)B * H;
    const int prep_smem = 4 * int(sizeof(PrepWarp<DK>));
    cudaError_t e = cudaFuncSetAttribute(gdn_chunked_prep_kernel<DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, prep_smem);
    if (e != cudaSuccess) return int(e);
    const int sms = device_sms();
    // one block a warp while that is a single wave of warps (576 blocks of the wider keys: 9.4 us for both kernels against 11.0)
    const int per = blocks <= 16ll * sms ? 1 : 2;
    gdn_chunked_prep_kernel<DK><<<unsigned((blocks + 4 * per - 1) / (4 * per)), 128, prep_smem, s>>>(
        static_cast<const __nv_bfloat16*>(q), static_cast<const __nv_bfloat16*>(k), g, beta, static_cast<uint8_t*>(ws), T, H, NB, blocks, per, scale);
    e = cudaGetLastError();
    if (e != cudaSuccess) return int(e);
    // The value columns of a sequence are independent: while sequences are too few to give every SM one, a sequence's columns are
    // split over CTAs.  While those are at most one an SM (four a sequence, then two), the chain form: its output warps have a
    // scheduler to themselves; beyond, two CTAs of the whole form, and from one sequence an SM on one.  Both kernels, 1,021
    // tokens, us, whole form split in two (DK 128 to 74 sequences: four) / chain form on four CTAs / on two: DK 64: 6 sequences of 700
    // 29.4 / 25.3 / 25.3, 18 40.5 / 33 / 35.5, 36 41.6 / 34 / 37, 48 41.7 / 42.6 / 37.7, 72 43.5 / 44 / 39.4, 96 61 / 59 / 63, 120 63 / 71 / 66;
    // DK 128: 6 of 700 37.5 / 29.4 / 37.5, 18 52 / 41.5 / 54, 36 54 / 44 / 56, 48 60 / 62 / 57.7, 72 63 / 65 / 61, 96 86 / 90 / 101.
    // Whole form in one CTA / two: DK 64, 1,024 tokens, 144 sequences 66 / 58; DK 128, 144 106 / 90, 288 of 2,048 343 / 348.
    if (4 * seqs <= sms) return launch_chain<DK, TO, 2>(q, k, v, ws, o, B, T, H, NB, scale, s);
    if (2 * seqs <= sms) return launch_chain<DK, TO, 4>(q, k, v, ws, o, B, T, H, NB, scale, s);
    if (seqs <= sms) return launch_scan<DK, TO, 1, 4, 4>(q, k, v, ws, o, B, T, H, NB, scale, s);
    // ring slots of a whole sequence, 3 / 4: 64 x 2,048, DK 64 248 / 254 us; 48 x 2,048, DK 128 314 / 309
    return launch_scan<DK, TO, DK == 64 ? 2 : 1, DK == 64 ? 4 : 8, DK == 64 ? 3 : 4>(q, k, v, ws, o, B, T, H, NB, scale, s);
}

}  // namespace
}  // namespace sb

extern "C" size_t shvk_gdn_chunked_workspace_bytes(int B, int T, int H) {
    if (B <= 0 || T <= 0 || H <= 0) return 0;
    return size_t(B) * size_t(H) * size_t((T + sb::CB - 1) / sb::CB) * size_t(sb::WS_BLOCK);
}

extern "C" int shvk_gdn_chunked(const void* q, const void* k, const void* v, const float* g, const float* beta, void* o,
                                int o_dtype, int B, int T, int H, int DK, int DV, float scale, void* workspace,
                                size_t workspace_bytes, void* stream) {
    using namespace sb;
    if (B <= 0 || T <= 0 || H <= 0) return 0;
    if (DV != CDV || (DK != 64 && DK != 128) || (o_dtype != DT_F32 && o_dtype != DT_BF16)) return int(cudaErrorInvalidValue);
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
         reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(workspace)) & 15)
        return int(cudaErrorInvalidValue);
    if (!workspace || workspace_bytes < shvk_gdn_chunked_workspace_bytes(B, T, H)) return int(cudaErrorInvalidValue);
    cudaStream_t s = cudaStream_t(stream);
    if (DK == 64) {
        return o_dtype == DT_F32 ? launch_chunked<64, float>(q, k, v, g, beta, o, workspace, B, T, H, scale, s)
                                 : launch_chunked<64, __nv_bfloat16>(q, k, v, g, beta, o, workspace, B, T, H, scale, s);
    }
    return o_dtype == DT_F32 ? launch_chunked<128, float>(q, k, v, g, beta, o, workspace, B, T, H, scale, s)
                             : launch_chunked<128, __nv_bfloat16>(q, k, v, g, beta, o, workspace, B, T, H, scale, s);
}

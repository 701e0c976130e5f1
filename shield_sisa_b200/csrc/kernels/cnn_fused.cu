// Fused frame-encoder kernels of the bf16 / fp16 modes (MobileNetV3-Large blocks on 320x180 crops; layer by layer the
// same network is cnn.cu).  The reference's CUDA engine runs every layer as a launch of its own (engine/cuda/engine.cu:338-403).
//
// What bounded the layered form (640 crops, 11.2 ms): every expanded map crossed HBM twice (two thirds of 46 MB per
// crop), and the 1x1 kernels spent three quarters of their time fetching, converting and parking operand slabs.  Here an
// expanded map never leaves the SM: a block of threads takes a spatial tile, rounds its input pixels (with the halo the
// depthwise filter needs) to the mode's 16-bit type once, and walks the expanded channels in chunks,
//     expand (mma.sync m16n8k16 -> fp32 in shared memory) | depthwise (fp32 FMA out of shared memory)
// and either rounds the chunk into the A operand of the projection, whose accumulators stay in registers over all chunks,
// or, where a squeeze-excite gate stands between (it needs the whole map), writes the fp32 map and its pooled sums.
// Every step rounds and sums as the layer kernels of cnn.cu do: 1x1 operands in the mode's 16-bit type, everything else
// float32, activations operation by operation, pooled sums over the same groups of pixels.  The maps are the same bits.
//
// mma.sync and not tcgen05: the products are 16 to 160 deep and 8 to 160 wide on tiles whose rows are gathered pixels;
// they are a third of these kernels' instructions, the depthwise filter and the activations are the rest.
//
// Weights of the 1x1 convolutions arrive as 16-bit fragments (shvk_cnn_pack_weights): a lane's values for an mma are
// contiguous, a warp's load is one coalesced row, and no shared memory or conversion is spent on them.
#include "device_utils.cuh"
#include "shv_cnn_kernels.h"

namespace sb {
size_t se_gate_frame_bytes(int C, int CS);       // shared memory of a frame in the gate's cluster form (asked by cnn.cu too)
int se_partial_sums(const float* x, float* partial, int F, int HW, int C, cudaStream_t s);   // cnn.cu
namespace {

// x * relu6(x + 3) / 6 of a pair, each step rounded as cnn.cu rounds it (div6).  Encoding 640 crops bf16 takes 6.09 ms; with
// x * saturate(x / 6 + 1/2), which rounds otherwise (1e-7 absolute near -3), 5.99.
__device__ __forceinline__ float2 hswish2(float2 x) {
    const float2 s = add2(x, make_float2(3.0f, 3.0f));
    const float2 p = mul2(x, make_float2(fminf(fmaxf(s.x, 0.0f), 6.0f), fminf(fmaxf(s.y, 0.0f), 6.0f)));
    return fma2(p, make_float2(SIXTH_HI, SIXTH_HI), mul2(p, make_float2(SIXTH_LO, SIXTH_LO)));
}
template <bool HS> __device__ __forceinline__ float2 act2(float2 x) { return HS ? hswish2(x) : make_float2(fmaxf(x.x, 0.0f), fmaxf(x.y, 0.0f)); }

template <typename HT> struct Half;
template <> struct Half<__nv_bfloat16> {
    static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
        __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<uint32_t*>(&v);
    }
    static __device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    }
};
template <> struct Half<__half> {
    static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
        __half2 v = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<uint32_t*>(&v);
    }
    static __device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    }
};

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }

__host__ __device__ constexpr int up(int a, int b) { return (a + b - 1) / b * b; }
__host__ __device__ constexpr int cmax(int a, int b) { return a > b ? a : b; }

// ---------------------------------------------------------------------------------------------------- depthwise
// One thread's share of a depthwise filter: two channels, PX adjacent output pixels of SR rows.  e points at the tile's
// float32 map (pitch P floats per pixel, IWA pixels per row) at the thread's first input pixel and channel pair; every
// input pixel is read once and used by all outputs it belongs to.  Per output the taps are visited row by row.
template <int KS, int S, int PX, int SR, int P, int IWA>
__device__ __forceinline__ void depthwise_pair(const float* e, const float2 (&w)[KS * KS], float2 (&acc)[SR][PX]) {
    constexpr int NIN = (PX - 1) * S + KS;
#pragma unroll
    for (int r = 0; r < SR; ++r)
#pragma unroll
        for (int p = 0; p < PX; ++p) acc[r][p] = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int iy = 0; iy < (SR - 1) * S + KS; ++iy) {
        float2 x[NIN];
#pragma unroll
        for (int j = 0; j < NIN; ++j) x[j] = *reinterpret_cast<const float2*>(e + (iy * IWA + j) * P);
#pragma unroll
        for (int r = 0; r < SR; ++r) {
            const int ky = iy - r * S;
            if (ky < 0 || ky >= KS) continue;
#pragma unroll
            for (int kx = 0; kx < KS; ++kx)
#pragma unroll
                for (int p = 0; p < PX; ++p) acc[r][p] = fma2(w[ky * KS + kx], x[p * S + kx], acc[r][p]);
        }
    }
}

// ---------------------------------------------------------------------------------------------------- inverted residual
// CIN -> CEXP (1x1, activation) -> depthwise KS x KS, stride S, activation -> COUT (1x1, + residual); COUT = 0: stop after
// the depthwise map (squeeze-excite blocks).  TH x TW output pixels per block of THREADS threads, CE expanded channels at a time.
template <int CIN_, int CEXP_, int COUT_, int KS_, int S_, int HI_, int WI_, int TH_, int TW_, int CE_, int PX_, int SR_, int NSPLIT_,
          bool HS_, bool RES_, bool AHEAD_, int MINB_, int THREADS_ = 256>
struct Block {
    static constexpr int CIN = CIN_, CEXP = CEXP_, COUT = COUT_, KS = KS_, S = S_, HI = HI_, WI = WI_, TH = TH_, TW = TW_, CE = CE_;
    static constexpr int PX = PX_, SR = SR_, NSPLIT = NSPLIT_, MINB = MINB_, THREADS = THREADS_, WARPS = THREADS_ / 32;
    static constexpr bool HS = HS_, RES = RES_, SE = COUT_ == 0, AHEAD = AHEAD_;
    static constexpr int PAD = (KS - 1) / 2, HO = (HI + 2 * PAD - KS) / S + 1, WO = (WI + 2 * PAD - KS) / S + 1;
    static constexpr int TY = (HO + TH - 1) / TH, TX = (WO + TW - 1) / TW, TILES = TY * TX;
    static constexpr int IH = (TH - 1) * S + KS, IW = (TW - 1) * S + KS;
    static constexpr int VH = IH < HI ? IH : HI, VW = IW < WI ? IW : WI;     // most input pixels of a tile that lie in the image
    static constexpr int VPX = VH * VW, MROWS = up(VPX, 16);
    static constexpr int KP = up(CIN, 16), KT = KP / 16, XP = KP + 8;        // 16-bit input tile: XP halves per pixel
    static constexpr int NT = CE / 8, NW = NT / NSPLIT;
    static constexpr int P = CE % 16 == 8 ? CE : CE + 8;                     // fp32 pitch = 8 mod 16 words: expand's stores miss each other's banks
    static constexpr int CHUNKS = (CEXP + CE - 1) / CE;
    static constexpr int OPX = TH * TW, OMT = (OPX + 15) / 16, ONT = cmax(COUT / 8, 1), CK = up(CE, 16), DP = CK + 8;
    static constexpr int KPAD = SE ? CEXP : up(CEXP, 64);                      // k of the projection weights as they are packed, for any CE
    static constexpr int KFILL = cmax((CK - CE) / 2, 1);                       // k padding of a chunk, in pairs
    static constexpr int UNITS = OMT * ONT, UPW = SE ? 1 : (UNITS + WARPS - 1) / WARPS;
    static constexpr int STRIPS = TH / SR, GX = TW / PX, ITEMS = CE / 2 * GX * STRIPS;
    static constexpr bool EARLY = !SE && ITEMS <= THREADS;   // a thread has one item, its channels are known before the chunk is
    // squeeze-excite: the pooled sums are taken over groups of 64 pixels in row order, as se_partial_kernel takes them.  A tile that
    // consists of whole groups sums them itself (POOL)
    static constexpr int GROUP = 64, GROUPS = (HO * WO + GROUP - 1) / GROUP, TGROUPS = (TH * TW + GROUP - 1) / GROUP;
    static constexpr bool POOL = SE && TW == WO && (TILES == 1 || (S == 1 && TH * TW % GROUP == 0));
    static constexpr int RUN = TW % 8 == 0 ? 8 : TW % 4 == 0 ? 4 : 2;        // pixels of a row that are together in a group
    static constexpr int E_BYTES = up(IH * IW * P * 4, 16), X_BYTES = up(MROWS * XP * 2, 16), T_BYTES = up(MROWS * 2, 16);
    static constexpr int D_BYTES = SE ? 0 : up(OMT * 16 * DP * 2, 16);
    static constexpr int SMEM = E_BYTES + X_BYTES + T_BYTES + D_BYTES;
    static_assert(CE % 8 == 0 && NT % NSPLIT == 0 && WARPS % NSPLIT == 0 && TW % PX == 0 && TH % SR == 0, "tile shape");
    static_assert(SE ? CEXP % CE == 0 : CK == CE || CHUNKS == 1, "channel chunks");
    static_assert(SE || (COUT % 8 == 0 && CHUNKS * CK <= KPAD), "output channels");
    static_assert(!SE || ITEMS <= THREADS, "a thread keeps its outputs until the tile's map is consumed");
    static_assert(VPX * VW < 65536, "pixel numbers");
    static_assert(!POOL || (TW % RUN == 0 && GROUP % RUN == 0), "groups");
};

struct BlockArgs {
    const float* x;            // [F][HI][WI][CIN]
    const uint2* we;           // expand weights, fragments [n tile][k tile][lane]
    const float* be;
    const float* wd;           // depthwise filter [KS * KS][CEXP]
    const float* bd;
    const uint2* wp;           // projection weights, fragments [n tile][k tile][lane]
    const float* bp;
    float* out;                // [F][HO][WO][COUT], or the depthwise map [F][HO][WO][CEXP]
    float* sums;               // squeeze-excite: [F][GROUPS][CEXP] sums of the map over groups of pixels
    int chunks_per_group;      // squeeze-excite: chunks a block takes (gridDim.y groups)
};

template <class C, typename HT>
__global__ void __launch_bounds__(C::THREADS, C::MINB) block_kernel(const BlockArgs a) {
    extern __shared__ __align__(16) uint8_t smem[];
    float* const E = reinterpret_cast<float*>(smem);
    uint16_t* const X = reinterpret_cast<uint16_t*>(smem + C::E_BYTES);
    uint16_t* const pos = reinterpret_cast<uint16_t*>(smem + C::E_BYTES + C::X_BYTES);   // E pixel of every input row of X
    uint8_t* const D = smem + C::E_BYTES + C::X_BYTES + C::T_BYTES;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int f = blockIdx.x / C::TILES, tile = blockIdx.x % C::TILES;
    const int oy0 = tile / C::TX * C::TH, ox0 = tile % C::TX * C::TW;
    const int iy0 = oy0 * C::S - C::PAD, ix0 = ox0 * C::S - C::PAD;
    const int vy0 = max(iy0, 0), vy1 = min(iy0 + C::IH, C::HI), vx0 = max(ix0, 0), vx1 = min(ix0 + C::IW, C::WI);
    const int vw = vx1 - vx0, nv = (vy1 - vy0) * vw;
    const float* const img = a.x + (long long)f * (C::HI * C::WI * C::CIN);
    const int first = C::SE ? blockIdx.y * a.chunks_per_group : 0;
    const int last = C::SE ? min(first + a.chunks_per_group, C::CHUNKS) : C::CHUNKS;

    // Input pixels of the tile, rounded to 16 bits; channels past CIN and the halo outside the image are zero.  Eight loads of a thread
    // fly together: one at a time, a tile waited for 9 to 20 round trips to L2, a third of the time of blocks 2 to 4.
    constexpr int Q4 = C::KP / 4, FLY = 8;
    const uint32_t per_row = (65536u + vw - 1) / vw;     // r / vw = r * per_row >> 16, exact while r * vw < 65536
    for (int i0 = tid; i0 < nv * Q4; i0 += FLY * C::THREADS) {
        float4 p[FLY];
        int at[FLY];
#pragma unroll
        for (int j = 0; j < FLY; ++j) {
            const int i = i0 + j * C::THREADS, r = i / Q4, q = i % Q4, vy = int(uint32_t(r) * per_row >> 16), vx = r - vy * vw;
            p[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            at[j] = r * C::XP + q * 4;
            if (i < nv * Q4) {
                if (C::CIN % 16 == 0 || q * 4 < C::CIN)
                    p[j] = __ldg(reinterpret_cast<const float4*>(img + ((vy0 + vy) * C::WI + vx0 + vx) * C::CIN + q * 4));
                if (q == 0) pos[r] = uint16_t((vy0 - iy0 + vy) * C::IW + (vx0 - ix0 + vx));
            }
        }
#pragma unroll
        for (int j = 0; j < FLY; ++j)
            if (i0 + j * C::THREADS < nv * Q4)
                *reinterpret_cast<uint2*>(X + at[j]) = make_uint2(Half<HT>::pack(p[j].x, p[j].y), Half<HT>::pack(p[j].z, p[j].w));
    }
    if (nv < C::IH * C::IW)
        for (int i = tid; i < C::E_BYTES / 16; i += C::THREADS) reinterpret_cast<uint4*>(E)[i] = make_uint4(0u, 0u, 0u, 0u);
    if (!C::SE && C::CK != C::CE)                    // projection k padding of a single chunk
        for (int i = tid; i < C::OMT * 16 * C::KFILL; i += C::THREADS)
            reinterpret_cast<uint32_t*>(D)[i / C::KFILL * (C::DP / 2) + C::CE / 2 + i % C::KFILL] = 0u;
    // Expand weights and biases of this warp's n tiles of a chunk.  AHEAD: asked for a phase early, before the barrier that ends the
    // previous chunk's filter, where the registers allow (blocks 7 / 8 / 11 / 12 / 13, 640 frames: 203 / 140 / 207 / 308 / 241 us without,
    // 195 / 132 / 195 / 290 / 229 with; blocks 4, 5 and 14 spill or gain nothing)
    const int ns = warp % C::NSPLIT;
    uint2 b[C::NW][C::KT];
    float2 bias[C::NW];
    auto load_expand = [&](int ch) {
#pragma unroll
        for (int n = 0; n < C::NW; ++n) {
            const int nt = ch * C::NT + ns * C::NW + n, col = nt * 8 + 2 * t;
#pragma unroll
            for (int k = 0; k < C::KT; ++k) b[n][k] = __ldg(a.we + (nt * C::KT + k) * 32 + lane);
            bias[n] = C::CEXP % C::CE == 0 || col < C::CEXP ? __ldg(reinterpret_cast<const float2*>(a.be + col)) : make_float2(0.0f, 0.0f);
        }
    };
    if (C::AHEAD) load_expand(first);
    float pacc[C::UPW][4];
#pragma unroll
    for (int u = 0; u < C::UPW; ++u)
#pragma unroll
        for (int e = 0; e < 4; ++e) pacc[u][e] = 0.0f;
    __syncthreads();

    const int mtiles = (nv + 15) >> 4;
    const uint32_t xrow = smem_addr(X) + uint32_t(((lane & 15) * C::XP + (lane >> 4) * 8) * 2);
    for (int ch = first; ch < last; ++ch) {
        // ---- expand: this warp's n tiles of the chunk for every (WARPS / NSPLIT)-th group of 16 input pixels
        {
            if (!C::AHEAD) load_expand(ch);
            for (int mt = warp / C::NSPLIT; mt < mtiles; mt += C::WARPS / C::NSPLIT) {
                float c[C::NW][4];
#pragma unroll
                for (int n = 0; n < C::NW; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) c[n][e] = 0.0f;
#pragma unroll
                for (int k = 0; k < C::KT; ++k) {
                    uint32_t af[4];
                    ldmatrix_x4(af, xrow + uint32_t((mt * 16 * C::XP + k * 16) * 2));
#pragma unroll
                    for (int n = 0; n < C::NW; ++n) Half<HT>::mma(c[n], af, b[n][k].x, b[n][k].y);
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = mt * 16 + g + h * 8;
                    if (r >= nv) continue;
                    float* const er = E + pos[r] * C::P + ns * C::NW * 8 + 2 * t;
#pragma unroll
                    for (int n = 0; n < C::NW; ++n)
                        *reinterpret_cast<float2*>(er + n * 8) = act2<C::HS>(add2(make_float2(c[n][2 * h], c[n][2 * h + 1]), bias[n]));
                }
            }
        }
        float2 w0[C::KS * C::KS], bias0;                     // depthwise weights, asked for before the barrier
        if constexpr (C::EARLY) {
            const int col = ch * C::CE + tid % (C::CE / 2) * 2;
            if (C::CEXP % C::CE == 0 || col < C::CEXP) {
#pragma unroll
                for (int k = 0; k < C::KS * C::KS; ++k) w0[k] = __ldg(reinterpret_cast<const float2*>(a.wd + k * C::CEXP + col));
                bias0 = __ldg(reinterpret_cast<const float2*>(a.bd + col));
            }
        }
        __syncthreads();
        // ---- depthwise
        auto depthwise = [&](int i, float2 (&v)[C::SR][C::PX], int& oy, int& ox, int& cp) {
            cp = i % (C::CE / 2);
            ox = i / (C::CE / 2) % C::GX * C::PX;
            oy = i / (C::CE / 2 * C::GX) * C::SR;
            const int col = ch * C::CE + cp * 2;
            if (C::CEXP % C::CE != 0 && col >= C::CEXP) {   // padding of the last chunk; its expanded values are NaN behind an infinite pixel
#pragma unroll
                for (int r = 0; r < C::SR; ++r)
#pragma unroll
                    for (int p = 0; p < C::PX; ++p) v[r][p] = make_float2(0.0f, 0.0f);
                return;
            }
            float2 w[C::KS * C::KS], bias;
            if constexpr (C::EARLY) {
#pragma unroll
                for (int k = 0; k < C::KS * C::KS; ++k) w[k] = w0[k];
                bias = bias0;
            } else {
#pragma unroll
                for (int k = 0; k < C::KS * C::KS; ++k) w[k] = __ldg(reinterpret_cast<const float2*>(a.wd + k * C::CEXP + col));
                bias = __ldg(reinterpret_cast<const float2*>(a.bd + col));
            }
            depthwise_pair<C::KS, C::S, C::PX, C::SR, C::P, C::IW>(E + (oy * C::S * C::IW + ox * C::S) * C::P + cp * 2, w, v);
#pragma unroll
            for (int r = 0; r < C::SR; ++r)
#pragma unroll
                for (int p = 0; p < C::PX; ++p) v[r][p] = act2<C::HS>(add2(v[r][p], bias));
        };
        float2 v[C::SR][C::PX];
        int oy, ox, cp;
        if constexpr (C::SE) {
            const bool mine = C::ITEMS == C::THREADS || tid < C::ITEMS;
            auto inside = [&](int r, int p) { return (C::HO % C::TH == 0 || oy0 + oy + r < C::HO) && (C::WO % C::TW == 0 || ox0 + ox + p < C::WO); };
            if (mine) {
                depthwise(tid, v, oy, ox, cp);
#pragma unroll
                for (int r = 0; r < C::SR; ++r)
#pragma unroll
                    for (int p = 0; p < C::PX; ++p)
                        if (inside(r, p))
                            *reinterpret_cast<float2*>(a.out + ((long long)(f * C::HO + oy0 + oy + r) * C::WO + ox0 + ox + p) * C::CEXP + ch * C::CE + cp * 2) = v[r][p];
            }
            if (C::AHEAD && ch + 1 < last) load_expand(ch + 1);
            __syncthreads();                             // the expanded chunk is consumed
            if constexpr (C::POOL) {
                // the outputs take the places of expanded pixels of the image (the next chunk writes those again, the halo stays zero)
                if (mine)
#pragma unroll
                    for (int r = 0; r < C::SR; ++r)
#pragma unroll
                        for (int p = 0; p < C::PX; ++p)
                            if (inside(r, p)) *reinterpret_cast<float2*>(E + ((oy + r + C::PAD) * C::IW + ox + p + C::PAD) * C::P + cp * 2) = v[r][p];
                __syncthreads();
                // A group's sum: eight partial sums of every eighth pixel, then those in order.  640 frames, us per launch with the maps
                // of blocks 5 / 11 / 12 / 13 / 14 summed here: 249 / 219 / 305 / 240 / 166; with sums per tile in the order of the
                // threads, which rounds otherwise, 235 / 195 / 268 / 218 / 158; block 4, whose tiles cut the groups, is read again
                // (332 -> 364).
                const int n = C::HO % C::TH == 0 ? C::TH * C::TW : min(C::TH, C::HO - oy0) * C::TW;
                for (int i = tid; i < C::CE * C::TGROUPS; i += C::THREADS) {
                    const int c = i % C::CE, s = C::TGROUPS == 1 ? 0 : i / C::CE;
                    float part[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) part[e] = 0.0f;
#pragma unroll
                    for (int q = 0; q < C::GROUP; q += C::RUN) {
                        const int p = s * C::GROUP + q;
                        const float* const row = E + ((p / C::TW + C::PAD) * C::IW + p % C::TW + C::PAD) * C::P + c;
                        if (p < n)                       // n is a multiple of RUN
#pragma unroll
                            for (int e = 0; e < C::RUN; ++e) part[(q + e) & 7] += row[e * C::P];
                    }
                    float t = part[0];
#pragma unroll
                    for (int e = 1; e < 8; ++e) t += part[e];
                    a.sums[((long long)f * C::GROUPS + tile * C::TGROUPS + s) * C::CEXP + ch * C::CE + c] = t;
                }
                __syncthreads();
            }
        } else {
            for (int i = tid; i < C::ITEMS; i += C::THREADS) {
                depthwise(i, v, oy, ox, cp);
#pragma unroll
                for (int r = 0; r < C::SR; ++r)
#pragma unroll
                    for (int p = 0; p < C::PX; ++p)
                        reinterpret_cast<uint32_t*>(D)[((oy + r) * C::TW + ox + p) * (C::DP / 2) + cp] = Half<HT>::pack(v[r][p].x, v[r][p].y);
            }
            if (C::AHEAD && ch + 1 < last) load_expand(ch + 1);
            __syncthreads();
            // ---- projection: this chunk's k range into the accumulators of the warp's (pixel group, n tile) units
            const uint32_t drow = smem_addr(D) + uint32_t(((lane & 15) * C::DP + (lane >> 4) * 8) * 2);
            constexpr int KC = C::CK / 16, KALL = C::KPAD / 16;
#pragma unroll
            for (int k = 0; k < KC; ++k)
#pragma unroll
                for (int u = 0; u < C::UPW; ++u) {
                    const int unit = warp + u * C::WARPS;
                    if (C::UNITS % C::WARPS != 0 && unit >= C::UNITS) break;
                    uint32_t af[4];
                    ldmatrix_x4(af, drow + uint32_t(((unit % C::OMT) * 16 * C::DP + k * 16) * 2));
                    const uint2 b = __ldg(a.wp + ((unit / C::OMT) * KALL + ch * KC + k) * 32 + lane);
                    Half<HT>::mma(pacc[u], af, b.x, b.y);
                }
        }
    }
    if constexpr (C::SE) return;
#pragma unroll
    for (int u = 0; u < C::UPW; ++u) {
        const int unit = warp + u * C::WARPS;
        if (C::UNITS % C::WARPS != 0 && unit >= C::UNITS) break;
        const int n = unit / C::OMT * 8 + 2 * t;
        const float2 bias = __ldg(reinterpret_cast<const float2*>(a.bp + n));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int p = unit % C::OMT * 16 + g + h * 8, oy = oy0 + p / C::TW, ox = ox0 + p % C::TW;
            if (p >= C::OPX || oy >= C::HO || ox >= C::WO) continue;
            float2 v = make_float2(pacc[u][2 * h] + bias.x, pacc[u][2 * h + 1] + bias.y);
            const long long at = ((long long)(f * C::HO + oy) * C::WO + ox) * C::COUT + n;
            if (C::RES) {
                const float2 r = *reinterpret_cast<const float2*>(a.x + at);
                v.x += r.x;
                v.y += r.y;
            }
            *reinterpret_cast<float2*>(a.out + at) = v;
        }
    }
}

// ---------------------------------------------------------------------------------------------------- stem + first block
// uint8 crop -> normalisation -> 3x3/2 convolution 3 -> 16, Hardswish -> depthwise 3x3, ReLU -> 1x1 16 -> 16, + the stem's
// output.  A block takes 10 x 32 output pixels: the 25 x 69 input pixels are looked up once into float32, the stem runs two
// pixels a thread with its filter as kernel parameters (an FMA takes one operand from the constant bank, so a tap costs no
// load; from shared memory it takes 670 us instead of 558), and its map stays in shared memory.  It is bound by issue: crops come
// as words (a byte at a time the index arithmetic was a third of it), four words a store, all loads of a thread in flight, four
// blocks an SM (three: 595).  640 crops 724 -> 558 us.
struct StemParams {
    float w[27 * 16];          // ((ky * 3 + kx) * 3 + ci) * 16 + co
    float b[16];
};
struct Stem {
    static constexpr int H = 90, W = 160, IMH = 180, IMW = 320, TH = 10, TW = 32, TILES = (H / TH) * (W / TW);
    static constexpr int SH = TH + 2, SW = TW + 2, UH = 2 * SH + 1, UW = 2 * SW + 1;   // stem map and input tile
    static constexpr int ULEAD = 3, UWORDS = (ULEAD + UW * 3 + 3) / 4, UP = UWORDS * 4;   // a tile row: whole words of the crop's row, the first ULEAD bytes unused
    static constexpr int P = 20, DP = 24, PX = 2, SR = 5;
    static constexpr int OMT = TH * TW / 16;
    static constexpr int S_BYTES = SH * SW * P * 4, U_BYTES = up(UH * UP * 4, 16), D_BYTES = TH * TW * DP * 2;
    static constexpr int SMEM = S_BYTES + cmax(U_BYTES, D_BYTES) + 768 * 4;
};

template <typename HT>
__global__ void __launch_bounds__(256, 4)
stem_block_kernel(const uint8_t* __restrict__ frames, const float* __restrict__ lut, const __grid_constant__ StemParams sp,
                  const float* __restrict__ wd, const float* __restrict__ bd, const uint2* __restrict__ wp,
                  const float* __restrict__ bp, float* __restrict__ out) {
    extern __shared__ __align__(16) uint8_t smem[];
    float* const M = reinterpret_cast<float*>(smem);                          // stem map, pitch P
    float* const U = reinterpret_cast<float*>(smem + Stem::S_BYTES);          // normalised input; D reuses it
    uint32_t* const D = reinterpret_cast<uint32_t*>(smem + Stem::S_BYTES);
    float* const L = reinterpret_cast<float*>(smem + Stem::S_BYTES + cmax(Stem::U_BYTES, Stem::D_BYTES));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int f = blockIdx.x / Stem::TILES, tile = blockIdx.x % Stem::TILES;
    const int oy0 = tile / (Stem::W / Stem::TW) * Stem::TH, ox0 = tile % (Stem::W / Stem::TW) * Stem::TW;
    const uint8_t* const img = frames + (long long)f * (Stem::IMH * Stem::IMW * 3);
    // stem pixel (sy, sx) of the tile is map pixel (oy0 - 1 + sy, ox0 - 1 + sx); its taps start at crop pixel 2 (.) - 1.  A thread's
    // words of the tile are all asked for before the first is looked up
    const int uy0 = 2 * (oy0 - 1) - 1, ux0 = 2 * (ox0 - 1) - 1;
    const bool words = (reinterpret_cast<uintptr_t>(frames) & 3) == 0;       // a crop's rows and a tile's first column are whole words then
    constexpr int WORDS = Stem::UH * Stem::UWORDS, EACH = (WORDS + 255) / 256;
    uint32_t raw[EACH];
    auto word_at = [&](int i, int& x3, int& y) {
        y = uy0 + i / Stem::UWORDS;
        x3 = ux0 * 3 - Stem::ULEAD + 4 * (i % Stem::UWORDS);
        return i < WORDS && y >= 0 && y < Stem::IMH && x3 >= 0 && x3 < Stem::IMW * 3;
    };
#pragma unroll
    for (int j = 0; j < EACH; ++j) {
        int x3, y;
        raw[j] = 0;
        if (word_at(tid + j * 256, x3, y)) {
            const uint8_t* const at = img + y * (Stem::IMW * 3) + x3;
            raw[j] = words ? __ldg(reinterpret_cast<const uint32_t*>(at)) : at[0] | at[1] << 8 | at[2] << 16 | uint32_t(at[3]) << 24;
        }
    }
    for (int i = tid; i < 768; i += 256) L[i] = __ldg(lut + i);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < EACH; ++j) {
        const int i = tid + j * 256, w = i % Stem::UWORDS;
        if (EACH * 256 != WORDS && i >= WORDS) break;
        int x3, y;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (word_at(i, x3, y)) {
            const uint32_t q = raw[j];
            const float* const l0 = L + w % 3 * 256;                          // byte k of the word has colour (w + k) % 3
            const float* const l1 = L + (w + 1) % 3 * 256;
            const float* const l2 = L + (w + 2) % 3 * 256;
            v = make_float4(l0[q & 255], l1[q >> 8 & 255], l2[q >> 16 & 255], l0[q >> 24]);
        }
        *reinterpret_cast<float4*>(U + i / Stem::UWORDS * Stem::UP + 4 * w) = v;
    }
    __syncthreads();
    // two pixels of a row a thread: a weight pair serves both
    for (int i2 = tid; i2 < Stem::SH * Stem::SW / 2; i2 += 256) {
        const int sy = i2 / (Stem::SW / 2), sx = i2 % (Stem::SW / 2) * 2;
        float2 acc[2][8];
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int c = 0; c < 8; ++c) acc[p][c] = make_float2(0.0f, 0.0f);
        const float* const u = U + 2 * sy * Stem::UP + Stem::ULEAD + 6 * sx;
#pragma unroll
        for (int ky = 0; ky < 3; ++ky) {
            float x[15];                                                      // the row's values of both pixels; all but the first in pairs
            x[0] = u[ky * Stem::UP];
#pragma unroll
            for (int j = 1; j < 15; j += 2) {
                const float2 q = *reinterpret_cast<const float2*>(u + ky * Stem::UP + j);
                x[j] = q.x;
                x[j + 1] = q.y;
            }
#pragma unroll
            for (int k = 0; k < 9; ++k)
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float2 w = make_float2(sp.w[(ky * 9 + k) * 16 + 2 * c], sp.w[(ky * 9 + k) * 16 + 2 * c + 1]);
#pragma unroll
                    for (int p = 0; p < 2; ++p) acc[p][c] = fma2(w, make_float2(x[k + 6 * p], x[k + 6 * p]), acc[p][c]);
                }
        }
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const int y = oy0 - 1 + sy, x = ox0 - 1 + sx + p;
            const bool in = y >= 0 && y < Stem::H && x >= 0 && x < Stem::W;       // the depthwise filter sees zeros outside the map
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float2 lo = hswish2(add2(acc[p][2 * q], make_float2(sp.b[4 * q], sp.b[4 * q + 1])));
                const float2 hi = hswish2(add2(acc[p][2 * q + 1], make_float2(sp.b[4 * q + 2], sp.b[4 * q + 3])));
                *reinterpret_cast<float4*>(M + (sy * Stem::SW + sx + p) * Stem::P + q * 4) = in ? make_float4(lo.x, lo.y, hi.x, hi.y) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        }
    }
    __syncthreads();
    {
        constexpr int GX = Stem::TW / Stem::PX;
        const int cp = tid % 8, gx = tid / 8 % GX, st = tid / (8 * GX);
        static_assert(8 * GX * (Stem::TH / Stem::SR) == 256, "one depthwise item per thread");
        float2 w[9], acc[Stem::SR][Stem::PX];
#pragma unroll
        for (int k = 0; k < 9; ++k) w[k] = __ldg(reinterpret_cast<const float2*>(wd + k * 16 + cp * 2));
        const float2 bias = __ldg(reinterpret_cast<const float2*>(bd + cp * 2));
        depthwise_pair<3, 1, Stem::PX, Stem::SR, Stem::P, Stem::SW>(M + (st * Stem::SR * Stem::SW + gx * Stem::PX) * Stem::P + cp * 2, w, acc);
#pragma unroll
        for (int r = 0; r < Stem::SR; ++r)
#pragma unroll
            for (int p = 0; p < Stem::PX; ++p)
                D[((st * Stem::SR + r) * Stem::TW + gx * Stem::PX + p) * (Stem::DP / 2) + cp] =
                    Half<HT>::pack(fmaxf(acc[r][p].x + bias.x, 0.0f), fmaxf(acc[r][p].y + bias.y, 0.0f));
    }
    __syncthreads();
    const uint32_t drow = smem_addr(D) + uint32_t(((lane & 15) * Stem::DP + (lane >> 4) * 8) * 2);
    const uint2 b0 = __ldg(wp + lane), b1 = __ldg(wp + 32 + lane);
#pragma unroll
    for (int u = 0; u < (Stem::OMT + 7) / 8; ++u) {
        const int mt = warp + u * 8;
        if (mt >= Stem::OMT) break;
        uint32_t af[4];
        ldmatrix_x4(af, drow + uint32_t(mt * 16 * Stem::DP * 2));
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            Half<HT>::mma(c, af, nt ? b1.x : b0.x, nt ? b1.y : b0.y);
            const int n = nt * 8 + 2 * t;
            const float2 bias = __ldg(reinterpret_cast<const float2*>(bp + n));
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int p = mt * 16 + g + h * 8, y = p / Stem::TW, x = p % Stem::TW;
                const float2 r = *reinterpret_cast<const float2*>(M + ((y + 1) * Stem::SW + x + 1) * Stem::P + n);
                *reinterpret_cast<float2*>(out + (((long long)f * Stem::H + oy0 + y) * Stem::W + ox0 + x) * 16 + n) =
                    make_float2(c[2 * h] + bias.x + r.x, c[2 * h + 1] + bias.y + r.y);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------------- squeeze-excite gate
// A cluster of eight blocks takes G frames.  Every block reduces the frames' pooled sums, computes an eighth of the hidden
// layer (a warp per unit, lanes over the channels, a weight row read once for all G frames), hands it to the other seven
// through distributed shared memory, and computes an eighth of the gates.  One block per frame read all 1.8 MB of the
// widest layer's weights through one SM: 52 us however few the frames, 210 us at 640; now 13 us and 109.
//
// Sums and roundings are those of se_gate_kernel: an output is a warp's, lane l sums the inputs l, l + 32, ... in order, then the
// lanes are added.  So weights come as coalesced 4-byte loads; the frames of a cluster lie next to each other in shared memory,
// one 128-bit read for all four.
template <int G> __device__ __forceinline__ void load_frames(const float* p, float (&v)[G]) {
    if constexpr (G == 4) {
        const float4 q = *reinterpret_cast<const float4*>(p);
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
#pragma unroll
        for (int i = 0; i < G; ++i) v[i] = p[i];
    }
}
// acc[u][fr] = sum over k of W[rows u][k] x[k][fr], each lane its share of k.  x has zeros up to a multiple of 32 GATE_BATCH, so that
// every batch is whole: the weights of GATE_BATCH steps are loaded before the first is used (an output is a chain of round trips
// to L2), and nothing is asked between the sums.
constexpr int GATE_BATCH = 8;
__host__ __device__ constexpr int gate_rows_padded(int k) { return up(k, 32 * GATE_BATCH); }
template <int G, int UNITS>
__device__ __forceinline__ void lane_sums(const float* __restrict__ W, int K, const int (&row)[UNITS], const float* x, int lane, float (&acc)[UNITS][G]) {
    const float* w[UNITS];
#pragma unroll
    for (int u = 0; u < UNITS; ++u) {
        w[u] = W + (long long)row[u] * K;
#pragma unroll
        for (int fr = 0; fr < G; ++fr) acc[u][fr] = 0.0f;
    }
#pragma unroll 1
    for (int k0 = lane; k0 < gate_rows_padded(K); k0 += 32 * GATE_BATCH) {
        float wv[GATE_BATCH][UNITS];
#pragma unroll
        for (int d = 0; d < GATE_BATCH; ++d)
#pragma unroll
            for (int u = 0; u < UNITS; ++u) wv[d][u] = k0 + 32 * d < K ? __ldg(w[u] + k0 + 32 * d) : 0.0f;
#pragma unroll
        for (int d = 0; d < GATE_BATCH; ++d) {
            float p[G];
            load_frames<G>(x + (k0 + 32 * d) * G, p);
#pragma unroll
            for (int u = 0; u < UNITS; ++u)
#pragma unroll
                for (int fr = 0; fr < G; ++fr) acc[u][fr] = fmaf(wv[d][u], p[fr], acc[u][fr]);
        }
    }
}
template <int G, int UNITS>
__global__ void __cluster_dims__(8, 1, 1) __launch_bounds__(256)
se_gate_cluster_kernel(const float* __restrict__ sums, const float* __restrict__ w1, const float* __restrict__ b1,
                       const float* __restrict__ w2, const float* __restrict__ b2, float* __restrict__ gate, int F, int tiles, float hw,
                       int C, int CS) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int CP = gate_rows_padded(C), CSP = gate_rows_padded(CS);
    float* const pooled = reinterpret_cast<float*>(smem);           // [CP][G]
    float* const hid = pooled + G * CP;                              // [CSP][G]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = blockIdx.x & 7;
    const int f0 = int(blockIdx.x >> 3) * G, nf = min(G, F - f0);
    for (int i = tid; i < G * C; i += 256) {
        const int fr = i / C, c = i - fr * C;
        float s = 0.0f;
        if (fr < nf) {
            const float* const p = sums + (long long)(f0 + fr) * tiles * C + c;
            int k = 0;
            for (; k + 4 < tiles; k += 5) {                          // five loads fly together: the wide early maps have 15 groups
                float v[5];
#pragma unroll
                for (int e = 0; e < 5; ++e) v[e] = __ldg(p + (k + e) * C);
#pragma unroll
                for (int e = 0; e < 5; ++e) s += v[e];
            }
            for (; k < tiles; ++k) s += __ldg(p + k * C);
        }
        pooled[c * G + fr] = s / hw;
    }
    for (int i = G * C + tid; i < G * CP; i += 256) pooled[i] = 0.0f;
    for (int i = G * CS + tid; i < G * CSP; i += 256) hid[i] = 0.0f;
    cluster_sync();                                                  // pooled is complete, and every block of the cluster runs
    // UNITS outputs of a warp at a time, so that their weight loads fly together: with one, an output costs a round trip to L2
    for (int j0 = rank * 8 + warp; j0 < CS; j0 += 64 * UNITS) {
        int row[UNITS];
        float acc[UNITS][G];
#pragma unroll
        for (int u = 0; u < UNITS; ++u) row[u] = min(j0 + 64 * u, CS - 1);
        lane_sums<G, UNITS>(w1, C, row, pooled, lane, acc);
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            const int j = j0 + 64 * u;
            if (j >= CS) break;
            const float bj = b1[j];
#pragma unroll
            for (int fr = 0; fr < G; ++fr) {
                const float v = fmaxf(warp_sum(acc[u][fr]) + bj, 0.0f);
                if (lane < 8) {                                      // lane r stores into block r of the cluster
                    const uint32_t local = smem_addr(hid + j * G + fr);
                    uint32_t remote;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(lane));
                    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(v) : "memory");
                }
            }
        }
    }
    cluster_sync();
    for (int c0 = rank * 8 + warp; c0 < C; c0 += 64 * UNITS) {
        int row[UNITS];
        float acc[UNITS][G];
#pragma unroll
        for (int u = 0; u < UNITS; ++u) row[u] = min(c0 + 64 * u, C - 1);
        lane_sums<G, UNITS>(w2, CS, row, hid, lane, acc);
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            const int c = c0 + 64 * u;
            if (c >= C) break;
#pragma unroll
            for (int fr = 0; fr < G; ++fr) acc[u][fr] = warp_sum(acc[u][fr]);
            if (lane == 0)
#pragma unroll
                for (int fr = 0; fr < G; ++fr)
                    if (fr < nf) gate[(long long)(f0 + fr) * C + c] = div6(fminf(fmaxf(acc[u][fr] + b2[c] + 3.0f, 0.0f), 6.0f));
        }
    }
}

// ---------------------------------------------------------------------------------------------------- 1x1 on rows
// out[m][n] = sum_k A[m][k] W[n][k] + b[n] (+ R[m][n]), A float32 scaled by a squeeze-excite gate per group of gate_rows
// rows, rounded to 16 bits, or already 16-bit.  A warp owns 16 rows and NT n tiles and is on its own: its A fragments come
// straight from memory into registers (the k order inside an mma is permuted so that a lane's values are one 16-byte load;
// the packed weights carry the same order), no shared memory, no barrier, STEP loads in flight.
// AHEAD = 0: a warp takes all n tiles of its rows, their weights come as they are used.  AHEAD > 0, for few rows: the n tiles are
// split over gridDim.y, and everything of a k step, weights included, is loaded AHEAD steps before it is used; the order of a
// sum is the same.
template <int NT, int AHEAD, typename HT>
__global__ void __launch_bounds__(128, AHEAD > 0 ? 2 : NT > 14 ? 3 : 4)
rows_gate_kernel(const float* __restrict__ A, const uint4* __restrict__ W, const float* __restrict__ bias, const float* __restrict__ gate,
                 int gate_rows, const float* R, float* out, int M, int N, int K) {
    constexpr int NP = (NT + 1) / 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int m0 = (blockIdx.x * 4 + warp) * 16;
    if (m0 >= M) return;
    const int ra = min(m0 + g, M - 1), rb = min(m0 + g + 8, M - 1);
    const float* const pa = A + (long long)ra * K + t * 4;
    const float* const pb = A + (long long)rb * K + t * 4;
    const float* const ga = gate + (long long)(ra / gate_rows) * K + t * 4;
    const float* const gb = gate + (long long)(rb / gate_rows) * K + t * 4;
    const int np0 = blockIdx.y * NP, npall = gridDim.y * NP;
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[n][e] = 0.0f;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const int kt = (K + 15) / 16;
    auto load = [&](float4 (&v)[4], int k) {
        const bool in = k < kt && k * 16 + t * 4 < K;
        v[0] = in ? __ldg(reinterpret_cast<const float4*>(pa + k * 16)) : zero;
        v[1] = in ? __ldg(reinterpret_cast<const float4*>(pb + k * 16)) : zero;
        v[2] = in ? __ldg(reinterpret_cast<const float4*>(ga + k * 16)) : zero;
        v[3] = in ? __ldg(reinterpret_cast<const float4*>(gb + k * 16)) : zero;
    };
    auto weight = [&](int k, int n) { return __ldg(W + ((long long)k * npall + np0 + n) * 32 + lane); };
    auto step = [&](const float4 (&v)[4], auto b_of) {
        uint32_t af[4];
        af[0] = Half<HT>::pack(v[0].x * v[2].x, v[0].y * v[2].y);
        af[1] = Half<HT>::pack(v[1].x * v[3].x, v[1].y * v[3].y);
        af[2] = Half<HT>::pack(v[0].z * v[2].z, v[0].w * v[2].w);
        af[3] = Half<HT>::pack(v[1].z * v[3].z, v[1].w * v[3].w);
#pragma unroll
        for (int n = 0; n < NP; ++n) {
            const uint4 b = b_of(n);
            Half<HT>::mma(acc[2 * n], af, b.x, b.y);
            if (2 * n + 1 < NT) Half<HT>::mma(acc[2 * n + 1 < NT ? 2 * n + 1 : 0], af, b.z, b.w);
        }
    };
    if constexpr (AHEAD == 0) {
        float4 v0[4], v1[4];
        load(v0, 0);
        for (int k = 0; k < kt; k += 2) {
            load(v1, k + 1);
            step(v0, [&](int n) { return weight(k, n); });
            load(v0, k + 2);
            if (k + 1 < kt) step(v1, [&](int n) { return weight(k + 1, n); });
        }
    } else {
        float4 v[AHEAD > 0 ? AHEAD : 1][4];
        uint4 w[AHEAD > 0 ? AHEAD : 1][NP];
        auto fetch = [&](int d, int k) {
            load(v[d], k);
#pragma unroll
            for (int n = 0; n < NP; ++n) w[d][n] = k < kt ? weight(k, n) : make_uint4(0u, 0u, 0u, 0u);
        };
#pragma unroll
        for (int d = 0; d < AHEAD; ++d) fetch(d, d);
        for (int k0 = 0; k0 < kt; k0 += AHEAD)
#pragma unroll
            for (int d = 0; d < AHEAD; ++d) {
                if (k0 + d >= kt) break;
                step(v[d], [&](int n) { return w[d][n]; });
                fetch(d, k0 + d + AHEAD);
            }
    }
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        const int col = blockIdx.y * (NP * 16) + n * 8 + 2 * t;
        const float2 bv = __ldg(reinterpret_cast<const float2*>(bias + col));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int m = m0 + g + h * 8;
            if (m >= M) continue;
            float2 v = make_float2(acc[n][2 * h] + bv.x, acc[n][2 * h + 1] + bv.y);
            const long long at = (long long)m * N + col;
            if (R) {
                const float2 r = *reinterpret_cast<const float2*>(R + at);
                v.x += r.x;
                v.y += r.y;
            }
            *reinterpret_cast<float2*>(out + at) = v;
        }
    }
}

// The same for many rows.  A warp still owns 16 rows and all n tiles, the sums are the same in the same order, but what a step reads comes
// through a ring of shared memory, RowsTile::STAGES stages of two k tiles: the rows of A as they are (float32, a warp reads only its
// own) and the weight fragments, once for all warps of the block.
template <int NT> struct RowsTile {
    static constexpr int NP = (NT + 1) / 2, STAGES = 4, W_BYTES = 2 * NP * 512;
    static constexpr int stage_bytes(int warps) { return warps * 16 * 128 + W_BYTES; }
};
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
template <int NT, typename HT>
__global__ void __launch_bounds__(256, 2)
rows_gate_tile_kernel(const float* __restrict__ A, const uint4* __restrict__ W, const float* __restrict__ bias, const float* __restrict__ gate,
                      int gate_rows, const float* R, float* out, int M, int N, int K) {
    using L = RowsTile<NT>;
    constexpr int NP = L::NP, STAGES = L::STAGES;
    extern __shared__ __align__(16) uint8_t smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3, rows = blockDim.x >> 1;
    const int mb = blockIdx.x * rows, m0 = mb + warp * 16, kt = (K + 15) / 16, ns = (kt + 1) / 2;
    const uint32_t sb = smem_addr(smem), stage_bytes = uint32_t(rows * 128 + L::W_BYTES);
    // 16-byte piece c of row r of a stage lies at piece c ^ 4 (r & 1): the lanes of two rows read all 32 banks at once
    const int cr = tid >> 3, cc = tid & 7, cstep = blockDim.x >> 3;
    const float* const gsrc = A + cc * 4;
    auto issue = [&](int s) {
        if (s < ns) {
            const uint32_t sa = sb + uint32_t(s % STAGES) * stage_bytes;
            const bool in = s * 32 + cc * 4 < K;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = cr + i * cstep;
                copy16(sa + uint32_t(r * 128 + ((cc ^ ((r & 1) << 2)) << 4)), in ? gsrc + (long long)min(mb + r, M - 1) * K + s * 32 : A, in);
            }
            const uint32_t sw = sa + uint32_t(rows * 128);
            const uint4* const ws = W + (long long)s * (2 * NP * 32);
            const int have = min(2, kt - 2 * s) * NP * 32;
            for (int i = tid; i < have; i += blockDim.x) copy16(sw + uint32_t(i * 16), ws + i, true);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int ra = min(m0 + g, M - 1), rb = min(m0 + g + 8, M - 1);
    const float* const ga = gate + (long long)(ra / gate_rows) * K + t * 4;
    const float* const gb = gate + (long long)(rb / gate_rows) * K + t * 4;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    auto gates = [&](float4 (&v)[2], int k) {
        const bool in = k * 16 + t * 4 < K;
        v[0] = in ? __ldg(reinterpret_cast<const float4*>(ga + k * 16)) : zero;
        v[1] = in ? __ldg(reinterpret_cast<const float4*>(gb + k * 16)) : zero;
    };
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[n][e] = 0.0f;
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) issue(s);
    float4 gv[2];
    gates(gv, 0);
    const uint32_t arow = uint32_t((warp * 16 + g) * 128);
    for (int s = 0; s < ns; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                                  // stage s has landed, stage s - 1 is read
        issue(s + STAGES - 1);
        const uint8_t* const st = smem + (s % STAGES) * stage_bytes;
        const uint4* const ws = reinterpret_cast<const uint4*>(st + rows * 128) + lane;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int k = 2 * s + h;
            if (k >= kt) break;
            const uint32_t piece = uint32_t(((h * 4 + t) ^ ((g & 1) << 2)) << 4);
            const float4 va = *reinterpret_cast<const float4*>(st + arow + piece), vb = *reinterpret_cast<const float4*>(st + arow + 8 * 128 + piece);
            const uint32_t af[4] = {Half<HT>::pack(va.x * gv[0].x, va.y * gv[0].y), Half<HT>::pack(vb.x * gv[1].x, vb.y * gv[1].y),
                                    Half<HT>::pack(va.z * gv[0].z, va.w * gv[0].w), Half<HT>::pack(vb.z * gv[1].z, vb.w * gv[1].w)};
            gates(gv, k + 1);
#pragma unroll
            for (int n = 0; n < NP; ++n) {
                const uint4 b = ws[(h * NP + n) * 32];
                Half<HT>::mma(acc[2 * n], af, b.x, b.y);
                if (2 * n + 1 < NT) Half<HT>::mma(acc[2 * n + 1 < NT ? 2 * n + 1 : 0], af, b.z, b.w);
            }
        }
    }
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        const int col = n * 8 + 2 * t;
        const float2 bv = __ldg(reinterpret_cast<const float2*>(bias + col));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int m = m0 + g + h * 8;
            if (m >= M) continue;
            float2 v = make_float2(acc[n][2 * h] + bv.x, acc[n][2 * h + 1] + bv.y);
            const long long at = (long long)m * N + col;
            if (R) {
                const float2 r = *reinterpret_cast<const float2*>(R + at);
                v.x += r.x;
                v.y += r.y;
            }
            *reinterpret_cast<float2*>(out + at) = v;
        }
    }
}

// The same with A already in the mode's 16-bit type [M][K], K a multiple of 32, no bias (the token projection).  A lane loads 16
// bytes, eight values of k; the first of two mma must have the lower sixteen of their 32 k, as in the layer kernel (which k share an
// mma shows in the rounding, their order in it does not), so lanes t and t + 2 exchange 8 bytes: 4 frames
// 5.1 us, 80 frames 12.8, 320 frames 35.7, 640 frames 41.9 (k permuted over both mma instead 4.6, 11.4, 31.6, 45.9; 8-byte loads 5.5,
// 16.1, 47.9, 50.7).
template <int NT, int AHEAD, typename HT>
__global__ void __launch_bounds__(128)
rows_h_kernel(const uint16_t* __restrict__ A, const uint4* __restrict__ W, float* __restrict__ out, int M, int N, int K) {
    constexpr int NP = NT / 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int m0 = (blockIdx.x * 4 + warp) * 16;
    if (m0 >= M) return;
    const uint16_t* const pa = A + (long long)min(m0 + g, M - 1) * K + t * 8;
    const uint16_t* const pb = A + (long long)min(m0 + g + 8, M - 1) * K + t * 8;
    const int np0 = blockIdx.y * NP, npall = gridDim.y * NP;
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[n][e] = 0.0f;
    const int ks = K / 32;
    auto weight = [&](int k, int h, int n) { return __ldg(W + ((long long)(2 * k + h) * npall + np0 + n) * 32 + lane); };
    const bool upper = (t & 2) != 0;
    // .x, .y: the lane's operand of the first mma, .z, .w: of the second
    auto exchange = [&](const uint4& v) {
        const uint32_t r0 = __shfl_xor_sync(0xffffffffu, upper ? v.x : v.z, 2), r1 = __shfl_xor_sync(0xffffffffu, upper ? v.y : v.w, 2);
        return upper ? make_uint4(r0, r1, v.z, v.w) : make_uint4(v.x, v.y, r0, r1);
    };
    auto step = [&](const uint4& ra, const uint4& rb, auto b_of) {
        const uint4 va = exchange(ra), vb = exchange(rb);
        const uint32_t a0[4] = {va.x, vb.x, va.y, vb.y}, a1[4] = {va.z, vb.z, va.w, vb.w};
#pragma unroll
        for (int n = 0; n < NP; ++n) {
            const uint4 b = b_of(0, n);
            Half<HT>::mma(acc[2 * n], a0, b.x, b.y);
            Half<HT>::mma(acc[2 * n + 1], a0, b.z, b.w);
        }
#pragma unroll
        for (int n = 0; n < NP; ++n) {
            const uint4 b = b_of(1, n);
            Half<HT>::mma(acc[2 * n], a1, b.x, b.y);
            Half<HT>::mma(acc[2 * n + 1], a1, b.z, b.w);
        }
    };
    if constexpr (AHEAD == 0) {
        uint4 va = __ldg(reinterpret_cast<const uint4*>(pa)), vb = __ldg(reinterpret_cast<const uint4*>(pb));
#pragma unroll 2
        for (int k = 0; k < ks; ++k) {
            const int kn = k + 1 < ks ? k + 1 : k;
            const uint4 na = __ldg(reinterpret_cast<const uint4*>(pa + kn * 32)), nb = __ldg(reinterpret_cast<const uint4*>(pb + kn * 32));
            step(va, vb, [&](int h, int n) { return weight(k, h, n); });
            va = na;
            vb = nb;
        }
    } else {
        uint4 va[AHEAD > 0 ? AHEAD : 1], vb[AHEAD > 0 ? AHEAD : 1], w[AHEAD > 0 ? AHEAD : 1][2][NP];
        auto fetch = [&](int d, int k) {
            const int kc = min(k, ks - 1);
            va[d] = __ldg(reinterpret_cast<const uint4*>(pa + kc * 32));
            vb[d] = __ldg(reinterpret_cast<const uint4*>(pb + kc * 32));
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int n = 0; n < NP; ++n) w[d][h][n] = weight(kc, h, n);
        };
#pragma unroll
        for (int d = 0; d < AHEAD; ++d) fetch(d, d);
        for (int k0 = 0; k0 < ks; k0 += AHEAD)
#pragma unroll
            for (int d = 0; d < AHEAD; ++d) {
                if (k0 + d >= ks) break;
                step(va[d], vb[d], [&](int h, int n) { return w[d][h][n]; });
                fetch(d, k0 + d + AHEAD);
            }
    }
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        const int col = (np0 * 2 + n) * 8 + 2 * t;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int m = m0 + g + h * 8;
            if (m < M) *reinterpret_cast<float2*>(out + (long long)m * N + col) = make_float2(acc[n][2 * h], acc[n][2 * h + 1]);
        }
    }
}

// ---------------------------------------------------------------------------------------------------- last convolution + pooling
// 1x1 160 -> 960, Hardswish, adaptive 4x4 average pooling of the 6 x 10 map, rounded to the 16-bit type the token projection
// reads it in.  A block takes a frame and 96 output channels; the map stays in shared memory.
struct Last {
    static constexpr int K = 160, KT = 10, XP = K + 8, N = 960, CE = 96, NT = CE / 8, P = CE + 8, PXS = 60;
    static constexpr int X_BYTES = 64 * XP * 2, SMEM = X_BYTES + PXS * P * 4;
};
template <typename HT>
__global__ void __launch_bounds__(256, 3)
last_pool_kernel(const float* __restrict__ x, const uint2* __restrict__ w, const float* __restrict__ b, uint16_t* __restrict__ pooled) {
    extern __shared__ __align__(16) uint8_t smem[];
    uint16_t* const X = reinterpret_cast<uint16_t*>(smem);
    float* const E = reinterpret_cast<float*>(smem + Last::X_BYTES);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3, f = blockIdx.x;
    const float* const img = x + (long long)f * (Last::PXS * Last::K);
    for (int i = tid; i < Last::PXS * Last::K / 4; i += 256) {
        const float4 p = *reinterpret_cast<const float4*>(img + i * 4);
        *reinterpret_cast<uint2*>(X + i / 40 * Last::XP + i % 40 * 4) = make_uint2(Half<HT>::pack(p.x, p.y), Half<HT>::pack(p.z, p.w));
    }
    // warp: one half of the n tiles, one of the four pixel groups
    const int mt = warp & 3, nt0 = (warp >> 2) * (Last::NT / 2);
    float c[Last::NT / 2][4];
#pragma unroll
    for (int n = 0; n < Last::NT / 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) c[n][e] = 0.0f;
    __syncthreads();
    const uint32_t xrow = smem_addr(X) + uint32_t(((mt * 16 + (lane & 15)) * Last::XP + (lane >> 4) * 8) * 2);
    const uint2* const wf = w + ((blockIdx.y * Last::NT + nt0) * Last::KT) * 32 + lane;
#pragma unroll 2
    for (int k = 0; k < Last::KT; ++k) {
        uint32_t af[4];
        ldmatrix_x4(af, xrow + uint32_t(k * 32));
#pragma unroll
        for (int n = 0; n < Last::NT / 2; ++n) {
            const uint2 bf = __ldg(wf + (n * Last::KT + k) * 32);
            Half<HT>::mma(c[n], af, bf.x, bf.y);
        }
    }
#pragma unroll
    for (int n = 0; n < Last::NT / 2; ++n) {
        const int col = (nt0 + n) * 8 + 2 * t;
        const float2 bv = __ldg(reinterpret_cast<const float2*>(b + blockIdx.y * Last::CE + col));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = mt * 16 + g + h * 8;
            if (r < Last::PXS) *reinterpret_cast<float2*>(E + r * Last::P + col) = hswish2(add2(make_float2(c[n][2 * h], c[n][2 * h + 1]), bv));
        }
    }
    __syncthreads();
    for (int i = tid; i < 16 * Last::CE / 2; i += 256) {
        const int cp = i % (Last::CE / 2), tok = i / (Last::CE / 2), r = tok >> 2, q = tok & 3;
        const int y0 = (r * 6) / 4, y1 = ((r + 1) * 6 + 3) / 4, x0 = (q * 10) / 4, x1 = ((q + 1) * 10 + 3) / 4;
        float2 s = make_float2(0.0f, 0.0f);
        for (int y = y0; y < y1; ++y)
            for (int xx = x0; xx < x1; ++xx) {
                const float2 v = *reinterpret_cast<const float2*>(E + (y * 10 + xx) * Last::P + cp * 2);
                s.x += v.x;
                s.y += v.y;
            }
        const float cnt = float((y1 - y0) * (x1 - x0));
        *reinterpret_cast<uint32_t*>(pooled + ((long long)f * 16 + tok) * Last::N + blockIdx.y * Last::CE + cp * 2) = Half<HT>::pack(s.x / cnt, s.y / cnt);
    }
}

//                CIN CEXP COUT K  S  HI  WI  TH  TW  CE PX SR NS  HS     RES    AHEAD  blocks/SM
using B2 = Block<16, 64, 24, 3, 2, 90, 160, 9, 8, 32, 2, 3, 1, false, false, true, 3>;
using B3 = Block<24, 72, 24, 3, 1, 45, 80, 9, 16, 72, 4, 3, 3, false, true, true, 2, 384>;
using B4 = Block<24, 72, 0, 5, 2, 45, 80, 6, 10, 24, 2, 3, 1, false, false, false, 3>;
using B5 = Block<40, 120, 0, 5, 1, 23, 40, 8, 40, 24, 4, 4, 1, false, false, false, 2>;
using B7 = Block<40, 240, 80, 3, 2, 23, 40, 6, 10, 48, 2, 3, 1, true, false, true, 2>;
using B8 = Block<80, 200, 80, 3, 1, 12, 20, 6, 20, 32, 4, 3, 2, true, true, true, 2>;
// few frames: smaller tiles, so that more SMs work, and for the fewest more channels at a time, so that fewer phases stand in a row
using B7F = Block<40, 240, 80, 3, 2, 23, 40, 3, 10, 80, 2, 3, 2, true, false, true, 2>;
using B8F = Block<80, 200, 80, 3, 1, 12, 20, 6, 10, 32, 2, 3, 2, true, true, true, 2>;
using B8S = Block<80, 200, 80, 3, 1, 12, 20, 3, 10, 64, 2, 3, 2, true, true, true, 2>;
using B9F = Block<80, 184, 80, 3, 1, 12, 20, 6, 10, 32, 2, 3, 2, true, true, true, 2>;
using B9S = Block<80, 184, 80, 3, 1, 12, 20, 3, 10, 64, 2, 3, 4, true, true, true, 2>;
using B9 = Block<80, 184, 80, 3, 1, 12, 20, 6, 20, 32, 4, 3, 2, true, true, true, 2>;
using B11 = Block<80, 480, 0, 3, 1, 12, 20, 12, 20, 32, 4, 4, 2, true, false, true, 2>;
using B12 = Block<112, 672, 0, 3, 1, 12, 20, 12, 20, 32, 4, 4, 2, true, false, true, 2>;
using B13 = Block<112, 672, 0, 5, 2, 12, 20, 6, 10, 32, 2, 2, 2, true, false, true, 2>;
using B14 = Block<160, 960, 0, 5, 1, 6, 10, 6, 10, 64, 5, 3, 4, true, false, false, 2>;

inline unsigned blocks_of(long long n, int per) { return unsigned((n + per - 1) / per); }
inline bool unaligned(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; }

template <class C, typename HT>
int launch_block(const BlockArgs& args, int F, cudaStream_t s) {
    static_assert(C::SMEM <= 227 * 1024, "shared memory");
    cudaError_t e = cudaFuncSetAttribute(block_kernel<C, HT>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    if (e != cudaSuccess) return int(e);
    BlockArgs a = args;
    dim3 grid(unsigned(F) * C::TILES, 1);
    if (C::SE) {
        // A block redoes the tile's input for its share of the channels, which costs about as much as three quarters of a chunk.  As many shares
        // as make the busiest SM's time least: n blocks there take n / 2 pairs, which share the SM at 1.25 times the time of one,
        // and the odd one.  us, one share / as the rule has it / 3 / 7: block 12, 48 frames 84 / 31 / 35 / 37, 96 frames 85 / 47 / 47 / 55, 256
        // frames 117 / 117 / 127 / 131, 640 frames 304 / 280 / 283 / 346.
        int groups = 1;
        float least = 1e30f;
        const int sms = device_sms();
        for (int g = 1; g <= C::CHUNKS; ++g) {
            const long long n = (grid.x * (long long)g + sms - 1) / sms;
            const float t = ((C::CHUNKS + g - 1) / g + 0.75f) * (1.25f * float(n / 2) + float(n % 2));
            if (t < least * 0.999f) { least = t; groups = g; }
        }
        a.chunks_per_group = (C::CHUNKS + groups - 1) / groups;
        grid.y = unsigned((C::CHUNKS + a.chunks_per_group - 1) / a.chunks_per_group);
    }
    block_kernel<C, HT><<<grid, C::THREADS, C::SMEM, s>>>(a);
    e = cudaGetLastError();
    if (e != cudaSuccess || !C::SE || C::POOL) return int(e);
    return se_partial_sums(a.out, a.sums, F, C::HO * C::WO, C::CEXP, s);
}

inline bool one_wave(long long blocks, int per_sm) { return blocks <= (long long)per_sm * device_sms(); }
template <typename HT>
int dispatch_block(int block, const BlockArgs& a, int F, cudaStream_t s) {
    switch (block) {
    case 2: return launch_block<B2, HT>(a, F, s);
    case 3: return launch_block<B3, HT>(a, F, s);
    case 4: return launch_block<B4, HT>(a, F, s);
    case 5: case 6: return launch_block<B5, HT>(a, F, s);
    // Whole blocks of the deeper maps have two to four tiles a frame, too few to fill the GPU with few frames.  us, large tiles / F / S:
    // block 7: 12 frames 20.2 / 16.1, 24 20.4 / 18, 40 27.9 / 26.2, 64 28.4 / 31.2; block 8: 12 26.2 / 17 / 14, 24 26 / 17.9 / 18,
    // 40 26.3 / 22.1 / 25.9, 64 26.1 / 22.1 / 30.5, 96 32.6 / 37.3.  The lines: two blocks an SM, and for S one.
    case 7: return one_wave(B7F::TILES * F, 2) ? launch_block<B7F, HT>(a, F, s) : launch_block<B7, HT>(a, F, s);
    case 8:
        return one_wave(B8S::TILES * F, 1) ? launch_block<B8S, HT>(a, F, s)
             : one_wave(B8F::TILES * F, 2) ? launch_block<B8F, HT>(a, F, s) : launch_block<B8, HT>(a, F, s);
    case 9: case 10:
        return one_wave(B9S::TILES * F, 1) ? launch_block<B9S, HT>(a, F, s)
             : one_wave(B9F::TILES * F, 2) ? launch_block<B9F, HT>(a, F, s) : launch_block<B9, HT>(a, F, s);
    case 11: return launch_block<B11, HT>(a, F, s);
    case 12: return launch_block<B12, HT>(a, F, s);
    case 13: return launch_block<B13, HT>(a, F, s);
    case 14: case 15: return launch_block<B14, HT>(a, F, s);
    default: return int(cudaErrorInvalidValue);
    }
}
int block_groups(int block) {
    switch (block) {
    case 4: return B4::GROUPS;
    case 5: case 6: return B5::GROUPS;
    case 11: return B11::GROUPS;
    case 12: return B12::GROUPS;
    case 13: return B13::GROUPS;
    case 14: case 15: return B14::GROUPS;
    default: return 0;
    }
}
// expanded channels a block walks (a multiple of its chunk), and the k range of its projection
void block_padding(int block, int* cols, int* k) {
#define SB_PAD(B) do { *cols = *k = B::KPAD; } while (0)
    *cols = *k = 0;
    switch (block) {
    case 2: SB_PAD(B2); break;
    case 3: SB_PAD(B3); break;
    case 4: SB_PAD(B4); break;
    case 5: case 6: SB_PAD(B5); break;
    case 7: SB_PAD(B7); break;
    case 8: SB_PAD(B8); break;
    case 9: case 10: SB_PAD(B9); break;
    case 11: SB_PAD(B11); break;
    case 12: SB_PAD(B12); break;
    case 13: SB_PAD(B13); break;
    case 14: case 15: SB_PAD(B14); break;
    default: break;
    }
#undef SB_PAD
}

}  // namespace
}  // namespace sb

// Host side: W [N][K] float32 -> 16-bit mma fragments.  order 0: fragments [n tile][k tile][lane] of 4 values, k as the
// instruction numbers it; order 1 / 2: [k tile][pair of n tiles][lane] of 8 values, k permuted inside a k tile so that a lane's
// operand A is four consecutive values of a row (1), or what it has of a tile after the exchange of rows_h_kernel (2: an even
// number of k tiles).
extern "C" size_t shvk_cnn_packed_bytes(int N, int K, int order) {
    if (N <= 0 || K <= 0 || order < 0 || order > 2) return 0;
    const size_t kt = size_t(order == 2 ? (K + 31) / 32 * 2 : (K + 15) / 16);
    return order == 0 ? size_t((N + 7) / 8) * kt * 32 * 8 : kt * size_t((N + 15) / 16) * 32 * 16;
}
extern "C" int shvk_cnn_pack_weights(const float* w, int N, int K, int order, int dtype, void* out) {
    if (!w || !out || !shvk_cnn_packed_bytes(N, K, order) || (dtype != sb::DT_BF16 && dtype != sb::DT_F16)) return int(cudaErrorInvalidValue);
    uint16_t* o = static_cast<uint16_t*>(out);
    auto put = [&](int n, int k) {
        const float v = n < N && k < K ? w[size_t(n) * K + k] : 0.0f;
        if (dtype == sb::DT_BF16) {
            const __nv_bfloat16 h = __float2bfloat16_rn(v);
            *o++ = *reinterpret_cast<const uint16_t*>(&h);
        } else {
            const __half h = __float2half_rn(v);
            *o++ = *reinterpret_cast<const uint16_t*>(&h);
        }
    };
    if (order == 0) {
        for (int nt = 0; nt < (N + 7) / 8; ++nt)
            for (int kt = 0; kt < (K + 15) / 16; ++kt)
                for (int lane = 0; lane < 32; ++lane)
                    for (int e = 0; e < 4; ++e) put(nt * 8 + lane / 4, kt * 16 + (e / 2) * 8 + (lane % 4) * 2 + e % 2);
    } else {
        const int kts = order == 2 ? (K + 31) / 32 * 2 : (K + 15) / 16;
        for (int kt = 0; kt < kts; ++kt)
            for (int np = 0; np < (N + 15) / 16; ++np)
                for (int lane = 0; lane < 32; ++lane)
                    for (int e = 0; e < 8; ++e) {
                        const int n = np * 16 + (e / 4) * 8 + lane / 4;
                        const int t = lane % 4, quad = order == 1 ? t : (t & 1) * 2 + (t >> 1);
                        put(n, kt * 16 + quad * 4 + e % 4);
                    }
    }
    return 0;
}

extern "C" int shvk_cnn_block_tiles(int block) { return sb::block_groups(block); }
extern "C" int shvk_cnn_block_launches(int block) { return block == 4 && !sb::B4::POOL ? 2 : 1; }
extern "C" void shvk_cnn_block_padding(int block, int* columns, int* k) { sb::block_padding(block, columns, k); }

extern "C" int shvk_cnn_block(int block, const float* x, const void* we, const float* be, const float* wd, const float* bd,
                              const void* wp, const float* bp, float* out, float* sums, int F, int dtype, void* stream) {
    if (F <= 0) return 0;
    const bool se = sb::block_groups(block) > 0;
    if (!x || !we || !be || !wd || !bd || !out || (se ? !sums : !wp || !bp) || out == x || sb::unaligned(x) || sb::unaligned(out) ||
        sb::unaligned(we) || (wp && sb::unaligned(wp)) || sb::unaligned(be) || sb::unaligned(wd) || sb::unaligned(bd) || (bp && sb::unaligned(bp)))
        return int(cudaErrorInvalidValue);
    const sb::BlockArgs a{x, static_cast<const uint2*>(we), be, wd, bd, static_cast<const uint2*>(wp), bp, out, sums, 0};
    if (dtype == sb::DT_BF16) return sb::dispatch_block<__nv_bfloat16>(block, a, F, cudaStream_t(stream));
    if (dtype == sb::DT_F16) return sb::dispatch_block<__half>(block, a, F, cudaStream_t(stream));
    return int(cudaErrorInvalidValue);
}

extern "C" int shvk_cnn_stem_block(const uint8_t* frames, const float* lut, const float* stem_w_host, const float* stem_b_host,
                                   const float* wd, const float* bd, const void* wp, const float* bp, float* out, int F, int dtype,
                                   void* stream) {
    if (F <= 0) return 0;
    if (!frames || !lut || !stem_w_host || !stem_b_host || !wd || !bd || !wp || !bp || !out || sb::unaligned(out) || sb::unaligned(wp) ||
        sb::unaligned(wd) || sb::unaligned(bd) || sb::unaligned(bp) || (dtype != sb::DT_BF16 && dtype != sb::DT_F16))
        return int(cudaErrorInvalidValue);
    sb::StemParams sp;
    for (int i = 0; i < 27 * 16; ++i) sp.w[i] = stem_w_host[i];
    for (int i = 0; i < 16; ++i) sp.b[i] = stem_b_host[i];
    const unsigned grid = unsigned(F) * sb::Stem::TILES;
    auto go = [&](auto kernel) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sb::Stem::SMEM);
        if (e != cudaSuccess) return int(e);
        kernel<<<grid, 256, sb::Stem::SMEM, cudaStream_t(stream)>>>(frames, lut, sp, wd, bd, static_cast<const uint2*>(wp), bp, out);
        return int(cudaGetLastError());
    };
    return dtype == sb::DT_BF16 ? go(sb::stem_block_kernel<__nv_bfloat16>) : go(sb::stem_block_kernel<__half>);
}

size_t sb::se_gate_frame_bytes(int C, int CS) {
    if (C > 1 << 20 || CS > 1 << 20) return ~size_t(0) / 8;             // nothing that fits, and nothing that overflows
    return size_t(gate_rows_padded(C) + gate_rows_padded(CS)) * sizeof(float);
}

extern "C" int shvk_cnn_se_gate_sums(const float* sums, const float* w1, const float* b1, const float* w2, const float* b2, float* gate,
                                     int F, int tiles, int HW, int C, int CS, void* stream) {
    if (F <= 0) return 0;
    if (!sums || !w1 || !b1 || !w2 || !b2 || !gate || tiles <= 0 || HW <= 0 || C <= 0 || CS <= 0 || (C & 3)) return int(cudaErrorInvalidValue);
    // Frames per cluster: one while that gives an SM three blocks or fewer (960 channels, one / four: 56 frames 18.7 / 27 us, 75 frames
    // 29.8 / 29.8, 112 frames 33 / 30), else four (a weight row serves four frames)
    const int sms = sb::device_sms(), G = 8LL * F <= 3 * sms ? 1 : 4;
    const size_t smem = size_t(G) * sb::se_gate_frame_bytes(C, CS);
    if (smem > 48 * 1024) return int(cudaErrorInvalidValue);
    const unsigned grid = sb::blocks_of(F, G) * 8;
    cudaStream_t s = cudaStream_t(stream);
    // Four outputs of a warp at a time up to two blocks an SM (960 channels, four / one: 75 frames 29.7 / 33.6 us, 130 frames 31.7 / 36.6);
    // beyond, other clusters hide the loads and the narrow maps pay for the registers (120 channels, 300 frames 14.1 / 11.4), so two:
    // a frame's values are read from shared memory once for both (640 frames, two / one: 960 channels 100 / 114 us, 480 55 / 60)
    auto go = [&](auto kernel) {
        kernel<<<grid, 256, smem, s>>>(sums, w1, b1, w2, b2, gate, F, tiles, float(HW), C, CS);
        return int(cudaGetLastError());
    };
    if (G == 1) return go(sb::se_gate_cluster_kernel<1, 4>);
    return grid <= 2u * sms ? go(sb::se_gate_cluster_kernel<4, 4>) : go(sb::se_gate_cluster_kernel<4, 2>);
}

namespace sb {
namespace {
template <typename HT>
int launch_rows_gate(const float* A, const uint4* W, const float* b, const float* gate, int gate_rows, const float* R, float* out, int M,
                     int N, int K, cudaStream_t s) {
    const unsigned gx = blocks_of(M, 64);
    // Few rows: a warp's chain of k steps is all the time there is, so its loads run ahead and the n tiles go to other blocks.  us,
    // whole / split: 160 channels of 960: 4 frames 41 / 15, 40 frames 64 / 18, 160 frames 64 / 43, 320 frames 75 / 87; 112 channels
    // of 480: 4 frames 23 / 10, 40 frames 33 / 24, 80 frames 33 / 39 (300 row blocks).
    const int sms = device_sms();
    const bool few = 12LL * gx <= 13 * sms;     // about a row block per SM
    auto go = [&](auto kernel, unsigned gy) {
        kernel<<<dim3(gx, gy), 128, 0, s>>>(A, W, b, gate, gate_rows, R, out, M, N, K);
        return int(cudaGetLastError());
    };
    // Rows of a block, 16 a warp: what leaves the busiest SM the fewest rows
    auto tiled = [&](auto kernel, auto layout) {
        int warps = 8;
        long long least = 1LL << 62;
        for (int w = 8; w >= 4; --w) {
            const long long rows = ((blocks_of(M, w * 16) + sms - 1) / sms) * (long long)w;
            if (rows < least) { least = rows; warps = w; }
        }
        const int smem = decltype(layout)::STAGES * decltype(layout)::stage_bytes(warps);
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, decltype(layout)::STAGES * decltype(layout)::stage_bytes(8));
        if (e != cudaSuccess) return int(e);
        kernel<<<blocks_of(M, warps * 16), warps * 32, smem, s>>>(A, W, b, gate, gate_rows, R, out, M, N, K);
        return int(cudaGetLastError());
    };
    // 40 channels of 72: three stages are too few for the ring to help (256 / 640 frames, direct / ring: 26.5 / 28.6, 61.4 / 61.3);
    // of 120: 67.5 / 57.4, 141 / 120; 112 of 480: 73.7 / 51, 170 / 118; 160 of 960: 69.6 / 48, 154 / 108
    switch (N) {
    case 40: return few ? go(rows_gate_kernel<5, 4, HT>, 1) : K > 96 ? tiled(rows_gate_tile_kernel<5, HT>, RowsTile<5>()) : go(rows_gate_kernel<5, 0, HT>, 1);
    case 112: return few ? go(rows_gate_kernel<2, 6, HT>, 7) : tiled(rows_gate_tile_kernel<14, HT>, RowsTile<14>());
    case 160: return few ? go(rows_gate_kernel<4, 6, HT>, 5) : tiled(rows_gate_tile_kernel<20, HT>, RowsTile<20>());
    default: return int(cudaErrorInvalidValue);
    }
}
}  // namespace
}  // namespace sb

extern "C" int shvk_cnn_rows_gate(const float* A, const void* W, const float* b, const float* gate, int gate_rows, const float* R,
                                  float* out, int M, int N, int K, int dtype, void* stream) {
    if (M <= 0) return 0;
    if (!A || !W || !b || !gate || gate_rows <= 0 || !out || K <= 0 || (K & 3) || sb::unaligned(A) || sb::unaligned(W) || sb::unaligned(b) ||
        sb::unaligned(gate) || (R && sb::unaligned(R)) || sb::unaligned(out))
        return int(cudaErrorInvalidValue);
    const uint4* w = static_cast<const uint4*>(W);
    if (dtype == sb::DT_BF16) return sb::launch_rows_gate<__nv_bfloat16>(A, w, b, gate, gate_rows, R, out, M, N, K, cudaStream_t(stream));
    if (dtype == sb::DT_F16) return sb::launch_rows_gate<__half>(A, w, b, gate, gate_rows, R, out, M, N, K, cudaStream_t(stream));
    return int(cudaErrorInvalidValue);
}

extern "C" int shvk_cnn_last_pool(const float* x, const void* w, const float* b, void* pooled, int F, int dtype, void* stream) {
    if (F <= 0) return 0;
    if (!x || !w || !b || !pooled || sb::unaligned(x) || sb::unaligned(w) || sb::unaligned(b) || sb::unaligned(pooled))
        return int(cudaErrorInvalidValue);
    auto go = [&](auto kernel) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sb::Last::SMEM);
        if (e != cudaSuccess) return int(e);
        kernel<<<dim3(unsigned(F), sb::Last::N / sb::Last::CE), 256, sb::Last::SMEM, cudaStream_t(stream)>>>(x, static_cast<const uint2*>(w), b,
                                                                                                     static_cast<uint16_t*>(pooled));
        return int(cudaGetLastError());
    };
    if (dtype == sb::DT_BF16) return go(sb::last_pool_kernel<__nv_bfloat16>);
    if (dtype == sb::DT_F16) return go(sb::last_pool_kernel<__half>);
    return int(cudaErrorInvalidValue);
}

extern "C" int shvk_cnn_token_proj(const void* pooled, const void* W, float* tokens, int rows, int dtype, void* stream) {
    if (rows <= 0) return 0;
    if (!pooled || !W || !tokens || sb::unaligned(pooled) || sb::unaligned(W) || sb::unaligned(tokens)) return int(cudaErrorInvalidValue);
    const uint16_t* A = static_cast<const uint16_t*>(pooled);
    const uint4* w = static_cast<const uint4*>(W);
    cudaStream_t s = cudaStream_t(stream);
    const unsigned gx = sb::blocks_of(rows, 64);
    // as in launch_rows_gate, up to a row block for about two SMs: 4 frames 26 / 9 us, 40 frames 55 / 12, 320 frames (80 blocks) 51 / 37
    const bool few = 11LL * gx <= 6 * sb::device_sms();
    auto go = [&](auto kernel, unsigned gy) {
        kernel<<<dim3(gx, gy), 128, 0, s>>>(A, w, tokens, rows, 384, 960);
        return int(cudaGetLastError());
    };
    if (dtype == sb::DT_BF16) return few ? go(sb::rows_h_kernel<2, 8, __nv_bfloat16>, 24) : go(sb::rows_h_kernel<8, 0, __nv_bfloat16>, 6);
    if (dtype == sb::DT_F16) return few ? go(sb::rows_h_kernel<2, 8, __half>, 24) : go(sb::rows_h_kernel<8, 0, __half>, 6);
    return int(cudaErrorInvalidValue);
}

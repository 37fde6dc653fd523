// Products of some tens to some hundreds of rows on the 5th-generation tensor cores with the weights as the operand in
// tensor memory: y[M, N] = x[M, K] * W[N, K]^T (+ bias), W in Q4_K (both orders), Q4_0, Q8_0, Q6_K or K-blocked MXFP4.
//
// What bounds it: the decode, about three instructions per weight and lane, then the tensor cores (a step of 128 weight
// rows x 64 k against 128 tokens is 256 clocks of them). The weights are the rows of the MMA (M = 128) and the tokens its
// columns (N = 16 .. 128), so that a decoding thread owns one weight row: its block headers stay in its registers, its
// raw bytes are its own row of a box in shared memory (conflict-free 16-byte reads), and the bf16 pairs it makes go
// straight into its lane of tensor memory (tcgen05.st) -- no swizzled stores to shared memory, no proxy fence, no reads
// of the weights by the tensor core through shared memory.
//   warps 0-7   decode: warps 0-3 the first, 4-7 the second 128 weights of every 256 (two 64-wide k steps each, four
//               operand stages of 32 columns in all), afterwards the epilogue;
//   warp 8      one thread streams the raw blocks of 128 rows x 256 weights (TMA boxes; Q6_K, whose 210-byte blocks no
//               tensor map can address, from the tiled copy, eight bulk copies);
//   warp 9      one thread issues the MMAs;
//   warp 10     bf16 activations: one thread streams their boxes;
//   warps 10-13 f32 activations: each converts every fourth k step to bf16 in the swizzled layout.
// Half of an SM's tensor memory and shared memory each, so that two CTAs share an SM and one decodes while the other
// starts or ends. K is split over the CTAs of a cluster where the tiles are few: every CTA leaves its sums in its own
// shared memory and adds up its share of the columns over the others' in rank order (no scratch buffer, no second launch).
// Weights are rounded to bf16 after an exact f32 decode, sums are f32.
// Every wait is bounded; a CTA that gives up records it, still meets its cluster and frees its tensor memory.
#include <cuda.h>
#include <cuda_bf16.h>
#include <limits.h>
#include <string.h>

#include <type_traits>

#include "decode.cuh"
#include "gemm_tc.h"
#include "skinny.h"
#include "sync.cuh"
#include "tcgen05.cuh"

namespace nnq {

constexpr int kTsDecodeWarps = 8;
constexpr int kTsLoadWarp = 8, kTsMmaWarp = 9, kTsXWarp = 10, kTsXWarps = 4;
constexpr int kTsMaxN = 128;         // tokens of a tile
constexpr int kTsMaxJobs = 8;
constexpr int kTsMaxX = 8;
constexpr int kTsSmem = 111 * 1024;  // two CTAs per SM
constexpr int kTsSmemMin = 80 * 1024;   // never three: their tensor memory would not fit, and clusters would wait for one another

// raw bytes of 128 rows x 256 weights in shared memory
template <int FMT>
struct TsGeom {
    static constexpr bool kTiled = FMT == NNQ_Q6_K;
    static constexpr int kPitch = FMT == NNQ_Q8_0 ? 272 : (FMT == NNQ_MXFP4_SPLIT ? 128 : (kTiled ? 210 : 144));
    static constexpr int kCopy = kTiled ? 8 * 3360 : 128 * kPitch;       // bytes that arrive
    static constexpr int kBytes = (kCopy + 1023) / 1024 * 1024;
    static constexpr int kStages = 2;
};

struct TsJob {
    CUtensorMap map;         // raw blocks as 32-bit words
    const uint8_t *tiled;    // Q6_K
    const uint8_t *scales;   // MXFP4
    const float *bias;
    void *y;
    int n, tile_begin;
};
struct TsParams {
    CUtensorMap xmap;
    TsJob job[kTsMaxJobs];
    const float *xf;         // f32 activations
    int njobs, m, k, nt, xstages, y_dt;
    int *status;
};

__device__ __forceinline__ void ts_tma_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void ts_st16(uint32_t addr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};"
        ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
          "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t ts_pack(float2 v) { return pack_bf16(v.x, v.y); }

// ---------------------------------------------------------------------------------
// The 32 weights of a sub-block as sixteen bf16 pairs, exactly as the f32 decode rounds them.
// ---------------------------------------------------------------------------------

// 32-bit word at halfword h of a row whose words from W0 on are in registers
template <int W0, int NW>
__device__ __forceinline__ uint32_t ts_word(const uint32_t (&w)[NW], int h) {
    return h & 1 ? __funnelshift_r(w[(h >> 1) - W0], w[(h >> 1) + 1 - W0], 16) : w[(h >> 1) - W0];
}

// eight four-bit codes of a word, low nibble first: (q - bias) * s (+ c) two at a time
template <bool ADD>
__device__ __forceinline__ void ts_nibbles(uint32_t q, float2 unbias, float2 s2, float2 c2, uint32_t *o) {
    const uint32_t lo = q & 0x0F0F0F0Fu, hi = (q >> 4) & 0x0F0F0F0Fu;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float2 c = make_float2(__uint_as_float(__byte_perm(lo, 0x4B000000u, 0x7540 + i)), __uint_as_float(__byte_perm(hi, 0x4B000000u, 0x7540 + i)));
        c = __fadd2_rn(c, unbias);
        o[i] = ts_pack(ADD ? __ffma2_rn(c, s2, c2) : __fmul2_rn(c, s2));   // (s q has 21 bits at most: the sum is rounded once either way)
    }
}

template <int FMT, int H>
struct TsDecode;   // H = which 128 of the 256 weights; sub<J>: sub-block J (0..7) of the 256

template <int H>
struct TsDecode<NNQ_Q4_K, H> {
    uint4 hdr;
    const uint4 *p;
    __device__ __forceinline__ void open(const uint8_t *stage, int row, const TsJob &, int, int, int) {
        p = reinterpret_cast<const uint4 *>(stage + row * 144);
        hdr = p[0];
    }
    template <int J>
    __device__ __forceinline__ void sub(uint32_t (&o)[16]) {
        const uint4 q = p[1 + J];
        const float d = f16_bits_to_f32((uint16_t)(hdr.x & 0xFFFFu)), dmin = f16_bits_to_f32((uint16_t)(hdr.x >> 16));
        const uint32_t sc = ((hdr.y >> (8 * (J >> 1) + 4 * (J & 1))) & 15u) | (((hdr.w >> (8 * (J >> 2) + 2 * (J & 3))) & 3u) << 4);
        const uint32_t mn = ((hdr.z >> (8 * (J >> 1) + 4 * (J & 1))) & 15u) | (((hdr.w >> (16 + 8 * (J >> 2) + 2 * (J & 3))) & 3u) << 4);
        const float s = __fmul_rn(d, u2f(sc)), m = __fmul_rn(dmin, u2f(mn));
        const float2 unbias = make_float2(-8388608.0f, -8388608.0f), s2 = make_float2(s, s), nm = make_float2(-m, -m);
        ts_nibbles<true>(q.x, unbias, s2, nm, o);
        ts_nibbles<true>(q.y, unbias, s2, nm, o + 4);
        ts_nibbles<true>(q.z, unbias, s2, nm, o + 8);
        ts_nibbles<true>(q.w, unbias, s2, nm, o + 12);
    }
};

template <int H>
struct TsDecode<NNQ_Q4_K_GGML, H> {
    uint4 hdr;
    const uint4 *p;
    __device__ __forceinline__ void open(const uint8_t *stage, int row, const TsJob &, int, int, int) {
        p = reinterpret_cast<const uint4 *>(stage + row * 144);
        hdr = p[0];
    }
    template <int J>
    __device__ __forceinline__ void sub(uint32_t (&o)[16]) {
        const uint4 q0 = p[1 + 2 * (J >> 1)], q1 = p[2 + 2 * (J >> 1)];
        const float d = f16_bits_to_f32((uint16_t)(hdr.x & 0xFFFFu)), dmin = f16_bits_to_f32((uint16_t)(hdr.x >> 16));
        const uint32_t S[3] = {hdr.y, hdr.z, hdr.w};
        auto sbyte = [&](int i) -> uint32_t { return (S[i >> 2] >> (8 * (i & 3))) & 0xFFu; };
        const uint32_t sc = J < 4 ? sbyte(J) & 63u : (sbyte(J + 4) & 15u) | ((sbyte(J & 3) >> 6) << 4);
        const uint32_t mn = J < 4 ? sbyte(J + 4) & 63u : (sbyte(J + 4) >> 4) | ((sbyte(J) >> 6) << 4);
        const float s = __fmul_rn(d, u2f(sc)), m = __fmul_rn(dmin, u2f(mn));
        const float2 unbias = make_float2(-8388608.0f, -8388608.0f), s2 = make_float2(s, s), nm = make_float2(-m, -m);
        const uint32_t qw[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
        for (int v = 0; v < 8; v++) {
            const uint32_t n = (J & 1 ? qw[v] >> 4 : qw[v]) & 0x0F0F0F0Fu;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                float2 c = make_float2(__uint_as_float(__byte_perm(n, 0x4B000000u, 0x7540 + 2 * i)), __uint_as_float(__byte_perm(n, 0x4B000000u, 0x7541 + 2 * i)));
                o[2 * v + i] = ts_pack(__ffma2_rn(__fadd2_rn(c, unbias), s2, nm));
            }
        }
    }
};

template <int H>
struct TsDecode<NNQ_Q4_0, H> {
    static constexpr int W0 = H ? 16 : 0;   // blocks 4H .. 4H+3: bytes 72H .. 72H+71
    uint32_t w[20];
    __device__ __forceinline__ void open(const uint8_t *stage, int row, const TsJob &, int, int, int) {
        const uint4 *p = reinterpret_cast<const uint4 *>(stage + row * 144) + W0 / 4;
#pragma unroll
        for (int i = 0; i < 5; i++) {
            const uint4 v = p[i];
            w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
        }
    }
    template <int J>
    __device__ __forceinline__ void sub(uint32_t (&o)[16]) {
        constexpr int h = 9 * J;
        const float d = f16_bits_to_f32((uint16_t)(w[(h >> 1) - W0] >> (16 * (h & 1))));
        const float2 unbias = make_float2(-8388616.0f, -8388616.0f), d2 = make_float2(d, d), none = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int v = 0; v < 4; v++) ts_nibbles<false>(ts_word<W0>(w, h + 1 + 2 * v), unbias, d2, none, o + 4 * v);
    }
};

template <int H>
struct TsDecode<NNQ_Q8_0, H> {
    const uint8_t *p;
    __device__ __forceinline__ void open(const uint8_t *stage, int row, const TsJob &, int, int, int) { p = stage + row * 272; }
    template <int J>
    __device__ __forceinline__ void sub(uint32_t (&o)[16]) {
        constexpr int h = 17 * J, W0 = (h / 2) & ~3;   // the block: halfwords h .. h+16, inside three or four 16-byte words
        constexpr int NV = ((h + 16) / 2) / 4 - W0 / 4 + 1;
        uint32_t w[4 * NV];
#pragma unroll
        for (int i = 0; i < NV; i++) {
            const uint4 v = reinterpret_cast<const uint4 *>(p)[W0 / 4 + i];
            w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
        }
        const float d = f16_bits_to_f32((uint16_t)(w[(h >> 1) - W0] >> (16 * (h & 1))));
        const float2 unbias = make_float2(-(8388608.0f + 128.0f), -(8388608.0f + 128.0f)), d2 = make_float2(d, d);
#pragma unroll
        for (int v = 0; v < 8; v++) {
            const uint32_t q = ts_word<W0>(w, h + 1 + 2 * v) ^ 0x80808080u;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                float2 c = make_float2(__uint_as_float(__byte_perm(q, 0x4B000000u, 0x7540 + 2 * i)), __uint_as_float(__byte_perm(q, 0x4B000000u, 0x7541 + 2 * i)));
                o[2 * v + i] = ts_pack(__fmul2_rn(__fadd2_rn(c, unbias), d2));
            }
        }
    }
};

// the tiled copy: 16 rows x 256 weights in 3360 bytes; a row's four words of a sub-block lie side by side
template <int H>
struct TsDecode<NNQ_Q6_K, H> {
    const uint8_t *tile;
    int r;
    float d;
    uint2 sc;
    __device__ __forceinline__ void open(const uint8_t *stage, int row, const TsJob &, int, int, int) {
        tile = stage + (row >> 4) * 3360;
        r = row & 15;
        sc = *reinterpret_cast<const uint2 *>(tile + 16 * r + 8 * H);   // the scales of this half's eight groups
        d = __half2float(reinterpret_cast<const __half *>(tile + 256)[r]);
    }
    template <int J>
    __device__ __forceinline__ void sub(uint32_t (&o)[16]) {
        const uint8_t *c = tile + 288 + 384 * J;
        const uint4 lo = *reinterpret_cast<const uint4 *>(c + 128 * (r >> 3) + 16 * (r & 7)), hi = *reinterpret_cast<const uint4 *>(c + 256 + 16 * (r & 7));
        const uint32_t two = (J & 2 ? sc.y : sc.x) >> (16 * (J & 1));
        const float sa = __fmul_rn(d, s8_to_f(two & 0xFFu)), sb = __fmul_rn(d, s8_to_f((two >> 8) & 0xFFu));
        const float2 s0 = make_float2(sa, sa), s1 = make_float2(sb, sb), unbias = make_float2(-8388640.0f, -8388640.0f);
        const uint32_t l[4] = {lo.x, lo.y, lo.z, lo.w}, h4[4] = {hi.x, hi.y, hi.z, hi.w};
        const int sh = r & 8;
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const uint32_t h = h4[t] >> sh;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t up = (i < 2 ? h << (4 - 2 * i) : h >> (2 * i - 4)) & 0x00300030u;
                const uint32_t q = ((l[t] >> (4 * i)) & 0x000F000Fu) | up;
                float2 v = make_float2(__uint_as_float(__byte_perm(q, 0x4B000000u, 0x7540)), __uint_as_float(__byte_perm(q, 0x4B000000u, 0x7542)));
                o[(i >> 1) * 8 + 2 * t + (i & 1)] = ts_pack(__fmul2_rn(__fadd2_rn(v, unbias), i < 2 ? s0 : s1));
            }
        }
    }
};

// codes of 256 weights: eight 16-byte words per row, 128-byte swizzle; scale bytes [n, k / 32] from global memory
template <int H>
struct TsDecode<NNQ_MXFP4_SPLIT, H> {
    const uint8_t *p;
    int x7;
    uint32_t e[4];
    __device__ __forceinline__ void open(const uint8_t *stage, int row, const TsJob &J, int grow, int unit, int blocks) {
        p = stage + row * 128;
        x7 = row & 7;
        const uint8_t *s = J.scales + (size_t)(grow < J.n ? grow : 0) * blocks;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int b = unit * 8 + 4 * H + i;
            e[i] = b < blocks ? __ldg(s + b) : 127u;
        }
    }
    template <int J>
    __device__ __forceinline__ void sub(uint32_t (&o)[16]) {
        const uint4 q = *reinterpret_cast<const uint4 *>(p + ((J ^ x7) << 4));
        const uint32_t sc = max(e[J & 3] << 7, 0x40u), s2 = sc | (sc << 16);   // 2^(e - 127) in bf16, e = 0: 2^-127
        const uint32_t w4[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int v = 0; v < 4; v++) {
            const uint32_t w = w4[v], sel = w & 0x77777777u;
            // E2M1 magnitudes as the two bytes of a bf16: 0, .5, 1, 1.5, 2, 3, 4, 6
            const uint32_t la = __byte_perm(0xC0800000u, 0xC0804000u, sel), ha = __byte_perm(0x3F3F3F00u, 0x40404040u, sel);
            const uint32_t lb = __byte_perm(0xC0800000u, 0xC0804000u, sel >> 16), hb = __byte_perm(0x3F3F3F00u, 0x40404040u, sel >> 16);
            const uint32_t m[4] = {__byte_perm(la, ha, 0x5140), __byte_perm(la, ha, 0x7362), __byte_perm(lb, hb, 0x5140), __byte_perm(lb, hb, 0x7362)};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t a = i < 2 ? w << (12 - 8 * i) : w >> (8 * i - 12), b = w << (24 - 8 * i);
                uint32_t u = m[i] | (a & 0x8000u) | (b & 0x80000000u);
                __nv_bfloat162 z = __hmul2(*reinterpret_cast<__nv_bfloat162 *>(&u), *reinterpret_cast<const __nv_bfloat162 *>(&s2));
                o[4 * v + i] = *reinterpret_cast<uint32_t *>(&z);
            }
        }
    }
};

template <int FMT, bool F32X>
__global__ void __launch_bounds__((kTsXWarp + (F32X ? kTsXWarps : 1)) * 32, 2)
gemm_ts_kernel(const __grid_constant__ TsParams P) {
    using G = TsGeom<FMT>;
    constexpr int W = G::kStages;
    extern __shared__ uint8_t ts_smem_raw[];
    uint8_t *smem = ts_smem_raw + (-smem_u32(ts_smem_raw) & 1023u);   // (stays an address in shared memory to the compiler)
    // w_full, w_empty [W], x_full, x_empty [8], a_full, a_empty [4], accumulators ready
    __shared__ __align__(8) uint64_t bars[2 * W + 2 * kTsMaxX + 9];
    __shared__ uint32_t tmem_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0);
    const uint32_t wf = smem_u32(bars), we = wf + 8 * W, xf = we + 8 * W, xe = xf + 8 * kTsMaxX, af = xe + 8 * kTsMaxX, ae = af + 32, acc = ae + 32;
    const int nt = P.nt, xstages = P.xstages, xbytes = nt * 128;
    uint8_t *xs = smem + W * G::kBytes;

    int j = 0;
#pragma unroll
    for (int i = 1; i < kTsMaxJobs; i++)
        if (i < P.njobs && (int)blockIdx.x >= P.job[i].tile_begin) j = i;
    const TsJob &J = P.job[j];
    const int n0 = ((int)blockIdx.x - J.tile_begin) * 128, m0 = (int)blockIdx.y * nt;
    // this CTA's units of 256 weights, and the 64-wide k steps in them
    const int units = (P.k + 255) >> 8, splits = (int)gridDim.z, rank = (int)blockIdx.z;
    const int u_lo = rank * units / splits, nu = (rank + 1) * units / splits - u_lo;
    const int steps = min((P.k >> 6) - 4 * u_lo, 4 * nu);

    if (tid == 0) {
        for (int i = 0; i < W; i++) {
            mbar_init(wf + 8 * i, 1);
            mbar_init(we + 8 * i, kTsDecodeWarps);
        }
        for (int i = 0; i < kTsMaxX; i++) {
            mbar_init(xf + 8 * i, 1);
            mbar_init(xe + 8 * i, 1);
        }
        for (int i = 0; i < 4; i++) {
            mbar_init(af + 8 * i, 4);
            mbar_init(ae + 8 * i, 1);
        }
        mbar_init(acc, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kTsMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)), "r"(256u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, tmem_s, 0), tmem_a = tmem + 128;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    bool ok = true;
    int issued = 0;   // copies under way, of the two threads that start them

    if (warp < kTsDecodeWarps) {
        // ---------------- decode ----------------
        const int half = warp >> 2, row = (warp & 3) * 32 + lane;
        const uint32_t mine = tmem_a + ((uint32_t)(warp & 3) << 21) + 64 * half;
        int slot = 0;
        uint32_t ph = 0;
        auto run = [&](auto hc) {
            constexpr int H = decltype(hc)::value;
            for (int u = 0; u < nu && ok; u++) {
                ok = __all_sync(0xFFFFFFFFu, mbar_wait_fast(wf + 8 * slot, ph));
                if (!ok) break;
                TsDecode<FMT, H> D;
                D.open(smem + slot * G::kBytes, row, J, n0 + row, u_lo + u, P.k >> 5);
                const int left = steps - 4 * u - 2 * H;   // k steps of this half that exist
                auto step = [&](auto sc) {
                    constexpr int S = decltype(sc)::value;   // 0 or 1: sub-blocks 4H + 2S, 4H + 2S + 1
                    uint32_t o[16];
                    D.template sub<4 * H + 2 * S>(o);
                    if (u) ok &= __all_sync(0xFFFFFFFFu, mbar_wait_fast(ae + 8 * (2 * H + S), (uint32_t)(u - 1) & 1u)) != 0;
                    tc_fence_after();
                    ts_st16(mine + 32 * S, o);
                    D.template sub<4 * H + 2 * S + 1>(o);
                    ts_st16(mine + 32 * S + 16, o);
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    tc_fence_before();
                    __syncwarp();
                    if (elect_one()) mbar_arrive(af + 8 * (2 * H + S));
                };
                if (left > 0) step(std::integral_constant<int, 0>{});
                if (left > 1) step(std::integral_constant<int, 1>{});
                __syncwarp();
                if (elect_one()) mbar_arrive(we + 8 * slot);
                if (++slot == W) {
                    slot = 0;
                    ph ^= 1u;
                }
            }
        };
        if (half) run(std::integral_constant<int, 1>{});
        else run(std::integral_constant<int, 0>{});
    } else if (warp == kTsLoadWarp) {
        // ---------------- weights ----------------
        if (lane == 0) {
            const int tiles16 = (J.n + 15) >> 4;   // row tiles of the tiled copy
            for (int u = 0; u < nu; u++) {
                const int s = u % W;
                if (u >= W) ok = mbar_wait_fast(we + 8 * s, ((uint32_t)(u / W) & 1u) ^ 1u);
                if (!ok) break;
                const uint32_t dst = smem_u32(smem + s * G::kBytes);
                if (G::kTiled) {
                    const int have = min(8, tiles16 - n0 / 16);
                    mbar_expect_tx(wf + 8 * s, have * 3360);
                    for (int i = 0; i < have; i++) bulk_g2s(dst + i * 3360, J.tiled + ((size_t)(n0 / 16 + i) * units + u_lo + u) * 3360, 3360, wf + 8 * s);
                } else {
                    mbar_expect_tx(wf + 8 * s, G::kCopy);
                    ts_tma_2d(dst, &J.map, (u_lo + u) * (G::kPitch / 4), n0, wf + 8 * s);
                }
                issued = u + 1;
            }
            // every copy has landed before this CTA's shared memory is used again or given back
            for (int i = max(0, issued - W); i < issued; i++) ok &= mbar_wait(wf + 8 * (i % W), (uint32_t)(i / W) & 1u);
        }
    } else if (warp == kTsMmaWarp) {
        // ---------------- MMA issuer (the warp waits together, one lane issues) ----------------
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(nt >> 3) << 17) | ((128u >> 4) << 24);
        int xslot = 0;
        uint32_t xph = 0;
        for (int kb = 0; kb < steps; kb++) {
            const int a = kb & 3;
            ok = __all_sync(0xFFFFFFFFu, mbar_wait_fast(xf + 8 * xslot, xph) && mbar_wait_fast(af + 8 * a, (uint32_t)(kb >> 2) & 1u));
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const uint64_t db = smem_desc(smem_u32(xs + xslot * xbytes));
#pragma unroll
                for (int k = 0; k < 4; k++) umma_ts(tmem, tmem_a + 32 * a + 8 * k, db + 2 * k, idesc, (kb | k) != 0);
                umma_commit(ae + 8 * a);
                umma_commit(xe + 8 * xslot);
            }
            __syncwarp();
            if (++xslot == xstages) {
                xslot = 0;
                xph ^= 1u;
            }
        }
        if (elect_one()) umma_commit(acc);
    } else if (!F32X) {
        // ---------------- activations (a thread of their own: neither ring waits for the other's consumers) ----------------
        if (lane == 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");   // they come from the kernel before this one
            int s = 0;
            uint32_t ph = 1;
            for (int kb = 0; kb < steps; kb++) {
                if (kb >= xstages) ok = mbar_wait_fast(xe + 8 * s, ph);
                if (!ok) break;
                mbar_expect_tx(xf + 8 * s, xbytes);
                ts_tma_2d(smem_u32(xs + s * xbytes), &P.xmap, (4 * u_lo + kb) * 64, m0, xf + 8 * s);
                issued = kb + 1;
                if (++s == xstages) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            for (int i = max(0, issued - xstages); i < issued; i++) ok &= mbar_wait(xf + 8 * (i % xstages), (uint32_t)(i / xstages) & 1u);
        }
    } else {
        // ---------------- f32 activations ----------------
        asm volatile("griddepcontrol.wait;" ::: "memory");
        // (never more warps than stages: a parity wait is only right while its warp cannot be two uses of a stage ahead)
        const int groups = min(kTsXWarps, xstages), c = lane & 7;
        for (int kb = warp - kTsXWarp; warp - kTsXWarp < groups && kb < steps && ok; kb += groups) {
            const int s = kb % xstages;
            if (kb >= xstages) ok = mbar_wait_fast(xe + 8 * s, ((uint32_t)(kb / xstages) & 1u) ^ 1u);
            if (!ok) break;
            uint8_t *dst = xs + s * xbytes;
            const float *src = P.xf + (size_t)(4 * u_lo + kb) * 64 + 8 * c;
            for (int r0 = lane >> 3; r0 < nt; r0 += 16) {   // rows r0, r0 + 4, + 8, + 12
                float4 a[4], b[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int t = m0 + r0 + 4 * i;
                    a[i] = b[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (t < P.m) {
                        a[i] = __ldg(reinterpret_cast<const float4 *>(src + (size_t)t * P.k));
                        b[i] = __ldg(reinterpret_cast<const float4 *>(src + (size_t)t * P.k) + 1);
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; i++)
                    *reinterpret_cast<uint4 *>(dst + swz(r0 + 4 * i, c)) =
                        make_uint4(pack_bf16(a[i].x, a[i].y), pack_bf16(a[i].z, a[i].w), pack_bf16(b[i].x, b[i].y), pack_bf16(b[i].z, b[i].w));
            }
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(xf + 8 * s);
        }
    }

    // ---------------- epilogue ----------------
    // all MMAs have ended (and with them every use of the rings): tensor memory lane = weight row, column = token
    __syncwarp();
    ok &= mbar_wait_fast(acc, 0);
    if (!ok) atomicExch(P.status, 1);
    __syncthreads();   // (the copies have landed: the rings may be overwritten)
    float *part = reinterpret_cast<float *>(smem);   // [nt][128]
    if (warp < kTsDecodeWarps) {
        asm volatile("griddepcontrol.wait;" ::: "memory");   // (returns at once) before any store
        tc_fence_after();
        const int row = (warp & 3) * 32 + lane;
        const bool live = n0 + row < J.n;
        const float bv = J.bias && live ? __ldg(J.bias + n0 + row) : 0.0f;
        for (int c0 = (warp >> 2) * 16; c0 < nt; c0 += 32) {
            uint32_t v[16];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                "tcgen05.wait::ld.sync.aligned;"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
                  "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                : "r"(tmem + ((uint32_t)(warp & 3) << 21) + (uint32_t)c0) : "memory");
            if (splits > 1) {
#pragma unroll
                for (int i = 0; i < 16; i++) part[(c0 + i) * 128 + row] = __uint_as_float(v[i]);
            } else if (live) {
#pragma unroll
                for (int i = 0; i < 16; i++)
                    if (m0 + c0 + i < P.m) {
                        const size_t at = (size_t)(m0 + c0 + i) * J.n + n0 + row;
                        const float f = __uint_as_float(v[i]) + bv;
                        if (P.y_dt == NNQ_F32) reinterpret_cast<float *>(J.y)[at] = f;
                        else reinterpret_cast<__nv_bfloat16 *>(J.y)[at] = __float2bfloat16_rn(f);
                    }
            }
        }
        tc_fence_before();
    }
    // A rank's share of the columns: a warp takes two at a time and asks all ranks for both before it adds (a read from another
    // CTA's shared memory takes about a microsecond when all do so: with four reads in flight a third of a launch of 4096 x 4096 x
    // 128 went here), then stores neighbouring rows. 4096 x 4096 at 33 / 128 rows 10.1 -> 9.0 / 14.2 -> 13.2 us.
    if (splits > 1) cluster_sync();
    if (splits > 1 && warp < kTsDecodeWarps) {
        const int lo = rank * nt / splits, hi = min((rank + 1) * nt / splits, P.m - m0), row = n0 + 4 * lane;
        const bool vec = (J.n & 3) == 0;
        float4 bv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (J.bias) {
            if (row < J.n) bv.x = __ldg(J.bias + row);
            if (row + 1 < J.n) bv.y = __ldg(J.bias + row + 1);
            if (row + 2 < J.n) bv.z = __ldg(J.bias + row + 2);
            if (row + 3 < J.n) bv.w = __ldg(J.bias + row + 3);
        }
        const uint32_t base = smem_u32(part) + 16 * lane;
        for (int c = lo + warp; c < hi; c += 2 * kTsDecodeWarps) {
            float4 p[2][8];
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int z = 0; z < 8; z++)
                    p[h][z] = z < splits && c + h * kTsDecodeWarps < hi ? ld_cluster_f4(cluster_addr(base + (uint32_t)((c + h * kTsDecodeWarps) * 512), (uint32_t)z))
                                                                        : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                if (c + h * kTsDecodeWarps >= hi) break;
                float4 f = p[h][0];
#pragma unroll
                for (int z = 1; z < 8; z++) {
                    f.x += p[h][z].x; f.y += p[h][z].y; f.z += p[h][z].z; f.w += p[h][z].w;
                }
                const float o[4] = {f.x + bv.x, f.y + bv.y, f.z + bv.z, f.w + bv.w};
                const size_t at = (size_t)(m0 + c + h * kTsDecodeWarps) * J.n + row;
                if (vec && row < J.n) {
                    if (P.y_dt == NNQ_F32) *reinterpret_cast<float4 *>(reinterpret_cast<float *>(J.y) + at) = make_float4(o[0], o[1], o[2], o[3]);
                    else *reinterpret_cast<uint2 *>(reinterpret_cast<__nv_bfloat16 *>(J.y) + at) = make_uint2(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]));
                } else {
                    for (int i = 0; i < 4; i++)
                        if (row + i < J.n) {
                            if (P.y_dt == NNQ_F32) reinterpret_cast<float *>(J.y)[at + i] = o[i];
                            else reinterpret_cast<__nv_bfloat16 *>(J.y)[at + i] = __float2bfloat16_rn(o[i]);
                        }
                }
            }
        }
    }
    if (splits > 1) {   // nobody leaves while its sums are read (they have been: the reads' values were used)
        __syncwarp();
        asm volatile("barrier.cluster.arrive.relaxed.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    __syncthreads();
    if (warp == kTsMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u) : "memory");
    }
}

// ---------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------

// Raw rows a tensor map can address: whole 16-byte words per row. Q6_K comes from the tiled copy.
bool gemm_ts_supported(const nnq_weight *w, int64_t m) {
    if (!w || m < 1 || w->n < 1 || w->n > INT_MAX - 128 || w->k < 64 || w->k > INT_MAX - 256) return false;
    switch (w->fmt) {
        case NNQ_Q4_K: case NNQ_Q4_K_GGML: case NNQ_Q4_0: case NNQ_Q8_0:
            return w->d_raw && w->k % 256 == 0 && ((uintptr_t)w->d_raw & 15u) == 0;
        case NNQ_MXFP4_SPLIT: return w->d_raw && w->d_scales && w->k % 64 == 0 && ((uintptr_t)w->d_raw & 15u) == 0;
        case NNQ_Q6_K: return w->tiled_layout == kTiledQ6K;
        default: return false;
    }
}

// Tokens of a tile at most. Q8_0's raw blocks leave room for two activation stages of 128 tokens, but the four warps that convert
// f32 rows work on one each. Tiles of up to 128 / of up to 80 tokens, and the fused decode of gemm_tc.cu, in us: 12288 x 4096 at
// 128 rows 82 / 55 / 69, at 256 187 / 95 / 108, at 1024 571 / 295 / 357; 4096 x 12288 at 512 rows 303 / 184 / 194; 1024 x 4096 at
// 128 rows 18 / 11 / 16.
static int ts_tile_tokens(int fmt, int x_dt) { return fmt == NNQ_Q8_0 && x_dt == NNQ_F32 ? 80 : kTsMaxN; }

template <int FMT>
static bool ts_w_map(const nnq_weight *w, CUtensorMap *map) {
    const bool mx = FMT == NNQ_MXFP4_SPLIT;
    const int64_t row_bytes = mx ? w->k / 2 : w->k / 256 * TsGeom<FMT>::kPitch;
    return encode_map_2d(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, w->d_raw, row_bytes / 4, w->n, row_bytes, TsGeom<FMT>::kPitch / 4, 128,
                         mx ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE);
}

// Ways to split K (CTAs of a cluster): the shortest estimate, in units of 256 weights of a CTA that has its SM for itself
// (1.35 us). Two CTAs on an SM take 1.6 per unit each; a CTA costs 3.3 beside its units (set-up, pipeline fill, epilogue).
// Clusters resident at once: what the occupancy query answers for a plain kernel with this shared memory on 148 SMs (for
// this one it counts one CTA per SM, but two run). Measured at 64 rows in us, 12288 x 4096: 30.9, 21.6, 29.0, 23.6 for one
// to four ways and 32.4 for eight; 4096 x 12288: 73.0, 43.9, 34.5, 26.6 and 19.9; 1024 x 4096: 24.4, 15.3, 12.7, 9.6 and 7.5.
static int ts_splits(int64_t tiles, int units, int sms) {
    static const int fit148[9] = {0, 296, 148, 93, 71, 56, 45, 37, 33};
    int best = 1;
    double least = 1e30;
    for (int s = 1; s <= 8 && s <= units; s++) {
        const int64_t slots = sms * fit148[s] / 148 > 0 ? sms * fit148[s] / 148 : 1, waves = (tiles + slots - 1) / slots;
        const int per_cta = (units + s - 1) / s;
        const double t = waves * (per_cta * (tiles * s <= sms ? 1.0 : 1.6) + 3.3);
        if (t < least - 1e-9) {
            least = t;
            best = s;
        }
    }
    return best;
}

template <int FMT, bool F32X>
static cudaError_t ts_launch(const TsParams &P, int tiles, int ttiles, int smem, int sms, cudaStream_t stream) {
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(gemm_ts_kernel<FMT, F32X>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTsSmem);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    const int splits = ts_splits((int64_t)tiles * ttiles, (P.k + 255) / 256, sms);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)tiles, (unsigned)ttiles, (unsigned)splits);
    cfg.blockDim = dim3((kTsXWarp + (F32X ? kTsXWarps : 1)) * 32);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = (unsigned)splits;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, gemm_ts_kernel<FMT, F32X>, P);
}

template <int FMT>
static nnq_status ts_run(nnq_ctx *ctx, const SkinnyJob *jobs, int count, int x_dt, int64_t m, int y_dt, cudaStream_t stream) {
    using G = TsGeom<FMT>;
    static_assert(G::kStages * G::kBytes + 2 * kTsMaxN * 128 + 1024 <= kTsSmem && kTsMaxN * 512 + 1024 <= kTsSmem, "shared memory");
    TsParams P;
    memset(&P, 0, sizeof(P));
    const int64_t k = jobs[0].w->k;
    int tiles = 0;
    for (int i = 0; i < count; i++) {
        const nnq_weight *w = jobs[i].w;
        TsJob &J = P.job[i];
        J.tiled = w->d_tiled;
        J.scales = w->d_scales;
        J.bias = jobs[i].bias;
        J.y = jobs[i].y;
        J.n = (int)w->n;
        J.tile_begin = tiles;
        tiles += (int)((w->n + 127) / 128);
        if (!G::kTiled && !ts_w_map<FMT>(w, &J.map)) return fail(ctx, NNQ_ERR_UNSUPPORTED, "tensor map of the weight");
    }
    P.njobs = count;
    P.m = (int)m;
    P.k = (int)k;
    P.y_dt = y_dt;
    P.status = ctx->d_status;
    // tokens in tiles of equal size
    const bool f32x = x_dt == NNQ_F32;
    const int most = ts_tile_tokens(FMT, x_dt);
    const int64_t ttiles = (m + most - 1) / most;
    P.nt = (int)(((m + ttiles - 1) / ttiles + 15) / 16 * 16);
    if (f32x) P.xf = static_cast<const float *>(jobs[0].x);
    else if (!encode_map_2d(&P.xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, jobs[0].x, k, m, 2 * k, 64, P.nt, CU_TENSOR_MAP_SWIZZLE_128B))
        return fail(ctx, NNQ_ERR_UNSUPPORTED, "tensor map of the activations");
    const int wbytes = G::kStages * G::kBytes;
    P.xstages = (kTsSmem - 1024 - wbytes) / (P.nt * 128);
    if (P.xstages > kTsMaxX) P.xstages = kTsMaxX;
    int smem = wbytes + P.xstages * P.nt * 128 + 1024;
    if (smem < P.nt * 512 + 1024) smem = P.nt * 512 + 1024;
    if (smem < kTsSmemMin) smem = kTsSmemMin;
    const cudaError_t e = f32x ? ts_launch<FMT, true>(P, tiles, (int)ttiles, smem, ctx->sm_count, stream) : ts_launch<FMT, false>(P, tiles, (int)ttiles, smem, ctx->sm_count, stream);
    ctx->launches++;
    return check_cuda(ctx, e, "tensor-memory product launch");
}

nnq_status launch_gemm_ts(nnq_ctx *ctx, const SkinnyJob *jobs, int count, int x_dt, int64_t m, int y_dt, cudaStream_t stream) {
    constexpr int64_t kRows = 1 << 22;   // of a launch: at most 65535 token tiles
    for (int64_t m0 = 0; m > kRows && m0 < m; m0 += kRows) {
        SkinnyJob part[kSkinnyMaxJobs];
        for (int i = 0; i < count; i++)
            part[i] = {jobs[i].w, static_cast<const uint8_t *>(jobs[i].x) + m0 * jobs[i].w->k * (x_dt == NNQ_F32 ? 4 : 2), jobs[i].bias,
                       static_cast<uint8_t *>(jobs[i].y) + m0 * jobs[i].w->n * (y_dt == NNQ_F32 ? 4 : 2)};
        nnq_status s = launch_gemm_ts(ctx, part, count, x_dt, m - m0 < kRows ? m - m0 : kRows, y_dt, stream);
        if (s != NNQ_OK || m0 + kRows >= m) return s;
    }
    int i = 0;
    while (i < count) {   // jobs of the same activations, K and format go out together
        int e = i + 1;
        while (e < count && e - i < kTsMaxJobs && jobs[e].x == jobs[i].x && jobs[e].w->k == jobs[i].w->k && jobs[e].w->fmt == jobs[i].w->fmt) e++;
        nnq_status s;
        switch (jobs[i].w->fmt) {
            case NNQ_Q4_K: s = ts_run<NNQ_Q4_K>(ctx, jobs + i, e - i, x_dt, m, y_dt, stream); break;
            case NNQ_Q4_K_GGML: s = ts_run<NNQ_Q4_K_GGML>(ctx, jobs + i, e - i, x_dt, m, y_dt, stream); break;
            case NNQ_Q4_0: s = ts_run<NNQ_Q4_0>(ctx, jobs + i, e - i, x_dt, m, y_dt, stream); break;
            case NNQ_Q8_0: s = ts_run<NNQ_Q8_0>(ctx, jobs + i, e - i, x_dt, m, y_dt, stream); break;
            case NNQ_Q6_K: s = ts_run<NNQ_Q6_K>(ctx, jobs + i, e - i, x_dt, m, y_dt, stream); break;
            case NNQ_MXFP4_SPLIT: s = ts_run<NNQ_MXFP4_SPLIT>(ctx, jobs + i, e - i, x_dt, m, y_dt, stream); break;
            default: return fail(ctx, NNQ_ERR_UNSUPPORTED, "no tensor-memory product for format %d", jobs[i].w->fmt);
        }
        if (s != NNQ_OK) return s;
        i = e;
    }
    return NNQ_OK;
}

}  // namespace nnq

// Large-prefill product (M >= 256 tokens): decode the weight once to bf16, then a plain bf16 GEMM
// on the 5th-generation tensor cores.
//
// With hundreds of activation rows per weight row the decode is a small part of the work: one pass
// over the raw blocks writes bf16 [N, K] into a scratch buffer owned by the context (0.56 + 2 bytes
// per weight at HBM speed; weights up to ~60 MB stay in L2 for the GEMM), and the GEMM main loop
// then does nothing but move tiles and issue MMAs:
//   * persistent CTAs (one per SM), output tiles of 256 x 256 by pairs of CTAs (or 128 x 256, 128 x 128 by one), k steps of
//     64 (one 128-byte swizzle row of bf16), a ring of 6 x (16 KB activation tile + 16 KB weight tile) per CTA;
//   * warp 0: one thread issues the TMA loads of both tiles (cp.async.bulk.tensor.2d, 128-byte
//     swizzle, zero fill beyond M / N) onto the stage's "full" barrier;
//   * warp 1 (of the pair's first CTA): an elected lane issues tcgen05.mma (M 256, N 256, K 16, bf16 x bf16 -> f32) into one of
//     two 256-column accumulators in tensor memory and commits the stage's "empty" barrier;
//   * warps 2..5: epilogue -- tcgen05.ld of the finished accumulator (each warp its quarter of
//     the 128 lanes), bias, conversion, stores -- while the MMA warp already fills the other
//     accumulator with the next tile.
// Tiles are numbered m-fastest, so the CTAs running at one time share a few weight tiles and the
// activation matrix stays in L2. Weights and activations are bf16: the 1e-2 tolerance class.
// Every barrier wait is bounded; a wait that runs out sets the context's status word, every role
// leaves its loop and the tensor memory is freed.
#include <cuda.h>
#include <cuda_bf16.h>
#include <string.h>

#include "decode.cuh"
#include "gemm_tc.h"
#include "sync.cuh"
#include "tcgen05.cuh"

namespace nnq {

// ---------------------------------------------------------------------------------
// raw blocks -> bf16 [N, K]
// ---------------------------------------------------------------------------------

constexpr int kDbThreads = 128;

// MXFP4 straight to bf16 bits, no f32 detour: a magnitude code m >= 2 is (1 + (m & 1) / 2) * 2^((m >> 1) - 1),
// m == 1 is 0.5, and the block scale is 2^(e - 127), so the product is the bf16 number with exponent field
// e - 1 + (m >> 1) and top mantissa bit (m & 1): bits = ((e - 1) << 7) + (m' << 6) with m' = m (0 for m == 1),
// zero for m == 0, sign on bit 15. Exact, hence equal to rounding the f32 decode; valid for 1 <= e <= 251
// (other exponents take the f32 path).
__device__ __forceinline__ uint32_t mx_bf16_one(uint32_t nib, uint32_t base) {
    const uint32_t m = nib & 7u;
    const uint32_t mp = m == 1u ? 0u : m;
    const uint32_t mag = m == 0u ? 0u : base + (mp << 6);
    return mag | ((nib & 8u) << 12);
}

template <bool HIGH_FIRST>
__device__ __forceinline__ void mx_chunk_bf16(const uint4 q, uint32_t e, uint4 *out4) {
    const uint32_t base = (e - 1u) << 7;
    const uint32_t qw[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int v = 0; v < 4; v++) {
        uint32_t p[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t byte = (qw[v] >> (8 * i)) & 0xFFu;
            const uint32_t even = HIGH_FIRST ? byte >> 4 : byte & 15u, odd = HIGH_FIRST ? byte & 15u : byte >> 4;
            p[i] = mx_bf16_one(even, base) | (mx_bf16_one(odd, base) << 16);
        }
        out4[v] = make_uint4(p[0], p[1], p[2], p[3]);
    }
}

template <int FMT, bool PAIR>
__global__ void __launch_bounds__(kDbThreads)
dequant_bf16_kernel(const uint8_t *__restrict__ src, const uint8_t *__restrict__ scales, int64_t nchunks,
                    uint4 *__restrict__ dst, int cpr, int half_rows, int pair) {
    // PAIR: row j goes to row 2j + pair (one of two weights whose rows alternate; nchunks < 2^31). Kernels of their own: as a branch this
    // took registers from the others (MXFP4: 87 -> 72 and spills)
    const int shift = (cpr & (cpr - 1)) == 0 ? __ffs(cpr) - 1 : -1;
    auto paired = [&](int64_t c) {
        const uint32_t row = shift >= 0 ? (uint32_t)c >> shift : (uint32_t)c / (uint32_t)cpr;
        return (int64_t)(2 * row + (uint32_t)pair) * cpr + ((uint32_t)c - row * (uint32_t)cpr);
    };
    if (FMT == NNQ_MXFP4_SPLIT || FMT == NNQ_MXFP4_GPTOSS) {
        // a thread owns one 32-weight chunk: 64 contiguous output bytes (two whole 32-byte sectors), written
        // with four 16-byte stores -- the integer decode needs no staging (measured: 366 -> 320 us for the
        // 282 MB of a gpt-oss gate / up tensor; the f32 decoders below are faster with the staged store)
        auto emit = [&](int64_t c, uint32_t e, const uint4 q) {
            uint4 o4[4];
            if (e >= 1u && e <= 251u) {
                mx_chunk_bf16<FMT == NNQ_MXFP4_GPTOSS>(q, e, o4);
            } else {
                float o[32];
                Decode<FMT>::chunk(src, scales, c, o);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    uint32_t p[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        __nv_bfloat162 v = __floats2bfloat162_rn(o[8 * j + 2 * i], o[8 * j + 2 * i + 1]);
                        p[i] = *reinterpret_cast<uint32_t *>(&v);
                    }
                    o4[j] = make_uint4(p[0], p[1], p[2], p[3]);
                }
            }
            // half_rows > 0: every group of 2 * half_rows weight rows (one expert's gate rows, then its up
            // rows) is written interleaved, gate row j to row 2j and up row j to row 2j + 1, so that a GEMM
            // tile holds both halves of an output column pair (the fused SwiGLU epilogue)
            int64_t oc = c;
            if (PAIR) {
                oc = paired(c);
            } else if (half_rows > 0) {   // nchunks < 2^31 here (checked by the launcher): 32-bit divisions
                const uint32_t c32 = (uint32_t)c, row = c32 / (uint32_t)cpr, cin = c32 - row * (uint32_t)cpr;
                const uint32_t ex = row / (2u * half_rows), r = row - ex * 2u * half_rows;
                const uint32_t r2 = r < (uint32_t)half_rows ? 2u * r : 2u * (r - half_rows) + 1u;
                oc = (int64_t)(ex * 2u * half_rows + r2) * cpr + cin;
            }
#pragma unroll
            for (int j = 0; j < 4; j++) dst[oc * 4 + j] = o4[j];
        };
        // two chunks per iteration: both loads are in flight before either is decoded
        const int64_t stride = (int64_t)gridDim.x * kDbThreads;
        int64_t c = (int64_t)blockIdx.x * kDbThreads + threadIdx.x;
        for (; c + stride < nchunks; c += 2 * stride) {
            const uint32_t e0 = __ldg(scales + c), e1 = __ldg(scales + c + stride);
            const uint4 q0 = __ldg(reinterpret_cast<const uint4 *>(src + c * 16));
            const uint4 q1 = __ldg(reinterpret_cast<const uint4 *>(src + (c + stride) * 16));
            emit(c, e0, q0);
            emit(c + stride, e1, q1);
        }
        if (c < nchunks) emit(c, __ldg(scales + c), __ldg(reinterpret_cast<const uint4 *>(src + c * 16)));
        return;
    }
    __shared__ uint4 tile[kDbThreads * 4 + 4];
    for (int64_t base = (int64_t)blockIdx.x * kDbThreads; base < nchunks; base += (int64_t)gridDim.x * kDbThreads) {
        const int64_t c = base + threadIdx.x;
        if (c < nchunks) {
            float o[32];
            Decode<FMT>::chunk(src, scales, c, o);   // the bit-exact decode, then round to nearest even
#pragma unroll
            for (int j = 0; j < 4; j++) {
                uint32_t p[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    __nv_bfloat162 v = __floats2bfloat162_rn(o[8 * j + 2 * i], o[8 * j + 2 * i + 1]);
                    p[i] = *reinterpret_cast<uint32_t *>(&v);
                }
                // chunk-local XOR swizzle: for a fixed j the 16-byte stores of a quarter warp fall into
                // eight different bank groups (unswizzled, threads 64 bytes apart share two of them)
                tile[threadIdx.x * 4 + (j ^ ((threadIdx.x >> 1) & 3))] = make_uint4(p[0], p[1], p[2], p[3]);
            }
        }
        __syncthreads();
        const int64_t remaining = nchunks - base;
        const int live = remaining < kDbThreads ? (int)remaining : kDbThreads;
        uint4 *out = dst + base * 4;
        if (PAIR) out = dst + (paired(base + (threadIdx.x >> 2)) - (threadIdx.x >> 2)) * 4;
        for (int idx = threadIdx.x; idx < live * 4; idx += kDbThreads) {
            out[idx] = tile[(idx & ~3) | ((idx & 3) ^ ((idx >> 3) & 3))];
            if (PAIR && idx + kDbThreads < live * 4) out = dst + (paired(base + ((idx + kDbThreads) >> 2)) - ((idx + kDbThreads) >> 2)) * 4;
        }
        __syncthreads();
    }
}

// Formats whose blocks are not aligned: Q6_K, Q8_0, Q4_0. Read byte by byte from global memory they are bound by L1 (88 % busy), so a
// warp brings 64 chunks, whole 16-byte units of any of them, to its own shared memory with asynchronous copies, the next 64 while
// it decodes; a lane makes a chunk from halfwords, 32 at a time, and they are stored through a tile in whole lines. Bound by memory
// then. 12288 x 4096, byte by byte / this, in us: Q6_K 32.6 / 27.0, Q8_0 39.4 / 22.7, Q4_0 28.8 / 21.1; 25600 x 5120 Q6_K 80.6 / 66.0
// (5.6 TB/s).
template <int FMT>
__host__ __device__ constexpr int staged_bytes() {   // of 64 chunks
    return FMT == NNQ_Q6_K ? 1680 : FMT == NNQ_Q8_0 ? 2176 : 1152;
}
template <int FMT>
__device__ __forceinline__ void staged_chunk(const uint8_t *raw, int c, float (&o)[32]) {
    if constexpr (FMT == NNQ_Q8_0) {
        Decode<NNQ_Q8_0>::chunk_halfwords(reinterpret_cast<const uint16_t *>(raw + 34 * c), o);
    } else if constexpr (FMT == NNQ_Q4_0) {
        // two weights (a byte) per step: the high nibble stays where it is, d / 16 (exact) is its factor
        const uint16_t *p = reinterpret_cast<const uint16_t *>(raw + 18 * c);
        const float d = f16_bits_to_f32(p[0]);
        const float2 unbias = make_float2(-(8388608.0f + 8.0f), -(8388608.0f + 128.0f)), d2 = make_float2(d, __fmul_rn(d, 0.0625f));
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t t = p[1 + i];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint32_t b = t >> (8 * h);
                const float2 v = __fmul2_rn(__fadd2_rn(make_float2(__uint_as_float((b & 0x0Fu) | 0x4B000000u), __uint_as_float((b & 0xF0u) | 0x4B000000u)), unbias), d2);
                o[4 * i + 2 * h] = v.x;
                o[4 * i + 2 * h + 1] = v.y;
            }
        }
    } else {
        // four weights per step: the two of a byte's low (high) nibbles side by side, q and 256 q'
        const uint16_t *p = reinterpret_cast<const uint16_t *>(raw + 210 * (c >> 3));
        const int j = c & 7;
        const float d = f16_bits_to_f32(p[104]);
        const uint32_t sc = p[96 + j];
        const float s[2] = {__fmul_rn(d, s8_to_f(sc & 0xFFu)), __fmul_rn(d, s8_to_f(sc >> 8))};
        const float2 unbias = make_float2(-(8388608.0f + 32.0f), -(8388608.0f + 8192.0f));
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t ql = p[8 * j + i], qh = (uint32_t)p[64 + 4 * j + (i >> 1)] >> (8 * (i & 1));
            const uint32_t a = (ql & 0x0F0Fu) | ((qh << 4) & 0x30u) | ((qh << 8) & 0x3000u);
            const uint32_t b = ((ql >> 4) & 0x0F0Fu) | ((qh << 2) & 0x30u) | ((qh << 6) & 0x3000u);
            const float2 s2 = make_float2(s[i >> 2], __fmul_rn(s[i >> 2], 0.00390625f));
            const float2 u = __fmul2_rn(__fadd2_rn(make_float2(__uint_as_float((a & 0xFFu) | 0x4B000000u), __uint_as_float((a & 0xFF00u) | 0x4B000000u)), unbias), s2);
            const float2 v = __fmul2_rn(__fadd2_rn(make_float2(__uint_as_float((b & 0xFFu) | 0x4B000000u), __uint_as_float((b & 0xFF00u) | 0x4B000000u)), unbias), s2);
            o[4 * i] = u.x;
            o[4 * i + 1] = v.x;
            o[4 * i + 2] = u.y;
            o[4 * i + 3] = v.y;
        }
    }
}

constexpr int kDbResident = 8;   // CTAs per SM (registers, shared memory)
template <int FMT>
__global__ void __launch_bounds__(kDbThreads, kDbResident)
dequant_staged_kernel(const uint8_t *__restrict__ src, int64_t nchunks, uint4 *__restrict__ dst, int cpr, int pair) {
    constexpr int UB = staged_bytes<FMT>(), W = kDbThreads / 32;
    __shared__ __align__(16) uint8_t raw[W][2][UB];
    __shared__ uint4 tile[W][128];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, shift = (cpr & (cpr - 1)) == 0 ? __ffs(cpr) - 1 : -1;
    const int64_t units = (nchunks + 63) / 64, total = nchunks * UB / 64, stride = (int64_t)gridDim.x * W;
    auto bring = [&](int64_t u, int buf) {
        if (u < units) {
            const int64_t off = u * UB;
            const int bytes = total - off < UB ? (int)(total - off) : UB;
            const uint32_t to = smem_u32(raw[warp][buf]);
#pragma unroll
            for (int i = 0; i < (UB / 16 + 31) / 32; i++)
                if (16 * (i * 32 + lane) + 16 <= bytes)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 16 * (i * 32 + lane)), "l"(src + off + 16 * (i * 32 + lane)) : "memory");
            const int at = (bytes & ~15) + lane;   // what is left of the last unit
            if (lane < (bytes & 15)) raw[warp][buf][at] = __ldg(src + off + at);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int buf = 0;
    int64_t u = (int64_t)blockIdx.x * W + warp;
    bring(u, 0);
    for (; u < units; u += stride, buf ^= 1) {
        bring(u + stride, buf ^ 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
#pragma unroll 1
        for (int h = 0; h < 2; h++) {
            const int64_t base = u * 64 + 32 * h;
            if (base + lane < nchunks) {
                float o[32];
                staged_chunk<FMT>(raw[warp][buf], 32 * h + lane, o);   // the bit-exact decode, then round to nearest even
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    uint32_t p[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) p[i] = pack_bf16(o[8 * j + 2 * i], o[8 * j + 2 * i + 1]);
                    tile[warp][lane * 4 + (j ^ ((lane >> 1) & 3))] = make_uint4(p[0], p[1], p[2], p[3]);   // (swizzle: as below)
                }
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int idx = 32 * i + lane;
                const int64_t c = base + (idx >> 2);
                if (c < nchunks) {
                    int64_t oc = c;
                    if (pair >= 0) {   // row j goes to row 2j + pair (nchunks < 2^30 here)
                        const uint32_t row = shift >= 0 ? (uint32_t)c >> shift : (uint32_t)c / (uint32_t)cpr;
                        oc = (int64_t)(2 * row + (uint32_t)pair) * cpr + ((uint32_t)c - row * (uint32_t)cpr);
                    }
                    dst[oc * 4 + (idx & 3)] = tile[warp][(idx & ~3) | ((idx & 3) ^ ((idx >> 3) & 3))];
                }
            }
            __syncwarp();
        }
    }
}

// nn-gptoss expert tensors [E, K, N] (MXFP4, 32-weight blocks along N, the even column in the high
// nibble) -> bf16 [E, N, K]: a CTA turns a tile of 64 KT (k) x 64 (n)
// through shared memory. Reads are whole sectors (32 bytes of a k row), writes 128 KT contiguous bytes per output row. Bound by the
// decode, which looks four magnitudes up at a time and stores pairs of k, then by the stores: both weights of 32 experts of 2880,
// KT = 1 / 3: 504 / 467 us (KT = 3 where K is a multiple of 192). half_rows > 0 interleaves the output rows of every expert (row j ->
// 2j, row half_rows + j -> 2j + 1), as the fused SwiGLU epilogue wants.
constexpr int kKnTile = 64;
template <int KT>
__global__ void __launch_bounds__(128 * KT)
dequant_kn_bf16_kernel(const uint8_t *__restrict__ data, const uint8_t *__restrict__ scales, __nv_bfloat16 *__restrict__ dst,
                       int K, int N, int half_rows) {
    __shared__ __align__(16) uint16_t tile[kKnTile][kKnTile * KT + 8];   // [n][k]; the odd 16 bytes keep 16-byte reads aligned
    const int e = blockIdx.z, k0 = blockIdx.y * kKnTile * KT, n0 = blockIdx.x * kKnTile;
    // this thread's pair of k rows and 16 of the 64 columns: it makes the pairs (k, k + 1) that lie side by side in the copy
    const int pair = (threadIdx.x & 31) + 32 * (threadIdx.x >> 7), part = (threadIdx.x >> 5) & 3;
    const size_t row = (size_t)e * K + k0 + 2 * pair;
    const uint2 qa = __ldg(reinterpret_cast<const uint2 *>(data + row * (size_t)(N / 2) + n0 / 2 + part * 8));
    const uint2 qb = __ldg(reinterpret_cast<const uint2 *>(data + (row + 1) * (size_t)(N / 2) + n0 / 2 + part * 8));
    const uint32_t ea = __ldg(scales + row * (size_t)(N / 32) + n0 / 32 + (part >> 1)), eb = __ldg(scales + (row + 1) * (size_t)(N / 32) + n0 / 32 + (part >> 1));
    // E2M1 magnitudes as the two bytes of a bf16 (0, .5, 1, 1.5, 2, 3, 4, 6), four per table look-up; the scale 2^(e - 127)
    // (e = 0: 2^-126) is an exact bf16 factor, e = 255 infinity
    const uint32_t scale = max(ea << 7, 0x80u) | (max(eb << 7, 0x80u) << 16);
    const uint32_t wa[2] = {qa.x, qa.y}, wb[2] = {qb.x, qb.y};
#pragma unroll
    for (int v = 0; v < 2; v++) {
#pragma unroll
        for (int h = 0; h < 2; h++) {   // two bytes: columns 8 v + 4 h .. + 3, the even one of a byte in its high nibble
            const uint32_t a = wa[v] >> (16 * h), b = wb[v] >> (16 * h), sa = a & 0x7777u, sb = b & 0x7777u;
            const uint32_t la = __byte_perm(0xC0800000u, 0xC0804000u, sa), ha = __byte_perm(0x3F3F3F00u, 0x40404040u, sa);
            const uint32_t lb = __byte_perm(0xC0800000u, 0xC0804000u, sb), hb = __byte_perm(0x3F3F3F00u, 0x40404040u, sb);
            const uint32_t a01 = __byte_perm(la, ha, 0x5140), a23 = __byte_perm(la, ha, 0x7362), b01 = __byte_perm(lb, hb, 0x5140), b23 = __byte_perm(lb, hb, 0x7362);
            const uint32_t m[4] = {__byte_perm(a01, b01, 0x5410), __byte_perm(a01, b01, 0x7632), __byte_perm(a23, b23, 0x5410), __byte_perm(a23, b23, 0x7632)};
#pragma unroll
            for (int i = 0; i < 4; i++) {   // nibble i of the two bytes is column i ^ 1
                uint32_t u = m[i] | ((a << (12 - 4 * i)) & 0x8000u) | ((b << (28 - 4 * i)) & 0x80000000u);
                const __nv_bfloat162 z = __hmul2(*reinterpret_cast<const __nv_bfloat162 *>(&u), *reinterpret_cast<const __nv_bfloat162 *>(&scale));
                *reinterpret_cast<__nv_bfloat162 *>(&tile[part * 16 + 8 * v + 4 * h + (i ^ 1)][2 * pair]) = z;
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kKnTile * 8 * KT; i += 128 * KT) {
        const int r = i / (8 * KT), c = i - r * (8 * KT), n = n0 + r;
        const int nn = half_rows > 0 ? (n < half_rows ? 2 * n : 2 * (n - half_rows) + 1) : n;
        *reinterpret_cast<uint4 *>(dst + ((size_t)e * N + nn) * K + k0 + c * 8) = *reinterpret_cast<const uint4 *>(&tile[r][c * 8]);
    }
}

template <int FMT>
static cudaError_t launch_dequant_bf16(const uint8_t *src, const uint8_t *scales, int64_t nchunks, void *dst, int sm_count,
                                       cudaStream_t stream, int cpr = 1, int half_rows = 0, int pair = -1) {
    if constexpr (FMT == NNQ_Q6_K || FMT == NNQ_Q8_0 || FMT == NNQ_Q4_0) {
        // From a unit for every resident warp on; below, the copy in between is one more wait (1024 x 5120 Q6_K, directly / staged:
        // 6.2 / 6.5 us). Persistent, every warp with the same number of units.
        constexpr int W = kDbThreads / 32;
        const int64_t units = (nchunks + 63) / 64, most = (int64_t)sm_count * kDbResident * W, rounds = (units + most - 1) / most;
        if (half_rows == 0 && units >= most && ((uintptr_t)src & 15u) == 0) {
            const int64_t ctas = (units + W * rounds - 1) / (W * rounds);
            dequant_staged_kernel<FMT><<<(int)ctas, kDbThreads, 0, stream>>>(src, nchunks, reinterpret_cast<uint4 *>(dst), cpr, pair);
            return cudaGetLastError();
        }
    }
    const int64_t want = (nchunks + kDbThreads - 1) / kDbThreads;
    const int64_t cap = (int64_t)sm_count * 16;
    int grid = (int)(want < cap ? want : cap);
    if (grid < 1) grid = 1;
    if (pair >= 0) dequant_bf16_kernel<FMT, true><<<grid, kDbThreads, 0, stream>>>(src, scales, nchunks, reinterpret_cast<uint4 *>(dst), cpr, half_rows, pair);
    else dequant_bf16_kernel<FMT, false><<<grid, kDbThreads, 0, stream>>>(src, scales, nchunks, reinterpret_cast<uint4 *>(dst), cpr, half_rows, pair);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------
// bf16 GEMM: y[M, N] = x[M, K] * Wd[N, K]^T (+ bias)
// ---------------------------------------------------------------------------------

// Tile 128 CG x BN x 64: CG = 2 CTAs of a cluster multiply one tile together (cta_group::2), or one CTA its own. BN = 256,
// or 128 where 256-wide tiles would leave SMs without a tile.
constexpr int kDgBM = 128, kDgBK = 64;
constexpr int kDgABytes = kDgBM * 128;
constexpr int kDgMaxOuts = 4;
constexpr int kDgSilu = 16;   // gate_kind: silu by expf and a rounded division
constexpr int kDgThreads = 192;
__host__ __device__ constexpr int dg_stage_bytes(int bn, int cg) { return kDgABytes + bn / cg * 128; }
__host__ __device__ constexpr int dg_stages(int, int cg) { return cg == 1 ? 4 : 6; }
static int dg_smem_bytes(int bn, int cg) { return dg_stages(bn, cg) * dg_stage_bytes(bn, cg) + 1024; }

__device__ __forceinline__ void dg_tma_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar) : "memory");
}
// the same into this CTA's shared memory, completion counted on a barrier of either CTA of the pair (a shared::cluster address)
__device__ __forceinline__ void dg_tma_2d_pair(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar) : "memory");
}

// A pair of CTAs (CG = 2) holds 128 rows of the activation tile and BN / 2 rows of the weight tile each: the tensor cores
// read both halves, so an operand byte is brought to shared memory and read from it once per 256 x 256 products instead of
// once per 128 x 256. With one CTA the two (48 KB in, 48 KB out per 64-wide k step of 512 tensor-core clocks) exceed what
// shared memory moves. The first CTA of the pair issues the MMAs; its "full" barriers count both CTAs' copies, its "empty" and "accumulator
// full" commits reach both CTAs, both CTAs' epilogues hand the accumulators back to it.
// 25600 x 5120 at 4096 rows: 739 -> 683 us (1.57 PFLOP/s), the seven products of such a layer in Q6_K 3.68 -> 3.42 ms, decode included.
// Outputs of weights that lie one behind the other (whole tiles each but the last): weight rows begin[i] .. begin[i + 1] are out i's.
struct DgOuts {
    void *y[kDgMaxOuts];
    const float *bias[kDgMaxOuts];
    int begin[kDgMaxOuts + 1], count;
};

template <int BN, int CG>
__global__ void __launch_bounds__(kDgThreads, 1)
gemm_dense_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap,
                  const __grid_constant__ DgOuts outs, int M, int N, int K, int y_dt, int *status,
                  __nv_bfloat16 *__restrict__ h_out, int gate_kind) {
    constexpr int kDgBN = BN, kDgStageBytes = dg_stage_bytes(BN, CG), kDgStages = dg_stages(BN, CG), kDgRows = kDgBM * CG;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // Tiles of 128 x 128 with timed waits and a generic address, the others with neither: decoded weights of 1024 x 4096 at 800 rows
    // with both / with the waits alone / with neither 23.7 / 25.0 / 25.6 us, 2048 x 6144 36.6 / 38.8 / 39.4; 4096 rows and more the other way by
    // up to 1 %.
    constexpr bool kTimed = BN == 128;
    uint8_t *smem = kTimed ? reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023) : smem_raw + (-smem_u32(smem_raw) & 1023u);
    __shared__ __align__(8) uint64_t bars[2 * kDgStages + 5];   // full, empty [kDgStages], acc_full[2], acc_empty[2], every MMA has ended
    __shared__ uint32_t tmem_base_s;

    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0);
    const uint32_t full_s = smem_u32(bars), empty_s = full_s + 8 * kDgStages;
    const uint32_t accf_s = empty_s + 8 * kDgStages, acce_s = accf_s + 16, done_s = acce_s + 16;
    const int rank = CG == 2 ? (int)cluster_rank() : 0;
    const int unit = blockIdx.x / CG, units = gridDim.x / CG;   // a unit multiplies one tile at a time
    const int m_tiles = (M + kDgRows - 1) / kDgRows, n_tiles = (N + kDgBN - 1) / kDgBN;
    const int tiles = m_tiles * n_tiles;
    const int nkb = K / kDgBK;
    // tile t -> this CTA's first row, first weight row
    auto locate = [&](int t, int &m0, int &n0) {
        m0 = t % m_tiles * kDgRows + rank * kDgBM;
        n0 = (t / m_tiles) * kDgBN;
    };

    if (tid == 0) {
        for (int s = 0; s < kDgStages; s++) {
            mbar_init(full_s + 8 * s, 1);
            mbar_init(empty_s + 8 * s, 1);
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(accf_s + 8 * a, 1);
            mbar_init(acce_s + 8 * a, 4 * CG);
        }
        mbar_init(done_s, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        if (CG == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(512u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(512u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if (CG == 2) cluster_sync();   // both CTAs' barriers are set up
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;
    bool ok = true;

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            const uint32_t count_s = CG == 2 ? cluster_addr(full_s, 0) : full_s;   // the barriers that count the copies
            int slot = 0;
            uint32_t phase = 0;
            long long filled = 0;
            for (int t = unit; t < tiles && ok; t += units) {
                int m0, n0;
                locate(t, m0, n0);
                const int w0 = n0 + rank * (BN / CG);
                for (int kb = 0; kb < nkb; kb++) {
                    if (filled >= kDgStages && !mbar_wait_fast<kTimed>(empty_s + 8 * slot, phase ^ 1u)) {
                        ok = false;
                        break;
                    }
                    const uint32_t a_s = smem_u32(smem + (size_t)slot * kDgStageBytes);
                    if (rank == 0) mbar_expect_tx(full_s + 8 * slot, CG * kDgStageBytes);
                    if (CG == 2) {
                        dg_tma_2d_pair(a_s, &xmap, kb * kDgBK, m0, count_s + 8 * slot);
                        dg_tma_2d_pair(a_s + kDgABytes, &wmap, kb * kDgBK, w0, count_s + 8 * slot);
                    } else {
                        dg_tma_2d(a_s, &xmap, kb * kDgBK, m0, full_s + 8 * slot);
                        dg_tma_2d(a_s + kDgABytes, &wmap, kb * kDgBK, w0, full_s + 8 * slot);
                    }
                    filled++;
                    if (++slot == kDgStages) {
                        slot = 0;
                        phase ^= 1u;
                    }
                }
            }
            // The last use of every stage: this CTA's copies have landed and been read, and the arrivals on its barriers, which
            // for the second CTA of a pair come from the first, are over. Behind a wait that ran out the stages may never be
            // given back; the copies are still waited for (by the CTA whose barriers count them).
            for (long long f = filled > kDgStages ? filled - kDgStages : 0; f < filled; f++) {
                const uint32_t s = (uint32_t)(f % kDgStages), p = (uint32_t)(f / kDgStages) & 1u;
                if (ok) ok = mbar_wait_fast<kTimed>(empty_s + 8 * s, p);
                if (!ok && rank == 0) mbar_wait(full_s + 8 * s, p);
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        // (the warp waits together, an elected lane issues: behind `lane == 0` the compiler loops over the active lanes around every
        // instruction that takes uniform registers)
        if (rank == 0) {
            // f32 accumulate, bf16 x bf16, both K-major, N = BN, M = 128 CG
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (((uint32_t)BN >> 3) << 17) | (((uint32_t)kDgRows >> 4) << 24);
            int slot = 0;
            uint32_t phase = 0;
            int it = 0;
            for (int t = unit; t < tiles && ok; t += units, it++) {
                const int a = it & 1;
                // the epilogue has read this accumulator's previous tile
                if (it >= 2) ok = __all_sync(0xFFFFFFFFu, mbar_wait_fast<kTimed>(acce_s + 8 * a, (uint32_t)(((it >> 1) - 1) & 1)));
                const uint32_t acc = tmem_base + (uint32_t)(a * kDgBN);
                for (int kb = 0; kb < nkb && ok; kb++) {
                    ok = __all_sync(0xFFFFFFFFu, mbar_wait_fast<kTimed>(full_s + 8 * slot, phase));
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t a_s = smem_u32(smem + (size_t)slot * kDgStageBytes);
                        const uint64_t da = smem_desc(a_s), db = smem_desc(a_s + kDgABytes);
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            if (CG == 2) umma_bf16_pair(acc, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
                            else umma_bf16(acc, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
                        }
                        if (CG == 2) umma_commit_pair(empty_s + 8 * slot);
                        else umma_commit(empty_s + 8 * slot);
                        if (kb == nkb - 1) {
                            if (CG == 2) umma_commit_pair(accf_s + 8 * a);
                            else umma_commit(accf_s + 8 * a);
                        }
                    }
                    __syncwarp();
                    if (++slot == kDgStages) {
                        slot = 0;
                        phase ^= 1u;
                    }
                }
            }
            if (elect_one()) {   // also behind a wait that ran out
                if (CG == 2) umma_commit_pair(done_s);
                else umma_commit(done_s);
            }
            __syncwarp();
        }
    } else {
        // ---------------- epilogue ----------------
        const uint32_t back_s = CG == 2 ? cluster_addr(acce_s, 0) : acce_s;
        const int q = warp & 3;   // the quarter of the 128 TMEM lanes this warp may read
        int it = 0;
        for (int t = unit; t < tiles && ok; t += units, it++) {
            const int a = it & 1;
            int m0, n0;
            locate(t, m0, n0);
            int out = 0;
            while (out + 1 < outs.count && n0 >= outs.begin[out + 1]) out++;
            void *const y = outs.y[out];
            const float *const bias = outs.bias[out];
            const int N = outs.begin[out + 1] - outs.begin[out];
            n0 -= outs.begin[out];
            if (!mbar_wait_fast<kTimed>(accf_s + 8 * a, (uint32_t)((it >> 1) & 1))) {
                ok = false;
                break;
            }
            tc_fence_after();
            const int row = m0 + q * 32 + lane;
#pragma unroll 1
            for (int cc = 0; cc < kDgBN / 32; cc++) {
                uint32_t v[32];
                tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(a * kDgBN + cc * 32), v);
                const int col0 = n0 + cc * 32;
                if (h_out) {
                    // interleaved gate / up columns (2j, 2j + 1): h[row, j] = f(g) * u in bf16, f silu or gelu; the bias of column c
                    // is the gate bias of c / 2 for even c and the up bias (second half of the bias row) for odd c
                    if (row < M && col0 < N) {
                        const int I = N >> 1;
                        uint32_t packed[8];
#pragma unroll
                        for (int p = 0; p < 16; p += 2) {
                            float hv[2];
#pragma unroll
                            for (int q2 = 0; q2 < 2; q2++) {
                                const int j = (col0 >> 1) + p + q2;
                                float gv = __uint_as_float(v[2 * (p + q2)]), uv = __uint_as_float(v[2 * (p + q2) + 1]);
                                if (bias && j < I) {
                                    gv += __ldg(bias + j);
                                    uv += __ldg(bias + I + j);
                                }
                                // kDgSilu: the numbers of the activation's own kernel (prompt_rows.cu). The others have the fast
                                // exponential and division, whose error grows with the argument (2^-22 relative near zero, 2^-20
                                // at -16; h is rounded to 2^-9). (The tanh form of gelu is x sigmoid(2 sqrt(2 / pi) (x + 0.044715 x^3)).)
                                if (gate_kind == kDgSilu) {
                                    hv[q2] = gv / (1.0f + expf(-gv)) * uv;
                                } else {
                                    const float sx = gate_kind == NNQ_ACT_GELU_TANH ? 1.5957691216057308f * fmaf(0.044715f * gv * gv, gv, gv) : gv;
                                    hv[q2] = __fdividef(gv, 1.0f + __expf(-sx)) * uv;
                                }
                            }
                            __nv_bfloat162 b2 = __floats2bfloat162_rn(hv[0], hv[1]);
                            packed[p >> 1] = *reinterpret_cast<uint32_t *>(&b2);
                        }
                        __nv_bfloat16 *dstp = h_out + (size_t)row * I + (col0 >> 1);
                        if (col0 + 32 <= N && (I & 7) == 0) {
                            reinterpret_cast<uint4 *>(dstp)[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
                            reinterpret_cast<uint4 *>(dstp)[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
                        } else {
                            const __nv_bfloat16 *pk = reinterpret_cast<const __nv_bfloat16 *>(packed);
                            for (int i = 0; i < 16; i++)
                                if ((col0 >> 1) + i < I) dstp[i] = pk[i];
                        }
                    }
                } else if (row < M && col0 < N) {
                    float f[32];
#pragma unroll
                    for (int i = 0; i < 32; i++) f[i] = __uint_as_float(v[i]) + (bias && col0 + i < N ? __ldg(bias + col0 + i) : 0.0f);
                    if (col0 + 32 <= N && (N & 7) == 0) {
                        if (y_dt == NNQ_F32) {
                            float4 *dst = reinterpret_cast<float4 *>(reinterpret_cast<float *>(y) + (size_t)row * N + col0);
#pragma unroll
                            for (int i = 0; i < 8; i++) dst[i] = make_float4(f[4 * i], f[4 * i + 1], f[4 * i + 2], f[4 * i + 3]);
                        } else {
                            uint4 *dst = reinterpret_cast<uint4 *>(reinterpret_cast<__nv_bfloat16 *>(y) + (size_t)row * N + col0);
#pragma unroll
                            for (int i = 0; i < 4; i++) {
                                uint32_t p[4];
#pragma unroll
                                for (int j = 0; j < 4; j++) {
                                    __nv_bfloat162 b2 = __floats2bfloat162_rn(f[8 * i + 2 * j], f[8 * i + 2 * j + 1]);
                                    p[j] = *reinterpret_cast<uint32_t *>(&b2);
                                }
                                dst[i] = make_uint4(p[0], p[1], p[2], p[3]);
                            }
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; i++) {
                            if (col0 + i < N) {
                                if (y_dt == NNQ_F32) reinterpret_cast<float *>(y)[(size_t)row * N + col0 + i] = f[i];
                                else reinterpret_cast<__nv_bfloat16 *>(y)[(size_t)row * N + col0 + i] = __float2bfloat16_rn(f[i]);
                            }
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (CG == 2) mbar_arrive_cluster(back_s + 8 * a);
                else mbar_arrive(acce_s + 8 * a);
            }
        }
    }
    if (!ok) atomicExch(status, 1);
    __syncthreads();
    // all MMAs have ended (in an aborted CTA too): shared and tensor memory may be given back
    if (warp == 1) mbar_wait(done_s, 0);
    // a CTA of a pair stays until the other one has no more use for its shared memory, barriers and tensor memory
    if (CG == 2) cluster_sync();
    if (warp == 1) {
        tc_fence_after();
        if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// ---------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------

typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                             const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                             CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeFn encode_fn() {
    static EncodeFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeFn>(p);
        cudaGetLastError();
    }
    return fn;
}

// bf16 [rows, k] row-major -> boxes of 64 x box_rows elements, 128-byte swizzle, zero fill outside
static bool make_map(const void *base, int64_t rows, int64_t k, int box_rows, CUtensorMap *map) {
    EncodeFn fn = encode_fn();
    if (!fn || ((uintptr_t)base & 15u) || (k * 2) % 16) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)k * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kDgBK, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1u, 1u};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool gemm_dense_shape_ok(const nnq_ctx *ctx, int64_t m, int64_t n, int64_t k, int x_dt) {
    static const char *env_min = diag_env("NNQ_DENSE_MIN_M");   // tuning aid
    const int64_t min_m = env_min ? atoll(env_min) : 256;
    return x_dt == NNQ_BF16 && m >= min_m && k >= kDgBK && k % kDgBK == 0 && n >= 1 && m < (1ll << 31) && n < (1ll << 31) && encode_fn() != nullptr;
}
bool gemm_dense_supported(const nnq_ctx *ctx, const nnq_weight *w, int64_t m, int x_dt) {
    if (!w || !w->d_raw || !gemm_dense_shape_ok(ctx, m, w->n, w->k, x_dt)) return false;
    // a bf16 weight is multiplied in place, the others are decoded into the scratch
    return (w->fmt == NNQ_BF16_DENSE && !((uintptr_t)w->d_raw & 15u)) || (ctx->d_dense && (size_t)w->n * (size_t)w->k * 2 <= ctx->dense_bytes);
}

nnq_status dense_scratch_reserve(nnq_ctx *ctx, int64_t n, int64_t k) {
    if (k < kDgBK || k % kDgBK) return NNQ_OK;
    const size_t need = (size_t)n * (size_t)k * 2;
    if (need <= ctx->dense_bytes) return NNQ_OK;
    cudaFree(ctx->d_dense);   // load time: synchronising here is fine
    ctx->d_dense = nullptr;
    ctx->dense_bytes = 0;
    nnq_status s = check_cuda(ctx, cudaMalloc(&ctx->d_dense, need), "cudaMalloc bf16 weight scratch");
    if (s != NNQ_OK) return s;
    ctx->dense_bytes = need;
    return NNQ_OK;
}

// Shape of a tile: its width and the CTAs that share it. Pair / single CTAs with 128 x 256 in us (waves of tiles in brackets):
// - pairs with 256 x 256, whose waves are 10 to 18 % shorter from K = 4096 on and about 5 % at 1024: 25600 x 5120 at 4096 rows
//   683 / 739 (22, 22), at 1300 rows 258 / 264 (9, 8), 151936 x 1024 at 2049 rows 572 / 577 (73, 69);
// - single CTAs with 128 x 256 where those need fewer waves by more than that (ragged rows): 4096 x 4096 at 1025 rows 47.8 / 33.0
//   (2, 1), 12288 x 4096 at 257 rows 51.4 / 38.7 (2, 1), at 1025 rows 93 / 86 (4, 3), 151936 x 1024 at 1025 rows 313 / 303 (41, 37);
// - and in the first wave on a weight just decoded, while both operands fit half of L2 (start-up counts, memory does not): with the
//   decode 4096 x 4096 at 640 rows 34.8 / 33.0, 5120 x 2048 at 640 25.6 / 24.6, 1024 x 4096 at 4096 31.4 / 30.1; but
//   4096 x 8192 at 640 61 / 70, 1024 x 12288 at 2600 69 / 80;
// - single CTAs with 128 x 128 where the large tiles would leave more than half of the SMs without work: 1024 x 4096 at 1024 rows,
//   256 x 128 by a pair / 128 x 128 by a CTA 25.6 / 22.8.
struct DgShape {
    int bn, cg;
};
static DgShape dg_pick(const nnq_ctx *ctx, int64_t m, int64_t n, int64_t k, bool decoded) {
    const int64_t wide = (n + 255) / 256, pair_tiles = (m + 255) / 256 * wide, tiles = (m + 127) / 128 * wide;
    if (4 * pair_tiles <= ctx->sm_count) return {128, 1};
    const int64_t pairs = ctx->sm_count / 2, pair_waves = (pair_tiles + pairs - 1) / pairs, waves = (tiles + ctx->sm_count - 1) / ctx->sm_count;
    if (decoded && waves == 1 && (m + n) * k * 2 <= 60ll << 20) return {256, 1};
    return 16 * pair_waves <= (k >= 2048 ? 18 : 17) * waves ? DgShape{256, 2} : DgShape{256, 1};
}

struct DgArgs {
    DgOuts outs;
    int m, n, k, y_dt;
    __nv_bfloat16 *h_out;
    int gate_kind;
};

template <int BN, int CG>
static nnq_status dg_launch(nnq_ctx *ctx, const CUtensorMap &xmap, const CUtensorMap &wmap, const DgArgs &a, int64_t tiles, cudaStream_t stream) {
    static bool configured[64] = {};
    const int smem = dg_smem_bytes(BN, CG);
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        nnq_status s = check_cuda(ctx, cudaFuncSetAttribute(gemm_dense_kernel<BN, CG>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem), "GEMM attribute");
        if (s != NNQ_OK) return s;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    const int64_t most = ctx->sm_count / CG;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(CG * (tiles < most ? tiles : most)));
    cfg.blockDim = dim3(kDgThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CG;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = CG == 2 ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_dense_kernel<BN, CG>, xmap, wmap, a.outs, a.m, a.n, a.k, a.y_dt, ctx->d_status, a.h_out, a.gate_kind);
    ctx->launches++;
    return check_cuda(ctx, e, "bf16 GEMM launch");
}

static nnq_status dg_launch_shape(nnq_ctx *ctx, DgShape shape, const CUtensorMap &xmap, const CUtensorMap &wmap, const DgArgs &a, int64_t tiles, cudaStream_t stream) {
    if (shape.cg == 2) return dg_launch<256, 2>(ctx, xmap, wmap, a, tiles, stream);
    return shape.bn == 256 ? dg_launch<256, 1>(ctx, xmap, wmap, a, tiles, stream) : dg_launch<128, 1>(ctx, xmap, wmap, a, tiles, stream);
}

// The GEMM alone: w_bf16 is a bf16 [n, k] weight in device memory (16-byte aligned), decoded: just before. h_out: see
// launch_gemm_dense_pairs.
static nnq_status dense_outs(nnq_ctx *ctx, const void *w_bf16, const void *x, const DgArgs &d, bool decoded, cudaStream_t stream) {
    CUtensorMap xmap, wmap;
    memset(&xmap, 0, sizeof(xmap));
    memset(&wmap, 0, sizeof(wmap));
    const DgShape shape = dg_pick(ctx, d.m, d.n, d.k, decoded);
    if (!make_map(x, d.m, d.k, kDgBM, &xmap) || !make_map(w_bf16, d.n, d.k, shape.bn / shape.cg, &wmap))
        return fail(ctx, NNQ_ERR_DISPATCH_FAILED, "tensor map creation failed");
    const int64_t rows = kDgBM * shape.cg, tiles = ((int64_t)d.m + rows - 1) / rows * (((int64_t)d.n + shape.bn - 1) / shape.bn);
    return dg_launch_shape(ctx, shape, xmap, wmap, d, tiles, stream);
}
static nnq_status dense_bf16(nnq_ctx *ctx, const void *w_bf16, const TcArgs &a, __nv_bfloat16 *h_out, int gate_kind, bool decoded, cudaStream_t stream) {
    const DgArgs d = {{{a.y}, {a.bias}, {0, (int)a.n}, 1}, (int)a.m, (int)a.n, (int)a.k, a.y_dt, h_out, gate_kind};
    return dense_outs(ctx, w_bf16, a.x, d, decoded, stream);
}

nnq_status launch_gemm_dense_bf16(nnq_ctx *ctx, const void *w_bf16, const TcArgs &a, cudaStream_t stream) { return dense_bf16(ctx, w_bf16, a, nullptr, 0, w_bf16 == ctx->d_dense, stream); }

nnq_status launch_gemm_dense_pairs(nnq_ctx *ctx, const TcArgs &a, __nv_bfloat16 *h_out, int gate_kind, cudaStream_t stream) {
    return dense_bf16(ctx, a.w, a, h_out, gate_kind, false, stream);
}

static cudaError_t decode_bf16(nnq_ctx *ctx, int fmt, const uint8_t *w, const uint8_t *scales, int64_t nchunks, void *dst, cudaStream_t stream, int cpr = 1, int half_rows = 0,
                               int pair = -1) {
    ctx->launches++;
    switch (fmt) {
#define NNQ_DB(F) case F: return launch_dequant_bf16<F>(w, scales, nchunks, dst, ctx->sm_count, stream, cpr, half_rows, pair)
        NNQ_DB(NNQ_Q4_0); NNQ_DB(NNQ_Q4_1); NNQ_DB(NNQ_Q8_0); NNQ_DB(NNQ_Q4_K); NNQ_DB(NNQ_Q4_K_GGML); NNQ_DB(NNQ_Q6_K);
        NNQ_DB(NNQ_MXFP4_CORE); NNQ_DB(NNQ_MXFP4_SPLIT); NNQ_DB(NNQ_MXFP4_GPTOSS); NNQ_DB(NNQ_Q5_0); NNQ_DB(NNQ_Q5_1);
        NNQ_DB(NNQ_Q2_K); NNQ_DB(NNQ_Q3_K); NNQ_DB(NNQ_Q5_K);
        NNQ_DB(NNQ_F32_DENSE); NNQ_DB(NNQ_BF16_DENSE);
#undef NNQ_DB
        default: return cudaErrorInvalidValue;
    }
}

nnq_status launch_gemm_dense(nnq_ctx *ctx, const TcArgs &a, cudaStream_t stream) {
    // a bf16 weight is its own decoded form
    if (a.fmt == NNQ_BF16_DENSE && !((uintptr_t)a.w & 15u)) return launch_gemm_dense_bf16(ctx, a.w, a, stream);
    const Geometry g = geometry(a.fmt);
    nnq_status s = check_cuda(ctx, decode_bf16(ctx, a.fmt, a.w, a.scales, a.n * (a.k / g.elems) * (g.elems / 32), ctx->d_dense, stream), "bf16 decode launch");
    return s != NNQ_OK ? s : launch_gemm_dense_bf16(ctx, ctx->d_dense, a, stream);
}

// Products of one input with weights of one format (query, key and value) as one GEMM over the decoded weights one behind the other:
// a narrow weight's tiles fill the last wave of a wide one instead of one of their own (4096, 1024 and 1024 rows of 4096 at 2048 tokens:
// three waves instead of two, one and one). Prompt of 2048 tokens through eight layers of the Qwen3-8B shape: 8.22 / 8.06 ms.
bool gemm_dense_batch_supported(const nnq_ctx *ctx, const SkinnyJob *jobs, int count, int64_t m, int x_dt) {
    if (count < 2 || count > kDgMaxOuts || jobs[0].w->fmt == NNQ_BF16_DENSE) return false;
    size_t bytes = 0;
    int64_t rows = 0;
    for (int i = 0; i < count; i++) {
        const nnq_weight *w = jobs[i].w;
        if (w->fmt != jobs[0].w->fmt || w->k != jobs[0].w->k || jobs[i].x != jobs[0].x || !gemm_dense_supported(ctx, w, m, x_dt) || (i + 1 < count && w->n % 256)) return false;
        bytes += (size_t)w->n * (size_t)w->k * 2;
        rows += w->n;
    }
    return bytes <= ctx->dense_bytes && rows < (1ll << 31);
}
nnq_status launch_gemm_dense_batch(nnq_ctx *ctx, const SkinnyJob *jobs, int count, int64_t m, int y_dt, cudaStream_t stream) {
    const int64_t k = jobs[0].w->k;
    const Geometry g = geometry(jobs[0].w->fmt);
    DgArgs d = {};
    d.outs.count = count;
    for (int i = 0; i < count; i++) {
        const nnq_weight *w = jobs[i].w;
        uint8_t *dst = static_cast<uint8_t *>(ctx->d_dense) + (size_t)d.outs.begin[i] * (size_t)k * 2;
        nnq_status s = check_cuda(ctx, decode_bf16(ctx, w->fmt, w->d_raw, w->d_scales, w->n * (k / g.elems) * (g.elems / 32), dst, stream), "bf16 decode launch");
        if (s != NNQ_OK) return s;
        d.outs.y[i] = jobs[i].y;
        d.outs.bias[i] = jobs[i].bias;
        d.outs.begin[i + 1] = d.outs.begin[i] + (int)w->n;
    }
    d.m = (int)m;
    d.n = d.outs.begin[count];
    d.k = (int)k;
    d.y_dt = y_dt;
    return dense_outs(ctx, ctx->d_dense, jobs[0].x, d, true, stream);
}

// Gate and up products of one input and the activation in one GEMM over the two weights decoded to alternating rows of the
// caller's buffer: the f32 products are neither written nor read, and no kernel multiplies them. Prompt of 2048
// tokens through eight layers of the Qwen3-8B shape (gate and up of 12288 x 4096), apart / together: 8.80 / 8.17 ms.
size_t gemm_dense_gate_up_bytes(const nnq_weight *gate, const nnq_weight *up) {
    if (!gate || !up || gate->fmt != up->fmt || gate->n != up->n || gate->k != up->k || gate->fmt == NNQ_BF16_DENSE || !gate->d_raw || !up->d_raw) return 0;
    return gate->n % 8 == 0 && gate->k >= kDgBK && gate->k % kDgBK == 0 && gate->n * (gate->k / 32) < (1ll << 30) ? (size_t)gate->n * (size_t)gate->k * 4 : 0;
}
nnq_status launch_gemm_dense_gate_up(nnq_ctx *ctx, const nnq_weight *gate, const nnq_weight *up, void *w_bf16, const void *x, int64_t m, __nv_bfloat16 *h_out, cudaStream_t stream) {
    const Geometry g = geometry(gate->fmt);
    const int64_t nchunks = gate->n * (gate->k / g.elems) * (g.elems / 32);
    const nnq_weight *w[2] = {gate, up};
    for (int i = 0; i < 2; i++) {
        nnq_status s = check_cuda(ctx, decode_bf16(ctx, w[i]->fmt, w[i]->d_raw, w[i]->d_scales, nchunks, w_bf16, stream, (int)(gate->k / 32), 0, i), "bf16 decode launch");
        if (s != NNQ_OK) return s;
    }
    const TcArgs a = {nullptr, nullptr, x, nullptr, nullptr, m, 2 * gate->n, gate->k, NNQ_BF16_DENSE, NNQ_BF16, NNQ_BF16};
    return dense_bf16(ctx, w_bf16, a, h_out, kDgSilu, true, stream);
}

bool gemm_dense_grouped_supported(const nnq_ctx *ctx, const TcGroupArgs &g) {
    if (g.kn && (g.fmt != NNQ_MXFP4_GPTOSS || g.n % kKnTile || g.k % kKnTile || ((uintptr_t)g.w & 15u))) return false;
    const bool room = g.pairs || (ctx->d_dense && (size_t)g.experts * (size_t)g.n * (size_t)g.k * 2 <= ctx->dense_bytes);
    return room && g.k >= kDgBK && g.k % kDgBK == 0 && g.experts >= 1 && g.experts <= kGeMaxGroups && g.rows_upper >= 1 && g.rows_upper < (1ll << 30) &&
           (int64_t)g.experts * g.n < (1ll << 31) && encode_fn() != nullptr;
}

bool gemm_dense_grouped_fuses_swiglu(const TcGroupArgs &g) {
    return g.h_out != nullptr && (g.pairs || g.fmt == NNQ_MXFP4_SPLIT || g.fmt == NNQ_MXFP4_GPTOSS) && g.n % 2 == 0 &&
           (int64_t)g.experts * g.n * (g.k / 32) < (1ll << 31);
}

nnq_status launch_gemm_dense_grouped(nnq_ctx *ctx, const TcGroupArgs &g, cudaStream_t stream) {
    // the experts' raw blocks are one contiguous [experts, N, K] tensor: one decode launch
    Geometry geo = geometry(g.fmt);
    const int64_t nchunks = (int64_t)g.experts * g.n * (g.k / geo.elems) * (geo.elems / 32);
    cudaError_t e = cudaSuccess;
    // SwiGLU in the GEMM's epilogue (g.h_out given): needs the gate / up rows interleaved in the decoded copy,
    // which the direct MXFP4 decode can write at no cost
    const bool fuse = gemm_dense_grouped_fuses_swiglu(g);
    const int cpr = (int)(g.k / 32), half = fuse ? (int)(g.n / 2) : 0;
    const void *w_bf16 = g.pairs ? (const void *)g.w : ctx->d_dense;
    if (g.pairs) {
        // bf16 experts are multiplied where they are
    } else if (g.kn) {
        const int kt = g.k % (3 * kKnTile) == 0 ? 3 : 1;
        const dim3 grid((unsigned)(g.n / kKnTile), (unsigned)(g.k / (kt * kKnTile)), (unsigned)g.experts);
        __nv_bfloat16 *dst = static_cast<__nv_bfloat16 *>(ctx->d_dense);
        if (kt == 3) dequant_kn_bf16_kernel<3><<<grid, 384, 0, stream>>>(g.w, g.scales, dst, (int)g.k, (int)g.n, half);
        else dequant_kn_bf16_kernel<1><<<grid, 128, 0, stream>>>(g.w, g.scales, dst, (int)g.k, (int)g.n, half);
        e = cudaGetLastError();
        ctx->launches++;
    } else {
        e = decode_bf16(ctx, g.fmt, g.w, g.scales, nchunks, ctx->d_dense, stream, cpr, half);
    }
    nnq_status s = check_cuda(ctx, e, "bf16 decode launch");
    if (s != NNQ_OK) return s;
    return launch_gemm_experts(ctx, g, w_bf16, fuse ? g.h_out : nullptr, stream);
}

}  // namespace nnq

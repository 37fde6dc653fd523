// Causal attention of a prompt's rows on the 5th-generation tensor cores with f32-class accuracy (Qwen3 layers: heads of 128, no
// window, bf16 decoders).
//
// q, k, v and the softmax weights are f32 and stay so in effect: every operand enters the tensor core as two f16 terms of the value
// scaled by a power of two (x = hi + lo, the remainder is below 2^-23 of x), a product is lo hi + hi lo + hi hi with f32 accumulation in
// tensor memory. Scores, maxima, exponentials, sums and the output accumulators are f32. Keys and values of a head share a power of
// two each, every query vector has its own, the softmax weights have kSpProb.
//
// What bounds it: the chain scores -> softmax -> weighted values of a key tile, about 1500 clocks of MMAs and 1300 of softmax for 128
// query vectors x 64 keys, and 64 KB of keys and values per tile from L2. So (1) a kernel in front splits keys and values once per
// layer, into images of the swizzled tiles as the MMAs read them (the tiles of a head are read by all its 64 query tiles of 2048 rows),
// and a tile is two bulk copies; (2) scores, softmax weights and weighted values have two places each in tensor memory, the weights are
// the operand that the MMA reads there: S(t + 2) and O(t) = P V are multiplied while the softmax of t + 1 runs.
// One CTA: 128 query vectors of one kv head (consecutive (row, query head of the group) pairs), key tiles of 64.
//   warps 0-3: softmax. Thread r owns query vector r: its 64 scores from tensor memory, maximum and sum, the weights as two f16 tiles
//              back to it; then adds the tile before's weighted values to its f32 accumulators.
//   warp 4, 6: a thread each copies keys / values, two stages.
//   warp 5:    one thread issues the MMAs.
// 2048 rows of the Qwen3-8B shape: 114 us and 15 for the two launches in front (307 and 5 with conversion by three warps of every
// CTA, the weights through shared memory and one place for each of S, P and O). Every wait is bounded.
#include <math.h>

#include <algorithm>

#include "blocks.cuh"
#include "pdl.cuh"
#include "sync.cuh"
#include "tcgen05.cuh"

namespace nnq {

constexpr int kSpKeys = 64, kSpRows = 128, kSpThreads = 224;
constexpr int kSpQAtom = kSpRows * 128, kSpKAtom = kSpKeys * 128;   // bytes of a tile of 64 columns (one swizzle row)
constexpr int kSpQ = 4 * kSpQAtom, kSpK = 4 * kSpKAtom, kSpV = 2 * 128 * 128;   // query tile, key and value image: two terms each
constexpr int kSpSmem = 1024 + kSpQ + 2 * (kSpK + kSpV);
constexpr uint32_t kSpCols = 512;   // S at 0 and 64, O at 128 and 256, P (hi, lo) at 384 and 448
constexpr float kSpLog2E = 1.4426950408889634f;
constexpr float kSpProb = 16384.0f;

// scale * x and scale * y as f16 pairs: the nearest values and the nearest values of what they leave
__device__ __forceinline__ void split2_f16(float x, float y, float scale, uint32_t &hi, uint32_t &lo) {
    const float2 v = __fmul2_rn(make_float2(x, y), make_float2(scale, scale));
    const __half2 h = __floats2half2_rn(v.x, v.y);
    const float2 r = __ffma2_rn(__half22float2(h), make_float2(-1.0f, -1.0f), v);
    const __half2 l = __floats2half2_rn(r.x, r.y);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}
// The power of two that brings the largest of some values (the bits of its absolute value) to 2^14 .. 2^15, and its inverse
// (largest values below 2^-112 are scaled like that one: the inverse stays a normal number).
__device__ __forceinline__ uint32_t top_exponent(uint32_t bits) { return min(max(bits >> 23, 15u), 254u); }
__device__ __forceinline__ float top_scale(uint32_t bits) { return __uint_as_float((268u - top_exponent(bits)) << 23); }
__device__ __forceinline__ float top_unscale(uint32_t bits) { return __uint_as_float((top_exponent(bits) - 14u) << 23); }
__device__ __forceinline__ uint32_t abs_bits4(float4 v) {
    const uint32_t all = 0x7FFFFFFFu;
    return max(max(__float_as_uint(v.x) & all, __float_as_uint(v.y) & all), max(__float_as_uint(v.z) & all, __float_as_uint(v.w) & all));
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// byte offset of element e (0 .. 63) of row r inside a swizzled tile of 128-byte rows
__device__ __forceinline__ uint32_t sp_at(int r, int e) { return swz(r, e >> 3) + 2 * (e & 7); }

// The bits of the largest absolute key and value of every tile of 64 keys, [kv heads, tiles]; a NaN is above an infinity.
__global__ void __launch_bounds__(256) attn_top_kernel(const float *__restrict__ kcache, const float *__restrict__ vcache, int cap, int keys, uint2 *__restrict__ top) {
    __shared__ uint32_t m[2];
    const int tid = threadIdx.x, key0 = blockIdx.x * kSpKeys, have = min(kSpKeys, keys - key0);
    pdl_release();
    if (tid < 2) m[tid] = 0;
    __syncthreads();
    pdl_prologue();
    const size_t at = ((size_t)blockIdx.y * cap + key0) * 128;
    uint32_t k = 0, v = 0;
#pragma unroll
    for (int i = 0; i < kSpKeys * 32 / 256; i++) {
        const int u = tid + 256 * i;
        if (u < have * 32) {
            k = max(k, abs_bits4(reinterpret_cast<const float4 *>(kcache + at)[u]));
            v = max(v, abs_bits4(reinterpret_cast<const float4 *>(vcache + at)[u]));
        }
    }
    k = __reduce_max_sync(0xFFFFFFFFu, k);
    v = __reduce_max_sync(0xFFFFFFFFu, v);
    if ((tid & 31) == 0) {
        atomicMax(&m[0], k);
        atomicMax(&m[1], v);
    }
    __syncthreads();
    if (tid == 0) top[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = make_uint2(m[0], m[1]);
}

// Images of the key tile (rows = keys: hi, lo of two 64-wide pieces) and the value tile (rows = dimensions: hi, lo), [kv heads from kv0 on, tiles].
__global__ void __launch_bounds__(256) attn_image_kernel(const float *__restrict__ kcache, const float *__restrict__ vcache, int cap, int keys, int kv0, const uint2 *__restrict__ top,
                                                         uint8_t *__restrict__ images) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tiles = gridDim.x, key0 = blockIdx.x * kSpKeys, have = min(kSpKeys, keys - key0);
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    pdl_release();
    pdl_prologue();
    const int kvh = kv0 + blockIdx.y;
    const uint2 m = attn_largest(top + (size_t)kvh * tiles, tiles);
    if (max(m.x, m.y) >= kNotFinite) return;
    const float k_scale = top_scale(m.x), v_scale = top_scale(m.y);
    const float *kb = kcache + ((size_t)kvh * cap + key0) * 128, *vb = vcache + ((size_t)kvh * cap + key0) * 128;
    uint8_t *dst = images + ((size_t)blockIdx.y * tiles + blockIdx.x) * (kSpK + kSpV);
    float4 k[8], x[4], y[4];
#pragma unroll
    for (int i = 0; i < 8; i++) k[i] = warp + 8 * i < have ? *reinterpret_cast<const float4 *>(kb + (warp + 8 * i) * 128 + 4 * lane) : zero;
    // values: a lane has a pair of keys and four dimensions of every 32
    const int j = 2 * lane;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int d = 4 * (warp + 8 * i);
        x[i] = j < have ? *reinterpret_cast<const float4 *>(vb + j * 128 + d) : zero;
        y[i] = j + 1 < have ? *reinterpret_cast<const float4 *>(vb + (j + 1) * 128 + d) : zero;
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int d = 4 * lane;
        uint2 hi, lo;
        split2_f16(k[i].x, k[i].y, k_scale, hi.x, lo.x);
        split2_f16(k[i].z, k[i].w, k_scale, hi.y, lo.y);
        uint8_t *p = dst + (d >> 6) * kSpKAtom + sp_at(warp + 8 * i, d & 63);
        *reinterpret_cast<uint2 *>(p) = hi;
        *reinterpret_cast<uint2 *>(p + 2 * kSpKAtom) = lo;
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float xv[4] = {x[i].x, x[i].y, x[i].z, x[i].w}, yv[4] = {y[i].x, y[i].y, y[i].z, y[i].w};
#pragma unroll
        for (int e = 0; e < 4; e++) {
            uint32_t hi, lo;
            split2_f16(xv[e], yv[e], v_scale, hi, lo);
            uint8_t *p = dst + kSpK + sp_at(4 * (warp + 8 * i) + e, j);
            *reinterpret_cast<uint32_t *>(p) = hi;
            *reinterpret_cast<uint32_t *>(p + kSpV / 2) = lo;
        }
    }
}

__device__ __forceinline__ void sp_st8(uint32_t addr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};"
                 ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(addr) : "memory");
}

__global__ void __launch_bounds__(kSpThreads, 1) attn_split_kernel(const WindowAttn a, int kv0, const uint2 *__restrict__ top, int all_tiles, const uint8_t *__restrict__ images, int *status) {
    extern __shared__ __align__(1024) uint8_t sp_smem_raw[];
    uint8_t *smem = sp_smem_raw + (-smem_u32(sp_smem_raw) & 1023u);
    __shared__ __align__(8) uint64_t bars[14];   // k_full, k_empty, v_full, v_empty, s_full, p_full, o_full: two each
    __shared__ uint32_t tmem_s;
    __shared__ float q_unscale[kSpRows];
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0);
    const uint32_t kf = smem_u32(bars), ke = kf + 16, vf = kf + 32, ve = kf + 48, sf = kf + 64, pf = kf + 80, of = kf + 96;
    // (the last rows first: they see the most keys)
    const int kvh = kv0 + blockIdx.x, group = a.heads / a.kv_heads, pairs = a.span.n * group, t0 = (gridDim.y - 1 - blockIdx.y) * kSpRows;
    const int last_pair = min(pairs, t0 + kSpRows) - 1, pos0 = a.span.pos0;
    const int tiles = (pos0 + last_pair / group) / kSpKeys + 1;
    pdl_release();
    pdl_prologue();
    const uint2 m2 = attn_largest(top + (size_t)kvh * all_tiles, all_tiles);
    if (max(m2.x, m2.y) >= kNotFinite) return;
    uint8_t *k_s = smem + kSpQ, *v_s = k_s + 2 * kSpK;
    const uint8_t *image = images + (size_t)blockIdx.x * all_tiles * (kSpK + kSpV);

    if (tid == 0) {
        for (int i = 0; i < 14; i++) mbar_init(kf + 8 * i, i >= 10 && i < 12 ? 4 : 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)), "r"(kSpCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    {
        // the 128 query vectors, a warp per vector and turn: a lane has four dimensions; all loads of a turn before the first store
        constexpr int QN = 10;
        for (int r0 = warp; r0 < kSpRows; r0 += 7 * QN) {
            float4 v[QN];
#pragma unroll
            for (int i = 0; i < QN; i++) {
                const int r = r0 + 7 * i, t = t0 + r;
                v[i] = r < kSpRows && t <= last_pair ? *reinterpret_cast<const float4 *>(a.qrot + ((size_t)(t / group) * a.heads + kvh * group + t % group) * 128 + 4 * lane)
                                                     : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
#pragma unroll
            for (int i = 0; i < QN; i++) {
                const int r = r0 + 7 * i, d = 4 * lane;
                if (r >= kSpRows) continue;
                const uint32_t big = __reduce_max_sync(0xFFFFFFFFu, abs_bits4(v[i]));
                const float scale = top_scale(big);
                if (lane == 0) q_unscale[r] = top_unscale(big);
                uint2 hi, lo;
                split2_f16(v[i].x, v[i].y, scale, hi.x, lo.x);
                split2_f16(v[i].z, v[i].w, scale, hi.y, lo.y);
                uint8_t *dst = smem + (d >> 6) * kSpQAtom + sp_at(r, d & 63);
                *reinterpret_cast<uint2 *>(dst) = hi;
                *reinterpret_cast<uint2 *>(dst + 2 * kSpQAtom) = lo;
            }
        }
        fence_async_smem();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, tmem_s, 0);
    bool ok = true;

    if (warp < 4) {
        // ---------------- softmax ----------------
        const int row = (t0 + tid) / group, my_hi = pos0 + row;   // the last key this vector sees (rows past the end are not stored)
        const float c = fmaxf(a.scale * kSpLog2E * q_unscale[tid] * top_unscale(m2.x), 1.2e-38f);   // (never 0: masked scores are infinite)
        const uint32_t base_t = tmem + ((uint32_t)(warp * 32) << 16);
        float acc[128];
#pragma unroll
        for (int i = 0; i < 128; i++) acc[i] = 0.0f;
        float m = -INFINITY, l = 0.0f, corr = 1.0f, late = 1.0f;   // late: the factor that belongs to the tile before's values
        auto add_values = [&](int t) {
            if (!__all_sync(0xFFFFFFFFu, mbar_wait_fast(of + 8 * (t & 1), (t >> 1) & 1))) {
                ok = false;
                return;
            }
            tc_fence_after();
#pragma unroll
            for (int b = 0; b < 4; b++) {
                uint32_t v[32];
                tmem_ld32(base_t + 128 + 128 * (t & 1) + b * 32, v);
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    const float2 r = __ffma2_rn(make_float2(acc[b * 32 + i], acc[b * 32 + i + 1]), make_float2(late, late),
                                                make_float2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])));
                    acc[b * 32 + i] = r.x;
                    acc[b * 32 + i + 1] = r.y;
                }
            }
        };
        for (int t = 0; t < tiles && ok; t++) {
            if (!__all_sync(0xFFFFFFFFu, mbar_wait_fast(sf + 8 * (t & 1), (t >> 1) & 1))) {
                ok = false;
                break;
            }
            tc_fence_after();
            uint32_t s[2][32];
            tmem_ld32(base_t + 64 * (t & 1), s[0]);
            tmem_ld32(base_t + 64 * (t & 1) + 32, s[1]);
            const int hi = my_hi - t * kSpKeys;   // visible keys of the tile: 0 .. hi
            if (!__all_sync(0xFFFFFFFFu, hi >= kSpKeys - 1)) {
#pragma unroll
                for (int i = 0; i < 64; i++) s[i >> 5][i & 31] = i <= hi ? s[i >> 5][i & 31] : __float_as_uint(-INFINITY);
            }
            float mt[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int i = 0; i < 64; i++) mt[i & 3] = fmaxf(mt[i & 3], __uint_as_float(s[i >> 5][i & 31]));
            const float mn = fmaxf(m, fmaxf(fmaxf(mt[0], mt[1]), fmaxf(mt[2], mt[3])) * c);   // finite: every vector sees the first key
            corr = m == mn ? 1.0f : exp2f(m - mn);
            float2 sum = make_float2(0.0f, 0.0f);
            const float2 c2 = make_float2(c, c), nb = make_float2(-mn, -mn);
            const uint32_t p_t = base_t + 384 + 64 * (t & 1);
#pragma unroll
            for (int ch = 0; ch < 4; ch++) {   // 16 weights
                uint32_t h[8], lw[8];
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    const int i = ch * 16 + 2 * e;
                    const float2 x = __ffma2_rn(make_float2(__uint_as_float(s[i >> 5][i & 31]), __uint_as_float(s[i >> 5][(i & 31) + 1])), c2, nb);
                    const float p0 = ex2(x.x), p1 = ex2(x.y);
                    sum = __fadd2_rn(sum, make_float2(p0, p1));
                    split2_f16(p0, p1, kSpProb, h[e], lw[e]);
                }
                sp_st8(p_t + 8 * ch, h);
                sp_st8(p_t + 32 + 8 * ch, lw);
            }
            l = fmaf(l, corr, sum.x + sum.y);
            m = mn;
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (elect_one()) mbar_arrive(pf + 8 * (t & 1));
            if (t) add_values(t - 1);
            late = corr;
        }
        if (ok) add_values(tiles - 1);
        if (ok && t0 + tid <= last_pair) {
            const int head = kvh * group + (t0 + tid) % group;
            const float inv = top_unscale(m2.y) * (1.0f / kSpProb) / l;
            uint4 *o = reinterpret_cast<uint4 *>(reinterpret_cast<__nv_bfloat16 *>(a.ffn.act) + (size_t)row * a.ffn.out_k + head * 128);
#pragma unroll
            for (int d = 0; d < 128; d += 8)
                o[d / 8] = make_uint4(pack_bf16(acc[d] * inv, acc[d + 1] * inv), pack_bf16(acc[d + 2] * inv, acc[d + 3] * inv),
                                      pack_bf16(acc[d + 4] * inv, acc[d + 5] * inv), pack_bf16(acc[d + 6] * inv, acc[d + 7] * inv));
        }
    } else if (warp == 5) {
        // ---------------- MMA issuer (the warp waits together, one lane issues) ----------------
        const uint32_t id_s = (1u << 4) | ((uint32_t)(kSpKeys >> 3) << 17) | ((128u >> 4) << 24);   // both operands f16
        const uint32_t id_o = (1u << 4) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
        const uint32_t qa = smem_u32(smem);
        auto scores = [&](int t) {   // the small products first, so that their sums are rounded at their size
            if (!__all_sync(0xFFFFFFFFu, mbar_wait_fast(kf + 8 * (t & 1), (t >> 1) & 1))) {
                ok = false;
                return;
            }
            tc_fence_after();
            if (elect_one()) {
                const uint32_t ka = smem_u32(k_s + (t & 1) * kSpK);
#pragma unroll
                for (int i = 0; i < 3; i++) {   // lo hi, hi lo, hi hi
                    const uint32_t qo = qa + (i == 0 ? 2 * kSpQAtom : 0), ko = ka + (i == 1 ? 2 * kSpKAtom : 0);
#pragma unroll
                    for (int at = 0; at < 2; at++) {
                        const uint64_t dq = smem_desc(qo + at * kSpQAtom), dk = smem_desc(ko + at * kSpKAtom);
#pragma unroll
                        for (int k = 0; k < 4; k++) umma_bf16(tmem + 64 * (t & 1), dq + 2 * k, dk + 2 * k, id_s, (i | at | k) != 0);
                    }
                }
                umma_commit(sf + 8 * (t & 1));
                umma_commit(ke + 8 * (t & 1));
            }
            __syncwarp();
        };
        scores(0);
        if (ok && tiles > 1) scores(1);
        for (int t = 0; t < tiles && ok; t++) {
            ok = __all_sync(0xFFFFFFFFu, mbar_wait_fast(pf + 8 * (t & 1), (t >> 1) & 1) && mbar_wait_fast(vf + 8 * (t & 1), (t >> 1) & 1));
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const uint32_t va = smem_u32(v_s + (t & 1) * kSpV), pa = tmem + 384 + 64 * (t & 1), oa = tmem + 128 + 128 * (t & 1);
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    const uint64_t dv = smem_desc(va + (i == 1 ? kSpV / 2 : 0));
#pragma unroll
                    for (int k = 0; k < 4; k++) umma_ts(oa, pa + (i == 0 ? 32 : 0) + 8 * k, dv + 2 * k, id_o, (i | k) != 0);
                }
                umma_commit(of + 8 * (t & 1));
                umma_commit(ve + 8 * (t & 1));
            }
            __syncwarp();
            if (t + 2 < tiles) scores(t + 2);   // (its place was read before the weights of t came)
        }
        if (!ok) {
            // MMAs that were issued may still read shared memory and write tensor memory: one more bounded wait
            if (elect_one()) umma_commit(sf);
            __syncwarp();
            for (int i = 0; i < 2; i++) mbar_wait(sf, i);
        }
    } else if (lane == 0) {
        // ---------------- keys (warp 4), values (warp 6) ----------------
        const bool values = warp == 6;
        const uint32_t full = values ? vf : kf, empty = values ? ve : ke, bytes = values ? kSpV : kSpK;
        const uint32_t dst = smem_u32(values ? v_s : k_s);
        const uint8_t *src = image + (values ? kSpK : 0);
        int issued = 0;
        for (int t = 0; t < tiles; t++) {
            if (t >= 2 && !mbar_wait_fast(empty + 8 * (t & 1), ((t >> 1) - 1) & 1)) {
                ok = false;
                break;
            }
            mbar_expect_tx(full + 8 * (t & 1), bytes);
            bulk_g2s(dst + (t & 1) * bytes, src + (size_t)t * (kSpK + kSpV), bytes, full + 8 * (t & 1));
            issued = t + 1;
        }
        // every copy has landed before the shared memory is given back
        for (int t = max(0, issued - 2); t < issued; t++) ok &= mbar_wait(full + 8 * (t & 1), (t >> 1) & 1);
    }
    if (!ok) atomicExch(status, 1);
    tc_fence_before();
    __syncthreads();
    if (warp == 5) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kSpCols) : "memory");
    }
}

int attn_tiles(int keys) { return (keys + kSpKeys - 1) / kSpKeys; }
size_t attn_image_bytes(int kv_heads, int keys) { return (size_t)kv_heads * attn_tiles(keys) * (kSpK + kSpV); }

bool attn_split_supported(const WindowAttn &a) {
    return a.ffn.act_dt == NNQ_BF16 && a.dim == 128 && a.vdim == 128 && a.dim_ld == 128 && a.vdim_ld == 128 && !a.gated && a.window >= a.cap &&
           a.span.pos0 + a.span.n <= a.cap && a.ffn.out_k % 8 == 0 && a.span.n * (a.heads / a.kv_heads) >= 32;
}

// Operands as two f16 terms hold 22 to 24 bits of every value that is at most 2^16 below the largest of its query vector, or of the
// head's keys or values (2^-39 of that largest below). Error of the outputs against 64 bits, f32 kernel / this / two bf16 terms: 4.8e-7 /
// 1.6e-7 / 1.7e-6 for 2048 rows of normal values, 1.2e-6 / 5.7e-7 / 9.5e-6 with four times the queries, 7.8e-7 / 3.6e-7 / 4.3e-6 for
// 4000 rows, 2.1e-7 / 1.8e-7 / 4.0e-6 for 9 rows behind 20. Kv heads with an infinity or a NaN are left to the f32 kernel.
// top: [kv_heads, attn_tiles(keys)], images: attn_image_bytes(held, keys), of `held` kv heads at a time.
nnq_status launch_attn_split(nnq_ctx *ctx, const WindowAttn &a, uint2 *top, uint8_t *images, int held, cudaStream_t st) {
    const int keys = a.span.pos0 + a.span.n, tiles = attn_tiles(keys), pairs = a.span.n * (a.heads / a.kv_heads);
    nnq_status s = check_cuda(ctx, cudaFuncSetAttribute(attn_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSpSmem), "attention shared memory");
    if (s != NNQ_OK) return s;
    launch_pdl(attn_top_kernel, dim3(tiles, a.kv_heads), dim3(256), st, a.kcache, a.vcache, a.cap, keys, top);
    for (int kv0 = 0; kv0 < a.kv_heads; kv0 += held) {
        const int heads = std::min(held, a.kv_heads - kv0);
        launch_pdl(attn_image_kernel, dim3(tiles, heads), dim3(256), st, a.kcache, a.vcache, a.cap, keys, kv0, top, images);
        launch_pdl_smem(attn_split_kernel, dim3(heads, (pairs + kSpRows - 1) / kSpRows), dim3(kSpThreads), kSpSmem, st, a, kv0, top, tiles, images, ctx->d_status);
        ctx->launches += 2;
    }
    ctx->launches++;
    return check_cuda(ctx, cudaGetLastError(), "prompt attention launch");
}

}  // namespace nnq

// The kernels between the products of a prompt's rows (Qwen3 layers): norms, rotation, activation, four elements per thread.
// In a file of their own: beside the kernels of the decode step they changed how the compiler schedules that step's attention
// (162 -> 146 registers, fewer loads in flight, 36 layers behind 2048 tokens 2.54 -> 2.60 ms).
#include <cuda_bf16.h>
#include <math.h>

#include "decoder_common.cuh"
#include "nnq_internal.h"

namespace nnq {

__device__ __forceinline__ void store_act4(void *p, int act_dt, size_t i4, float4 v) {
    if (act_dt == NNQ_F32) {
        reinterpret_cast<float4 *>(p)[i4] = v;
    } else {
        __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
        reinterpret_cast<uint2 *>(p)[i4] = make_uint2(*reinterpret_cast<uint32_t *>(&a), *reinterpret_cast<uint32_t *>(&b));
    }
}

// Many rows of silu(g) * u, four elements per thread (widths in whole groups of four): bound by memory, 10 bytes per element
// (2048 rows of 12288: 252 MB). Eight layers of the Qwen3-8B shape over 2048
// tokens, one element per thread / this: 0.96 / 0.32 ms.
__global__ void __launch_bounds__(256)
dec_silu_mul_rows_kernel(const float4 *__restrict__ g, const float4 *__restrict__ u, void *__restrict__ mid, int act_dt, int64_t n4) {
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n4; i += (int64_t)gridDim.x * 256) {
        const float4 x = g[i], y = u[i];
        store_act4(mid, act_dt, i, make_float4((x.x / (1.0f + expf(-x.x))) * y.x, (x.y / (1.0f + expf(-x.y))) * y.y, (x.z / (1.0f + expf(-x.z))) * y.z,
                                               (x.w / (1.0f + expf(-x.w))) * y.w));
    }
}

// The rows below in one pass over memory, the row's elements in registers: widths in whole groups of four up to 8192, rows of the
// embedding on 8-byte boundaries. 16 norms of 2048 rows of 4096, two passes over scalars / this: 0.56 / 0.32 ms.
template <int MAXV>
__global__ void __launch_bounds__(256)
dec_norm_rows4_kernel(float *__restrict__ h, const float *__restrict__ delta, const __nv_bfloat16 *__restrict__ embed, const int *__restrict__ tokens,
                      const float *__restrict__ w, float eps, void *__restrict__ xn, int act_dt, int hidden) {
    __shared__ float red[32];
    const size_t r = blockIdx.x;
    const int n4 = hidden >> 2;
    float4 *hr = reinterpret_cast<float4 *>(h + r * hidden);
    const float4 *dr = reinterpret_cast<const float4 *>(delta ? delta + r * hidden : nullptr);
    const uint2 *er = reinterpret_cast<const uint2 *>(embed ? embed + (size_t)tokens[r] * hidden : nullptr);
    float4 v[MAXV];
    float ss = 0.0f;
#pragma unroll
    for (int j = 0; j < MAXV; j++) {
        const int i = threadIdx.x + 256 * j;
        v[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (i < n4) {
            if (er) {
                const uint2 e = er[i];
                v[j] = make_float4(__uint_as_float(e.x << 16), __uint_as_float(e.x & 0xFFFF0000u), __uint_as_float(e.y << 16), __uint_as_float(e.y & 0xFFFF0000u));
            } else {
                const float4 a = hr[i], b = dr[i];
                v[j] = make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
            }
            hr[i] = v[j];
        }
        ss = fmaf(v[j].x, v[j].x, fmaf(v[j].y, v[j].y, fmaf(v[j].z, v[j].z, fmaf(v[j].w, v[j].w, ss))));
    }
    const float rms = sqrtf(block_sum(ss, red) / (float)hidden + eps);
    char *xr = reinterpret_cast<char *>(xn) + r * hidden * (act_dt == NNQ_F32 ? 4 : 2);
#pragma unroll
    for (int j = 0; j < MAXV; j++) {
        const int i = threadIdx.x + 256 * j;
        if (i < n4) {
            const float4 a = reinterpret_cast<const float4 *>(w)[i];
            store_act4(xr, act_dt, i, make_float4((v[j].x / rms) * a.x, (v[j].y / rms) * a.y, (v[j].z / rms) * a.z, (v[j].w / rms) * a.w));
        }
    }
}

// Heads of 128: a warp per head of a row, four dimensions per lane (the pair of a dimension, 64 on, is 16 lanes away), eight
// heads per CTA: 0.57 -> 0.20 ms for eight layers of 2048 rows. Same numbers as dec_qk_rope_rows_kernel (decoder.cu) but for the order of the sum
// of squares.
__global__ void __launch_bounds__(256)
dec_qk_rope_rows128_kernel(const float *__restrict__ q, const float *__restrict__ k, const float *__restrict__ v, const float *__restrict__ qw,
                           const float *__restrict__ kw, const float *__restrict__ cosv, const float *__restrict__ sinv, int pos0, float eps,
                           float *__restrict__ qrot, float *__restrict__ kcache, float *__restrict__ vcache, int n_heads, int n_kv, int rows, int max_seq) {
    const int lane = threadIdx.x & 31, heads = n_heads + 2 * n_kv;
    const int64_t unit = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (unit >= (int64_t)rows * heads) return;
    const int row = (int)(unit / heads), head = (int)(unit - (int64_t)row * heads), pos = pos0 + row;
    const size_t qoff = (size_t)row * n_heads * 128, kvoff = (size_t)row * n_kv * 128;
    if (head >= n_heads + n_kv) {
        const int kvh = head - n_heads - n_kv;
        reinterpret_cast<float4 *>(vcache + ((size_t)kvh * max_seq + pos) * 128)[lane] = reinterpret_cast<const float4 *>(v + kvoff + kvh * 128)[lane];
        return;
    }
    const bool is_q = head < n_heads;
    const float4 x = reinterpret_cast<const float4 *>(is_q ? q + qoff + head * 128 : k + kvoff + (head - n_heads) * 128)[lane];
    float ss = fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, x.w * x.w)));
#pragma unroll
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
    const float rms = sqrtf(ss / 128.0f + eps);
    const float4 w = reinterpret_cast<const float4 *>(is_q ? qw : kw)[lane];
    const float a[4] = {(x.x / rms) * w.x, (x.y / rms) * w.y, (x.z / rms) * w.z, (x.w / rms) * w.w};
    const float4 c4 = reinterpret_cast<const float4 *>(cosv + (size_t)pos * 64)[lane & 15], s4 = reinterpret_cast<const float4 *>(sinv + (size_t)pos * 64)[lane & 15];
    const float c[4] = {c4.x, c4.y, c4.z, c4.w}, sn[4] = {s4.x, s4.y, s4.z, s4.w};
    float y[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float b = __shfl_xor_sync(0xFFFFFFFFu, a[i], 16);
        y[i] = lane < 16 ? a[i] * c[i] - b * sn[i] : b * sn[i] + a[i] * c[i];
    }
    float *dst = is_q ? qrot + qoff + head * 128 : kcache + ((size_t)(head - n_heads) * max_seq + pos) * 128;
    reinterpret_cast<float4 *>(dst)[lane] = make_float4(y[0], y[1], y[2], y[3]);
}

void launch_norm_rows4(float *h, const float *delta, const __nv_bfloat16 *embed, const int *tokens, const float *w, float eps, void *xn, int act_dt, int hidden, int rows,
                       cudaStream_t st) {
    if (hidden <= 4096) dec_norm_rows4_kernel<4><<<rows, 256, 0, st>>>(h, delta, embed, tokens, w, eps, xn, act_dt, hidden);
    else dec_norm_rows4_kernel<8><<<rows, 256, 0, st>>>(h, delta, embed, tokens, w, eps, xn, act_dt, hidden);
}

void launch_qk_rope_rows128(const float *q, const float *k, const float *v, const float *qw, const float *kw, const float *cosv, const float *sinv, int pos0, float eps,
                            float *qrot, float *kcache, float *vcache, int n_heads, int n_kv, int rows, int max_seq, cudaStream_t st) {
    const int64_t units = (int64_t)rows * (n_heads + 2 * n_kv);
    dec_qk_rope_rows128_kernel<<<(unsigned)((units + 7) / 8), 256, 0, st>>>(q, k, v, qw, kw, cosv, sinv, pos0, eps, qrot, kcache, vcache, n_heads, n_kv, rows, max_seq);
}

void launch_silu_mul_rows(nnq_ctx *ctx, const float *g, const float *u, void *mid, int act_dt, int64_t total, cudaStream_t st) {
    const int64_t want = (total / 4 + 255) / 256, most = 16 * (int64_t)ctx->sm_count;
    dec_silu_mul_rows_kernel<<<(unsigned)(want < most ? want : most), 256, 0, st>>>((const float4 *)g, (const float4 *)u, mid, act_dt, total / 4);
}

}  // namespace nnq

// Products of the rows of a mixture-of-experts block, hundreds per expert, with decoded bf16 weights: for every expert e and routed row r
// of it, out[r, :] = x[r, :] * W_e^T (+ bias_e), or the gated activation of interleaved gate / up rows.
//
// As gemm_dense.cu (persistent pairs of CTAs, cta_group::2, rings of TMA boxes, two accumulators in tensor memory), with the weights
// as the rows of the MMA and the routed rows as its columns: an expert's rows come in any number, and the columns of an MMA come in
// steps of 32, its rows in steps of 256. An expert's rows are dealt to tiles of at most 256 of equal size; a tile costs the tensor cores
// what it holds (its copies are boxes of 128 routed rows for each CTA, whatever it holds).
// Bound by the tensor cores: 16384 routed rows of 32 experts, 2880 x 5760 and 2880 x 2880, 660 us (1.24 PFLOP/s); with the routed rows
// as the rows of single CTAs' MMAs, 128 at a time, it was 912.
// The epilogue finds a weight row in a lane and a routed row in a column: a warp stores 32 neighbouring values of one routed row.
#include <cuda.h>
#include <cuda_bf16.h>
#include <string.h>

#include "decoder_common.cuh"
#include "gemm_tc.h"
#include "sync.cuh"
#include "tcgen05.cuh"

namespace nnq {

constexpr int kGeThreads = 192, kGeStages = 6, kGeHalf = 128 * 128, kGeStageBytes = 2 * kGeHalf;   // 128 weight rows, 128 routed rows, 64 of k
constexpr int kGeSmem = kGeStages * kGeStageBytes + 1024, kGeCols = 256;

__device__ __forceinline__ void ge_tma_pair(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar) : "memory");
}

__global__ void __launch_bounds__(kGeThreads, 1)
gemm_experts_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, const float *__restrict__ bias, float *__restrict__ y, int N, int K,
                    int *status, const int *__restrict__ offsets, int groups, __nv_bfloat16 *__restrict__ h_out, float swiglu_limit) {
    extern __shared__ __align__(1024) uint8_t ge_smem_raw[];
    uint8_t *smem = ge_smem_raw + (-smem_u32(ge_smem_raw) & 1023u);
    __shared__ __align__(8) uint64_t bars[2 * kGeStages + 5];   // full, empty [kGeStages], acc_full[2], acc_empty[2], every MMA has ended
    __shared__ uint32_t tmem_base_s;
    __shared__ int tile_begin[kGeMaxGroups + 1], row_begin[kGeMaxGroups + 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0);
    const uint32_t full_s = smem_u32(bars), empty_s = full_s + 8 * kGeStages;
    const uint32_t accf_s = empty_s + 8 * kGeStages, acce_s = accf_s + 16, done_s = acce_s + 16;
    const int rank = (int)cluster_rank(), unit = blockIdx.x / 2, units = gridDim.x / 2;   // a pair multiplies one tile at a time
    for (int e = tid; e <= groups; e += kGeThreads) row_begin[e] = offsets[e];
    __syncthreads();
    if (tid == 0) {
        int acc = 0;
        for (int e = 0; e < groups; e++) {
            tile_begin[e] = acc;
            acc += (row_begin[e + 1] - row_begin[e] + kGeCols - 1) / kGeCols;
        }
        tile_begin[groups] = acc;
        for (int s = 0; s < kGeStages; s++) {
            mbar_init(full_s + 8 * s, 1);
            mbar_init(empty_s + 8 * s, 1);
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(accf_s + 8 * a, 1);
            mbar_init(acce_s + 8 * a, 8);
        }
        mbar_init(done_s, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();   // both CTAs' barriers are set up
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xFFFFFFFFu, tmem_base_s, 0);
    const int n_tiles = (N + 255) / 256, tiles = tile_begin[groups] * n_tiles, nkb = K / 64;
    // tile t -> (expert, first routed row, columns, rows that exist, this CTA's first weight row). Expert by expert, the tiles of a
    // weight tile side by side: the pairs work on a few experts at a time, whose rows stay in L2 (weight tiles of all experts in
    // turn had the routed rows, 94 MB for 4096 tokens, read again from memory for each: 871 us).
    auto locate = [&](int t, int &e, int &m0, int &cols, int &cnt, int &n0) {
        e = 0;
        while (e + 1 < groups && t >= tile_begin[e + 1] * n_tiles) e++;
        const int rows = row_begin[e + 1] - row_begin[e], parts = tile_begin[e + 1] - tile_begin[e], i = t - tile_begin[e] * n_tiles, nt = i / parts;
        cols = ((rows + parts - 1) / parts + 31) / 32 * 32;
        m0 = row_begin[e] + (i - nt * parts) * cols;
        cnt = min(cols, row_begin[e + 1] - m0);   // (may be nothing: the columns are rounded up)
        n0 = nt * 256 + rank * 128;
    };
    bool ok = true;

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            const uint32_t count_s = cluster_addr(full_s, 0);   // the barriers that count the copies
            int slot = 0;
            uint32_t phase = 0;
            long long filled = 0;
            for (int t = unit; t < tiles && ok; t += units) {
                int e, m0, cols, cnt, n0;
                locate(t, e, m0, cols, cnt, n0);
                const int w0 = e * N + n0, x0 = m0 + rank * (cols / 2);
                for (int kb = 0; kb < nkb; kb++) {
                    if (filled >= kGeStages && !mbar_wait_fast(empty_s + 8 * slot, phase ^ 1u)) {
                        ok = false;
                        break;
                    }
                    const uint32_t a_s = smem_u32(smem + (size_t)slot * kGeStageBytes);
                    if (rank == 0) mbar_expect_tx(full_s + 8 * slot, 2 * kGeStageBytes);
                    ge_tma_pair(a_s, &wmap, kb * 64, w0, count_s + 8 * slot);
                    ge_tma_pair(a_s + kGeHalf, &xmap, kb * 64, x0, count_s + 8 * slot);
                    filled++;
                    if (++slot == kGeStages) {
                        slot = 0;
                        phase ^= 1u;
                    }
                }
            }
            // The last use of every stage: this CTA's copies have landed and been read, and the arrivals on its barriers, which for the
            // second CTA come from the first, are over. Behind a wait that ran out the stages may never be given back; the copies are
            // still waited for (by the CTA whose barriers count them).
            for (long long f = filled > kGeStages ? filled - kGeStages : 0; f < filled; f++) {
                const uint32_t s = (uint32_t)(f % kGeStages), p = (uint32_t)(f / kGeStages) & 1u;
                if (ok) ok = mbar_wait_fast(empty_s + 8 * s, p);
                if (!ok && rank == 0) mbar_wait(full_s + 8 * s, p);
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (the warp waits together, one lane issues) ----------------
        if (rank == 0) {
            int slot = 0, it = 0;
            uint32_t phase = 0;
            for (int t = unit; t < tiles && ok; t += units, it++) {
                const int a = it & 1;
                int e, m0, cols, cnt, n0;
                locate(t, e, m0, cols, cnt, n0);
                const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(cols >> 3) << 17) | ((256u >> 4) << 24);
                // the epilogue has read this accumulator's previous tile
                if (it >= 2) ok = __all_sync(0xFFFFFFFFu, mbar_wait_fast(acce_s + 8 * a, (uint32_t)(((it >> 1) - 1) & 1)));
                const uint32_t acc = tmem_base + (uint32_t)(a * kGeCols);
                for (int kb = 0; kb < nkb && ok; kb++) {
                    ok = __all_sync(0xFFFFFFFFu, mbar_wait_fast(full_s + 8 * slot, phase));
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t a_s = smem_u32(smem + (size_t)slot * kGeStageBytes);
                        const uint64_t da = smem_desc(a_s), db = smem_desc(a_s + kGeHalf);
#pragma unroll
                        for (int k = 0; k < 4; k++) umma_bf16_pair(acc, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
                        umma_commit_pair(empty_s + 8 * slot);
                        if (kb == nkb - 1) umma_commit_pair(accf_s + 8 * a);
                    }
                    __syncwarp();
                    if (++slot == kGeStages) {
                        slot = 0;
                        phase ^= 1u;
                    }
                }
            }
            if (elect_one()) umma_commit_pair(done_s);   // also behind a wait that ran out
            __syncwarp();
        }
    } else {
        // ---------------- epilogue ----------------
        const uint32_t back_s = cluster_addr(acce_s, 0);
        const int q = warp & 3, I = N >> 1;   // the quarter of the 128 TMEM lanes this warp may read
        int it = 0;
        for (int t = unit; t < tiles && ok; t += units, it++) {
            const int a = it & 1;
            int e, m0, cols, cnt, n0;
            locate(t, e, m0, cols, cnt, n0);
            const int row = n0 + q * 32 + lane;
            const bool live = row < N;
            float b = 0.0f;
            if (bias && live) b = __ldg(bias + (size_t)e * N + (h_out ? (row & 1 ? I : 0) + (row >> 1) : row));
            if (!__all_sync(0xFFFFFFFFu, mbar_wait_fast(accf_s + 8 * a, (uint32_t)((it >> 1) & 1)))) {
                ok = false;
                break;
            }
            tc_fence_after();
#pragma unroll 1
            for (int c0 = 0; c0 < cnt; c0 += 32) {
                uint32_t v[32];
                tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(a * kGeCols + c0), v);
                const int left = cnt - c0;   // routed rows of these 32 columns
                if (h_out) {
                    // Interleaved gate / up rows (2j, 2j + 1) lie in neighbouring lanes: an even lane forms h = clamp(silu(g), +-limit) * u of
                    // every even column, an odd one of every odd column. (Fast exponential and division, 2^-22 relative near zero, 2^-20
                    // at -16: far below the bf16 rounding of h.)
                    __nv_bfloat16 *h = h_out + (size_t)(m0 + c0 + (lane & 1)) * I + (row >> 1);
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        const float x0 = __uint_as_float(v[i]) + b, x1 = __uint_as_float(v[i + 1]) + b;
                        const float got = __shfl_xor_sync(0xFFFFFFFFu, lane & 1 ? x0 : x1, 1);
                        const float g = lane & 1 ? got : x0, u = lane & 1 ? x1 : got;
                        const float s = fminf(fmaxf(__fdividef(g, 1.0f + __expf(-g)), -swiglu_limit), swiglu_limit);
                        if (live && i + (lane & 1) < left) h[(size_t)i * I] = __float2bfloat16_rn(s * u);
                    }
                } else if (live) {
                    float *o = y + (size_t)(m0 + c0) * N + row;
                    if (left >= 32) {
#pragma unroll
                        for (int i = 0; i < 32; i++) o[(size_t)i * N] = __uint_as_float(v[i]) + b;
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; i++)
                            if (i < left) o[(size_t)i * N] = __uint_as_float(v[i]) + b;
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(back_s + 8 * a);
        }
    }
    if (!ok) atomicExch(status, 1);
    __syncthreads();
    // all MMAs have ended (in an aborted CTA too): shared and tensor memory may be given back
    if (warp == 1) mbar_wait(done_s, 0);
    cluster_sync();   // a CTA stays until the other one has no more use for its shared memory, barriers and tensor memory
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// w_bf16: [experts, n, k]; h_out given: the activation of interleaved gate / up rows instead of y.
nnq_status launch_gemm_experts(nnq_ctx *ctx, const TcGroupArgs &g, const void *w_bf16, __nv_bfloat16 *h_out, cudaStream_t stream) {
    CUtensorMap xmap, wmap;
    memset(&xmap, 0, sizeof(xmap));
    memset(&wmap, 0, sizeof(wmap));
    if (!encode_map_2d(&xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, g.x_bf16, g.k, g.rows_upper, 2 * g.k, 64, 128, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !encode_map_2d(&wmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, w_bf16, g.k, (int64_t)g.experts * g.n, 2 * g.k, 64, 128, CU_TENSOR_MAP_SWIZZLE_128B))
        return fail(ctx, NNQ_ERR_DISPATCH_FAILED, "tensor map creation failed");
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        nnq_status s = check_cuda(ctx, cudaFuncSetAttribute(gemm_experts_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGeSmem), "GEMM attribute");
        if (s != NNQ_OK) return s;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(ctx->sm_count / 2 * 2));   // (the number of tiles is known on the device only)
    cfg.blockDim = dim3(kGeThreads);
    cfg.dynamicSmemBytes = kGeSmem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_experts_kernel, xmap, wmap, g.bias, reinterpret_cast<float *>(g.y), (int)g.n, (int)g.k, ctx->d_status, g.offsets, g.experts,
                                             h_out, g.swiglu_limit);
    ctx->launches++;
    return check_cuda(ctx, e, "expert GEMM launch");
}

}  // namespace nnq

// ksplit.cu -- products of the tensor-core GEMMs cut along K: how many parts, and the pass that adds them up.
#include "common.cuh"
#include "pdl.cuh"

namespace b200q {

// dst[n][m] = sum over the K parts, part 0 first: V consecutive rows a thread, a column of dst per blockIdx.y
template <int V>
__global__ void __launch_bounds__(256)
ksplit_sum_kernel(const float *__restrict__ parts, int ksplit, int64_t part_stride, int M, float *__restrict__ dst, int64_t ldd) {
    pdl_trigger();
    pdl_wait();
    const int m = ((int)blockIdx.x * 256 + (int)threadIdx.x) * V;
    if (m >= M) return;
    const float *p = parts + (int64_t)blockIdx.y * M + m;
    float *o = dst + (int64_t)blockIdx.y * ldd + m;
    if (V == 4) {
        float4 acc = *reinterpret_cast<const float4 *>(p);
        for (int z = 1; z < ksplit; ++z) {
            const float4 v = *reinterpret_cast<const float4 *>(p + z * part_stride);
            acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        }
        *reinterpret_cast<float4 *>(o) = acc;
    } else {
        float acc = *p;
        for (int z = 1; z < ksplit; ++z) acc += p[z * part_stride];
        *o = acc;
    }
}

// Into how many parts to cut K: the schedule's length in nanoseconds, rounds of units over the SMs plus, for more than one
// part, the pass that adds them (a launch and its traffic). t: a k-step (one raw stage) and a unit of the kernel, see common.cuh.
// Of 20 shapes (tiles 4 to 256, 4 to 74 steps) in each of the seven types, timed at every number of parts with the kernels as they are, the
// choice is 0.6 % from the fastest on average, at most 14 % (Q6_K 11008x4096 x 100 tokens: 35 us whole, 31 in three parts; the next
// worst is Q5_K at the same size, 8 %).
int choose_ksplit(const b200q_ctx *ctx, int64_t tiles, int64_t steps, KsplitTimes t, int64_t outputs, int64_t most, int64_t chunks) {
    int best_ks = 1;
    int64_t best = 0;
    if (ctx->no_ksplit) return 1;
    for (int ks = 1; ks <= most && (ks == 1 || steps / ks >= 2); ++ks) {
        const int64_t len = chunks * schedule_ns(ctx, tiles, steps, ks, t) + ksplit_sum_ns(ks, outputs);
        if (ks == 1 || len < best) { best = len; best_ks = ks; }
    }
    return best_ks;
}

// The number of parts (1: the product stays whole) and where they go. Where the scratch cannot be had, on a full device or inside a
// capture that would have to grow it, the product is cut into what the block there is holds.
int plan_ksplit(b200q_ctx *ctx, int64_t tiles, int64_t steps, KsplitTimes t, int64_t M, int64_t N, float **parts, int64_t chunks) {
    Workspace *ws = &ctx->moe_ws[9];
    const size_t part = sizeof(float) * (size_t)(N * M);
    int ks = choose_ksplit(ctx, tiles, steps, t, M * N, MOST_PARTS, chunks);
    if (ks > 1 && !ws_try_reserve(ctx, ws, part * ks)) {
        const size_t hold = ws->cap / part;                 // (less than ks)
        ks = choose_ksplit(ctx, tiles, steps, t, M * N, hold < 1 ? 1 : (int64_t)hold, chunks);
    }
    *parts = (float *)ws->ptr;
    return ks;
}

b200q_status launch_ksplit_sum(b200q_ctx *ctx, const float *parts, int ksplit, int64_t part_stride, int64_t M, int64_t N, float *dst, int64_t ldd) {
    // four rows a thread where every part's and dst's columns start on 16 bytes
    const bool vec = M % 4 == 0 && ldd % 4 == 0 && (uintptr_t)dst % 16 == 0;
    for (int64_t n0 = 0; n0 < N; n0 += 65535) {
        const unsigned nn = (unsigned)(N - n0 < 65535 ? N - n0 : 65535);
        const float *p = parts + n0 * M;
        float *o = dst + n0 * ldd;
        B200Q_CUDA(ctx, vec ? launch_pdl(!ctx->no_pdl, ksplit_sum_kernel<4>, dim3((unsigned)((M / 4 + 255) / 256), nn), dim3(256), 0, ctx->stream, p, ksplit,
                                         part_stride, (int)M, o, ldd)
                            : launch_pdl(!ctx->no_pdl, ksplit_sum_kernel<1>, dim3((unsigned)((M + 255) / 256), nn), dim3(256), 0, ctx->stream, p, ksplit,
                                         part_stride, (int)M, o, ldd));
        B200Q_CUDA(ctx, cudaGetLastError());
    }
    count(ctx, ST_GEMM_KSPLIT);
    return B200Q_OK;
}

}  // namespace b200q

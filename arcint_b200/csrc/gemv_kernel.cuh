// gemv_kernel.cuh -- the decode GEMV kernel template (see gemv.cu for the description).
#pragma once

#include "gemv_core.cuh"
#include "pdl.cuh"

namespace b200q {

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// index of column c of the second column group (0 when there is no second group, so the
// never-used instantiation still indexes inside its arrays)
template <int NCG, int NC2> __host__ __device__ constexpr int second_group_index(int c) {
    return (NC2 > 0 && c < NC2) ? NCG + c : 0;
}

// MUL_MAT_ID view of the same kernel: the "columns" of a unit are the pairs of one route
// tile (all of one expert), so a unit is (tile, row batch) and its weight base, activation
// columns and output addresses come from the tile. Pair p = t*n_used + i has expert
// ids[t][i], activation column (i % ne11) + t*ne11 and output dst + t*ld2 + i*ld1
// (the reference's ID_PROLOGUE, marfrit/arcint contrib/llama.cpp/patches/
// 0000-01-kquant-integer-dpas.patch:3917-3934).
struct GemvId {
    const int32_t *tiles;      // [n][4]: expert, first pair, count, - ; NULL: direct mode, tile p = pair p
    const int32_t *n_tiles;    // device scalar (direct mode: unused)
    const int32_t *pairs;      // pairs sorted by expert (direct mode: unused)
    const uint8_t *ids;        // direct mode: ids[t][i] at ids + t*ids_stride + 4*i
    size_t         ids_stride;
    int            n_pairs, n_expert;
    int            n_used, ne11;
    size_t         expert_stride;   // bytes between expert matrices
    int64_t        ld1, ld2;        // dst strides of slot i and token t, in floats
    // a second product over the same activation and route in the same launch (gate and up of a feed-forward block): from the first one's
    // weights and results to its own, in bytes and floats (n_mat = 1: none)
    int            n_mat;
    int64_t        w_off, dst_off;
};

// How a product's rows lie: every row a 16-byte multiple from a 16-byte start; rows whose starts are only a multiple of what
// the lane code needs (gemv_row_align); anything else.
enum { GEMV_ROWS_BYTES = 0, GEMV_ROWS_ALIGNED = 1, GEMV_ROWS_SHIFTED = 2 };
// the start alignment with which the lane code takes a row: words at any even byte, 8 bytes (IQ4_XS), 16 (Q4_K, Q5_K)
__host__ __device__ constexpr int gemv_row_align(int type) {
    return type == B200Q_TYPE_Q4_K || type == B200Q_TYPE_Q5_K ? 16 : type == B200Q_TYPE_IQ4_XS ? 8 : 2;
}
// all_starts: the matrix address and every stride between rows (and experts) or-ed together
inline int gemv_row_mode(int type, size_t all_starts, size_t row_bytes) {
    if (all_starts % 16 == 0 && row_bytes % 16 == 0) return GEMV_ROWS_ALIGNED;
    return all_starts % (size_t)gemv_row_align(type) == 0 ? GEMV_ROWS_SHIFTED : GEMV_ROWS_BYTES;
}
template <int TYPE> __host__ __device__ constexpr int gemv_kernel_slot(int rows) { return GemvStage<TYPE>::SLOT + (rows == GEMV_ROWS_SHIFTED ? 16 : 0); }

// One warp owns a batch of B consecutive rows at a time and walks the row in stages of 2048
// weights. For each stage it holds the activation side (64 codes per lane and column, scales,
// block sums) in registers and runs the B staged row chunks against it, so the activation
// loads, address arithmetic and pipeline bookkeeping are paid once per B rows. The chunks
// arrive through a per-warp ring of NSETS sets of B slots filled with 16-byte asynchronous
// copies: NSETS-1 sets are in flight while the current one is consumed. More
// than four columns are taken as two column groups over the same staged set.
// ROWS: how the rows lie (gemv_row_mode): 16-byte aligned, shifted (a row's stage starts anywhere in a 16-byte unit: the
// copies start at the boundary below and the lane code adds the remainder; a copy never leaves the 16-byte units that
// hold the row's own bytes) or fetched two bytes at a time.
template <int TYPE, int NC, int B, int WARPS, int NSETS, int ROWS, bool ID>
__global__ void __launch_bounds__(WARPS * 32)
gemv_kernel(const uint8_t *__restrict__ W, size_t row_stride, int M, int nblk, GemvAct act,
            float *__restrict__ dst, int ldd, GemvId id) {
    typedef GemvFmt<TYPE> F;
    typedef GemvStage<TYPE> S;
    constexpr int NCG = NC <= 4 ? NC : (NC + 1) / 2;      // columns of the first group
    constexpr int NC2 = NC - NCG;                         // columns of the second group (0: none)
    constexpr int N2 = NC2 > 0 ? NC2 : 1;
    constexpr int SLOT = gemv_kernel_slot<TYPE>(ROWS);
    constexpr int PIECES = (S::BYTES + (ROWS == GEMV_ROWS_SHIFTED ? 15 : 0) + 511) / 512;        // 16-byte copies per lane and chunk
    extern __shared__ __align__(16) uint8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint8_t *ring = smem + warp * (NSETS * B * SLOT);
    if (ID) pdl_wait();                  // the route (tile lists, counts) comes from the kernel before

    const int row_bytes = nblk * F::BLK_B;
    const int nstages = (nblk + F::STAGE_BLOCKS - 1) / F::STAGE_BLOCKS;
    const int n_bt = (M + B - 1) / B;                     // row batches per matrix
    const bool direct = ID && id.tiles == nullptr;
    const int n_tiles = ID ? (direct ? id.n_pairs : __ldg(id.n_tiles)) : 1, n_units = n_tiles * n_bt * (ID ? id.n_mat : 1);
    // direct mode: the expert of pair p, read from ids and clamped like the reference's route kernel
    auto pair_expert = [&](int p) {
        const int t = p / id.n_used, i = p - t * id.n_used;
        const int e = __ldg(reinterpret_cast<const int32_t *>(id.ids + (size_t)t * id.ids_stride) + i);
        return min(max(e, 0), id.n_expert - 1);
    };
    const int gw = blockIdx.x * WARPS + warp, tw = gridDim.x * WARPS;

    // producer cursor: unit and stage of the next set to fetch, and its place in the ring
    int p_u = gw, p_s = 0, p_set = 0;
    auto issue = [&]() {
        if (p_u < n_units) {
            const int off = p_s * S::BYTES;
            const int bytes = min((int)S::BYTES, row_bytes - off);
            const int row0 = (ID ? p_u % n_bt : p_u) * B;
            const uint8_t *src = W + (size_t)row0 * row_stride + off;
            if (ID) {
                const int t = p_u / n_bt, tile = t < n_tiles ? t : t - n_tiles;
                src += (size_t)(direct ? pair_expert(tile) : __ldg(id.tiles + 4 * tile)) * id.expert_stride + (t < n_tiles ? 0 : id.w_off);
            }
            uint8_t *d = ring + p_set * (B * SLOT);
#pragma unroll
            for (int r = 0; r < B; ++r) {
                if (row0 + r < M) {              // rows past the end keep stale bytes; never stored
                    if (ROWS == GEMV_ROWS_SHIFTED) {
                        const int sh = (int)((uintptr_t)src & 15);
#pragma unroll
                        for (int j = 0; j < PIECES; ++j) {
                            const int b = lane * 16 + j * 512;
                            if (b < sh + bytes) cp_async16(d + b, src - sh + b);
                        }
                    } else if (ROWS == GEMV_ROWS_ALIGNED) {
#pragma unroll
                        for (int j = 0; j < PIECES; ++j) {
                            const int b = lane * 16 + j * 512;
                            if (b < bytes) cp_async16(d + b, src + b);
                        }
                    } else {
                        for (int b = lane * 2; b < bytes; b += 64)
                            *reinterpret_cast<uint16_t *>(d + b) = *reinterpret_cast<const uint16_t *>(src + b);
                    }
                }
                src += row_stride;
                d += SLOT;
            }
            if (++p_s == nstages) { p_s = 0; p_u += tw; }
        }
        p_set = p_set + 1 == NSETS ? 0 : p_set + 1;
        cp_async_commit();
    };

    float acc[B][NC];
#pragma unroll
    for (int i = 0; i < NSETS - 1; ++i) issue();
    // the first weight stages are in flight; the activation (the quantizer's output) and dst (which
    // an earlier kernel may still be writing or reading) are touched only after this
    if (!ID) pdl_wait();
    int c_set = 0;
    for (int u = gw; u < n_units; u += tw) {
        // this unit's columns: where each reads its activation and writes its result
        int cols[NC];
        int64_t outs[NC];
        int ncol = NC;
        uintptr_t wbase = (uintptr_t)W;                    // where the unit's matrix begins (shifted rows)
        if (ID) {
            const int tile2 = u / n_bt, tile = tile2 < n_tiles ? tile2 : tile2 - n_tiles;
            const int first = direct ? tile : __ldg(id.tiles + 4 * tile + 1);
            ncol = direct ? 1 : __ldg(id.tiles + 4 * tile + 2);
            if (ROWS == GEMV_ROWS_SHIFTED) wbase += (size_t)(direct ? pair_expert(tile) : __ldg(id.tiles + 4 * tile)) * id.expert_stride + (tile2 < n_tiles ? 0 : id.w_off);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const int p = direct ? tile : __ldg(id.pairs + first + min(c, ncol - 1));   // short tiles repeat their last pair
                const int t = p / id.n_used, i = p - t * id.n_used;
                cols[c] = (i % id.ne11) + t * id.ne11;
                outs[c] = t * id.ld2 + i * id.ld1 + (tile2 < n_tiles ? 0 : id.dst_off);
            }
        } else {
#pragma unroll
            for (int c = 0; c < NC; ++c) { cols[c] = c; outs[c] = (int64_t)c * ldd; }
        }
        int cols1[NCG], cols2[N2];
#pragma unroll
        for (int c = 0; c < NCG; ++c) cols1[c] = cols[c];
#pragma unroll
        for (int c = 0; c < N2; ++c) cols2[c] = cols[second_group_index<NCG, NC2>(c)];
#pragma unroll
        for (int r = 0; r < B; ++r)
#pragma unroll
            for (int c = 0; c < NC; ++c) acc[r][c] = 0.f;
        const int row0 = (ID ? u % n_bt : u) * B;
        uint32_t shift[B];                                 // a stage is a multiple of 16 bytes: the same for all of a row's
#pragma unroll
        for (int r = 0; r < B; ++r) shift[r] = ROWS == GEMV_ROWS_SHIFTED ? (uint32_t)(wbase + (size_t)(row0 + r) * row_stride) & 15u : 0u;
        for (int s = 0; s < nstages; ++s) {
            __syncwarp();                    // every lane is done with the set about to be refilled
            issue();
            cp_async_wait<NSETS - 1>();      // all but the NSETS-1 newest sets have landed
            __syncwarp();
            const uint8_t *set = ring + c_set * (B * SLOT);
            c_set = c_set + 1 == NSETS ? 0 : c_set + 1;
            {
                GemvX<NCG> X;
                gemv_load_x<TYPE, NCG>(lane, s, nblk, act, cols1, X);
#pragma unroll
                for (int r = 0; r < B; ++r) {
                    float a[NCG];
#pragma unroll
                    for (int c = 0; c < NCG; ++c) a[c] = acc[r][c];
                    gemv_lane_row<TYPE, NCG>(reinterpret_cast<const uint32_t *>(set + r * SLOT), lane, X, a, shift[r]);
#pragma unroll
                    for (int c = 0; c < NCG; ++c) acc[r][c] = a[c];
                }
            }
            if (NC2 > 0) {
                GemvX<N2> X;
                gemv_load_x<TYPE, N2>(lane, s, nblk, act, cols2, X);
#pragma unroll
                for (int r = 0; r < B; ++r) {
                    float a[N2];
#pragma unroll
                    for (int c = 0; c < N2; ++c) a[c] = acc[r][second_group_index<NCG, NC2>(c)];
                    gemv_lane_row<TYPE, N2>(reinterpret_cast<const uint32_t *>(set + r * SLOT), lane, X, a, shift[r]);
#pragma unroll
                    for (int c = 0; c < N2; ++c)
                        if (c < NC2) acc[r][second_group_index<NCG, NC2>(c)] = a[c];
                }
            }
        }
#pragma unroll
        for (int r = 0; r < B; ++r)
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                float v = acc[r][c];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
                if (lane == 0 && row0 + r < M && c < ncol) dst[outs[c] + row0 + r] = v;
            }
    }
    // this block's work is done: once every block is here the next kernel of the stream may be
    // scheduled (any earlier and its blocks would take this wave's places on the SMs)
    pdl_trigger();
    cp_async_wait<0>();
}

}  // namespace b200q

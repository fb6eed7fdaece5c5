// tc_common.cuh -- PTX wrappers shared by the tensor-core (tcgen05) kernels: mbarriers with
// bounded waits, bulk copies, tensor-memory loads, UMMA descriptors, packed f32x2 arithmetic.
#pragma once

#include <stdint.h>

namespace b200q {
namespace tc {

// Polls of a bounded wait. A try_wait that fails has the hardware hold the thread for about 4 us (1000, 65,536 and 2^20 of them took 4.1,
// 259 and 4148 ms on B200), so a wait gives up after some four seconds.
constexpr uint32_t SPIN_LIMIT = 1u << 20;

// K-major, no swizzle, 128 rows: 8 rows x 16 bytes are one contiguous 128-byte core matrix; the
// two 16-byte halves of K=32 (int8) are LBO apart, the sixteen 8-row groups SBO apart.
constexpr uint32_t LBO = 16 * 128, SBO = 128;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// one arrival for the whole warp: the lanes' earlier writes and fences are ordered before it by
// the warp barrier. Barriers counted in warps take 32 times fewer serialized updates than
// barriers counted in threads, which matters when a handoff happens every few hundred clocks.
__device__ __forceinline__ void mbar_arrive_warp(uint32_t bar, int lane) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait: false when the limit ran out or another role already gave up. Kept small and not unrolled: there is one at every
// handoff, and unrolled four times (the compiler's choice) they made up most of a GEMM's 80 KB of code, whose warps then waited
// for instructions (1.5 warps of five per issue).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    uint32_t i = 0;
    bool ok;
#pragma unroll 1
    do {
        ok = mbar_try(bar, parity);
    } while (!ok && ((++i & 63) || (i < SPIN_LIMIT && !*abort_flag)));
    if (!ok) *abort_flag = 1;
    return ok;
}
// the same for a whole warp: every lane finishes its own bounded wait, then the warp agrees
// on the outcome, so the warp-synchronous instructions that follow never see a split warp
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    return __all_sync(0xFFFFFFFFu, mbar_wait(bar, parity, abort_flag) ? 1 : 0) != 0;
}
// Two barriers, usually both ready: one look and one vote cost a warp what a wait for one of them does, some 100 clk.
__device__ __forceinline__ bool mbar_ready_warp(uint32_t bar0, uint32_t parity0, uint32_t bar1, uint32_t parity1) {
    const bool a = mbar_try(bar0, parity0), b = mbar_try(bar1, parity1);
    return __all_sync(0xFFFFFFFFu, a && b ? 1 : 0) != 0;
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// One tiled tensor-map copy of a [rows x bytes] box of the packed weight matrix (a 2-D view in
// 32-bit elements): x in elements (x * 4 is a multiple of 16), y the first row; rows past the
// matrix arrive as zeros and still count toward the barrier's byte total. No multicast.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void *tmap, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(tmap), "r"(x), "r"(y), "r"(bar) : "memory");
}
// the same box out of matrix z of a stack of matrices (the experts of MUL_MAT_ID): rows past the
// matrix's own M arrive as zeros, they never come from the next matrix
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const void *tmap, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const void *tmap) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(tmap) : "memory");
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(LBO >> 4) << 16) | ((uint64_t)(SBO >> 4) << 32) | (1ull << 46);
}
// the same with the two strides given: lbo between the 16-byte halves of K, sbo between 8-row groups
__device__ __forceinline__ uint64_t umma_desc2(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46);
}
// the descriptor of an address `bytes` on (shared-memory addresses stay below 2^18, so the sum carries nowhere)
__device__ __forceinline__ uint64_t umma_desc_on(uint64_t desc, uint32_t bytes) {
    return (desc & 0xFFFFFFFF00000000ull) | (uint32_t)((uint32_t)desc + (bytes >> 4));
}
__device__ __forceinline__ void tmem_ld32(uint32_t addr, uint32_t (&v)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
                   "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
                   "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                 : "r"(addr) : "memory");
}
// 16-byte shared load kept where it is written (volatile asm keeps program order), so the
// compiler does not hoist a whole block's worth of scale loads into live registers
__device__ __forceinline__ float4 lds128(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}
// two f32 lanes per register pair: Blackwell's packed FP32 instructions halve the issue slots
// of the scale-accumulate (the FP32 pipe still does two lanes' worth of work per instruction)
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 f2_pack(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_unpack(f32x2 v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 f2_fma(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 f2_mul(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 f2_add(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// two 64-bit shared loads kept in program order (see lds128)
__device__ __forceinline__ void lds128_f2(uint32_t addr, f32x2 &a, f32x2 &b) {
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr));
}
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&v)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(addr) : "memory");
}
// the same 32-bit value into sixteen consecutive columns of the warp's 32 lanes
__device__ __forceinline__ void tmem_st16_const(uint32_t addr, uint32_t v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
                 "{%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// The MMAs and commits of an issuing warp. They are issued by one elected lane, but by predicate and not by a branch: inside
// `if (lane == 0)` the compiler takes every operand for a per-thread value and moves it into uniform registers one instruction
// at a time (a 64-column MMA after another: 61 clk in a branch, 32 by predicate, its own time). With that, and the role branches
// on a warp index that the compiler knows to be uniform, Q4_K 11008x4096 x 512 tokens went from 97.6 to 80.9 us. `leader` is
// elect_one(); the other operands are the same in all lanes (tensor-memory addresses that come out of shared memory by way
// of a shuffle).
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(p));
    return p;
}
// D (+)= A x B^T with A in tensor memory (halves)
__device__ __forceinline__ void umma_ts(uint32_t leader, uint32_t d, uint32_t a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
                 "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(db), "r"(idesc), "r"(accumulate), "r"(leader) : "memory");
}
// ... and with A in shared memory
template <bool F16>
__device__ __forceinline__ void umma_ss(uint32_t leader, uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    if (F16)
        asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
                     "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                     ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(leader) : "memory");
    else
        asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
                     "@q tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
                     ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(leader) : "memory");
}
__device__ __forceinline__ void tc_commit_one(uint32_t leader, uint32_t bar) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
                 "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar), "r"(leader) : "memory");
}
// sixteen registers of each lane into sixteen consecutive columns of the warp's 32 lanes
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
                 "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
// one register of each lane into one column of the warp's 32 lanes
__device__ __forceinline__ void tmem_st1(uint32_t addr, uint32_t v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(addr), "r"(v) : "memory");
}
// a compile-time number as an argument
template <int V> struct Int { enum { value = V }; };

// 32 columns of the sixteen lanes at the address: of every eight columns lane l gets columns 2 (l & 3), + 1 of row l / 4 in
// two registers and of row l / 4 + 8 in the next two
__device__ __forceinline__ void tmem_ld_16x256_x4(uint32_t addr, uint32_t (&v)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(addr) : "memory");
}
__device__ __forceinline__ f32x2 lds64_f2(uint32_t addr) {
    f32x2 a;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(a) : "r"(addr));
    return a;
}
__device__ __forceinline__ void sts64_f2(uint32_t addr, f32x2 v) { asm volatile("st.shared.b64 [%0], %1;" ::"r"(addr), "l"(v) : "memory"); }
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Optional self-profile (compile with -DB200Q_TC_PROF): every role adds up the clocks it spends in
// each kind of barrier wait and one block prints them when it ends -- who waits for whom.
#ifdef B200Q_TC_PROF
#define PROF_DECL long long prof_[8] = {0, 0, 0, 0, 0, 0, 0, 0}; const long long prof_t0_ = clock64();
#define WAITP(slot, b, par) ([&]() { const long long t_ = clock64(); const bool r_ = mbar_wait_warp(b, par, abortp); prof_[slot] += clock64() - t_; return r_; }())
#define PROF_DUMP(role) if (lane == 0 && blockIdx.x == 1 && blockIdx.y == (gridDim.y > 1 ? 1 : 0)) printf("%s warp %2d total %lld waits: rawF %lld rawE %lld actF %lld actE %lld aF %lld aE %lld accF %lld accE %lld\n", role, warp, clock64() - prof_t0_, prof_[0], prof_[1], prof_[2], prof_[3], prof_[4], prof_[5], prof_[6], prof_[7]);
#else
#define PROF_DECL
#define WAITP(slot, b, par) mbar_wait_warp(b, par, abortp)
#define PROF_DUMP(role)
#endif
#define WAITP2(slot0, b0, par0, slot1, b1, par1) (mbar_ready_warp(b0, par0, b1, par1) || (WAITP(slot0, b0, par0) && WAITP(slot1, b1, par1)))

}  // namespace tc
}  // namespace b200q

// Inline-PTX wrappers for the sm_100a features the joint-attention kernels use:
// mbarrier, TMA tiled loads (plain cp.async.bulk.tensor into the issuing CTA only),
// tensor memory (TMEM) allocation and access, and tcgen05 MMA issue/commit.
//
// Every wait on an mbarrier is bounded: on expiry the caller gets `false`, records
// an error and leaves the kernel through its normal exit (TMEM is freed there).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace f2k::ptx {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ----------------------------------------------------------------------------
// mbarrier
// ----------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred P;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, P;\n\t"
        "}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// One look, without waiting: is the phase of this parity complete?
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred P;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, P;\n\t"
        "}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// One look at two barriers, both round trips in flight together: are both phases complete?
__device__ __forceinline__ bool mbar_test2(uint32_t bar_a, uint32_t parity_a, uint32_t bar_b, uint32_t parity_b) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred P, Q;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 Q, [%3], %4;\n\t"
        "and.pred P, P, Q;\n\t"
        "selp.u32 %0, 1, 0, P;\n\t"
        "}\n"
        : "=r"(ok)
        : "r"(bar_a), "r"(parity_a), "r"(bar_b), "r"(parity_b)
        : "memory");
    return ok != 0;
}

// Bounded wait. `abort_flag` is a CTA-shared word any role sets when it gives up;
// it is polled so that one expired wait releases every other waiter quickly.
// Returns false when the limit ran out or the CTA is aborting. The limit is kept on the
// SM cycle counter and only looked at every 256 polls: the fast path is nothing but
// try_wait (reading a timer on every miss would sit on the critical path of every
// hand-over between the roles).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity,
                                          volatile uint32_t* abort_flag, long long limit_cycles) {
    long long t0 = 0;
    for (uint32_t spins = 1;; ++spins) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((spins & 255u) == 0u) {
            if (*abort_flag != 0u) return false;
            const long long now = clock64();
            if (t0 == 0) {
                t0 = now;
            } else if (now - t0 > limit_cycles) {
                *abort_flag = 1u;
                return false;
            }
        }
    }
}

// Bounded wait on a word in global memory that someone else - a copy engine, a stream memory
// operation, a kernel on another GPU - sets to `value` (or to the value of a later call: the
// comparison is "not before", modulo 2^32). Same contract as mbar_wait.
__device__ __forceinline__ bool global_flag_wait(const unsigned int* flag, unsigned int value,
                                                 volatile uint32_t* abort_flag, long long limit_cycles) {
    long long t0 = 0;
    for (uint32_t spins = 1;; ++spins) {
        unsigned int v;
        asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
        if ((int)(v - value) >= 0) return true;
        if ((spins & 63u) == 0u) {
            if (*abort_flag != 0u) return false;
            const long long now = clock64();
            if (t0 == 0) {
                t0 = now;
            } else if (now - t0 > limit_cycles) {
                *abort_flag = 1u;
                return false;
            }
        }
        __nanosleep(200);
    }
}

// Store with release semantics at system scope: everything this thread has observed or written
// (and fenced) before it is visible to whoever acquires the word, on this GPU or another.
__device__ __forceinline__ void st_release_sys(unsigned int* p, unsigned int v) {
    asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Called by one thread of every CTA after a CTA-wide barrier that follows the CTA's last global
// store: the last CTA of the grid to arrive publishes `value` to the `n` words flags[]. When
// `failed` (a status word some CTA of this launch may have set before it arrived here) is not
// zero, `value` goes to fail_flags[] first. The counter (zero before the launch) is zero again
// afterwards.
__device__ __forceinline__ void grid_done_publish(unsigned int* counter, unsigned int n_ctas,
                                                  unsigned int* const* flags, unsigned int* const* fail_flags,
                                                  int n, unsigned int value, const int* failed) {
    __threadfence_system();
    const unsigned int seen = atomicAdd(counter, 1u);
    if (seen == n_ctas - 1u) {
        atomicExch(counter, 0u);
        __threadfence_system();
        if (failed != nullptr && *reinterpret_cast<const volatile int*>(failed) != 0) {
            for (int i = 0; i < n; ++i)
                if (fail_flags[i] != nullptr) st_release_sys(fail_flags[i], value);
            __threadfence_system();
        }
        for (int i = 0; i < n; ++i) st_release_sys(flags[i], value);
    }
}

// Programmatic dependent launch: until every kernel this launch depends on has completed and its writes
// are visible (at once in a launch without the attribute).
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ----------------------------------------------------------------------------
// TMA (tiled, 4-D, global -> shared, completion on an mbarrier). One destination CTA.
// ----------------------------------------------------------------------------
__device__ __forceinline__ void tma_load_4d(uint32_t dst_smem, const void* tmap, uint32_t bar,
                                            int c0, int c1, int c2, int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(dst_smem), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar),
          "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}

// 16-byte accesses to shared memory by shared-space address.
__device__ __forceinline__ void st_shared_v4(uint32_t addr, const uint4& v) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}

// Untiled bulk copies (no multicast): global -> this CTA's shared memory with completion on an
// mbarrier, and shared -> global (this GPU's memory or a peer's) tracked by the issuing thread's
// bulk groups. Addresses 16-byte aligned, sizes multiples of 16 bytes.
__device__ __forceinline__ void bulk_load(uint32_t dst_smem, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst_smem), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void bulk_store(void* dst, uint32_t src_smem, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                 ::"l"(dst), "r"(src_smem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// until at most kPending of this thread's bulk groups still have to READ their shared-memory source
template <int kPending>
__device__ __forceinline__ void bulk_wait_read() {
    asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(kPending) : "memory");
}
// until at most kPending of this thread's bulk groups are incomplete (their writes performed)
template <int kPending>
__device__ __forceinline__ void bulk_wait() {
    asm volatile("cp.async.bulk.wait_group %0;" ::"n"(kPending) : "memory");
}
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }

// ----------------------------------------------------------------------------
// Tensor memory
// ----------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(dst_smem), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tc_fence_before_sync() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after_sync() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tmem_wait_ld() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_wait_st() {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// 32 lanes x 32-bit, 32 consecutive columns: thread i of the warp receives columns
// [col, col+32) of TMEM lane (lane_base + i).
__device__ __forceinline__ void tmem_ld_x32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
          "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
          "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st_x32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
          "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
          "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
          "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
          "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st_x16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
          "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
          "r"(r[14]), "r"(r[15])
        : "memory");
}

// ----------------------------------------------------------------------------
// tcgen05 MMA (kind::f16: bf16 x bf16 -> fp32 in TMEM), one issuing thread
// ----------------------------------------------------------------------------
// Shared-memory matrix descriptor, 128-byte swizzle. Fields (bits):
//   [0,14)  start address >> 4        [16,30) leading-dimension byte offset >> 4
//   [32,46) stride-dimension byte offset >> 4      [46,48) descriptor version = 1
//   [61,64) layout type, 2 = SWIZZLE_128B
__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t smem_addr, uint32_t lbo_bytes,
                                                   uint32_t sbo_bytes) {
    const uint32_t lo = ((smem_addr & 0x3FFFFu) >> 4) | ((lbo_bytes >> 4) << 16);
    const uint32_t hi = (sbo_bytes >> 4) | (1u << 14) | (2u << 29);
    return (static_cast<uint64_t>(hi) << 32) | lo;
}

// Instruction descriptor for kind::f16 with bf16 operands and fp32 accumulation.
//   [4,6) D format (1 = f32)   [7,10) A format (1 = bf16)   [10,13) B format (1 = bf16)
//   [15] A major (0 = K)       [16] B major (0 = K, 1 = MN)
//   [17,23) N >> 3             [24,29) M >> 4
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int m, int n, bool b_mn_major) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn_major ? 1u : 0u) << 16) |
           (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

// The issuing warp runs converged and every operand is warp-uniform; one elected lane issues.
// (A divergent single-lane branch would force the operands out of the uniform datapath and cost
// tens of cycles per MMA on a warp that shares its scheduler with the softmax warps.)

// D[tmem] = A[smem] * B[smem] over 8 k-steps of 16 elements: descriptors advance by 2 (32 bytes) inside
// a 128-byte swizzled row of 64 elements, and by 1024 (16 KiB) to the second box of 64.
__device__ __forceinline__ void umma_ss_x8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc) {
    asm volatile(
        "{\n\t"
        ".reg .pred pe, fresh, more;\n\t"
        ".reg .b64 a, b;\n\t"
        "elect.sync _|pe, 0xffffffff;\n\t"
        "setp.ne.b32 fresh, 0, 0;\n\t"
        "setp.eq.b32 more, 0, 0;\n\t"
        "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, fresh;\n\t"
        "add.s64 a, %1, 2;\n\t"
        "add.s64 b, %2, 2;\n\t"
        "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, more;\n\t"
        "add.s64 a, %1, 4;\n\t"
        "add.s64 b, %2, 4;\n\t"
        "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, more;\n\t"
        "add.s64 a, %1, 6;\n\t"
        "add.s64 b, %2, 6;\n\t"
        "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, more;\n\t"
        "add.s64 a, %1, 1024;\n\t"
        "add.s64 b, %2, 1024;\n\t"
        "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, more;\n\t"
        "add.s64 a, %1, 1026;\n\t"
        "add.s64 b, %2, 1026;\n\t"
        "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, more;\n\t"
        "add.s64 a, %1, 1028;\n\t"
        "add.s64 b, %2, 1028;\n\t"
        "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, more;\n\t"
        "add.s64 a, %1, 1030;\n\t"
        "add.s64 b, %2, 1030;\n\t"
        "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, more;\n\t"
        "}\n"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc)
        : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem] over 4 k-steps of 16: 8 columns of A and 2048 bytes of B each.
__device__ __forceinline__ void umma_ts_x4(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                           uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred pe, p, more;\n\t"
        ".reg .b32 a;\n\t"
        ".reg .b64 b;\n\t"
        "elect.sync _|pe, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.eq.b32 more, 0, 0;\n\t"
        "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "add.s32 a, %1, 8;\n\t"
        "add.s64 b, %2, 128;\n\t"
        "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, more;\n\t"
        "add.s32 a, %1, 16;\n\t"
        "add.s64 b, %2, 256;\n\t"
        "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, more;\n\t"
        "add.s32 a, %1, 24;\n\t"
        "add.s64 b, %2, 384;\n\t"
        "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, more;\n\t"
        "}\n"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrive (count 1) on `bar` once every tcgen05 operation the elected lane issued before the
// commit has completed. elect.sync picks the same lane every time for a full warp, so the
// commit tracks the MMAs issued through umma_ss_x8 / umma_ts_x4.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile(
        "{\n\t"
        ".reg .pred pe;\n\t"
        "elect.sync _|pe, 0xffffffff;\n\t"
        "@pe tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t"
        "}\n"
        ::"r"(bar) : "memory");
}

// ----------------------------------------------------------------------------
// Register budget: a warpgroup (4 consecutive warps) raises or lowers its per-thread
// register count; the total over the CTA must stay within what it was launched with.
// ----------------------------------------------------------------------------
template <int kRegs>
__device__ __forceinline__ void setmaxnreg_inc() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegs));
}
template <int kRegs>
__device__ __forceinline__ void setmaxnreg_dec() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegs));
}

// ----------------------------------------------------------------------------
// Small math helpers
// ----------------------------------------------------------------------------
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// Packed fp32 pairs: (d0, d1) = (a0, a1) * (b0, b1) + (c0, c1) in one instruction.
__device__ __forceinline__ void fma2(float& d0, float& d1, float a0, float a1, float b0, float b1,
                                     float c0, float c1) {
    asm("{\n\t"
        ".reg .b64 ra, rb, rc, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\t"
        "mov.b64 rb, {%4, %5};\n\t"
        "mov.b64 rc, {%6, %7};\n\t"
        "fma.rn.f32x2 rd, ra, rb, rc;\n\t"
        "mov.b64 {%0, %1}, rd;\n\t"
        "}\n"
        : "=f"(d0), "=f"(d1)
        : "f"(a0), "f"(a1), "f"(b0), "f"(b1), "f"(c0), "f"(c1));
}
__device__ __forceinline__ void add2(float& d0, float& d1, float a0, float a1, float b0, float b1) {
    asm("{\n\t"
        ".reg .b64 ra, rb, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\t"
        "mov.b64 rb, {%4, %5};\n\t"
        "add.rn.f32x2 rd, ra, rb;\n\t"
        "mov.b64 {%0, %1}, rd;\n\t"
        "}\n"
        : "=f"(d0), "=f"(d1)
        : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Two fp32 -> packed bf16x2 (round to nearest even); `lo` lands in bits [0,16).
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

}  // namespace f2k::ptx

// Inline-PTX wrappers shared by the tensor-core kernels: mbarrier, TMA (cp.async.bulk.tensor),
// tcgen05 MMA / commit / TMEM loads, shared-memory matrix descriptors.  sm_100a only.
#pragma once
#include <cuda.h>
#include <stdint.h>

#include "common.h"

namespace dnb {

// Default bound of every device-side wait, in SM clock cycles (about one second).  The bound travels in the
// kernels' argument blocks, so a caller (or a test) can shorten it for one plan.
constexpr long long WAIT_LIMIT_CYCLES = 2000000000LL;

// ------------------------------------------------------------------ PTX wrappers
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity)
{
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    return done;
}

// Bounded wait by ONE polling lane per warp; the result is broadcast to the warp.  Returns false when
// the wait expired or another role aborted.  Polling goes through shared memory, which the tensor
// cores read their operands from: one lane per warp polls, with a hardware suspend hint, and waiters
// that are not latency-critical back off with nanosleep between polls.
__device__ __forceinline__ uint32_t mbar_try_wait_hint(uint32_t bar, uint32_t parity, uint32_t hint_ns)
{
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(bar), "r"(parity), "r"(hint_ns) : "memory");
    return done;
}

// Bounded wait for a loop that a whole warp runs in step (the TMA and MMA roles): every lane polls, the vote makes the
// outcome, and with it the loop's control flow and all its counters, uniform in the compiler's eyes.  Such a loop keeps
// its addresses, coordinates and descriptors in uniform registers, where the TMA and MMA instructions want them; with one
// lane running the loop alone each of them was moved there operand by operand (an iteration of the MMA role then took
// 680-860 clocks, of the TMA role 460-520, whatever the tensor pipe and the memory could do).
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int *abort_flag, int *status, int code,
                                               long long limit = WAIT_LIMIT_CYCLES)
{
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    const long long t0 = clock64();
    int spins = 0;
    while (!__all_sync(0xffffffffu, mbar_try_wait_hint(bar, parity, 1000u))) {
        if ((++spins & 0x3f) == 0) {
            if (__any_sync(0xffffffffu, *abort_flag != 0)) return false;
            if (__any_sync(0xffffffffu, clock64() - t0 > limit)) {
                if ((threadIdx.x & 31) == 0) {
                    *abort_flag = 1;
                    atomicCAS(status, 0, code);
                }
                return false;
            }
        }
    }
    return true;
}
// One lane of a converged warp, the same one every time.
__device__ __forceinline__ bool elect_one()
{
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag, int *status, int code,
                                          unsigned backoff_ns = 0, long long limit = WAIT_LIMIT_CYCLES)
{
    int ok = 1;
    if ((threadIdx.x & 31) == 0) {
        if (!mbar_try_wait(bar, parity)) {
            const long long t0 = clock64();
            int spins = 0;
            while (!mbar_try_wait_hint(bar, parity, 2000u)) {
                if (backoff_ns) __nanosleep(backoff_ns);
                if ((++spins & 0x3f) == 0) {
                    if (*abort_flag) { ok = 0; break; }
                    if (clock64() - t0 > limit) {
                        *abort_flag = 1;
                        atomicCAS(status, 0, code);
                        ok = 0;
                        break;
                    }
                }
            }
        }
    }
    ok = __shfl_sync(0xffffffffu, ok, 0);
    return ok != 0;
}

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0, int c1, int c2, int c3)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0, int c1, int c2)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}

// Shared-memory matrix descriptor, K-major operand whose rows are `row_bytes`
// long and equal to the swizzle span; 8-row groups are 8*row_bytes apart.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t addr, int row_bytes)
{
    const uint64_t layout = row_bytes == 128 ? 2 : (row_bytes == 64 ? 4 : 6);  // SWIZZLE_128B / 64B / 32B
    uint64_t d = (uint64_t)((addr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;                                  // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)((8 * row_bytes) >> 4) << 32;             // stride byte offset between 8-row groups
    d |= (uint64_t)1 << 46;                                  // descriptor version for sm_100
    d |= layout << 61;
    return d;
}

// The operand kind is a template parameter on purpose: with a run-time `if` the compiler predicates ALL the
// tcgen05.mma instructions, and the predicated-off ones still occupy the tensor pipe's issue path.
// KIND: 0 kind::tf32 (f32 operands), 1 kind::f16 (bf16 operands), 2 kind::i8 (int8 operands, int32 accumulators).
enum { MMA_TF32 = 0, MMA_BF16 = 1, MMA_I8 = 2 };
template <int KIND>
__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate)
{
    if (KIND == MMA_BF16) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
    } else if (KIND == MMA_I8) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
    }
}
// Instruction descriptor of a dense K-major x K-major MMA of m rows and n columns: accumulator format (bits 4-5: f32,
// or s32 for int8), operand formats (bits 7-9 and 10-12: tf32 = 2, bf16 = 1, signed int8 = 1), n / 8 from bit 17, m / 16 from bit 24.
template <int KIND>
__device__ __forceinline__ uint32_t mma_idesc(uint32_t m, uint32_t n)
{
    const uint32_t cfmt = KIND == MMA_I8 ? 2u : 1u, fmt = KIND == MMA_TF32 ? 2u : 1u;
    return (cfmt << 4) | (fmt << 7) | (fmt << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}
__device__ __forceinline__ void umma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// ------------------------------------------------------------------ programmatic dependent launch
// A kernel launched with the programmatic-stream-serialization attribute may start while the kernel before it in the
// stream is still draining: its CTAs take SMs as they free up and run their set-up (barriers, TMEM, tensor-map
// fetch); grid_dependency_wait() then holds them until the previous kernel has finished and its writes are visible.
// Nothing a previous kernel wrote may be read, and nothing it may still read may be written, before that wait.
// launch_dependents() lets the kernel after this one be scheduled the same way.  Both are no-ops in a plain launch.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// ... from a kernel of many short blocks: where it fills the GPU, early successors would only take room from its own blocks.
__device__ __forceinline__ void launch_dependents_if_small()
{
    if ((unsigned long long)gridDim.x * gridDim.y * gridDim.z <= (unsigned long long)EARLY_BLOCKS) launch_dependents();
}

// ------------------------------------------------------------------ CTA pairs (cta_group::2)
// Two CTAs of a cluster of two run one MMA of 256 rows: each holds 128 rows of A and half of B's columns in its own
// shared memory and its 128 rows of the accumulator in its own TMEM; the even CTA (cluster rank 0) issues the MMAs.
// Shared-memory addresses of a CTA in a cluster carry its rank from bit 24 up; clearing that bit names the same
// offset in the even CTA.  No load here is shared between CTAs: each CTA loads its own operands.
constexpr uint32_t PAIR_LEADER_MASK = 0xFEFFFFFFu;

__device__ __forceinline__ uint32_t cluster_ctarank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// All threads of every CTA of the cluster (release / acquire: barrier initialisations before it are visible after it).
__device__ __forceinline__ void cluster_sync_all()
{
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
// The same barrier in the even CTA of the pair, as a shared::cluster address.
__device__ __forceinline__ uint32_t leader_bar(uint32_t bar) { return bar & PAIR_LEADER_MASK; }
__device__ __forceinline__ void mbar_arrive_leader(uint32_t bar)
{
    asm volatile(
        "{\n\t.reg .b32 rem;\n\t"
        "mapa.shared::cluster.u32 rem, %0, 0;\n\t"
        "mbarrier.arrive.shared::cluster.b64 _, [rem];\n\t}"
        ::"r"(bar) : "memory");
}
// Loads of a CTA pair: the data lands in the executing CTA's shared memory, the bytes are counted on the even CTA's barrier.
__device__ __forceinline__ void tma_load_4d_pair(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0, int c1, int c2, int c3)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(dst), "l"(map), "r"(leader_bar(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0, int c1, int c2)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(map), "r"(leader_bar(bar)), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
// `rows` consecutive pixels of the map's bounding box (w innermost, then h, then images) from (x, y, image) on, as the map was made
__device__ __forceinline__ void tma_load_im2col_4d_pair(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c, int x, int y, int image)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.im2col.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2], {%7, %8};"
        ::"r"(dst), "l"(map), "r"(leader_bar(bar)), "r"(c), "r"(x), "r"(y), "r"(image), "h"((uint16_t)0), "h"((uint16_t)0) : "memory");
}
template <int KIND>
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate)
{
    if (KIND == MMA_BF16) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
    } else if (KIND == MMA_I8) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
    }
}
// Arrives on the barrier at this offset in BOTH CTAs of the pair once the MMAs issued so far have retired (an
// mbarrier arrive, not a load: the only cluster-wide signal in the kernel).
__device__ __forceinline__ void umma_commit_pair(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// TMA store of one staged output chunk (shared -> global), bulk-group completion.
__device__ __forceinline__ void tma_store_4d(const CUtensorMap *map, uint32_t src, int c0, int c1, int c2, int c3)
{
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
                 ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap *map, uint32_t src, int c0, int c1)
{
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
                 ::"l"(map), "r"(src), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_read0() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_read1() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// 16 bytes from global to shared memory, or 16 zero bytes; completes in groups
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool in)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// a whole 32-byte sector, 32-byte aligned
__device__ __forceinline__ void st_global_32(void *dst, const uint32_t (&v)[8])
{
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"l"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
// asks for `bytes` (a multiple of 16) at a 16-byte aligned address to be brought into L2
__device__ __forceinline__ void prefetch_l2(const void *src, uint32_t bytes)
{
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}
// barrier among the 128 epilogue threads only (barrier 0 is __syncthreads)
__device__ __forceinline__ void epilogue_bar() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

}  // namespace dnb

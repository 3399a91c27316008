// Building blocks shared by the tensor-core kernels: mbarrier, TMA and tcgen05 wrappers, the shared-memory operand
// descriptor of a K-major tile of 128-byte rows (64 values of 16 bits) with 128-byte swizzle, and the host-side tensor-map encoder.
#pragma once
#include <cuda.h>

#include <type_traits>

#include "g2d_common.cuh"

namespace g2d {

constexpr int MT = 128;                    // macro tile edge
constexpr int KC = 32;                     // floats per 128-byte swizzle row
constexpr int STAGES = 3;
constexpr int TC_THREADS = 192;
constexpr long long WAIT_CYCLES = 2000000000LL;  // about a second

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// false on time-out.  Between polls the warp sleeps for `nap` nanoseconds: several CTAs of an update kernel share an SM, and the
// warps that work should not lose issue slots to those that wait.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, unsigned nap = 32, long long limit = WAIT_CYCLES) {
    const long long start = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - start > limit) return false;
        __nanosleep(nap);
    }
    return true;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// K-major operand tile of 128-byte rows, 128-byte swizzle: 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3FFF);   // start address
    d |= (uint64_t)1 << 16;                       // leading byte offset (unused with swizzle)
    d |= (uint64_t)(1024 >> 4) << 32;             // stride byte offset
    d |= (uint64_t)1 << 46;                       // descriptor version
    d |= (uint64_t)2 << 61;                       // SWIZZLE_128B
    return d;
}
// 32 consecutive accumulator columns of this warp's 32 tensor-memory lanes (one row per thread)
__device__ __forceinline__ void tmem_load_32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_load_16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ---- 16-bit operands: K-major tiles of 64 values = 128 bytes per row, the same swizzle and descriptor as above ----
constexpr int KH = 64;                     // k per chunk
constexpr int HTILE_BYTES = MT * KH * 2;   // 16 KB: 128 rows
// D fp32, A and B 16 bits (format 0: fp16, 1: bf16), both K-major, M = 128, N = nt
__host__ __device__ constexpr uint32_t idesc_16(int nt, uint32_t format, int mt = MT) {
    return (1u << 4) | (format << 7) | (format << 10) | ((uint32_t)(nt >> 3) << 17) | ((uint32_t)(mt >> 4) << 24);
}
__device__ __forceinline__ void umma_16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// ---- shared state of a CTA of TC_THREADS threads: warp 0 loads, warp 1 issues the MMAs, warps 2-5 read the accumulators ----
struct TcRing {
    uint64_t full[STAGES], empty[STAGES], accum;
    uint32_t tmem_slot;
    int failed;
};

// ---- two CTAs of a cluster on one product (cta_group::2): M = N = 256, 128 rows of A and of B in each CTA, so that a CTA fills shared memory with 256
// rows for its 128 x 256 of the product, where one on its own fills it with 384.  CTA 0 leads: it issues the MMAs for both. ----
__device__ __forceinline__ uint32_t leaders(uint64_t *bar) {  // the same barrier of CTA 0
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(bar)));
    return r;
}
__device__ __forceinline__ void mbar_arrive_at(uint32_t bar) { asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory"); }
// as mbar_wait, for what a thread of the other CTA may have arrived at
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t *bar, uint32_t parity, unsigned nap = 32, long long limit = WAIT_CYCLES) {
    const long long start = clock64();
    for (;;) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
        if (clock64() - start > limit) return false;
        __nanosleep(nap);
    }
}
// into this CTA's shared memory, counted at a barrier of either CTA
__device__ __forceinline__ void tma_load_2d_duo(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void umma_16_duo(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit_duo(uint64_t *bar) {  // arrives at the barrier of both CTAs
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}

// For one CTA or two
template <bool DUO>
__device__ __forceinline__ void mma(uint32_t tmem_d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t accumulate) {
    if (DUO) umma_16_duo(tmem_d, umma_desc(a), umma_desc(b), idesc, accumulate);
    else umma_16(tmem_d, umma_desc(a), umma_desc(b), idesc, accumulate);
}
template <bool DUO>
__device__ __forceinline__ void commit(uint64_t *bar) {
    if (DUO) umma_commit_duo(bar);
    else umma_commit(bar);
}
template <bool DUO>
__device__ __forceinline__ void tmem_alloc(uint32_t *slot, uint32_t cols) {  // one warp (of each CTA)
    if (DUO) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
}
template <bool DUO>
__device__ __forceinline__ void tmem_free(uint32_t tmem, uint32_t cols) {
    if (DUO) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
}
// One thread, after a time-out in a pair of CTAs: a load of this CTA may count at a barrier that nobody awaits any more, and a commit be on its way
// to the other CTA.  They land within microseconds; a millisecond on, the shared memory may be given back.
__device__ __forceinline__ void let_it_land() {
    const long long start = clock64();
    while (clock64() - start < WAIT_CYCLES / 1000) __nanosleep(1000);
}
// a launch of clusters of two CTAs along x, counted here
template <typename Job>
inline int launch_duo(void (*kernel)(Job), dim3 grid, int threads, size_t smem, cudaStream_t stream, const Job &job) {
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = dim3((unsigned)threads);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeClusterDimension;
    attribute.val.clusterDim.x = 2;
    attribute.val.clusterDim.y = attribute.val.clusterDim.z = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, job) == cudaSuccess ? check_launch() : G2D_ERR_CUDA;
}

// All threads: barriers, tensor-memory allocation of `cols` columns (by warp 1); returns the accumulator's address.
__device__ __forceinline__ uint32_t tc_ring_setup(TcRing &ring, uint32_t cols) {
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&ring.full[s], 1);
            mbar_init(&ring.empty[s], 1);
        }
        mbar_init(&ring.accum, 1);
        ring.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if ((threadIdx.x >> 5) == 1) tmem_alloc<false>(&ring.tmem_slot, cols);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return ring.tmem_slot;
}

// All threads: release tensor memory; returns whether a wait ran out (meaningful in every thread).
__device__ __forceinline__ bool tc_ring_teardown(TcRing &ring, uint32_t tmem, uint32_t cols) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if ((threadIdx.x >> 5) == 1) {
        if (ring.failed) {
            // give outstanding loads and MMAs a bounded chance to land before the memory they target is released
            if ((threadIdx.x & 31) == 0) mbar_wait(&ring.accum, 0);
            __syncwarp();
        }
    }
    if ((threadIdx.x >> 5) == 1) tmem_free<false>(tmem, cols);
    return ring.failed != 0;
}

// ---- results as reductions of 32 x 32 boxes ----
// A warp that holds one row per lane writes its box to shared memory (128-byte rows, the TMA's swizzle: no bank conflicts) and
// one reduction adds it to global memory.  The same additions as red.global.add.v4 from every lane touch 32 rows with every
// instruction and half a sector each.
constexpr int BOX_BYTES = 32 * 32 * 4;
__device__ __forceinline__ void box_store4(uint32_t box, int row, int group, float a, float b, float c, float d) {  // columns 4 group ..
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(box + row * 128 + ((group ^ (row & 7)) << 4)), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ void box_store1(uint32_t box, int row, int column, float v) {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(box + row * 128 + (((column >> 2) ^ (row & 7)) << 4) + (column & 3) * 4), "f"(v) : "memory");
}
__device__ __forceinline__ void box_reduce_add(const CUtensorMap *map, uint32_t box, int x, int y) {  // one lane, after fence and __syncwarp
    asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2}], [%3];"
                 ::"l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(box)
                 : "memory");
}
__device__ __forceinline__ void box_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void box_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// A 32 x 32 block of results through two boxes of 16 rows (4 KB of shared memory in turn): one is filled while the TMA still reads
// the other.  With one box of 32 rows the warp waited for it every time, and the eight warps took 6000 cycles for the results of a
// 128 x 256 tile, twice what the two accumulators of the pipeline hide (factors of 28672 and 8192: 97.1 -> 94.3 ms, the far updates of
// 8192 x 28672 alone: 28.9 -> 27.7 ms).
// v: the 32 values of the lane's row or, TRANSPOSED, of its column.
constexpr int HALF_BOX_ROWS = 16, HALF_BOX_BYTES = HALF_BOX_ROWS * 128;
__device__ __forceinline__ void half_box_free() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }  // all but the latest
template <bool TRANSPOSED>
__device__ __forceinline__ void add_block(const CUtensorMap *map, uint32_t box, int lane, const float *v, float factor, int x, int y, bool inside, int rows) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t half = box + h * HALF_BOX_BYTES;
        if (lane == 0) half_box_free();
        __syncwarp();
        if (TRANSPOSED) {
#pragma unroll
            for (int r = 0; r < HALF_BOX_ROWS; ++r) box_store1(half, r, lane, factor * v[h * HALF_BOX_ROWS + r]);
        } else if ((lane >> 4) == h) {
#pragma unroll
            for (int g = 0; g < 8; ++g) box_store4(half, lane & 15, g, factor * v[4 * g], factor * v[4 * g + 1], factor * v[4 * g + 2], factor * v[4 * g + 3]);
        }
        box_fence();
        __syncwarp();
        if (lane == 0) {
            if (inside && y + h * HALF_BOX_ROWS < rows) box_reduce_add(map, half, x, y + h * HALF_BOX_ROWS);
            box_commit();  // a group per half, reduced or not: half_box_free counts them
        }
    }
}
__device__ __forceinline__ void box_wait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// ---- pipeline for 16-bit pairs: A[128 x k] B[NT x k]^T as hi hi + lo hi + hi lo ----
// CTA of PAIR_THREADS threads: warp 0 loads, warp 1 issues the MMAs, eight warps read the accumulators.  The k range is cut into
// slices of SLICE chunks with two accumulators in turn: the tensor cores add into their fp32 accumulator with truncation, which
// biases long sums, so a slice is accumulated in tensor memory and the slices are added up in registers, round to nearest,
// under the MMAs of the next.  A reading warp has 32 rows (q = warp % 4) and half of the columns.
constexpr int PAIR_THREADS = 320;
template <int NT>
constexpr int pair_stage_bytes = 2 * HTILE_BYTES + 2 * NT * KH * 2;
constexpr int PAIR_BOXES = 8 * BOX_BYTES;  // one per reading warp, where the results leave as boxes
template <int NSTAGE>
struct PairRing {
    uint64_t full[NSTAGE], empty[NSTAGE], acc_full[2], acc_empty[2];
    uint64_t drained;  // after a time-out: every MMA that was issued has completed
    uint32_t tmem;
    int failed;
};

// A CTA takes several tiles, one after the other, so that a tile's loads and MMAs run while the results of the one before leave.
// next(number, tile): the CTA's tile of that number, false past the last.  load(tile, chunk, destination, barrier): A_hi, A_lo,
// B_hi, B_lo tiles one after the other.  finish(tile, q, lane, first column, totals, 4 KB of shared memory of the warp's own
// behind the stages).  DUO: by two CTAs of a cluster whose tiles differ in i0 only; load brings half of B's rows and counts at the barrier
// of CTA 0.  scale(tile, slice, q, column), optional: what a slice's sums are multiplied by, the same for 64 columns.
// Returns whether a wait ran out (of `limit` cycles; those that only let what is in flight come to its end have the usual limit).
struct PairTile {
    int i0, j0, chunks;
    int k0 = 0, which = 0;  // first k and a number of the caller's
};
struct PairNoScale {};
template <int NT, int NSTAGE, int SLICE, bool DUO = false, typename Next, typename Load, typename Finish, typename Scale = PairNoScale>
__device__ __forceinline__ bool pair_gemm(PairRing<NSTAGE> &ring, uint32_t smem_base, Next next, Load load, Finish finish, Scale scale = Scale(), long long limit = WAIT_CYCLES) {
    constexpr bool SCALED = !std::is_same<Scale, PairNoScale>::value;
    constexpr int B_BYTES = NT * KH * 2 / (DUO ? 2 : 1), STAGE = 2 * HTILE_BYTES + 2 * B_BYTES, MINE = NT / 2;
    constexpr uint32_t COLS = 2 * NT, DESC = idesc_16(NT, 0, DUO ? 2 * MT : MT);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = DUO ? (int)cluster_rank() : 0;
    const auto await = [](uint64_t *bar, uint32_t parity, unsigned nap, long long cycles) { return DUO ? mbar_wait_cluster(bar, parity, nap, cycles) : mbar_wait(bar, parity, nap, cycles); };
    const auto wait = [&](uint64_t *bar, uint32_t parity, unsigned nap = 32) { return await(bar, parity, nap, limit); };
    if (threadIdx.x == 0) {
        for (int s = 0; s < NSTAGE; ++s) {
            mbar_init(&ring.full[s], 1);
            mbar_init(&ring.empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&ring.acc_full[s], 1);
            mbar_init(&ring.acc_empty[s], DUO ? 16 : 8);  // one arrival per reading warp, of both CTAs at the leader's
        }
        mbar_init(&ring.drained, 1);
        ring.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc<DUO>(&ring.tmem, COLS);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (DUO) {
        __syncwarp();
        cluster_sync();
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = ring.tmem;
    // the roles count chunks and slices over all tiles of the CTA: stages and accumulators are used in turn throughout
    if (warp == 0) {
        if (lane == 0) {
            PairTile tile;
            int c = 0;
            for (int it = 0; !ring.failed && next(it, tile); ++it) {
                for (int ch = 0; ch < tile.chunks; ++ch, ++c) {
                    const int stage = c % NSTAGE, round = c / NSTAGE;
                    if (round > 0 && !wait(&ring.empty[stage], (round - 1) & 1)) { ring.failed = 1; break; }
                    // DUO: both CTAs' bytes count at the leader's barrier (they may do so before it expects them: the phase waits for its arrival)
                    if (rank == 0) mbar_expect_tx(&ring.full[stage], DUO ? 2 * STAGE : STAGE);
                    load(tile, ch, smem_base + stage * STAGE, &ring.full[stage]);
                }
            }
            // the last loads (DUO: both CTAs') have landed, or had their time to, before their shared memory is given back, whatever became of the MMAs
            if (rank == 0)
                for (int k = max(c - NSTAGE, 0); k < c; ++k) await(&ring.full[k % NSTAGE], (k / NSTAGE) & 1, 32, WAIT_CYCLES);
            if (DUO && !ring.failed) {
                // the leader's commits arrive here as well: none may be under way when this CTA ends (those of the accumulators are awaited below)
                for (int k = max(c - NSTAGE, 0); k < c; ++k)
                    if (!wait(&ring.empty[k % NSTAGE], (k / NSTAGE) & 1)) ring.failed = 1;
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            PairTile tile;
            int c = 0, slice = 0;
            for (int it = 0; !ring.failed && next(it, tile); ++it) {
                for (int ch = 0; ch < tile.chunks; ++ch, ++c) {
                    const int stage = c % NSTAGE, round = c / NSTAGE, buf = slice & 1;
                    const bool opens = ch % SLICE == 0, closes = ch % SLICE == SLICE - 1 || ch == tile.chunks - 1;
                    // the accumulator must have been read out by the warps of the slice two before
                    if (opens && slice >= 2 && !wait(&ring.acc_empty[buf], ((slice >> 1) - 1) & 1)) { ring.failed = 1; break; }
                    if (!wait(&ring.full[stage], round & 1)) { ring.failed = 1; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t d = tmem + (uint32_t)(buf * NT);
                    const uint32_t a_hi = smem_base + stage * STAGE, a_lo = a_hi + HTILE_BYTES, b_hi = a_hi + 2 * HTILE_BYTES, b_lo = b_hi + B_BYTES;
#pragma unroll
                    for (int ks = 0; ks < KH / 16; ++ks) {
                        const uint32_t off = ks * 32;  // 16 values = 32 bytes along the swizzled row
                        mma<DUO>(d, a_hi + off, b_hi + off, DESC, (opens && ks == 0) ? 0u : 1u);
                        mma<DUO>(d, a_lo + off, b_hi + off, DESC, 1u);
                        mma<DUO>(d, a_hi + off, b_lo + off, DESC, 1u);
                    }
                    commit<DUO>(&ring.empty[stage]);  // arrives when the MMAs above have read the stage
                    if (closes) {
                        commit<DUO>(&ring.acc_full[buf]);  // arrives when the slice is complete in tensor memory
                        ++slice;
                    }
                }
            }
            // every MMA that was issued completes, or has its time to, before what it reads and writes is given back: all of them closed a slice, but for
            // those before a time-out
            if (ring.failed) {
                commit<DUO>(&ring.drained);
                await(&ring.drained, 0, 32, WAIT_CYCLES);
            } else if (slice > 0) {
                await(&ring.acc_full[(slice - 1) & 1], ((slice - 1) >> 1) & 1, 32, WAIT_CYCLES);
            }
        }
    } else {
        const int q = warp & 3, c0 = ((warp - 2) >> 2) * MINE;
        PairTile tile;
        int slice = 0;
        bool go = true;
        for (int it = 0; go && next(it, tile); ++it) {
            const int slices = (tile.chunks + SLICE - 1) / SLICE;
            float total[MINE];
#pragma unroll
            for (int x = 0; x < MINE; ++x) total[x] = 0.f;
            for (int s = 0; s < slices; ++s, ++slice) {
                const int buf = slice & 1;
                float factor[MINE / 64];  // of this slice's columns, on their way while the slice is awaited
                if constexpr (SCALED) {
#pragma unroll
                    for (int g = 0; g < MINE / 64; ++g) factor[g] = scale(tile, s, q, c0 + g * 64);
                }
                const bool ok = wait(&ring.acc_full[buf], (slice >> 1) & 1, 64);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (!ok) ring.failed = 1;
                go = __all_sync(0xffffffffu, ok && !ring.failed);  // warp-uniform: the tensor-memory loads are warp-wide
                if (!go) break;
#pragma unroll
                for (int cb = 0; cb < MINE / 16; ++cb) {  // 16 at a time: 128 totals and 32 more do not fit the 168 registers
                    uint32_t v[16];
                    tmem_load_16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * NT + c0 + cb * 16), v);
#pragma unroll
                    for (int x = 0; x < 16; ++x) {
                        if constexpr (SCALED) total[cb * 16 + x] = fmaf(__uint_as_float(v[x]), factor[cb / 4], total[cb * 16 + x]);
                        else total[cb * 16 + x] += __uint_as_float(v[x]);
                    }
                }
                // this warp has read the accumulator: hand it back to the MMA warp
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    if (DUO) mbar_arrive_at(leaders(&ring.acc_empty[buf]));
                    else mbar_arrive(&ring.acc_empty[buf]);
                }
            }
            if (go) finish(tile, q, lane, c0, total, smem_base + (uint32_t)(NSTAGE * STAGE + (warp - 2) * BOX_BYTES));
        }
        box_wait();  // results that are still on their way out of shared memory
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (DUO) {
        // neither CTA leaves while the other's MMAs may read its shared memory or arrive at its barriers
        if (threadIdx.x == 0 && ring.failed) let_it_land();
        __syncwarp();
        cluster_sync();
    }
    if (warp == 1) tmem_free<DUO>(tmem, COLS);
    return ring.failed != 0;
}

// Tiles of 128 x NT that touch the lower triangle, row by row: row I has I * 128 / NT + 1 of them.
template <int NT>
__host__ __device__ inline int64_t lower_tiles(int64_t rows) {  // of the first `rows` tile rows
    return NT == 256 ? (rows / 2) * (rows / 2 + 1) + (rows % 2) * (rows / 2 + 1) : rows * (rows + 1) / 2;
}
// Tiles of 256 x 256: tile rows 2 a and 2 a + 1 together, a triangle of squares again.
__host__ __device__ inline int64_t duo_tiles(int64_t row_pairs) { return lower_tiles<128>(row_pairs); }
template <int NT>
__device__ __forceinline__ void lower_tile(int64_t lin, int &I, int &J) {
    if (NT == 256) {  // rows 2 a and 2 a + 1 have a + 1 tiles each
        int64_t a = (int64_t)((sqrt(4.0 * (double)lin + 1.0) - 1.0) / 2.0);
        while ((a + 1) * (a + 2) <= lin) ++a;
        while (a * (a + 1) > lin) --a;
        const int64_t rest = lin - a * (a + 1);
        I = (int)(2 * a + rest / (a + 1));
        J = (int)(rest % (a + 1));
    } else {
        int64_t a = (int64_t)((sqrt(8.0 * (double)lin + 1.0) - 1.0) / 2.0);
        while ((a + 1) * (a + 2) / 2 <= lin) ++a;
        while (a * (a + 1) / 2 > lin) --a;
        I = (int)a;
        J = (int)(lin - a * (a + 1) / 2);
    }
}
// Whole waves over the 148 SMs decide.  A 128 x 256 tile takes 1.5 times as long as a 128 x 128 one (80 against 60 % of the tensor rate for
// twice the work); two CTAs take 1.25 times as long for 256 x 256, but such tiles fill a wave less well.  Gram of 8192 samples, in us, with
// 128 x 128, 128 x 256 and 256 x 256: 169, 170, 200 at n = 2048 (1, 1 and 1 waves), 296, 237, 367 at 2944 (2, 1, 2), 410, 403, 373 at 3072
// (3, 2, 2), 550, 433, 408 at 4096 (4, 2, 2), 809, 641, 750 at 5248 (6, 3, 4), 2000, 1690, 1540 at 8192 (15, 8, 8).
enum TileChoice { SQUARE_TILES, WIDE_TILES, DUO_TILES };
inline TileChoice tiles_that_pay(int64_t square, int64_t wide, int64_t duo = 0) {  // duo: 0 where two CTAs do not share a tile
    const int64_t s = 4 * ceil_div(square, (int64_t)148), w = 6 * ceil_div(wide, (int64_t)148), d = 5 * ceil_div(duo, (int64_t)74);
    return duo > 0 && d <= s && d <= w ? DUO_TILES : w <= s ? WIDE_TILES : SQUARE_TILES;
}

// ---- host side: tensor maps ----
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult result;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &result) == cudaSuccess &&
            result == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
    return fn;
}

// row-major fp32 matrix [rows][cols]; boxes of box_rows rows x 32 columns, 128-byte swizzle, zero fill outside
static bool make_map(CUtensorMap *map, const float *base, int64_t rows, int64_t cols, int box_rows = MT, int64_t pitch = 0) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)(pitch ? pitch : cols) * sizeof(float)};
    const cuuint32_t box[2] = {KC, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float *>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// row-major 16-bit matrix [rows][cols] whose rows are `pitch` values apart (0: cols); boxes of box_rows rows x 64 columns
static bool make_map_16(CUtensorMap *map, const void *base, int64_t rows, int64_t cols, int box_rows, bool bf16 = false, int64_t pitch = 0) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)(pitch ? pitch : cols) * 2};
    const cuuint32_t box[2] = {KH, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return fn(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(base), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace g2d

// The near update of the sweep (see g2d_band_tc.cu): what its two kernels share.
#pragma once

#include <type_traits>

#include "g2d_tc.cuh"

namespace g2d {

constexpr int BN = 64;                               // N of the MMA: one tile
constexpr int BB_BYTES = BN * KH * 2;                // 8 KB
constexpr int BAND_BYTES = 2 * HTILE_BYTES + 2 * BB_BYTES;  // A_hi, A_lo, B_hi, B_lo: 48 KB, so several CTAs per SM

struct BandTargetMaps {
    CUtensorMap l_hi, l_lo, ut_hi, ut_lo;  // A operands: boxes of 128 rows
    CUtensorMap et_hi, et_lo, c_hi, c_lo;  // B operands: boxes of 64 rows
    CUtensorMap y, c;                      // planes that receive the right and the down feedback, boxes of 32 x 32
};
struct BandFields {
    const float *l_scale, *c_scale, *e_scale, *u_scale;
    int nI, nJ;                            // tiles per column / per row
    int m, n;
    int s, t0, t1;
    int outer_macro, lag_macro;            // > 0: targets that the far update of the source's macro group reaches are left out
    int *error_flag;
    const float *l, *u, *e, *c_from;       // for the products with wide tiles: the float values
    float *y_to, *c_to;                    // and the targets
    int64_t ldl, ldu, ld;
    // for the ring
    int longest, slots;                    // tiles along the longer side; pairs along the moving index that can hold a target
    const int *wide_count;
};
struct BandJob : BandTargetMaps, BandFields {};

// A job: two neighbouring tiles as targets, and their source tile.
struct BandTarget {
    bool right, valid_a, valid_b;
    int fixed, k_tile, t_a;  // tile column (down) or row (right); tile of the source along k; first target along the moving index
};
// x: tile column (down jobs) or tile row (right jobs), y: pair slot along the target range.  False where nothing is to be done.
__device__ __forceinline__ bool band_target(const BandFields &job, int x, int y, bool right, BandTarget &t) {
    const int fixed_count = right ? job.nI : job.nJ, moving_count = right ? job.nJ : job.nI;
    if (x >= fixed_count) return false;
    const int first = max(job.t0 - x, 0);
    const int pair = (first >> 1) + y;                   // tiles 2 pair, 2 pair + 1 along the moving index
    const int t_a = 2 * pair, t_b = 2 * pair + 1;
    t.valid_a = t_a < moving_count && t_a + x >= job.t0 && t_a + x <= job.t1;
    t.valid_b = t_b < moving_count && t_b + x >= job.t0 && t_b + x <= job.t1;
    if (!t.valid_a && !t.valid_b) return false;
    t.k_tile = job.s - x;                                // it lies before both targets
    if (t.k_tile < 0 || t.k_tile >= moving_count) return false;
    if (job.outer_macro > 0) {
        // both targets lie in one macro tile
        const int w_source = (t.k_tile >> 1) + (x >> 1), w_target = pair + (x >> 1);
        const int reach = (w_source / job.outer_macro + 1) * job.outer_macro + job.lag_macro;  // the far update starts here
        if (w_target >= reach) return false;
    }
    t.right = right;
    t.fixed = x;
    t.t_a = t_a;
    return true;
}
// negative where the source tile is wide
__device__ __forceinline__ float band_source_scale(const BandFields &job, const BandTarget &t) {
    return t.right ? job.c_scale[(int64_t)t.fixed * job.nJ + t.k_tile] : job.e_scale[(int64_t)t.k_tile * job.nJ + t.fixed];
}

// The product with a wide source tile (see TcPlanes), in float32 from the float values, by the whole CTA: 128 (r) x 64 (x) results,
// both operands staged whole where the tensor cores' operands would lie, 4 x 4 results per thread at a time.  Few registers: the
// kernel's other path shares SMs.  The rare path.
constexpr int WIDE_R = 128, WIDE_X = 64;
static_assert((WIDE_R + WIDE_X) * TILE * 4 <= BAND_BYTES, "the float operands fit where the 16-bit ones lie");
__device__ __forceinline__ void wide_product(const BandFields &job, bool right, int a_row, int b_row, int k0, bool valid_a, bool valid_b, float *As) {
    float *const Bs = As + TILE * WIDE_R;  // As[k][r], Bs[k][x]
    const int r_end = right ? job.n : job.m, x_end = right ? job.m : job.n;
    for (int idx = threadIdx.x; idx < TILE * WIDE_R; idx += TC_THREADS) {  // neighbouring threads along the rows of the source
        const int r = right ? idx % WIDE_R : idx / TILE, k = right ? idx / WIDE_R : idx % TILE;
        const int64_t at = a_row + r;
        As[k * WIDE_R + r] = at < r_end ? (right ? job.u[(int64_t)(k0 + k) * job.ldu + at] : job.l[at * job.ldl + k0 + k]) : 0.f;
    }
    for (int idx = threadIdx.x; idx < TILE * WIDE_X; idx += TC_THREADS) {
        const int x = right ? idx / TILE : idx % WIDE_X, k = right ? idx % TILE : idx / WIDE_X;
        const int64_t at = b_row + x;
        Bs[k * WIDE_X + x] = at < x_end ? (right ? job.c_from[at * job.ld + k0 + k] : job.e[(int64_t)(k0 + k) * job.ld + at]) : 0.f;
    }
    __syncthreads();
#pragma unroll 1
    for (int block = threadIdx.x; block < (WIDE_R / 4) * (WIDE_X / 4); block += TC_THREADS) {
        const int r0 = (right ? block % (WIDE_R / 4) : block / (WIDE_X / 4)) * 4, x0 = (right ? block / (WIDE_R / 4) : block % (WIDE_X / 4)) * 4;
        if (!(r0 < TILE ? valid_a : valid_b)) continue;
        float acc[4][4] = {};
#pragma unroll 2
        for (int k = 0; k < TILE; ++k) {
            const float4 p = *reinterpret_cast<const float4 *>(As + k * WIDE_R + r0), q = *reinterpret_cast<const float4 *>(Bs + k * WIDE_X + x0);
            const float pv[4] = {p.x, p.y, p.z, p.w}, qv[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int x = 0; x < 4; ++x) acc[r][x] = fmaf(pv[r], qv[x], acc[r][x]);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int64_t at_r = a_row + r0 + r, at_x = b_row + x0 + x;
                if (at_r >= r_end || at_x >= x_end) continue;
                if (right) job.y_to[at_x * job.ld + at_r] += acc[r][x];
                else job.c_to[at_r * job.ld + at_x] += acc[r][x];
            }
    }
}

// The same by a ring's CTA, which has an SM to itself, THREADS threads and often several such products in a row: latency bound.  So eight
// results by four per thread, operand loads issued sixteen at a time and stored without bank conflicts (the row of k has its groups
// of four in another order), targets read sixteen at a time.  Sums in the same order.  3900 x 4100 with rows of two units, where every
// product is of this kind: 15.1 ms with the form above, 11.3 with this one, 11.8 with the updates on a side stream.
__device__ __forceinline__ int wide_at(int k, int at) { return at ^ ((k & 7) << 2); }  // `at` in the row of k
// SIZE values of each of TILE source indices k from k0 on: the `from` rows of `pitch` values run along k (ROW_K) or along the values
template <int THREADS, int SIZE, bool ROW_K>
__device__ __forceinline__ void wide_stage(float *to, const float *from, int64_t pitch, int64_t first, int64_t end, int k0) {
    constexpr int UN = 16;
    static_assert(TILE * SIZE % (UN * THREADS) == 0, "whole trips");
    for (int base = threadIdx.x; base < TILE * SIZE; base += UN * THREADS) {
        float v[UN];
        int at[UN];
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const int idx = base + u * THREADS;
            // along k: a warp takes eight k of four rows, whole sectors that go to distinct banks
            const int k = ROW_K ? (idx & 7) | (idx >> 2 & 56) : idx / SIZE, r = ROW_K ? (idx >> 3 & 3) | (idx >> 8) << 2 : idx % SIZE;
            at[u] = k * SIZE + wide_at(k, r);
            v[u] = first + r < end ? from[ROW_K ? (first + r) * pitch + k0 + k : (k0 + k) * pitch + first + r] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < UN; ++u) to[at[u]] = v[u];
    }
}
template <int THREADS, bool RIGHT>
__device__ __forceinline__ void wide_product_alone(const BandFields &job, const BandTarget &t, float *As) {
    constexpr int PARTS = WIDE_R / 8;                   // eight rows r, four columns x per thread
    static_assert(THREADS == PARTS * (WIDE_X / 4), "a thread has one block of results");
    float *const Bs = As + TILE * WIDE_R;               // As[k][r], Bs[k][x]
    const int64_t a_row = (int64_t)t.t_a * TILE, b_row = (int64_t)t.fixed * TILE, r_end = RIGHT ? job.n : job.m, x_end = RIGHT ? job.m : job.n;
    const int k0 = t.k_tile * TILE, tid = threadIdx.x;
    wide_stage<THREADS, WIDE_R, !RIGHT>(As, RIGHT ? job.u : job.l, RIGHT ? job.ldu : job.ldl, a_row, r_end, k0);
    wide_stage<THREADS, WIDE_X, RIGHT>(Bs, RIGHT ? job.c_from : job.e, job.ld, b_row, x_end, k0);
    __syncthreads();
    // neighbouring threads along the rows of the target; the second group of four rows r is R_STEP further
    const int r0 = RIGHT ? tid % PARTS * 4 : tid / (WIDE_X / 4) * 8, x0 = (RIGHT ? tid / PARTS : tid % (WIDE_X / 4)) * 4;
    constexpr int R_STEP = RIGHT ? WIDE_R / 2 : 4;
    float acc[8][4] = {};
#pragma unroll 8
    for (int k = 0; k < TILE; ++k) {
        const float4 q = *reinterpret_cast<const float4 *>(Bs + k * WIDE_X + wide_at(k, x0));
        const float qv[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const float4 p = *reinterpret_cast<const float4 *>(As + k * WIDE_R + wide_at(k, r0 + g * R_STEP));
            const float pv[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int x = 0; x < 4; ++x) acc[4 * g + r][x] = fmaf(pv[r], qv[x], acc[4 * g + r][x]);
        }
    }
    float *const to = RIGHT ? job.y_to : job.c_to;
#pragma unroll
    for (int g = 0; g < 2; ++g) {
        const bool valid = r0 + g * R_STEP < TILE ? t.valid_a : t.valid_b;
        float old[4][4];
#pragma unroll
        for (int pass = 0; pass < 2; ++pass)
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const int64_t at_r = a_row + r0 + g * R_STEP + r, at_x = b_row + x0 + x;
                    if (!valid || at_r >= r_end || at_x >= x_end) continue;
                    float *const p = to + (RIGHT ? at_x * job.ld + at_r : at_r * job.ld + at_x);
                    if (pass == 0) old[r][x] = *p;
                    else *p = old[r][x] + acc[4 * g + r][x];
                }
    }
}

// ---- the parts of a job, down and right ones apart: which tensor maps a TMA instruction takes is fixed where the code is compiled.
// (Chosen in the ring's loop, under one lane, compiled code lost boxes of right jobs: their targets stayed without them.  The cause
// is not known.) ----
template <bool RIGHT>
__device__ __forceinline__ void band_load(const BandTargetMaps &maps, const BandTarget &t, uint32_t dst, uint64_t *full) {
    const int k = t.k_tile * TILE, a_row = t.t_a * TILE, b_row = t.fixed * TILE;
    mbar_expect_tx(full, BAND_BYTES);
    tma_load_2d(dst, RIGHT ? &maps.ut_hi : &maps.l_hi, k, a_row, full);
    tma_load_2d(dst + HTILE_BYTES, RIGHT ? &maps.ut_lo : &maps.l_lo, k, a_row, full);
    tma_load_2d(dst + 2 * HTILE_BYTES, RIGHT ? &maps.c_hi : &maps.et_hi, k, b_row, full);
    tma_load_2d(dst + 2 * HTILE_BYTES + BB_BYTES, RIGHT ? &maps.c_lo : &maps.et_lo, k, b_row, full);
}
__device__ __forceinline__ void band_mma(uint32_t d, uint32_t operands, uint64_t *accum) {
    constexpr uint32_t DESC = idesc_16(BN, 0);
    const uint32_t s_a_hi = operands, s_a_lo = s_a_hi + HTILE_BYTES, s_b_hi = s_a_hi + 2 * HTILE_BYTES, s_b_lo = s_b_hi + BB_BYTES;
#pragma unroll
    for (int ks = 0; ks < KH / 16; ++ks) {
        const uint32_t off = ks * 32;  // 16 values = 32 bytes along the swizzled row
        umma_16(d, umma_desc(s_a_hi + off), umma_desc(s_b_hi + off), DESC, ks == 0 ? 0u : 1u);
        umma_16(d, umma_desc(s_a_lo + off), umma_desc(s_b_hi + off), DESC, 1u);
        umma_16(d, umma_desc(s_a_hi + off), umma_desc(s_b_lo + off), DESC, 1u);
    }
    umma_commit(accum);  // arrives when every MMA so far has completed
}
// What the results of reading warp q (lanes 32 q .. of tensor memory; lanes 0-63 belong to the first tile, 64-127 to the second) are
// multiplied by
template <bool RIGHT>
__device__ __forceinline__ float band_factor(const BandFields &job, const BandTarget &t, int q, float source_scale) {
    const int target = t.t_a + (q >> 1);  // tile row (down) or column (right) of this warp's results
    return source_scale * (RIGHT ? job.u_scale[(int64_t)target * job.nJ + t.k_tile] : job.l_scale[(int64_t)target * job.nI + t.k_tile]);
}
// The accumulator's rows of this warp, through two boxes per warp where the operands lay, and off as reductions (one group of lane 0)
template <bool RIGHT>
__device__ __forceinline__ void band_results(const BandTargetMaps &maps, const BandFields &job, const BandTarget &t, int q, int lane, float factor, uint32_t accumulator, uint32_t operands) {
    const uint32_t boxes = operands + (uint32_t)(q * 2 * BOX_BYTES);
    const int along = t.t_a * TILE + q * 32;  // row (down) or column (right) of lane 0
#pragma unroll
    for (int cb = 0; cb < BN / 32; ++cb) {
        uint32_t v[32];
        tmem_load_32(accumulator + ((uint32_t)(q * 32) << 16) + (uint32_t)(cb * 32), v);
        const uint32_t box = boxes + cb * BOX_BYTES;
        if (!RIGHT) {
#pragma unroll
            for (int g = 0; g < 8; ++g)
                box_store4(box, lane, g, factor * __uint_as_float(v[4 * g]), factor * __uint_as_float(v[4 * g + 1]), factor * __uint_as_float(v[4 * g + 2]),
                           factor * __uint_as_float(v[4 * g + 3]));
        } else {
            // transposed product: consecutive lanes hold consecutive columns of one row of Y
#pragma unroll
            for (int x = 0; x < 32; ++x) box_store1(box, x, lane, factor * __uint_as_float(v[x]));
        }
    }
    box_fence();
    __syncwarp();
    if (lane == 0) {
#pragma unroll
        for (int cb = 0; cb < BN / 32; ++cb) {
            const int across = t.fixed * TILE + cb * 32;  // first column (down) or row (right) of the box
            if (along < (RIGHT ? job.n : job.m) && across < (RIGHT ? job.m : job.n))
                box_reduce_add(RIGHT ? &maps.y : &maps.c, boxes + cb * BOX_BYTES, RIGHT ? along : across, RIGHT ? across : along);
        }
        box_commit();
    }
}
// The jobs of one of `ctas` CTAs, down jobs first, until body(std::bool_constant<right>, target) is false.
template <typename Body>
__device__ __forceinline__ void band_jobs(const BandFields &job, int cta, int ctas, Body body) {
    const int half = job.longest * job.slots;
    BandTarget t;
    int index = cta;
    for (; index < half; index += ctas)
        if (band_target(job, index % job.longest, index / job.longest, false, t) && !body(std::false_type{}, t)) return;
    for (index -= half; index < half; index += ctas)
        if (band_target(job, index % job.longest, index / job.longest, true, t) && !body(std::true_type{}, t)) return;
}

// All jobs of a near update, dealt out to `ctas` CTAs of 256 threads that have shared memory to themselves: warp 0 loads, warp 1 issues the
// MMAs, warps 2 to 5 read the accumulators and send the results off, through BAND_STAGES stages of 48 KB and as many accumulators.  Jobs with
// wide source tiles come last, by the whole CTA.  Every target entry belongs to one job.
// A stage and its accumulator go round together: the four reading warps arrive at `empty` once they have read the accumulator and the TMA
// has read their boxes; the loading lane waits for that and arrives at `full`; the MMAs that overwrite the accumulator wait for `full`.
constexpr int BAND_STAGES = 3;
constexpr uint32_t BAND_RING_COLS = 256;
constexpr int BAND_RING_SMEM = BAND_STAGES * BAND_BYTES + 1024;
struct BandRing {
    uint64_t full[BAND_STAGES], accum[BAND_STAGES], empty[BAND_STAGES];
    uint32_t tmem;
    int failed, wide;
};
// A function of its own: in line with the tiles' code in one kernel it made the tiles slower, the more the longer it was (777 x 1333: 1123 us in
// line, 1147 with the longer products of wide tiles, 1118 apart).
static __device__ __noinline__ void band_ring_cta(const BandJob &parameters, BandRing &ring, uint32_t smem_base, float *smem_floats, int cta, int ctas) {
    // in registers: through the reference, every field is loaded again behind every barrier (8192 x 8192: 11.76 -> 11.51 ms; two sweeps of
    // 4096 x 4096 on two streams: 2607 -> 2560 us each)
    const BandFields job = parameters;
    const BandTargetMaps &maps = parameters;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < BAND_STAGES; ++s) {
            mbar_init(&ring.full[s], 1);
            mbar_init(&ring.accum[s], 1);
            mbar_init(&ring.empty[s], 4);  // one arrival per reading warp
        }
        ring.failed = 0;
        ring.wide = *job.wide_count;  // one answer for the CTA: the tiles of the moment may be counting
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ring.tmem)), "r"(BAND_RING_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = ring.tmem;
    int c = 0;  // jobs so far: stages and accumulators are used in turn
    if (warp == 0) {
        if (lane == 0) {
            band_jobs(job, cta, ctas, [&](auto right, const BandTarget &t) {
                if (band_source_scale(job, t) < 0.f) return true;
                const int stage = c % BAND_STAGES, round = c / BAND_STAGES;
                if (round > 0 && !mbar_wait(&ring.empty[stage], (round - 1) & 1)) ring.failed = 1;
                if (*(volatile int *)&ring.failed) return false;
                band_load<decltype(right)::value>(maps, t, smem_base + stage * BAND_BYTES, &ring.full[stage]);
                ++c;
                return true;
            });
            // the last loads have landed (or had their time to) before their shared memory is released, whatever became of the MMAs
            for (int back = 1; back <= BAND_STAGES && back <= c; ++back) mbar_wait(&ring.full[(c - back) % BAND_STAGES], ((c - back) / BAND_STAGES) & 1);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            band_jobs(job, cta, ctas, [&](auto, const BandTarget &t) {
                if (band_source_scale(job, t) < 0.f) return true;
                const int stage = c % BAND_STAGES, round = c / BAND_STAGES;
                if (!mbar_wait(&ring.full[stage], round & 1)) ring.failed = 1;
                if (*(volatile int *)&ring.failed) return false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                band_mma(tmem + stage * BN, smem_base + stage * BAND_BYTES, &ring.accum[stage]);
                ++c;
                return true;
            });
            // on time-out, give what is in flight a bounded chance to land before its memory is released
            if (ring.failed && c > 0) mbar_wait(&ring.accum[(c - 1) % BAND_STAGES], ((c - 1) / BAND_STAGES) & 1);
        }
    } else if (warp < 6) {
        const int q = warp & 3;
        band_jobs(job, cta, ctas, [&](auto right, const BandTarget &t) {
            constexpr bool RIGHT = decltype(right)::value;
            const float source_scale = band_source_scale(job, t);
            if (source_scale < 0.f) return true;
            const int stage = c % BAND_STAGES, round = c / BAND_STAGES;
            ++c;
            const bool mine = q < 2 ? t.valid_a : t.valid_b;  // warp-uniform
            const float factor = mine ? band_factor<RIGHT>(job, t, q, source_scale) : 0.f;
            const bool ok = mbar_wait(&ring.accum[stage], round & 1, 64);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (!ok) ring.failed = 1;
            if (!__all_sync(0xffffffffu, ok && !*(volatile int *)&ring.failed)) return false;  // warp-uniform: the tensor-memory loads are warp-wide
            if (mine) {
                band_results<RIGHT>(maps, job, t, q, lane, factor, tmem + (uint32_t)(stage * BN), smem_base + stage * BAND_BYTES);
                if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            }
            // this warp is done with the stage and its accumulator
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&ring.empty[stage]);
            return true;
        });
        box_wait();
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BAND_RING_COLS) : "memory");
    if (ring.wide != 0 && !ring.failed)
        band_jobs(job, cta, ctas, [&](auto right, const BandTarget &t) {
            if (band_source_scale(job, t) >= 0.f) return true;
            wide_product_alone<256, decltype(right)::value>(job, t, smem_floats);
            __syncthreads();
            return true;
        });
    if (threadIdx.x == 0 && ring.failed && job.error_flag) atomicExch(job.error_flag, 1);
}

// The near update of the tile anti-diagonal s into the anti-diagonals t0 .. t1; false where it has no targets.
bool make_band_job(BandJob &job, const BandTcMaps *maps, const TcPlanes &planes, int64_t m, int64_t n, int s, int t0, int t1, int outer_macro, int lag_macro);

}  // namespace g2d

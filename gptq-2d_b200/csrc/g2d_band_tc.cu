// Feedback between tiles on the tensor cores for the pipelined schedule (float only).
//
// A band update carries the finished tiles of the tile anti-diagonal s (sources) into the tiles of the anti-diagonals t0..t1
// (targets), t0 >= s + 2:
//     down :  C[I, J] += L[I, k] E[k, J],   k = s - J      (same column of tiles)
//     right:  Y[I, J] += C[I, k] U[k, J],   k = s - I      (same row of tiles)
// The source tile of a target depends on its column (down) or its row (right) only, so a CTA takes two tiles that share
// it: a down job owns 128 rows x 64 columns (tile rows I, I + 1 of column J), a right job 64 rows x 128 columns, the
// latter formed transposed (Y^T = U^T C^T) so that the 128 side is again the M side of the MMA.  Each product is one chunk of
// tcgen05.mma kind::f16 with M = 128, N = 64, k = 64 on the fp16 pairs that the macro updates use, the two tiles' scales
// applied as the accumulator is read; the results leave as TMA reductions of 32 x 32 boxes.
// Every target entry is owned by one CTA of one launch and launches that share targets are ordered by the caller: the result does
// not depend on scheduling.  Latency bound (one TMA round trip, 12 MMAs, one reduction): several CTAs share an SM.
#include "g2d_band_tc.cuh"

namespace g2d {

constexpr uint32_t BAND_TMEM_COLS = 64;
// grid: x = tile column (down jobs) or tile row (right jobs), y = pair slot along the target range, z = 0 down, 1 right
// Which tensor maps an instruction takes is chosen by whole warps, before one lane goes on alone (see g2d_band_tc.cuh).  The text is the
// kernel's own: short, and with its exits one after the other, since many CTAs have nothing to do (8192 x 28672: 56.9 ms; on
// the ring's functions, compiled for down and right jobs apart, 57.2).
__global__ void __launch_bounds__(TC_THREADS) band_tc_kernel(const __grid_constant__ BandJob job) {
    extern __shared__ unsigned char tc_smem_raw[];
    __shared__ __align__(8) uint64_t full_bar, accum_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    const bool right = blockIdx.z != 0;
    const int fixed = blockIdx.x;                        // J (down) or I (right)
    const int fixed_count = right ? job.nI : job.nJ, moving_count = right ? job.nJ : job.nI;
    if (fixed >= fixed_count) return;
    const int first = max(job.t0 - fixed, 0);
    const int pair = (first >> 1) + (int)blockIdx.y;     // tiles 2 pair, 2 pair + 1 along the moving index
    const int t_a = 2 * pair, t_b = 2 * pair + 1;
    bool valid_a = t_a < moving_count && t_a + fixed >= job.t0 && t_a + fixed <= job.t1;
    bool valid_b = t_b < moving_count && t_b + fixed >= job.t0 && t_b + fixed <= job.t1;
    if (!valid_a && !valid_b) return;
    const int k_tile = job.s - fixed;                    // the source tile along k; it lies before both targets
    if (k_tile < 0 || k_tile >= moving_count) return;
    if (job.outer_macro > 0) {
        // both targets lie in one macro tile
        const int w_source = (k_tile >> 1) + (fixed >> 1), w_target = pair + (fixed >> 1);
        const int reach = (w_source / job.outer_macro + 1) * job.outer_macro + job.lag_macro;  // the far update starts here
        if (w_target >= reach) return;
    }
    const int a_row = t_a * TILE;                        // first of the 128 rows of the A operand
    const int b_row = fixed * TILE;                      // first of the 64 rows of the B operand
    const CUtensorMap *a_hi = right ? &job.ut_hi : &job.l_hi, *a_lo = right ? &job.ut_lo : &job.l_lo;
    const CUtensorMap *b_hi = right ? &job.c_hi : &job.et_hi, *b_lo = right ? &job.c_lo : &job.et_lo;

    // asked for here, used behind the set-up: negative where the source tile is wide
    const float source_scale = right ? job.c_scale[(int64_t)fixed * job.nJ + k_tile] : job.e_scale[(int64_t)k_tile * job.nJ + fixed];

    const uint32_t smem_base = (smem_u32(tc_smem_raw) + 1023u) & ~1023u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(&full_bar, 1);
        mbar_init(&accum_bar, 1);
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(BAND_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;

    if (source_scale < 0.f) {
        wide_product(job, right, a_row, b_row, k_tile * TILE, valid_a, valid_b, reinterpret_cast<float *>(tc_smem_raw + (smem_base - smem_u32(tc_smem_raw))));
    } else if (warp == 0) {
        if (lane == 0) {
            const int k = k_tile * TILE;
            mbar_expect_tx(&full_bar, BAND_BYTES);
            tma_load_2d(smem_base, a_hi, k, a_row, &full_bar);
            tma_load_2d(smem_base + HTILE_BYTES, a_lo, k, a_row, &full_bar);
            tma_load_2d(smem_base + 2 * HTILE_BYTES, b_hi, k, b_row, &full_bar);
            tma_load_2d(smem_base + 2 * HTILE_BYTES + BB_BYTES, b_lo, k, b_row, &full_bar);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            if (mbar_wait(&full_bar, 0)) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                constexpr uint32_t DESC = idesc_16(BN, 0);
                const uint32_t s_a_hi = smem_base, s_a_lo = s_a_hi + HTILE_BYTES, s_b_hi = s_a_hi + 2 * HTILE_BYTES, s_b_lo = s_b_hi + BB_BYTES;
#pragma unroll
                for (int ks = 0; ks < KH / 16; ++ks) {
                    const uint32_t off = ks * 32;  // 16 values = 32 bytes along the swizzled row
                    umma_16(tmem, umma_desc(s_a_hi + off), umma_desc(s_b_hi + off), DESC, ks == 0 ? 0u : 1u);
                    umma_16(tmem, umma_desc(s_a_lo + off), umma_desc(s_b_hi + off), DESC, 1u);
                    umma_16(tmem, umma_desc(s_a_hi + off), umma_desc(s_b_lo + off), DESC, 1u);
                }
                umma_commit(&accum_bar);  // arrives when every MMA has completed
            } else {
                failed = 1;
            }
        }
    } else {
        // epilogue warps: lanes 32 q .. 32 q + 31 of tensor memory, q = warp % 4; lanes 0-63 belong to tile a, 64-127 to tile b
        const int q = warp & 3;
        const bool mine = q < 2 ? valid_a : valid_b;             // warp-uniform
        const int target = q < 2 ? t_a : t_b;                    // tile row (down) or column (right) of this warp's results
        float factor = 0.f;
        if (mine)
            factor = source_scale * (right ? job.u_scale[(int64_t)target * job.nJ + k_tile] : job.l_scale[(int64_t)target * job.nI + k_tile]);
        const bool ok = mbar_wait(&accum_bar, 0, 256);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (!ok) failed = 1;
        const bool go = __all_sync(0xffffffffu, ok && !failed);  // warp-uniform: the tensor-memory loads are warp-wide
        if (go && mine) {
            // the operands have been multiplied: their shared memory takes the results, two boxes per warp
            const uint32_t boxes = smem_base + (uint32_t)(q * 2 * BOX_BYTES);
            const int along = a_row + q * 32;                    // row (down) or column (right) of lane 0
#pragma unroll
            for (int cb = 0; cb < BN / 32; ++cb) {
                uint32_t v[32];
                tmem_load_32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(cb * 32), v);
                const uint32_t box = boxes + cb * BOX_BYTES;
                if (!right) {
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
            const CUtensorMap *const to = right ? &job.y : &job.c;
            const int along_end = right ? job.n : job.m, across_end = right ? job.m : job.n;
            box_fence();
            __syncwarp();
            if (lane == 0) {
#pragma unroll
                for (int cb = 0; cb < BN / 32; ++cb) {
                    const int across = b_row + cb * 32;          // first column (down) or row (right) of the box
                    if (along < along_end && across < across_end) box_reduce_add(to, boxes + cb * BOX_BYTES, right ? along : across, right ? across : along);
                }
                box_commit();
                box_wait();
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        if (failed) {
            // give outstanding loads and MMAs a bounded chance to land before the memory they target is released
            if (lane == 0) mbar_wait(&accum_bar, 0);
            __syncwarp();
        }
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BAND_TMEM_COLS) : "memory");
    }
    if (threadIdx.x == 0 && failed && job.error_flag) atomicExch(job.error_flag, 1);
}

// Tensor maps of one sweep; encoded once and reused by every band launch.
struct BandMaps {
    CUtensorMap l_hi, l_lo, ut_hi, ut_lo, et_hi, et_lo, c_hi, c_lo, y, c;
};
static_assert(sizeof(BandMaps) <= sizeof(BandTcMaps::bytes), "opaque tensor-map storage is too small");

int band_tc_prepare(BandTcMaps *opaque, const TcPlanes &pl, float *y, float *c, int64_t m, int64_t n, int64_t ld) {
    BandMaps *maps = reinterpret_cast<BandMaps *>(opaque);
    opaque->y = y;
    opaque->c = c;
    if (!make_map_16(&maps->l_hi, pl.l_hi, m, m, MT, false, pl.ldm) || !make_map_16(&maps->l_lo, pl.l_lo, m, m, MT, false, pl.ldm) ||
        !make_map_16(&maps->ut_hi, pl.ut_hi, n, n, MT, false, pl.ldn) || !make_map_16(&maps->ut_lo, pl.ut_lo, n, n, MT, false, pl.ldn) ||
        !make_map_16(&maps->et_hi, pl.et_hi, n, m, BN, false, pl.ldm) || !make_map_16(&maps->et_lo, pl.et_lo, n, m, BN, false, pl.ldm) ||
        !make_map_16(&maps->c_hi, pl.c_hi, m, n, BN, false, pl.ldn) || !make_map_16(&maps->c_lo, pl.c_lo, m, n, BN, false, pl.ldn) ||
        !make_map(&maps->y, y, m, n, 32, ld) || !make_map(&maps->c, c, m, n, 32, ld))
        return G2D_ERR_CUDA;
    static PerDeviceOnce configured;
    // Several CTAs of this kernel share an SM, with one another and with other kernels' CTAs.  It asks for the largest
    // shared-memory carve-out: an SM that a kernel with a smaller one had configured takes no CTA beside it that needs
    // more until it has drained.
    return configured.run([&] {
        return cudaFuncSetAttribute(band_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BAND_BYTES + 1024) == cudaSuccess &&
               cudaFuncSetAttribute(band_tc_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) == cudaSuccess;
    });
}

bool make_band_job(BandJob &job, const BandTcMaps *opaque, const TcPlanes &pl, int64_t m, int64_t n, int s, int t0, int t1, int outer_macro, int lag_macro) {
    const BandMaps *maps = reinterpret_cast<const BandMaps *>(opaque);
    job.l_hi = maps->l_hi; job.l_lo = maps->l_lo; job.ut_hi = maps->ut_hi; job.ut_lo = maps->ut_lo;
    job.et_hi = maps->et_hi; job.et_lo = maps->et_lo; job.c_hi = maps->c_hi; job.c_lo = maps->c_lo;
    job.y = maps->y; job.c = maps->c;
    job.l_scale = pl.l_scale; job.c_scale = pl.c_scale; job.e_scale = pl.e_scale; job.u_scale = pl.u_scale;
    job.nI = (int)ceil_div(m, (int64_t)TILE); job.nJ = (int)ceil_div(n, (int64_t)TILE);
    job.m = (int)m; job.n = (int)n;
    const int waves = job.nI + job.nJ - 1;
    if (t1 > waves - 1) t1 = waves - 1;
    if (t1 < t0) return false;
    job.s = s; job.t0 = t0; job.t1 = t1;
    job.outer_macro = outer_macro; job.lag_macro = lag_macro;
    job.error_flag = pl.error_flag; job.wide_count = pl.wide_count;
    job.l = pl.l; job.u = pl.u; job.e = pl.e; job.c_from = pl.c;
    job.y_to = opaque->y; job.c_to = opaque->c;
    job.ldl = pl.ldl; job.ldu = pl.ldu; job.ld = pl.ld;
    // pairs along the moving index that can hold a target: at most (t1 - t0) / 2 + 2, never more than the matrix has
    job.longest = job.nI > job.nJ ? job.nI : job.nJ;
    job.slots = (t1 - t0) / 2 + 2;
    if (job.slots > (job.longest + 1) / 2) job.slots = (job.longest + 1) / 2;
    return true;
}

int launch_band_tc(const BandTcMaps *maps, const TcPlanes &pl, int64_t m, int64_t n, int s, int t0, int t1, int outer_macro, int lag_macro, cudaStream_t stream) {
    if (t1 >= t0 && t0 < s + 2) return G2D_ERR_BAD_ARGUMENT;
    BandJob job;
    if (!make_band_job(job, maps, pl, m, n, s, t0, t1, outer_macro, lag_macro)) return G2D_OK;
    band_tc_kernel<<<dim3((unsigned)job.longest, (unsigned)job.slots, 2), TC_THREADS, BAND_BYTES + 1024, stream>>>(job);
    return check_launch();
}

}  // namespace g2d

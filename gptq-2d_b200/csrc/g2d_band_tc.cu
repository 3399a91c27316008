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

// grid: x = tile column (down jobs) or tile row (right jobs), y = pair slot along the target range, z = 0 down, 1 right
constexpr uint32_t BAND_TMEM_COLS = 64;
__global__ void __launch_bounds__(TC_THREADS) band_tc_kernel(const __grid_constant__ BandJob job) {
    extern __shared__ unsigned char tc_smem_raw[];
    __shared__ __align__(8) uint64_t full_bar, accum_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    BandTarget t;
    if (!band_target(job, blockIdx.x, blockIdx.y, blockIdx.z != 0, t)) return;

    // asked for here, used behind the set-up: negative where the source tile is wide
    const float source_scale = band_source_scale(job, t);

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

    auto body = [&](auto right) {
        constexpr bool RIGHT = decltype(right)::value;
        if (source_scale < 0.f) {
            wide_product<TC_THREADS>(job, RIGHT, t.t_a * TILE, t.fixed * TILE, t.k_tile * TILE, t.valid_a, t.valid_b,
                                     reinterpret_cast<float *>(tc_smem_raw + (smem_base - smem_u32(tc_smem_raw))));
        } else if (warp == 0) {
            if (lane == 0) band_load<RIGHT>(job, t, smem_base, &full_bar);
        } else if (warp == 1) {
            if (lane == 0) {
                if (mbar_wait(&full_bar, 0)) {
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    band_mma(tmem, smem_base, &accum_bar);
                } else {
                    failed = 1;
                }
            }
        } else {
            const int q = warp & 3;
            const bool mine = q < 2 ? t.valid_a : t.valid_b;         // warp-uniform
            const float factor = mine ? band_factor<RIGHT>(job, t, q, source_scale) : 0.f;
            const bool ok = mbar_wait(&accum_bar, 0, 256);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (!ok) failed = 1;
            const bool go = __all_sync(0xffffffffu, ok && !failed);  // warp-uniform: the tensor-memory loads are warp-wide
            if (go && mine) {
                band_results<RIGHT>(job, t, q, lane, factor, tmem, smem_base);
                if (lane == 0) box_wait();
            }
        }
    };
    if (blockIdx.z != 0) body(std::true_type{});
    else body(std::false_type{});
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

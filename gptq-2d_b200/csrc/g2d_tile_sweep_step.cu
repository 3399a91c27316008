// A step of the pipelined schedule in one launch (float, one matrix): the first CTAs sweep the tiles of the anti-diagonal S, and the others, on
// the SMs that the tiles leave free, carry out the near update of the anti-diagonal before.  The two do not depend on each other: the update's
// targets start at S + 1.  Bound by the tiles' serial chain, about 24 us.  On streams of their own (g2d_tile_sweep.cu, g2d_band_tc.cu) a step took
// 7 us of events between the two on top of it; in one launch that starts early, 1024 x 1024 takes 0.84 ms in place of 0.95, 2048 x 2048 1.72 in
// place of 1.97, 8192 x 8192 11.1 in place of 11.8.  A warp issues an instruction every ninth cycle; 2.0 of
// those nine it waits for instructions to arrive, 2.3 at barriers (4096 x 4096): how long the kernel's text is, and where its parts lie,
// shows in its time.
#include "g2d_band_tc.cuh"
#include "g2d_tile_sweep.cuh"

namespace g2d {

template <typename F, int KIND>
__global__ void __launch_bounds__(TTH, 1) sweep_step_kernel(const __grid_constant__ SweepArgs<F> P, int S, int i_first, int tiles, const __grid_constant__ BandJob job) {
    extern __shared__ __align__(16) unsigned char g2d_smem[];
    if ((int)blockIdx.x >= tiles) {
        __shared__ __align__(8) BandRing ring;
        after_the_launch_before();
        const uint32_t base = (smem_u32(g2d_smem) + 1023u) & ~1023u;
        band_ring_cta(job, ring, base, reinterpret_cast<float *>(g2d_smem + (base - smem_u32(g2d_smem))), (int)blockIdx.x - tiles, (int)gridDim.x - tiles);
        return;
    }
    constexpr int i_step = 1;
#define G2D_JOINT 1
#include "g2d_tile_body.cuh"
#undef G2D_JOINT
}

template <int KIND>
static int launch_step_kind(const SweepArgs<float> &args, int S, const BandJob &job, cudaStream_t stream) {
    static PerDeviceOnce configured;
    constexpr size_t smem = tile_smem<float> > BAND_RING_SMEM ? tile_smem<float> : BAND_RING_SMEM;
    if (configured.run([&] { return cudaFuncSetAttribute(sweep_step_kernel<float, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess; }) != G2D_OK)
        return G2D_ERR_CUDA;
    const int i_lo = S - args.nJ + 1 > 0 ? S - args.nJ + 1 : 0, i_hi = S + 1 < args.nI ? S + 1 : args.nI, tiles = i_hi - i_lo;
    // Updating CTAs: as many as there are SMs left, but sixteen jobs each, which the ring takes in 5 to 12 us of the tiles' 25.  More of them keep SMs
    // from the far updates (4 us of set-up and first loads each): 1, 8, 16 and 24 jobs at least, in us: 2048 x 2048 1732, 1719, 1721, 1764;
    // 4096 x 4096 3747, 3708, 3709, 3804; 8192 x 8192 11120, 11103, 11041, 10985.
    constexpr int JOBS_EACH = 16;
    const int jobs = 2 * job.longest * job.slots, free_sms = 148 - tiles, updating = (jobs + JOBS_EACH - 1) / JOBS_EACH;  // at most 128 tiles take this schedule
    if (free_sms < 1) return G2D_ERR_BAD_ARGUMENT;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3((unsigned)(tiles + (updating < free_sms ? updating : free_sms)));
    config.blockDim = dim3(TTH);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    if (cudaLaunchKernelEx(&config, sweep_step_kernel<float, KIND>, args, S, i_lo, tiles, job) != cudaSuccess) return G2D_ERR_CUDA;
    return check_launch();
}

int launch_sweep_step(const SweepArgs<float> &args, int S, const BandTcMaps *maps, const TcPlanes &planes, int s, int t0, int t1, int outer_macro, int lag_macro,
                      cudaStream_t stream) {
    BandJob job;
    if (s + 1 != S || !make_band_job(job, maps, planes, args.m, args.n, s, t0, t1, outer_macro, lag_macro)) return G2D_ERR_BAD_ARGUMENT;
    switch (args.kind) {
    case G2D_Q_ROUND: return launch_step_kind<G2D_Q_ROUND>(args, S, job, stream);
    case G2D_Q_AFFINE: return launch_step_kind<G2D_Q_AFFINE>(args, S, job, stream);
    case G2D_Q_FORCED: return launch_step_kind<G2D_Q_FORCED>(args, S, job, stream);
    default: return G2D_ERR_UNSUPPORTED;
    }
}

}  // namespace g2d

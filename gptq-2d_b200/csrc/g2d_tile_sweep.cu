// Fused tile sweep: one CTA rounds one TILE x TILE tile of the matrix, with the quantizer inside.
//
// Replaces, for the quantizers this library knows, the per-stage quantizer call and
// _push_kernel of the reference (gptq_2d.py:243-346, driven from :1342-1374).  Any order that
// respects "above and to the left first" gives the reference's result in exact arithmetic
// (gptq_2d_reference.py:166-200 prove it for two other orders), so the sweep is organised for
// the hardware instead of by global anti-diagonals:
//
//   * the host launches one grid per tile anti-diagonal; the tiles of one anti-diagonal are
//     independent, all feedback from earlier tiles is already in Y (right) and C (down);
//   * inside the CTA the tile lives in shared memory; the 16 x 16 sub-tiles are taken on a sub-tile wavefront: the
//     up to four sub-tiles of one sub-tile anti-diagonal are swept in registers by four warps.  These are the critical
//     path of the whole sweep and do little but the rounding stages: four helper warps carry the rest while a sub-tile
//     anti-diagonal is swept (the quantizer parameters of the next one, the feedback of finished sub-tiles into sub-tiles
//     two or more anti-diagonals ahead, the feedback for the neighbour tiles); between two sweeps both form the one
//     product pair per sub-tile that cannot be formed earlier, from the anti-diagonal just swept into the next one;
//   * inside a sub-tile half of a warp's lanes own the columns (the down feedback, "C"), the other half the rows (the right
//     feedback, "Y"), skewed so that the entries of an anti-diagonal sit in register 0 of every lane when their stage
//     comes: a push moves the accumulators down by one register.  One shuffle per stage exchanges the two sums of an
//     entry.  The feedback coefficients of a sub-tile come from zero-padded copies of the diagonal blocks of L and U^T,
//     so the pushes need no bounds predicates: out-of-range pushes multiply by zero;
//   * pipelined schedule: a tile also adds the far-feedback planes as it loads, and the feedback between neighbour
//     tiles of consecutive tile anti-diagonals travels as a push: the helper warps of tile (I, J) form, from the
//     errors and the completed C in shared memory,  L[I + 1, I] E[I, J]  and  C[I, J] U[J, J + 1]  while the tile is
//     still being swept and store them into two planes of their own, which the tiles (I + 1, J) and (I, J + 1) add
//     as they load one launch later.  No load from another tile's results sits on a tile's critical path.
#include "g2d_tile_sweep.cuh"

namespace g2d {

template <typename F, int KIND>
__global__ void __launch_bounds__(TTH, 1) tile_sweep_kernel(SweepArgs<F> P, int S, int i_first, int i_step) {
    extern __shared__ __align__(16) unsigned char g2d_smem[];
#define G2D_JOINT 0
#include "g2d_tile_body.cuh"
#undef G2D_JOINT
}

template <typename F, int KIND>
static int launch_kind(const SweepArgs<F> &args, int S, int parity, cudaStream_t stream) {
    // the opt-in to more than 48 KB of dynamic shared memory is per device
    static PerDeviceOnce configured;
    constexpr size_t smem = tile_smem<F>;
    // and the largest shared-memory carve-out, like the update kernels that run on the neighbouring SMs
    if (configured.run([&] {
            return cudaFuncSetAttribute(tile_sweep_kernel<F, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess &&
                   cudaFuncSetAttribute(tile_sweep_kernel<F, KIND>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) == cudaSuccess;
        }) != G2D_OK)
        return G2D_ERR_CUDA;
    const int i_lo = S - args.nJ + 1 > 0 ? S - args.nJ + 1 : 0;
    const int i_hi = S + 1 < args.nI ? S + 1 : args.nI;
    // parity 0: every tile of the anti-diagonal; 1: tiles with even row and column index; 2: odd row and column index
    int first = i_lo, step = 1, count = i_hi - i_lo;
    if (parity != 0) {
        const int want = parity == 1 ? 0 : 1;
        if ((S & 1) != 0) return G2D_OK;  // row + column parity is even for both selections
        first = i_lo + (((i_lo & 1) != want) ? 1 : 0);
        step = 2;
        count = first < i_hi ? (i_hi - first + 1) / 2 : 0;
    }
    if (count <= 0) return G2D_OK;
    dim3 grid((unsigned)count, (unsigned)(args.batch < 65535 ? args.batch : 65535));
    tile_sweep_kernel<F, KIND><<<grid, TTH, smem, stream>>>(args, S, first, step);
    return check_launch();
}

template <typename F>
int launch_tile_sweep(const SweepArgs<F> &args, int S, cudaStream_t stream, int parity) {
    switch (args.kind) {
    case G2D_Q_ROUND: return launch_kind<F, G2D_Q_ROUND>(args, S, parity, stream);
    case G2D_Q_AFFINE: return launch_kind<F, G2D_Q_AFFINE>(args, S, parity, stream);
    case G2D_Q_FORCED: return launch_kind<F, G2D_Q_FORCED>(args, S, parity, stream);
    default: return G2D_ERR_UNSUPPORTED;
    }
}

bool load_tile_sweep() {
    cudaFuncAttributes attributes;
    return cudaFuncGetAttributes(&attributes, tile_sweep_kernel<float, G2D_Q_AFFINE>) == cudaSuccess;
}

template int launch_tile_sweep<float>(const SweepArgs<float> &, int, cudaStream_t, int);
template int launch_tile_sweep<double>(const SweepArgs<double> &, int, cudaStream_t, int);

}  // namespace g2d

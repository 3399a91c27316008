// Feedback between tiles of any size on FFMA / DFMA, for the overlapped schedule (float64, batches, super-entries):
//
//     down :  C[i, j] += sum_k L[i, k] E[k, j],     right:  Y[i, j] += sum_k C[i, k] U[k, j]
//
// with the finished tiles of the tile anti-diagonals s0 .. s1-1 as sources and the tiles of t0 .. t1-1 as targets.  A tile is
// TR x TC entries; the sources of a target lie in whole tiles of its column (down) and its row (right), so both products
// run over one contiguous range of k and need no masks (the errors keep their natural layout, as everywhere).
//
// One CTA of 256 threads forms one product for one 64 x 64 block of a target tile, 4 x 4 outputs per thread, k in chunks of
// sixteen staged through shared memory, the next chunk on its way from global memory meanwhile.  These launches hold few
// CTAs (an anti-diagonal of tiles) and the next tile launch waits for them, so it is a CTA's latency that counts: 256
// threads instead of the 64 of band_update_kernel (which is built for many CTAs) and the two products in CTAs of their own
// take a rank-64 float64 update from 62 to 14 us.
#include "g2d_common.cuh"

namespace g2d {

constexpr int KB = 16;        // k per chunk
constexpr int UTH = 256;      // threads
constexpr int ULD = 64 + 4;   // shared row stride

template <typename F>
__global__ void __launch_bounds__(UTH) block_update_kernel(BlockUpdateArgs<F> A, int nI, int nJ, int row_parts, int col_parts) {
    __shared__ __align__(16) F As[2][KB * ULD];
    __shared__ __align__(16) F Bs[2][KB * ULD];
    const int wave = A.t0 + (int)blockIdx.y;
    const int lo = max(0, wave - nJ + 1), hi = min(wave + 1, nI);
    int x = (int)blockIdx.x;
    const int cp = x % col_parts;
    x /= col_parts;
    const int rp = x % row_parts;
    const int TI = lo + x / row_parts, TJ = wave - TI;
    if (TI >= hi) return;
    const int64_t m = A.m, n = A.n;
    const int64_t i0 = (int64_t)TI * A.TR + rp * 64, j0 = (int64_t)TJ * A.TC + cp * 64;
    const int rows = (int)min((int64_t)64, min(m, (int64_t)(TI + 1) * A.TR) - i0), cols = (int)min((int64_t)64, min(n, (int64_t)(TJ + 1) * A.TC) - j0);
    if (rows <= 0 || cols <= 0) return;
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;

    for (int64_t z = blockIdx.z; z < 2 * A.batch; z += gridDim.z) {
        const int64_t batch = z >> 1;
        const bool right = z & 1;
        const int64_t k_lo = right ? (int64_t)max(0, A.s0 - TI) * A.TC : (int64_t)max(0, A.s0 - TJ) * A.TR;
        const int64_t k_hi = right ? min(n, (int64_t)min(A.s1 - TI, TJ) * A.TC) : min(m, (int64_t)min(A.s1 - TJ, TI) * A.TR);
        if (k_hi <= k_lo) continue;
        const int64_t plane = batch * m * n;
        const F *a = right ? A.c_from + plane + i0 * n : A.l + (A.l_off ? A.l_off[batch] : 0) + i0 * m;
        const F *b = right ? A.u + (A.u_off ? A.u_off[batch] : 0) + j0 : A.e + plane + j0;
        const int64_t lda = right ? n : m;
        F *out = (right ? A.y : A.c) + plane + i0 * n + j0;
        F ra[4], rb[4];
        auto fetch = [&](int64_t k0) {
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int id = t * UTH + tid;
                const int row = id >> 4, ka = id & 15, kb = id >> 6, col = id & 63;
                ra[t] = row < rows && k0 + ka < k_hi ? a[row * lda + k0 + ka] : (F)0;
                rb[t] = col < cols && k0 + kb < k_hi ? b[(k0 + kb) * n + col] : (F)0;
            }
        };
        auto stash = [&](int buf) {
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int id = t * UTH + tid;
                As[buf][(id & 15) * ULD + (id >> 4)] = ra[t];
                Bs[buf][(id >> 6) * ULD + (id & 63)] = rb[t];
            }
        };
        F acc[4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[r][c] = (F)0;
        fetch(k_lo);
        stash(0);
        __syncthreads();
        int buf = 0;
        for (int64_t k0 = k_lo; k0 < k_hi; k0 += KB) {
            const bool more = k0 + KB < k_hi;
            if (more) fetch(k0 + KB);
#pragma unroll
            for (int kk = 0; kk < KB; ++kk) {
                F av[4], bv[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) av[r] = As[buf][kk * ULD + ty * 4 + r];
#pragma unroll
                for (int c = 0; c < 4; ++c) bv[c] = Bs[buf][kk * ULD + tx * 4 + c];
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[r][c] += av[r] * bv[c];
            }
            if (more) stash(buf ^ 1);
            __syncthreads();
            buf ^= 1;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (ty * 4 + r < rows && tx * 4 + c < cols) out[(int64_t)(ty * 4 + r) * n + tx * 4 + c] += acc[r][c];
    }
}

template <typename F>
int launch_block_update(const BlockUpdateArgs<F> &A, cudaStream_t stream) {
    const int nI = (int)ceil_div(A.m, A.TR), nJ = (int)ceil_div(A.n, A.TC), waves = nI + nJ - 1;
    const int t1 = A.t1 < waves ? A.t1 : waves;
    if (t1 <= A.t0 || A.s1 <= A.s0) return G2D_OK;
    const int row_parts = (int)ceil_div(A.TR, 64), col_parts = (int)ceil_div(A.TC, 64);
    const int64_t longest = (nI < nJ ? nI : nJ);
    dim3 grid((unsigned)(longest * row_parts * col_parts), (unsigned)(t1 - A.t0), (unsigned)(2 * A.batch < 65535 ? 2 * A.batch : 65534));
    block_update_kernel<F><<<grid, UTH, 0, stream>>>(A, nI, nJ, row_parts, col_parts);
    return check_launch();
}

template int launch_block_update<float>(const BlockUpdateArgs<float> &, cudaStream_t);
template int launch_block_update<double>(const BlockUpdateArgs<double> &, cudaStream_t);

}  // namespace g2d

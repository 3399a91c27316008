// Feedback between macro tiles on the tensor cores (float only): tcgen05.mma kind::f16 on fp16 pairs with accumulators in
// tensor memory, operands brought into shared memory by TMA (cp.async.bulk.tensor, 128-byte swizzle).
//
// One CTA owns one 128 x 128 target macro tile and forms both products of the band update
//     down :  C[I, J] += sum_k L[I, k] E[k, J]      right:  Y[I, J] += sum_k C[I, k] U[k, J]
// over the k ranges that hold the sources of the macro anti-diagonals s0..s1-1 (whole 128-blocks, no masks).
// float32 fidelity comes from the split of every operand into hi + lo with 11 significant bits each under a power of two per
// 64 x 64 tile (see split_half) and three products per k step, hi hi + lo hi + hi lo.  A slice of k is one tile wide, so the
// product of the two tiles' scales is a constant of a slice and of 64 rows and columns: it rides on the additions that
// add the slices up in registers.  All four operand kinds are stored K-major for the MMA: L and C as they are (rows x k), E and U
// transposed (columns x k); the split copies of L and U^T are made once per sweep by the kernels at the end of this file,
// those of E^T and C by the tile sweep as it finishes a tile.
//
// Bound: the shared-memory port (a 128 x 128 x 16 MMA reads its 8 KB in exactly the 64 cycles it takes, and the operands' arrival
// shares the port: 60 % of the tensor rate); with tf32 pairs that was 60 % of half the rate and twice the bytes.  128 x 256
// tiles would reach 80 %, but the k ranges of two neighbouring macro columns differ.  Each product's results leave as TMA
// reductions while the next product is multiplied.  With the near updates converted alike,
// the sweep of 8192 x 28672 went from 96 to 70 ms.
#include "g2d_tc.cuh"

namespace g2d {

constexpr int RB_I = 8, RB_J = 16;  // rasterisation block of the far updates: 128 macro tiles, about one wave of CTAs
constexpr int MACRO_STAGES = 3;

struct TcMaps {
    CUtensorMap l_hi, l_lo, c_hi, c_lo;      // A operands: [rows][k]
    CUtensorMap et_hi, et_lo, ut_hi, ut_lo;  // B operands: [columns][k]
    CUtensorMap y, c;                        // targets, boxes of 32 x 32
};
struct MacroScales {
    const float *l, *c, *e, *u;
    int nI, nJ;  // 64 x 64 tiles
    int m, n;
};

__global__ void __launch_bounds__(PAIR_THREADS, 1) macro_update_tc_kernel(const __grid_constant__ TcMaps maps, const MacroScales S, int nI2, int nJ2, int s0,
                                                                          int s1, int t_first, int s_end, int raster, int *error_flag) {
    constexpr int NT = 128, MINE = NT / 2;
    extern __shared__ unsigned char tc_smem_raw[];
    __shared__ __align__(8) PairRing<MACRO_STAGES> ring;
    // Target macro tile.  With gridDim.y > 1, blockIdx.y selects the macro anti-diagonal and blockIdx.x the tile on it
    // (few anti-diagonals: near updates).  Otherwise the whole macro grid is walked in RB_I x RB_J blocks, so that the
    // CTAs resident at one time cover a compact patch and share their L / C row strips and E^T / U^T column strips in L2.
    int I2, J2;
    if (raster == 0) {
        const int W = t_first + (int)blockIdx.y;
        const int ti_lo = max(0, W - nJ2 + 1), ti_hi = min(W + 1, nI2);
        I2 = ti_lo + (int)blockIdx.x;
        if (W >= s_end || I2 >= ti_hi) return;
        J2 = W - I2;
    } else {
        const int blocks_j = (nJ2 + RB_J - 1) / RB_J;
        const int blk = (int)blockIdx.x / (RB_I * RB_J), within = (int)blockIdx.x % (RB_I * RB_J);
        I2 = (blk / blocks_j) * RB_I + within / RB_J;
        J2 = (blk % blocks_j) * RB_J + within % RB_J;
        if (I2 >= nI2 || J2 >= nJ2 || I2 + J2 < t_first || I2 + J2 >= s_end) return;
    }
    // source macro rows (down) and macro columns (right) of the band
    const int kd_lo = max(s0 - J2, 0), kd_hi = min(s1 - J2, I2);
    const int kr_lo = max(s0 - I2, 0), kr_hi = min(s1 - I2, J2);
    const int chunks_d = kd_hi > kd_lo ? (kd_hi - kd_lo) * (MT / KH) : 0;
    const int chunks_r = kr_hi > kr_lo ? (kr_hi - kr_lo) * (MT / KH) : 0;
    if (chunks_d + chunks_r == 0) return;
    const uint32_t smem_base = (smem_u32(tc_smem_raw) + 1023u) & ~1023u;
    auto next = [&](int it, PairTile &t) {  // the down product, then the right one (`which`), each where it has sources
        const int which = it + (chunks_d == 0 ? 1 : 0);
        if (which > 1 || (which == 1 && chunks_r == 0)) return false;
        t = PairTile{I2 * MT, J2 * MT, which ? chunks_r : chunks_d, (which ? kr_lo : kd_lo) * MT, which};
        return true;
    };
    auto load = [&](const PairTile &t, int ch, uint32_t dst, uint64_t *bar) {
        const int k = t.k0 + ch * KH;
        tma_load_2d(dst, t.which ? &maps.c_hi : &maps.l_hi, k, t.i0, bar);
        tma_load_2d(dst + HTILE_BYTES, t.which ? &maps.c_lo : &maps.l_lo, k, t.i0, bar);
        tma_load_2d(dst + 2 * HTILE_BYTES, t.which ? &maps.ut_hi : &maps.et_hi, k, t.j0, bar);
        tma_load_2d(dst + 3 * HTILE_BYTES, t.which ? &maps.ut_lo : &maps.et_lo, k, t.j0, bar);
    };
    auto scale = [&](const PairTile &t, int slice, int q, int column) {
        const int k = t.k0 / TILE + slice, i = min(t.i0 / TILE + (q >> 1), S.nI - 1), j = min((t.j0 + column) / TILE, S.nJ - 1);
        return t.which ? S.c[(int64_t)i * S.nJ + k] * S.u[(int64_t)j * S.nJ + k] : S.l[(int64_t)i * S.nI + k] * S.e[(int64_t)k * S.nJ + j];
    };
    auto finish = [&](const PairTile &t, int q, int lane, int c0, float (&total)[MINE], uint32_t box) {
#pragma unroll
        for (int cb = 0; cb < MINE / 32; ++cb) {
            if (lane == 0) box_free();
            __syncwarp();
#pragma unroll
            for (int g = 0; g < 8; ++g) box_store4(box, lane, g, total[cb * 32 + g * 4], total[cb * 32 + g * 4 + 1], total[cb * 32 + g * 4 + 2], total[cb * 32 + g * 4 + 3]);
            box_fence();
            __syncwarp();
            if (lane == 0 && t.i0 + q * 32 < S.m && t.j0 + c0 + cb * 32 < S.n) {
                // one CTA owns each target entry, so the reduction needs no read-back and stays deterministic; what lies outside the
                // matrix is not written
                box_reduce_add(t.which ? &maps.y : &maps.c, box, t.j0 + c0 + cb * 32, t.i0 + q * 32);
                box_commit();
            }
        }
    };
    const bool failed = pair_gemm<NT, MACRO_STAGES, 1>(ring, smem_base, next, load, finish, scale);
    if (threadIdx.x == 0 && failed && error_flag) atomicExch(error_flag, 1);
}

// ---- one-time operand preparation: a 64 x 64 tile per CTA, strictly below the diagonal tiles (no update reads the others) ----

// Tile (I, K), K < I, of a lower triangle of nT tile rows from a linear index
__device__ __forceinline__ void below_diagonal(int64_t lin, int &I, int &K) {
    int64_t a = (int64_t)((sqrt(8.0 * (double)lin + 1.0) - 1.0) / 2.0);
    while ((a + 1) * (a + 2) / 2 <= lin) ++a;
    while (a * (a + 1) / 2 > lin) --a;
    I = (int)a + 1;
    K = (int)(lin - a * (a + 1) / 2);
}

// UPPER: U (row-major), transposed: out[j][k] = U[k][j]; else L: out[i][k] = L[i][k].  HBM bound: 4 bytes in, 4 out per entry.
template <bool UPPER>
__global__ void __launch_bounds__(256) split_tile_kernel(const float *__restrict__ src, int64_t pitch, int64_t size, int nT, __half *__restrict__ hi,
                                                         __half *__restrict__ lo, int64_t ld, float *__restrict__ scales) {
    __shared__ float tile[TILE][TILE + 1];
    __shared__ unsigned part[8];
    int I, K;
    below_diagonal(blockIdx.x, I, K);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // source block: rows a0 .., columns b0 ..
    const int64_t a0 = (int64_t)(UPPER ? K : I) * TILE, b0 = (int64_t)(UPPER ? I : K) * TILE;
    const bool vec = pitch % 4 == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0 && b0 + TILE <= size;
    unsigned most = 0u;
#pragma unroll
    for (int t = 0; t < TILE * TILE / 4 / 256; ++t) {
        const int idx = t * 256 + tid, r = idx / (TILE / 4), c = (idx % (TILE / 4)) * 4;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (a0 + r < size) {
            const float *p = src + (a0 + r) * pitch + b0 + c;
            if (vec) {
                const float4 f = *reinterpret_cast<const float4 *>(p);
                v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
            } else {
#pragma unroll
                for (int x = 0; x < 4; ++x) v[x] = b0 + c + x < size ? p[x] : 0.f;
            }
        }
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            most = max(most, __float_as_uint(v[x]) & 0x7fffffffu);
            if (UPPER) tile[c + x][r] = v[x];
            else tile[r][c + x] = v[x];
        }
    }
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0) part[warp] = most;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; ++w) most = max(most, part[w]);
    const int e = range_exponent(__uint_as_float(most));
    if (tid == 0) scales[(int64_t)I * nT + K] = power_of_two(e);
    const float by = power_of_two(-e);
#pragma unroll
    for (int t = 0; t < TILE * TILE / 8 / 256; ++t) {
        const int idx = t * 256 + tid, r = idx / (TILE / 8), c = (idx % (TILE / 8)) * 8;
        if ((int64_t)I * TILE + r >= size) continue;
        __align__(16) __half h[8];
        __align__(16) __half l[8];
#pragma unroll
        for (int x = 0; x < 8; ++x) split_half(tile[r][c + x] * by, h[x], l[x]);
        const int64_t at = ((int64_t)I * TILE + r) * ld + (int64_t)K * TILE + c;  // K < I: whole tiles of columns
        *reinterpret_cast<uint4 *>(hi + at) = *reinterpret_cast<const uint4 *>(h);
        *reinterpret_cast<uint4 *>(lo + at) = *reinterpret_cast<const uint4 *>(l);
    }
}

// ---- host side ---------------------------------------------------------------------------------------

int tc_prepare_operands(const float *l, int64_t ldl, const float *u, int64_t ldu, int64_t m, int64_t n, const TcPlanes &pl, cudaStream_t stream) {
    const int nI = (int)ceil_div(m, (int64_t)TILE), nJ = (int)ceil_div(n, (int64_t)TILE);
    const int64_t below_l = (int64_t)nI * (nI - 1) / 2, below_u = (int64_t)nJ * (nJ - 1) / 2;
    if (below_l > 0x7fffffff || below_u > 0x7fffffff) return G2D_ERR_TOO_LARGE;
    if (below_l > 0) {
        split_tile_kernel<false><<<(unsigned)below_l, 256, 0, stream>>>(l, ldl, m, nI, pl.l_hi, pl.l_lo, pl.ldm, pl.l_scale);
        if (check_launch() != G2D_OK) return G2D_ERR_CUDA;
    }
    if (below_u > 0) {
        split_tile_kernel<true><<<(unsigned)below_u, 256, 0, stream>>>(u, ldu, n, nJ, pl.ut_hi, pl.ut_lo, pl.ldn, pl.u_scale);
        if (check_launch() != G2D_OK) return G2D_ERR_CUDA;
    }
    return G2D_OK;
}

static_assert(sizeof(TcMaps) <= sizeof(MacroTcMaps), "opaque tensor-map storage is too small");
constexpr size_t MACRO_SMEM = (size_t)MACRO_STAGES * pair_stage_bytes<128> + PAIR_BOXES + 1024;

// Tensor maps of one sweep (encoded once, reused by every macro update of the sweep) and the kernels' one-time set-up.
int macro_tc_prepare(MacroTcMaps *opaque, const TcPlanes &pl, float *y, float *c, int64_t m, int64_t n, int64_t ld) {
    TcMaps &maps = *reinterpret_cast<TcMaps *>(opaque);
    if (!make_map_16(&maps.l_hi, pl.l_hi, m, m, MT, false, pl.ldm) || !make_map_16(&maps.l_lo, pl.l_lo, m, m, MT, false, pl.ldm) ||
        !make_map_16(&maps.c_hi, pl.c_hi, m, n, MT, false, pl.ldn) || !make_map_16(&maps.c_lo, pl.c_lo, m, n, MT, false, pl.ldn) ||
        !make_map_16(&maps.et_hi, pl.et_hi, n, m, MT, false, pl.ldm) || !make_map_16(&maps.et_lo, pl.et_lo, n, m, MT, false, pl.ldm) ||
        !make_map_16(&maps.ut_hi, pl.ut_hi, n, n, MT, false, pl.ldn) || !make_map_16(&maps.ut_lo, pl.ut_lo, n, n, MT, false, pl.ldn) ||
        !make_map(&maps.y, y, m, n, 32, ld) || !make_map(&maps.c, c, m, n, 32, ld))
        return G2D_ERR_CUDA;
    static PerDeviceOnce configured;
    return configured.run([&] { return cudaFuncSetAttribute(macro_update_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MACRO_SMEM) == cudaSuccess; });
}

// Sources: the macro anti-diagonals s0..s1-1; targets: t_first..s_end-1 (t_first >= s1).
int launch_macro_update_tc(const MacroTcMaps *opaque, const TcPlanes &pl, int64_t m, int64_t n, int s0, int s1, int s_end, cudaStream_t stream, int t_first) {
    const TcMaps &maps = *reinterpret_cast<const TcMaps *>(opaque);
    if (t_first < s1) t_first = s1;
    const int nI2 = (int)ceil_div(m, MT), nJ2 = (int)ceil_div(n, MT);
    if (s_end <= t_first) return G2D_OK;
    const int raster = s_end - t_first > 8 ? 1 : 0;
    dim3 grid((unsigned)(nI2 < nJ2 ? nI2 : nJ2), (unsigned)(s_end - t_first));
    if (raster) {
        const int64_t blocks = ceil_div(nI2, RB_I) * ceil_div(nJ2, RB_J);
        grid = dim3((unsigned)(blocks * RB_I * RB_J), 1);
    }
    const MacroScales scales{pl.l_scale, pl.c_scale, pl.e_scale, pl.u_scale, (int)ceil_div(m, (int64_t)TILE), (int)ceil_div(n, (int64_t)TILE), (int)m, (int)n};
    macro_update_tc_kernel<<<grid, PAIR_THREADS, MACRO_SMEM, stream>>>(maps, scales, nI2, nJ2, s0, s1, t_first, s_end, raster, pl.error_flag);
    return check_launch();
}

}  // namespace g2d

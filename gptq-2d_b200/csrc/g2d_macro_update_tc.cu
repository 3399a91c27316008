// Feedback between macro tiles on the tensor cores (float only): tcgen05.mma kind::f16 on fp16 pairs with accumulators in
// tensor memory, operands brought into shared memory by TMA (cp.async.bulk.tensor, 128-byte swizzle).
//
// A CTA owns one 128 x 128 target macro tile, or 2 x 2 of them, and forms both products of the band update
//     down :  C[I, J] += sum_k L[I, k] E[k, J]      right:  Y[I, J] += sum_k C[I, k] U[k, J]
// over the k ranges that hold the sources of the macro anti-diagonals s0..s1-1 (whole 128-blocks, no masks).
// float32 fidelity comes from the split of every operand into hi + lo with 11 significant bits each under a power of two per
// 64 x 64 tile (see split_half) and three products per k step, hi hi + lo hi + hi lo.  A slice of k is one tile wide, so the
// product of the two tiles' scales is a constant of a slice and of 64 rows and columns: it rides on the additions that
// add the slices up in registers.  All four operand kinds are stored K-major for the MMA: L and C as they are (rows x k), E and U
// transposed (columns x k); the split copies of L and U^T are made once per sweep by the kernels at the end of this file,
// those of E^T and C by the tile sweep as it finishes a tile.
//
// Bound: the L2 and the shared-memory port that operands come through (with tf32 pairs twice the bytes at half the tensor rate),
// and for a short source range what a CTA spends on its first loads and its last results.  Results leave as TMA reductions while the
// next product is multiplied.
#include "g2d_tc.cuh"

namespace g2d {

constexpr int RB_I = 8, RB_J = 16;  // rasterisation block: 128 macro tiles
constexpr int MACRO_STAGES = 3, MACRO_WIDE_STAGES = 2;

struct TcMaps {
    CUtensorMap l_hi, l_lo, c_hi, c_lo;      // [rows][k]
    CUtensorMap et_hi, et_lo, ut_hi, ut_lo;  // [columns][k]
    CUtensorMap y, c;                        // targets, boxes of 16 x 32
};
struct MacroScales {
    const float *l, *c, *e, *u;
    int nI, nJ;  // 64 x 64 tiles
    int m, n;
};

// What a launch covers: sources and targets, in macro tiles.
struct MacroRange {
    int nI2, nJ2, s0, s1, t_first, s_end;  // t_first >= s1
    __host__ __device__ bool target(int I2, int J2) const { return I2 < nI2 && J2 >= 0 && J2 < nJ2 && I2 + J2 >= t_first && I2 + J2 < s_end; }
    // the source macro rows of a target's column `across` (down) or macro columns of its row (right); every one lies before the
    // target, so they do not depend on its other index
    __device__ bool sources(int across, int &k, int &count) const {
        k = max(s0 - across, 0);
        count = s1 - across - k;
        return count > 0;
    }
    // Rasterisation blocks of block row b that can hold a target with a source (I2 or J2 below s1): the first and past the last
    __host__ __device__ void row(int b, int &first, int &last) const {
        const int i_lo = b * RB_I, i_hi = i_lo + RB_I < nI2 ? i_lo + RB_I : nI2;
        int j_lo = t_first - (i_hi - 1), j_hi = s_end - i_lo;
        if (j_lo < 0) j_lo = 0;
        if (j_hi > nJ2) j_hi = nJ2;
        if (i_lo >= s1 && j_hi > s1) j_hi = s1;
        first = j_lo / RB_J;
        last = j_hi > j_lo ? (j_hi + RB_J - 1) / RB_J : first;
    }
};

// Few anti-diagonals of targets: one macro tile per CTA, the down product and then the right one.  It is the part of a far update
// that the tile launches wait for, so what counts is that it ends soon.
__global__ void __launch_bounds__(PAIR_THREADS, 1) macro_update_tc_kernel(const __grid_constant__ TcMaps maps, const MacroScales S, const MacroRange R,
                                                                          int *error_flag) {
    constexpr int NT = 128, MINE = NT / 2;
    extern __shared__ unsigned char tc_smem_raw[];
    __shared__ __align__(8) PairRing<MACRO_STAGES> ring;
    const int I2 = blockIdx.y, J2 = R.t_first - I2 + (int)blockIdx.x;
    int k, macros;
    if (!R.target(I2, J2) || (!R.sources(J2, k, macros) && !R.sources(I2, k, macros))) return;
    const uint32_t smem_base = (smem_u32(tc_smem_raw) + 1023u) & ~1023u;
    auto next = [&, which = 0](int, PairTile &t) mutable {
        for (; which < 2; ++which) {
            int k, macros;
            if (R.sources(which ? I2 : J2, k, macros)) {
                t = PairTile{I2 * MT, J2 * MT, macros * (MT / KH), k * MT, which++};
                return true;
            }
        }
        return false;
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
            // one CTA owns each target entry, so the reduction needs no read-back and stays deterministic; what lies outside the
            // matrix is not written
            const int x = t.j0 + c0 + cb * 32;
            add_block<false>(t.which ? &maps.y : &maps.c, box, lane, total + cb * 32, 1.f, x, t.i0 + q * 32, x < S.n, S.m);
        }
    };
    const bool failed = pair_gemm<NT, MACRO_STAGES, 1>(ring, smem_base, next, load, finish, scale);
    if (threadIdx.x == 0 && failed && error_flag) atomicExch(error_flag, 1);
}

// Many anti-diagonals: 2 x 2 macro tiles per CTA as four products of M = 128, N = 256.  The source range of a down product depends
// on the column only, so two macro rows share it (the product is formed transposed, C^T = E^T L^T, which puts them on the N side),
// and that of a right product on the row only.  Wide products leave the shared-memory port at 80 % of the tensor rate instead of
// 60 %, and four of them per CTA hide what a CTA spends on its first loads and its last results: alone on the GPU at 8192 x 28672
// 233 TFLOP/s with a macro tile per CTA, 304 now (rank 512; 386 at rank 1024).  A target outside the launch's anti-diagonals is multiplied but not written.
// The targets are walked in RB_I x RB_J blocks, block row after block row, so that the CTAs resident at one time share
// their row and column strips in L2.
__global__ void __launch_bounds__(PAIR_THREADS, 1) macro_update_wide_kernel(const __grid_constant__ TcMaps maps, const MacroScales S, const MacroRange R,
                                                                            int *error_flag) {
    constexpr int NT = 256, MINE = NT / 2, SHARES = RB_I * RB_J / 4;
    extern __shared__ unsigned char tc_smem_raw[];
    __shared__ __align__(8) PairRing<MACRO_WIDE_STAGES> ring;
    int block = (int)blockIdx.x / SHARES, row = 0, first, last;
    for (R.row(0, first, last); block >= last - first; R.row(++row, first, last)) block -= last - first;
    const int within = (int)blockIdx.x % SHARES;
    const int I2 = row * RB_I + within / (RB_J / 2) * 2, J2 = (first + block) * RB_J + within % (RB_J / 2) * 2;
    // product x: down into column J2 + x, right into row I2 + x - 2
    auto product = [&](int x, PairTile &t) {
        const int which = x >> 1, half = x & 1;
        const bool wanted = which ? R.target(I2 + half, J2) || R.target(I2 + half, J2 + 1) : R.target(I2, J2 + half) || R.target(I2 + 1, J2 + half);
        int k, macros;
        if (!wanted || !R.sources((which ? I2 : J2) + half, k, macros)) return false;
        t = PairTile{((which ? I2 : J2) + half) * MT, (which ? J2 : I2) * MT, macros * (MT / KH), k * MT, which};
        return true;
    };
    PairTile any;
    if (!product(0, any) && !product(1, any) && !product(2, any) && !product(3, any)) return;
    const uint32_t smem_base = (smem_u32(tc_smem_raw) + 1023u) & ~1023u;
    auto next = [&, x = 0](int, PairTile &t) mutable {
        while (x < 4)
            if (product(x++, t)) return true;
        return false;
    };
    auto load = [&](const PairTile &t, int ch, uint32_t dst, uint64_t *bar) {
        const int k = t.k0 + ch * KH;
        tma_load_2d(dst, t.which ? &maps.c_hi : &maps.et_hi, k, t.i0, bar);
        tma_load_2d(dst + HTILE_BYTES, t.which ? &maps.c_lo : &maps.et_lo, k, t.i0, bar);
        for (int h = 0; h < 2; ++h) {
            tma_load_2d(dst + (2 + h) * HTILE_BYTES, t.which ? &maps.ut_hi : &maps.l_hi, k, t.j0 + h * MT, bar);
            tma_load_2d(dst + (4 + h) * HTILE_BYTES, t.which ? &maps.ut_lo : &maps.l_lo, k, t.j0 + h * MT, bar);
        }
    };
    auto scale = [&](const PairTile &t, int slice, int q, int column) {
        const int k = t.k0 / TILE + slice, a = t.i0 / TILE + (q >> 1), b = (t.j0 + column) / TILE;
        if (t.which) return S.c[(int64_t)min(a, S.nI - 1) * S.nJ + k] * S.u[(int64_t)min(b, S.nJ - 1) * S.nJ + k];
        return S.l[(int64_t)min(b, S.nI - 1) * S.nI + k] * S.e[(int64_t)k * S.nJ + min(a, S.nJ - 1)];
    };
    auto finish = [&](const PairTile &t, int q, int lane, int c0, float (&total)[MINE], uint32_t box) {
        // the warp's columns lie in one macro tile
        const int fixed = t.i0 / MT, moving = (t.j0 + c0) / MT;
        if (!(t.which ? R.target(fixed, moving) : R.target(moving, fixed))) return;
#pragma unroll
        for (int cb = 0; cb < MINE / 32; ++cb) {
            const int a = t.i0 + q * 32, b = t.j0 + c0 + cb * 32;
            if (t.which) add_block<false>(&maps.y, box, lane, total + cb * 32, 1.f, b, a, b < S.n, S.m);
            else add_block<true>(&maps.c, box, lane, total + cb * 32, 1.f, a, b, a < S.n, S.m);
        }
    };
    const bool failed = pair_gemm<NT, MACRO_WIDE_STAGES, 1>(ring, smem_base, next, load, finish, scale);
    if (threadIdx.x == 0 && failed && error_flag) atomicExch(error_flag, 1);
}

// ---- far products with wide tiles (see TcPlanes), in float32 from the float values ----
// A few CTAs behind every far update, which leave again where the sweep has no wide tile (a load: about 2 us beside the tile launch
// of the moment; behind the near updates, which the tile launches wait for sooner, the same launch took 1.5 % of a sweep).
// Else each walks over the targets, looks for sources among the wide tiles and adds their products, 64 x 64 targets at a time, 4 x 4 per
// thread, both operands of a source tile staged whole.  One CTA owns each target and the launch follows its update on one stream: a
// fixed order of additions.  The rare path: FFMA, about a tenth of the tensor cores' rate.
constexpr int WTH = 256, WLD = TILE + 4;
__global__ void __launch_bounds__(WTH) wide_update_kernel(TcPlanes P, MacroRange R, float *y, float *c, int m, int n) {
    __shared__ __align__(16) float As[TILE * WLD], Bs[TILE * WLD];
    __shared__ int wide;  // one answer for the CTA: the tile launch of the moment may be counting
    if (threadIdx.x == 0) wide = *P.wide_count;
    __syncthreads();
    if (wide == 0) return;
    const int nI = (m + TILE - 1) / TILE, nJ = (n + TILE - 1) / TILE, longest = min(nI, nJ);
    const int d0 = 2 * R.t_first, d1 = min(2 * R.s_end, nI + nJ - 2);  // tile anti-diagonals that can hold targets
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    for (int64_t at = blockIdx.x; at < (int64_t)(d1 - d0 + 1) * longest; at += gridDim.x) {
        const int d = d0 + (int)(at / longest), TI = max(0, d - nJ + 1) + (int)(at % longest), TJ = d - TI;
        if (TI >= nI || TJ < 0 || !R.target(TI >> 1, TJ >> 1)) continue;
        const int64_t i0 = (int64_t)TI * TILE, j0 = (int64_t)TJ * TILE;
        for (int right = 0; right < 2; ++right) {
            int k0, macros;
            if (!R.sources((right ? TI : TJ) >> 1, k0, macros)) continue;
            float acc[4][4] = {};
            bool any = false;
            for (int k = 2 * k0; k < 2 * (k0 + macros); ++k) {
                if ((right ? P.c_scale[(int64_t)TI * nJ + k] : P.e_scale[(int64_t)k * nJ + TJ]) >= 0.f) continue;  // the same for the whole CTA
                any = true;
                const int64_t kk = (int64_t)k * TILE;
                const float *const a = right ? P.c + i0 * P.ld + kk : P.l + i0 * P.ldl + kk, *const b = right ? P.u + kk * P.ldu + j0 : P.e + kk * P.ld + j0;
                const int64_t lda = right ? P.ld : P.ldl, ldb = right ? P.ldu : P.ld;
                __syncthreads();  // the products before have been formed
                for (int idx = tid; idx < TILE * TILE; idx += WTH) {
                    const int r = idx / TILE, x = idx % TILE;
                    As[x * WLD + r] = i0 + r < m ? a[r * lda + x] : 0.f;
                    Bs[r * WLD + x] = j0 + x < n ? b[r * ldb + x] : 0.f;
                }
                __syncthreads();
#pragma unroll 8
                for (int x = 0; x < TILE; ++x) {
                    const float4 p = *reinterpret_cast<const float4 *>(As + x * WLD + ty * 4), q = *reinterpret_cast<const float4 *>(Bs + x * WLD + tx * 4);
                    const float pv[4] = {p.x, p.y, p.z, p.w}, qv[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                    for (int r = 0; r < 4; ++r)
#pragma unroll
                        for (int s = 0; s < 4; ++s) acc[r][s] = fmaf(pv[r], qv[s], acc[r][s]);
                }
            }
            if (!any) continue;
            float *const out = right ? y : c;
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    if (i0 + ty * 4 + r < m && j0 + tx * 4 + s < n) out[(i0 + ty * 4 + r) * P.ld + j0 + tx * 4 + s] += acc[r][s];
        }
    }
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
            const unsigned size = __float_as_uint(v[x]) & 0x7fffffffu;
            most = max(most, size < 0x7f800000u ? size : 0u);  // infinities and NaN stay what they are under any scale
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

static_assert(sizeof(TcMaps) <= sizeof(MacroTcMaps::bytes), "opaque tensor-map storage is too small");
constexpr size_t MACRO_SMEM = (size_t)MACRO_STAGES * pair_stage_bytes<128> + PAIR_BOXES + 1024;
constexpr size_t MACRO_WIDE_SMEM = (size_t)MACRO_WIDE_STAGES * pair_stage_bytes<256> + PAIR_BOXES + 1024;

// Tensor maps of one sweep (encoded once, reused by every macro update of the sweep) and the kernels' one-time set-up.
int macro_tc_prepare(MacroTcMaps *opaque, const TcPlanes &pl, float *y, float *c, int64_t m, int64_t n, int64_t ld) {
    TcMaps &maps = *reinterpret_cast<TcMaps *>(opaque);
    opaque->y = y;
    opaque->c = c;
    if (!make_map_16(&maps.l_hi, pl.l_hi, m, m, MT, false, pl.ldm) || !make_map_16(&maps.l_lo, pl.l_lo, m, m, MT, false, pl.ldm) ||
        !make_map_16(&maps.c_hi, pl.c_hi, m, n, MT, false, pl.ldn) || !make_map_16(&maps.c_lo, pl.c_lo, m, n, MT, false, pl.ldn) ||
        !make_map_16(&maps.et_hi, pl.et_hi, n, m, MT, false, pl.ldm) || !make_map_16(&maps.et_lo, pl.et_lo, n, m, MT, false, pl.ldm) ||
        !make_map_16(&maps.ut_hi, pl.ut_hi, n, n, MT, false, pl.ldn) || !make_map_16(&maps.ut_lo, pl.ut_lo, n, n, MT, false, pl.ldn) ||
        !make_map(&maps.y, y, m, n, HALF_BOX_ROWS, ld) || !make_map(&maps.c, c, m, n, HALF_BOX_ROWS, ld))
        return G2D_ERR_CUDA;
    static PerDeviceOnce configured;
    return configured.run([&] {
        return cudaFuncSetAttribute(macro_update_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MACRO_SMEM) == cudaSuccess &&
               cudaFuncSetAttribute(macro_update_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MACRO_WIDE_SMEM) == cudaSuccess;
    });
}

// Sources: the macro anti-diagonals s0..s1-1; targets: t_first..s_end-1 (t_first >= s1).
int launch_macro_update_tc(const MacroTcMaps *opaque, const TcPlanes &pl, int64_t m, int64_t n, int s0, int s1, int s_end, cudaStream_t stream, int t_first) {
    const TcMaps &maps = *reinterpret_cast<const TcMaps *>(opaque);
    if (t_first < s1) t_first = s1;
    if (s_end <= t_first) return G2D_OK;
    const MacroRange range{(int)ceil_div(m, MT), (int)ceil_div(n, MT), s0, s1, t_first, s_end};
    const MacroScales scales{pl.l_scale, pl.c_scale, pl.e_scale, pl.u_scale, (int)ceil_div(m, (int64_t)TILE), (int)ceil_div(n, (int64_t)TILE), (int)m, (int)n};
    // The wide kernel's CTAs take about 60 us each: they need to be several per SM, or the launch ends in a long last wave and the
    // tile launches wait for SMs (2048 x 2048: 1.94 ms against 1.88).  Up to RB_I anti-diagonals its blocks would be nearly empty.
    int64_t blocks = 0;
    if (s_end - t_first > RB_I)
        for (int b = 0, first, last; b * RB_I < range.nI2; ++b) {
            range.row(b, first, last);
            blocks += last - first;
        }
    if (blocks * (RB_I * RB_J / 4) < 4 * 148) {
        if (range.nI2 > 65535) return G2D_ERR_TOO_LARGE;
        macro_update_tc_kernel<<<dim3((unsigned)(s_end - t_first), (unsigned)range.nI2), PAIR_THREADS, MACRO_SMEM, stream>>>(maps, scales, range, pl.error_flag);
    } else {
        macro_update_wide_kernel<<<(unsigned)(blocks * (RB_I * RB_J / 4)), PAIR_THREADS, MACRO_WIDE_SMEM, stream>>>(maps, scales, range, pl.error_flag);
    }
    if (check_launch() != G2D_OK) return G2D_ERR_CUDA;
    wide_update_kernel<<<2 * 148, WTH, 0, stream>>>(pl, range, opaque->y, opaque->c, (int)m, (int)n);
    return check_launch();
}

}  // namespace g2d

// Band update: apply the errors of the stages s0..s1-1 to the stages s1..s_end-1 as dense products.
//
//     down :  C[i, j] += sum_k L[i, k] E[k, j]   over the sources (k, j) of the band
//     right:  Y[i, j] += sum_k C[i, k] U[k, j]   over the sources (i, k) of the band
//
// with stage(i, j) = i / P + j / Q.  This is the work of _repack_errors_kernel + _flush_down_kernel +
// _flush_right_kernel of the reference (gptq_2d.py:632-1057).  The errors stay in their natural
// [m, n] layout and there is no repacking pass.  In tile mode (P = Q = TILE, used by the fused sweep) stages are tile
// anti-diagonals, every operand block is either wholly inside or wholly outside the band and the k range of a target
// tile is exact; the plain (P = Q = 1) and general modes serve the generic path with masks (second kernel).
//
// Tile mode: one CTA of 64 threads owns one 64 x 64 target tile; each thread accumulates 8 x 8 outputs in
// registers, operands are staged 16 k at a time.
#include "g2d_common.cuh"

namespace g2d {

constexpr int BT = 64;       // target tile edge
constexpr int BK = 16;       // k chunk
constexpr int BTH = 64;      // threads per CTA
constexpr int BLD = BT + 4;  // shared row stride of the staged operands

// Thread (ty, tx) of the 8 x 8 thread grid owns rows ty*4 + {0..3} and 32 + ty*4 + {0..3} (columns likewise with tx),
// so that its shared-memory reads are two 16-byte vectors that never collide with its neighbours'.
__device__ __forceinline__ int own(int t, int x) { return x < 4 ? t * 4 + x : 32 + t * 4 + (x - 4); }

// Edge tiles in tile mode: acc[8][8] += A[i0.., k_lo..k_hi) * B[k_lo..k_hi), j0..) with zeros outside the matrix.
template <typename F>
__device__ __forceinline__ void band_product(F (&acc)[8][8], const F *__restrict__ A, int64_t lda, const F *__restrict__ B, int64_t ldb,
                                             int64_t i0, int64_t j0, int64_t rows, int64_t cols, int64_t k_lo, int64_t k_hi, F *As, F *Bs) {
    const int tid = threadIdx.x, ty = tid >> 3, tx = tid & 7;
    for (int64_t k0 = k_lo; k0 < k_hi; k0 += BK) {
        // stage A transposed (As[kk][row]) and B (Bs[kk][col])
        for (int idx = tid; idx < BT * BK; idx += BTH) {
            const int row = idx / BK, kk = idx % BK;
            As[kk * BLD + row] = i0 + row < rows && k0 + kk < k_hi ? A[(i0 + row) * lda + k0 + kk] : (F)0;
        }
        for (int idx = tid; idx < BT * BK; idx += BTH) {
            const int kk = idx / BT, col = idx % BT;
            Bs[kk * BLD + col] = j0 + col < cols && k0 + kk < k_hi ? B[(k0 + kk) * ldb + j0 + col] : (F)0;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            F a[8], b[8];
#pragma unroll
            for (int x = 0; x < 8; ++x) a[x] = As[kk * BLD + own(ty, x)];
#pragma unroll
            for (int y = 0; y < 8; ++y) b[y] = Bs[kk * BLD + own(tx, y)];
#pragma unroll
            for (int x = 0; x < 8; ++x)
#pragma unroll
                for (int y = 0; y < 8; ++y) acc[x][y] += a[x] * b[y];
        }
        __syncthreads();
    }
}

template <typename F>
__device__ __forceinline__ void ld4(const F *p, F (&v)[4]);
template <>
__device__ __forceinline__ void ld4<float>(const float *p, float (&v)[4]) {
    const float4 t = *reinterpret_cast<const float4 *>(p);
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
template <>
__device__ __forceinline__ void ld4<double>(const double *p, double (&v)[4]) {
    const double2 a = *reinterpret_cast<const double2 *>(p), b = *reinterpret_cast<const double2 *>(p + 2);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
template <typename F>
__device__ __forceinline__ void st4(F *p, const F (&v)[4]);
template <>
__device__ __forceinline__ void st4<float>(float *p, const float (&v)[4]) {
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
template <>
__device__ __forceinline__ void st4<double>(double *p, const double (&v)[4]) {
    *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
    *reinterpret_cast<double2 *>(p + 2) = make_double2(v[2], v[3]);
}

// Interior tiles in tile mode: no masks, 16-byte vector loads, the next k chunk travels from global memory to
// registers while the current one is multiplied out of shared memory (two shared buffers, one barrier per chunk).
// Thread (ty, tx) owns rows ty*4 + {0..3} and 32 + ty*4 + {0..3}, columns tx*4 + {0..3} and 32 + tx*4 + {0..3}:
// acc[x][y] with x, y < 4 the first group and >= 4 the second.
template <typename F>
__device__ __forceinline__ void band_product_fast(F (&acc)[8][8], const F *__restrict__ A, int64_t lda, const F *__restrict__ B,
                                                  int64_t ldb, int64_t i0, int64_t j0, int64_t k_lo, int64_t k_hi, F *As, F *Bs) {
    const int tid = threadIdx.x, ty = tid >> 3, tx = tid & 7;
    constexpr int BUF = BK * BLD;
    F ra[4][4], rb[4][4];
    auto fetch = [&](int64_t k0) {
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int id = t * BTH + tid;
            ld4(A + (i0 + (id >> 2)) * lda + k0 + (id & 3) * 4, ra[t]);
            ld4(B + (k0 + (id >> 4)) * ldb + j0 + (id & 15) * 4, rb[t]);
        }
    };
    auto stash = [&](int buf) {
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int id = t * BTH + tid;
            const int row = id >> 2, kq = (id & 3) * 4;
#pragma unroll
            for (int x = 0; x < 4; ++x) As[buf * BUF + (kq + x) * BLD + row] = ra[t][x];
            st4(Bs + buf * BUF + (id >> 4) * BLD + (id & 15) * 4, rb[t]);
        }
    };
    fetch(k_lo);
    stash(0);
    __syncthreads();
    int buf = 0;
    for (int64_t k0 = k_lo; k0 < k_hi; k0 += BK) {
        const bool more = k0 + BK < k_hi;
        if (more) fetch(k0 + BK);
        const F *as = As + buf * BUF, *bs = Bs + buf * BUF;
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            F a[8], b[8];
            F t4[4];
            ld4(as + kk * BLD + ty * 4, t4);
#pragma unroll
            for (int x = 0; x < 4; ++x) a[x] = t4[x];
            ld4(as + kk * BLD + 32 + ty * 4, t4);
#pragma unroll
            for (int x = 0; x < 4; ++x) a[4 + x] = t4[x];
            ld4(bs + kk * BLD + tx * 4, t4);
#pragma unroll
            for (int x = 0; x < 4; ++x) b[x] = t4[x];
            ld4(bs + kk * BLD + 32 + tx * 4, t4);
#pragma unroll
            for (int x = 0; x < 4; ++x) b[4 + x] = t4[x];
#pragma unroll
            for (int x = 0; x < 8; ++x)
#pragma unroll
                for (int y = 0; y < 8; ++y) acc[x][y] += a[x] * b[y];
        }
        if (more) stash(buf ^ 1);
        __syncthreads();
        buf ^= 1;
    }
}

template <typename F>
__global__ void __launch_bounds__(BTH) band_update_kernel(BandArgs<F> P, int nTI, int nTJ, int a_lo) {
    __shared__ __align__(16) F As[2 * BK * BLD];
    __shared__ __align__(16) F Bs[2 * BK * BLD];
    // blockIdx.y selects a target tile anti-diagonal, blockIdx.x a tile on it
    const int A = a_lo + (int)blockIdx.y;
    const int ti_lo = max(0, A - nTJ + 1), ti_hi = min(A + 1, nTI);
    const int TI = ti_lo + (int)blockIdx.x;
    if (TI >= ti_hi) return;
    const int TJ = A - TI;
    const int64_t m = P.m, n = P.n;
    const int64_t i0 = (int64_t)TI * BT, j0 = (int64_t)TJ * BT;
    const int tid = threadIdx.x, ty = tid >> 3, tx = tid & 7;
    // the k ranges of the tile's sources: whole tiles above it (down) and to its left (right)
    int64_t dk_lo = max((P.s0 - TJ) * BT, (int64_t)0), dk_hi = min(min((P.s1 - TJ) * BT, m), (int64_t)TI * BT);
    int64_t rk_lo = max((P.s0 - TI) * BT, (int64_t)0), rk_hi = min(min((P.s1 - TI) * BT, n), (int64_t)TJ * BT);
    if (P.filter == 2 && !((TI & 1) && (TJ & 1))) return;
    if (P.filter == 1) {
        // single-stage use: the down source is tile (dk_lo / 64, TJ), the right source tile (TI, rk_lo / 64)
        if ((TJ & 1) || ((dk_lo / BT) & 1)) dk_hi = dk_lo;
        if ((TI & 1) || ((rk_lo / BT) & 1)) rk_hi = rk_lo;
    }

    for (int64_t batch = blockIdx.z; batch < P.batch; batch += gridDim.z) {
        F *yg = P.y + batch * m * n, *cg = P.c + batch * m * n;
        const F *eg = P.e + batch * m * n;
        const F *lg = P.l + (P.l_off ? P.l_off[batch] : 0);
        const F *ug = P.u + (P.u_off ? P.u_off[batch] : 0);
        // interior tiles take the vectorised, double-buffered product
        const bool fast = i0 + BT <= m && j0 + BT <= n && m % 4 == 0 && n % 4 == 0 &&
                          ((reinterpret_cast<uintptr_t>(yg) | reinterpret_cast<uintptr_t>(cg) | reinterpret_cast<uintptr_t>(eg) |
                            reinterpret_cast<uintptr_t>(lg) | reinterpret_cast<uintptr_t>(ug)) % (4 * sizeof(F)) == 0);
        for (int right = 0; right < 2; ++right) {
            // the right product reads C only on sources of the band, which no CTA of this launch writes
            const int64_t k_lo = right ? rk_lo : dk_lo, k_hi = right ? rk_hi : dk_hi;
            if (k_lo >= k_hi) continue;
            F acc[8][8];
#pragma unroll
            for (int x = 0; x < 8; ++x)
#pragma unroll
                for (int y = 0; y < 8; ++y) acc[x][y] = (F)0;
            const F *a = right ? cg : lg, *b = right ? ug : eg;
            const int64_t lda = right ? n : m;
            if (fast) band_product_fast<F>(acc, a, lda, b, n, i0, j0, k_lo, k_hi, As, Bs);
            else band_product<F>(acc, a, lda, b, n, i0, j0, m, n, k_lo, k_hi, As, Bs);
            F *out = right ? yg : cg;
#pragma unroll
            for (int x = 0; x < 8; ++x) {
                const int64_t i = i0 + own(ty, x);
#pragma unroll
                for (int y = 0; y < 8; ++y) {
                    const int64_t j = j0 + own(tx, y);
                    if (i < m && j < n) out[i * n + j] += acc[x][y];
                }
            }
        }
    }
}

// Band update with element masks (P x Q super-entries, any stages): the flushes of the stage-by-stage engines.
//
// The sources of a target are a window of k that moves with its super-entry column (down) or row (right), so a tile of
// targets takes the union of its windows and zeros outside each: the wider the tile against the band, the more of the union is
// zeros.  Bands of few stages therefore use tiles of 16 rows, wide ones tiles of 64; 256 threads, k in chunks staged in
// shared memory with the next chunk on its way, masks from bounds that a thread computes once for the rows and columns
// it stages (in place of divisions per element: 1 ms per flush before, 10 to 100 us now at 512 x 2048 under 1 x 32
// super-entries).  The terms of a sum keep their order, ascending in k, and the down sum is added before the right one.
// What bounds a flush of few stages is the row of chunks that a CTA takes one after the other: 23 at 512 x 2048 as 1 x 32 (rows of 8 x 32 k
// shifted against each other).  A flush of eight stages there took 45 us with 64-bit bounds, single reads of B and products of zeros, 36 now
// (512 x 2048 as 1 x 32 whole: 4970 us with two CTAs per SM, 4680 with three, 5890 with four).  Fewer threads with 4 x 4 targets read half as
// much from shared memory and are slower (64 x 16 targets 76 us, 128 x 16 63 us).
// SKIP: a warp passes over the chunks outside the windows of its rows.  Worth its branch where the rows of a tile lie in many super-entries:
// 512 x 2048 as 1 x 32 4680 us with and 4890 without it, 256 x 1024 as 4 x 128 1870 and 1830.
constexpr int MTH = 256;
template <typename F, int BM, bool SKIP>
__global__ void __launch_bounds__(MTH, BM == 16 && SKIP ? 3 : 1) band_masked_kernel(BandArgs<F> P) {
    constexpr int CK = sizeof(F) == sizeof(float) ? 32 : 16;  // k per chunk
    constexpr int NR = BM / 16;                               // rows per thread; 4 columns
    constexpr int LA = BM * CK / MTH, LB = 64 * CK / MTH;     // elements of A and B staged per thread
    constexpr int ALD = BM + 1, BLD2 = 64 + 4;
    __shared__ __align__(16) F As[2][CK * ALD];
    __shared__ __align__(16) F Bs[2][CK * BLD2];
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int64_t m = P.m, n = P.n;
    const int64_t i0 = (int64_t)blockIdx.y * BM, i1 = min(i0 + BM, m) - 1;
    for (int64_t batch = blockIdx.z; batch < P.batch; batch += gridDim.z) {
        const int64_t behind = P.skew != nullptr ? P.skew[batch] : 0;
        const int64_t s0 = P.s0 - behind, s1 = P.s1 - behind, s_end = P.s_end - behind;
        // tile columns that can hold targets of these rows start at column block s1 - (last row block)
        const int64_t first = max((int64_t)0, s1 - i1 / P.P) * P.Q / 64;
        const int64_t j0 = (first + blockIdx.x) * 64, j1 = min(j0 + 64, n) - 1;
        if (j0 >= n || i0 / P.P + j0 / P.Q >= s_end || i1 / P.P + j1 / P.Q < s1) continue;
        F *yg = P.y + batch * m * n, *cg = P.c + batch * m * n;
        const F *eg = P.e + batch * m * n;
        const F *lg = P.l + (P.l_off ? P.l_off[batch] : 0);
        const F *ug = P.u + (P.u_off ? P.u_off[batch] : 0);
        bool target[NR][4];
#pragma unroll
        for (int r = 0; r < NR; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int64_t i = i0 + ty * NR + r, j = j0 + tx * 4 + c, st = i / P.P + j / P.Q;
                target[r][c] = i < m && j < n && st >= s1 && st < s_end;
            }
        for (int right = 0; right < 2; ++right) {
            // union of the windows; sources lie in super-entry rows above / columns left of the targets
            const int64_t near_hi = right ? (s1 - i0 / P.P) * P.Q : (s1 - j0 / P.Q) * P.P, far_lo = right ? (s0 - i1 / P.P) * P.Q : (s0 - j1 / P.Q) * P.P;
            const int64_t k_lo = max(far_lo, (int64_t)0), k_hi = right ? min(min(near_hi, n), j1 / P.Q * P.Q) : min(min(near_hi, m), i1 / P.P * P.P);
            if (k_lo >= k_hi) continue;
            // bounds of k, from k_lo on, for the rows of A and the columns of B that this thread stages
            const int count = (int)(k_hi - k_lo);
            const auto place = [&](int64_t k) { return (int)min(max(k - k_lo, (int64_t)0), (int64_t)count); };
            int a_lo[LA], a_hi[LA];
            const F *pa[LA];
#pragma unroll
            for (int t = 0; t < LA; ++t) {
                const int64_t i = i0 + (t * MTH + tid) / CK;
                pa[t] = (right ? cg + i * n : lg + i * m) + k_lo;
                a_lo[t] = right ? place((s0 - i / P.P) * P.Q) : 0;
                a_hi[t] = i >= m ? 0 : place(right ? (s1 - i / P.P) * P.Q : i / P.P * P.P);
            }
            const int64_t jb = j0 + (tid & 63);
            const int b_lo = right ? 0 : place((s0 - jb / P.Q) * P.P);
            const int b_hi = jb >= n ? 0 : place(right ? jb / P.Q * P.Q : (s1 - jb / P.Q) * P.P);
            const F *pb = (right ? ug : eg) + k_lo * n + jb;
            F ra[LA], rb[LB];
            auto fetch = [&](int k0) {
#pragma unroll
                for (int t = 0; t < LA; ++t) {
                    const int k = k0 + (tid & (CK - 1));
                    ra[t] = k >= a_lo[t] && k < a_hi[t] ? pa[t][k] : (F)0;
                }
#pragma unroll
                for (int t = 0; t < LB; ++t) {
                    const int k = k0 + t * (MTH / 64) + (tid >> 6);
                    rb[t] = k >= b_lo && k < b_hi ? pb[k * n] : (F)0;
                }
            };
            // the k of the rows that this warp holds: outside them every product is a zero (the windows of a down product go by columns)
            constexpr int WARP_ROWS = 2 * NR;
            const int64_t row = i0 + (tid >> 5) * WARP_ROWS;
            const int mine_lo = right ? place((s0 - (row + WARP_ROWS - 1) / P.P) * P.Q) : 0, mine_hi = right ? place((s1 - row / P.P) * P.Q) : count;
            auto stash = [&](int buf) {
#pragma unroll
                for (int t = 0; t < LA; ++t) As[buf][(tid & (CK - 1)) * ALD + (t * MTH + tid) / CK] = ra[t];
#pragma unroll
                for (int t = 0; t < LB; ++t) Bs[buf][(t * (MTH / 64) + (tid >> 6)) * BLD2 + (tid & 63)] = rb[t];
            };
            F acc[NR][4];
#pragma unroll
            for (int r = 0; r < NR; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[r][c] = (F)0;
            fetch(0);
            stash(0);
            __syncthreads();
            int buf = 0;
            for (int k0 = 0; k0 < count; k0 += CK) {
                const bool more = k0 + CK < count;
                if (more) fetch(k0 + CK);
                if (!SKIP || (k0 < mine_hi && k0 + CK > mine_lo)) {
#pragma unroll
                    for (int kk = 0; kk < CK; ++kk) {
                        F av[NR], bv[4];
#pragma unroll
                        for (int r = 0; r < NR; ++r) av[r] = As[buf][kk * ALD + ty * NR + r];
                        ld4(&Bs[buf][kk * BLD2 + tx * 4], bv);
#pragma unroll
                        for (int r = 0; r < NR; ++r)
#pragma unroll
                            for (int c = 0; c < 4; ++c) acc[r][c] += av[r] * bv[c];
                    }
                }
                if (more) stash(buf ^ 1);
                __syncthreads();
                buf ^= 1;
            }
#pragma unroll
            for (int r = 0; r < NR; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (target[r][c]) {
                        const int64_t at = (i0 + ty * NR + r) * n + j0 + tx * 4 + c;
                        if (!right) cg[at] += acc[r][c];
                        if (right || P.down_into_y) yg[at] += acc[r][c];
                    }
        }
    }
}

template <typename F>
int launch_band_update(const BandArgs<F> &args, cudaStream_t stream) {
    const unsigned batches = (unsigned)(args.batch < 65535 ? args.batch : 65535);
    if (args.mode == BAND_TILE) {
        const int nTI = (int)ceil_div(args.m, BT), nTJ = (int)ceil_div(args.n, BT);
        if (args.s_end <= args.s1) return G2D_OK;
        dim3 grid((unsigned)(nTI < nTJ ? nTI : nTJ), (unsigned)(args.s_end - args.s1), batches);
        band_update_kernel<F><<<grid, BTH, 0, stream>>>(args, nTI, nTJ, (int)args.s1);
        return check_launch();
    }
    // 64-row tiles when the band's windows are at least as wide as what a tile of that many rows adds to them (512 x 2048 as 1 x 32 with
    // the line at 16, 64 and 256 rows: 5880, 5881 and 5695 us)
    BandArgs<F> a = args;
    if (a.mode == BAND_PLAIN) a.P = a.Q = 1;
    const int BM = (a.s1 - a.s0) * a.P >= 64 || a.m > 16 * 65535 ? 64 : 16;
    int64_t across = ceil_div((a.s_end - a.s1 + BM / a.P + 2) * a.Q, 64) + 2;  // tile columns that the targets of a tile row can touch
    const int64_t all = ceil_div(a.n, 64), down = ceil_div(a.m, BM);
    if (across > all) across = all;
    if (down > 65535) return G2D_ERR_TOO_LARGE;
    dim3 grid((unsigned)across, (unsigned)down, batches);
    const bool skip = BM >= 16 * a.P;
    if (BM == 64) {
        if (skip) band_masked_kernel<F, 64, true><<<grid, MTH, 0, stream>>>(a);
        else band_masked_kernel<F, 64, false><<<grid, MTH, 0, stream>>>(a);
    } else {
        if (skip) band_masked_kernel<F, 16, true><<<grid, MTH, 0, stream>>>(a);
        else band_masked_kernel<F, 16, false><<<grid, MTH, 0, stream>>>(a);
    }
    return check_launch();
}

template int launch_band_update<float>(const BandArgs<float> &, cudaStream_t);
template int launch_band_update<double>(const BandArgs<double> &, cudaStream_t);

}  // namespace g2d

// Factor preparation: the unit (block) lower triangular L with M^{-1} = L Lambda L^T for a symmetric positive
// definite M, i.e. ldl_of_inverse + _unit_diagonal_blocks of the reference (gptq_2d_reference.py:29-49), which
// there is torch.linalg.cholesky + solve_triangular.  Same three steps, blocked by 64 and written for the GPU:
//
//   1. reverse-order Cholesky  M = T^T T  (T lower triangular; T^T is the reference's upper factor Um), from the
//      last block row to the first: factor the diagonal block in one CTA (and invert it), solve the block row to
//      its left as a product with that inverse, subtract the block row's Gram from the part still to factor;
//   2. Lf = T^{-1} (= Um^{-T}) by block forward substitution, one block row per launch:
//      Lf[i, j] = -T[i, i]^{-1} sum_{k = j .. i-1} T[i, k] Lf[k, j],  Lf[i, i] = T[i, i]^{-1};
//   3. out = Lf D^{-1} with D the size x size diagonal blocks of Lf: identity diagonal blocks, zeros above.
//
// M is overwritten (its lower triangle becomes T).  A non-positive pivot stores its 1-based index in *flag.
#include <mutex>

#include <type_traits>

#include "g2d_common.cuh"

namespace g2d {

constexpr int FB = 64;        // block edge
constexpr int FK = 16;        // k chunk of the tile products
constexpr int FLD = FB + 4;   // shared row stride
constexpr int FTH = 64;       // threads of a tile-product CTA (8 x 8 outputs each)

__device__ __forceinline__ int own8(int t, int x) { return x < 4 ? t * 4 + x : 32 + t * 4 + (x - 4); }

// acc[8][8] += sum_{k < K} A(i, k) B(k, j) for the 64 x 64 tile of this CTA; la / lb return 0 outside the matrix.
template <typename F, typename LA, typename LB>
__device__ __forceinline__ void tile_product(F (&acc)[8][8], int64_t K, LA la, LB lb, F *As, F *Bs, bool a_k_contiguous) {
    const int tid = threadIdx.x, ty = tid >> 3, tx = tid & 7;
    for (int64_t k0 = 0; k0 < K; k0 += FK) {
        F ra[FB * FK / FTH], rb[FB * FK / FTH];
#pragma unroll
        for (int t = 0; t < FB * FK / FTH; ++t) {
            const int idx = t * FTH + tid;
            const int i = a_k_contiguous ? idx / FK : idx % FB, kk = a_k_contiguous ? idx % FK : idx / FB;
            ra[t] = k0 + kk < K ? la(i, k0 + kk) : (F)0;
            const int kb = idx / FB, j = idx % FB;
            rb[t] = k0 + kb < K ? lb(k0 + kb, j) : (F)0;
        }
        __syncthreads();  // the previous chunk has been consumed
#pragma unroll
        for (int t = 0; t < FB * FK / FTH; ++t) {
            const int idx = t * FTH + tid;
            const int i = a_k_contiguous ? idx / FK : idx % FB, kk = a_k_contiguous ? idx % FK : idx / FB;
            As[kk * FLD + i] = ra[t];
            Bs[(idx / FB) * FLD + idx % FB] = rb[t];
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < FK; ++kk) {
            F a[8], b[8];
#pragma unroll
            for (int x = 0; x < 8; ++x) a[x] = As[kk * FLD + own8(ty, x)];
#pragma unroll
            for (int y = 0; y < 8; ++y) b[y] = Bs[kk * FLD + own8(tx, y)];
#pragma unroll
            for (int x = 0; x < 8; ++x)
#pragma unroll
                for (int y = 0; y < 8; ++y) acc[x][y] += a[x] * b[y];
        }
    }
    __syncthreads();
}

// Up to two factorizations advance together, block step by block step, in the same launches (the steps are chains of
// short dependent kernels, so a second matrix rides along almost for free).  Problem z of a launch is blockIdx.y, or
// folded into blockIdx.x where the grid is three-dimensional already.  Block rows are taken in groups of GROUP
// (the trailing update of a tensor-core problem is applied once per group), and the problems are lined up so that
// their groups end at the same steps: with block-row counts rounded up to a multiple of GROUP, the launch for block
// row s of the largest problem serves block row s - (steps - rounded count) of a smaller one.
constexpr int GROUP = 4;
template <typename F>
struct LdlProblem {
    F *a, *out, *tinv, *w;
    int64_t n;
    int *flag;
    int tc;                       // trailing updates of whole groups run on the tensor cores (float)
    __half *pt_hi[2], *pt_lo[2];  // [n][2 GROUP * 64] transposed, scaled split panels of the even and odd pairs of groups
};
template <typename F>
struct LdlBatch {
    LdlProblem<F> p[2];
    int count;
    int steps;  // block rows of the largest problem, rounded up to a multiple of GROUP
};
__host__ __device__ inline int padded_block_rows(int64_t n) { return (int)(ceil_div(ceil_div(n, (int64_t)64), (int64_t)GROUP) * GROUP); }
#define LDL_PROBLEM(z)                                        \
    const LdlProblem<F> Q = (z) ? B.p[1] : B.p[0];            \
    F *const a = Q.a;                                         \
    const int64_t n = Q.n;                                    \
    const int kb = step_down - (B.steps - padded_block_rows(n)); \
    if (kb < 0 || (int64_t)kb * FB >= n) return;

template <typename F>
__device__ __forceinline__ void zero_acc(F (&acc)[8][8]) {
#pragma unroll
    for (int x = 0; x < 8; ++x)
#pragma unroll
        for (int y = 0; y < 8; ++y) acc[x][y] = (F)0;
}

// ---- products with one block row (at most 64 rows): 64 x 64 outputs, 4 x 4 per thread ----
// acc[4][4] += sum_{k < K} A(k, 4 ty ..) B(k, 4 tx ..); both operands are staged whole (float; double in two halves) with
// coalesced rows, so a CTA waits for memory once: these launches are short and the next step waits for them.
constexpr int CTH = 256;
constexpr int CLD = FB + 4;
template <typename F>
constexpr int chain_k = sizeof(F) == 4 ? 64 : 32;
template <typename F, typename LA, typename LB>
__device__ __forceinline__ void chain_product(F (&acc)[4][4], int K, LA la, LB lb, F *As, F *Bs) {
    constexpr int CK = chain_k<F>, PER = CK * FB / CTH;
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    for (int k0 = 0; k0 < K; k0 += CK) {
        F ra[PER], rb[PER];
#pragma unroll
        for (int t = 0; t < PER; ++t) {
            const int idx = t * CTH + tid, k = k0 + idx / FB, c = idx % FB;
            ra[t] = k < K ? la(k, c) : (F)0;
            rb[t] = k < K ? lb(k, c) : (F)0;
        }
        __syncthreads();  // the previous half has been consumed
#pragma unroll
        for (int t = 0; t < PER; ++t) {
            const int idx = t * CTH + tid;
            As[(idx / FB) * CLD + idx % FB] = ra[t];
            Bs[(idx / FB) * CLD + idx % FB] = rb[t];
        }
        __syncthreads();
#pragma unroll 16
        for (int k = 0; k < CK; ++k) {
            F p[4], q[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) p[x] = As[k * CLD + ty * 4 + x];
#pragma unroll
            for (int y = 0; y < 4; ++y) q[y] = Bs[k * CLD + tx * 4 + y];
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int y = 0; y < 4; ++y) acc[x][y] += p[x] * q[y];
        }
    }
}

// ---- step 1a: factor the diagonal block kb (bs x bs), M_kk = T_kk^T T_kk, and invert T_kk ----
// One CTA of 256 threads; sixteen rows are factored at a time, the last ones first.  Warp 0 holds their columns 0 .. r0 + 15 in
// registers, two per lane, and eliminates row after row: the columns of the pivots go through shared memory to all lanes one pivot ahead, the
// pivot row is scaled and stored as a row of T.  Then all threads subtract the rows' Gram from what is left.  At the end four
// warps invert the four 16 x 16 diagonal blocks of T by columns, and two doubling levels join them.  Bound by the chain of 64
// pivots.  A pivot took 290 cycles while its own column had to come through shared memory before its root, 20 thousand of the 37 thousand
// cycles of a block at n = 8192; with every lane forming the next pivot itself the factors of 1024 and 1024 take 590 us in place of 637, 2048 and 3000
// 1.63 ms in place of 1.78, 8192 and 8192 7.08 ms in place of 7.47.
constexpr int DTH = 256;
constexpr int DS = 16;          // rows factored at a time
constexpr int DLDS = FB + 4;    // shared row stride: rows are 16-byte multiples
template <typename F>
constexpr int diag_smem = (int)sizeof(F) * (2 * FB * DLDS + FB * FB / 4);

// sqrt(d), its reciprocal and 1 / d of a pivot.  float: from the reciprocal square root approximation with one Newton-Raphson step
// and a residual correction each, without the branches of the exact divisions: three of those were 500 of a step's 750
// cycles.  Largest error over all mantissas, at exponents from -126 to 127: root 0.5 ulp (0.75 below 2^-124), inverse root
// 1.0, inverse 0.5 (of the subnormal where it is one, as for the division).
__device__ __forceinline__ void pivot_roots(float d, float &root, float &inv_root, float &inv) {
    float r;
    asm("rsqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(d));
    r = fmaf(0.5f * r, fmaf(-(d * r), r, 1.f), r);
    const float s = d * r;
    root = fmaf(fmaf(-s, s, d), 0.5f * r, s);
    inv_root = r;
    const float q = r * r;
    inv = fmaf(fmaf(-d, q, 1.f), q, q);
}
// double: the chain takes the reciprocal only.  Rows are stored as they are and scaled sixteen at a time, a pivot's roots per lane (all
// three roots of a pivot in the chain: 640 x 640 in 64 x 64 blocks 1098 us, 1008 with one barrier per pivot over the whole block).
__device__ __forceinline__ void pivot_roots(double d, double &root, double &inv_root, double &inv) {
    root = d;
    inv_root = 1.0;
    inv = 1.0 / d;
}

// Float: the CTAs behind the first bring the block row's tiles left of the diagonal up to date with the block rows of its group that are
// finished, tile j = blockIdx.x - 1.  They only need the diagonal block after it is factored, so they run beside the factorization
// and a step has two launches.  (With a launch of its own that carried every finished block row into the rest of the group, and launches that wait for
// the last CTA of the one before: 1024 and 1024 797 us against 693, 8192 and 8192 8.77 ms against 7.64, 8192 and 28672 96.0 - 99.5
// against 88.3 - 97.5.  An entry gets the same products in the same order, so the results are the same bits.)
template <typename F>
__device__ __forceinline__ void update_row_tile(const LdlProblem<F> &Q, int kb, int j, F *As, F *Bs) {
    F *const a = Q.a;
    const int64_t n = Q.n, r0 = (int64_t)kb * FB, c0 = (int64_t)j * FB;
    const int last = min(kb / GROUP * GROUP + GROUP, (int)((n + FB - 1) / FB)) - 1;
    if (last <= kb) return;
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    F left[4][4];  // block rows follow, so all 64 rows of this one are there
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) left[x][y] = a[(r0 + ty * 4 + x) * n + c0 + tx * 4 + y];
    for (int k = last; k > kb; --k) {
        const int64_t o = (int64_t)k * FB;
        F acc[4][4] = {};
        chain_product<F>(acc, (int)min((int64_t)FB, n - o), [&](int kk, int i) { return a[(o + kk) * n + r0 + i]; }, [&](int kk, int c) { return a[(o + kk) * n + c0 + c]; }, As, Bs);
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
            for (int y = 0; y < 4; ++y) left[x][y] -= acc[x][y];
    }
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) a[(r0 + ty * 4 + x) * n + c0 + tx * 4 + y] = left[x][y];
}

template <typename F>
__global__ void __launch_bounds__(DTH) ldl_diag_kernel(LdlBatch<F> B, int step_down) {
    after_the_launch_before();
    LDL_PROBLEM(blockIdx.y)
    F *const tinv = Q.tinv;
    int *const flag = Q.flag;
    extern __shared__ __align__(16) unsigned char ldl_smem[];
    F *const S = reinterpret_cast<F *>(ldl_smem);  // the block (lower triangle), later T
    if constexpr (std::is_same<F, float>::value)
        if (blockIdx.x > 0) {
            if ((int)blockIdx.x <= kb) update_row_tile<F>(Q, kb, (int)blockIdx.x - 1, S, S + chain_k<F> * CLD);
            return;
        }
    F *const V = S + FB * DLDS;                    // inverse of T, lower triangle
    F *const Wt = V + FB * DLDS;                   // intermediate product of a doubling level
    __shared__ __align__(16) F column[2][DS];  // the pivot's column of the even and odd steps
    __shared__ F pivots[FB];                   // 1 / T[r][r]
    __shared__ int bad;
    constexpr int VLD = DLDS;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t o = (int64_t)kb * FB;
    const int bs = (int)min((int64_t)FB, n - o);
    if (tid == 0) bad = FB + 1;  // none
    F loaded[FB * FB / DTH];
#pragma unroll
    for (int t = 0; t < FB * FB / DTH; ++t) {
        const int idx = t * DTH + tid, r = idx / FB, c = idx % FB;
        // identity beyond a ragged block: its steps change nothing and the inverse stays finite
        loaded[t] = r < bs && c <= r ? a[(o + r) * n + o + c] : (r >= bs && r == c ? (F)1 : (F)0);
    }
#pragma unroll
    for (int t = 0; t < FB * FB / DTH; ++t) {
        const int idx = t * DTH + tid, r = idx / FB, c = idx % FB;
        S[r * DLDS + c] = loaded[t];
        V[r * VLD + c] = (F)0;
    }
    __syncthreads();
#pragma unroll 1
    for (int r0 = FB - DS; r0 >= 0; r0 -= DS) {
        if (warp == 0) {
            const int owner = r0 & 16;       // first of the lanes that hold the rows' own columns
            const bool second = r0 >= 32;    // columns 32 .. r0 + 15 are there
            const int c0 = second ? lane + 32 : lane, c1 = c0 ^ 32;
            F v0[DS], v1[DS];                // register r: row r0 + r of columns c0 (the set with the rows' own) and c1 (by symmetry where it lies above the diagonal)
#pragma unroll
            for (int r = 0; r < DS; ++r) {
                const int row = r0 + r;
                v0[r] = row >= c0 ? S[row * DLDS + c0] : S[c0 * DLDS + row];
                v1[r] = row >= c1 ? S[row * DLDS + c1] : S[c1 * DLDS + row];
            }
            // Every lane has the pivot's column (w) and the one of the pivot after it (u, not yet updated with this one): a lane
            // then forms the next pivot itself, and the way through shared memory, which brings the column after that, runs beside
            // the pivot's root.
            F w[DS], u[DS];
            if ((lane | 1) == owner + DS - 1) {
#pragma unroll
                for (int r = 0; r < DS; ++r) column[lane & 1][r] = v0[r];
            }
            __syncwarp();
#pragma unroll
            for (int r = 0; r < DS; ++r) {
                w[r] = column[1][r];
                u[r] = column[0][r];
            }
            __syncwarp();
            int worst = FB + 1;
            // The row that is eliminated sits in the last register: a step moves the others up by one, so that all steps are the
            // same instructions and fit the instruction cache.  (fma: left to the compiler, the last row's update can lie in another block of the
            // program than its product, and is rounded twice.)
#pragma unroll 2
            for (int j = DS - 1; j >= 0; --j) {
                F root, inv_root, inv;
                pivot_roots(w[DS - 1], root, inv_root, inv);
                worst = worst > FB && r0 + j < bs && !(w[DS - 1] > (F)0) ? r0 + j + 1 : worst;  // the first: its root makes the later ones NaN
                const F f0 = v0[DS - 1] * inv, f1 = v1[DS - 1] * inv, fu = u[DS - 1] * inv;
                // what lies right of the diagonal is stored along and never read
                F *const row = S + (r0 + j) * DLDS;
                row[c0] = c0 == r0 + j ? root : v0[DS - 1] * inv_root;
                if (second) row[c1] = v1[DS - 1] * inv_root;
                pivots[r0 + j] = inv_root;
                F *const col = column[j & 1];
#pragma unroll
                for (int r = DS - 1; r > 0; --r) v0[r] = fma(-f0, w[r - 1], v0[r - 1]);
                if (lane == owner + j - 2) {
#pragma unroll
                    for (int r = 0; r < DS; ++r) col[r] = v0[r];
                }
                __syncwarp();
#pragma unroll
                for (int r = DS - 1; r > 0; --r) {
                    v1[r] = fma(-f1, w[r - 1], v1[r - 1]);
                    w[r] = fma(-fu, w[r - 1], u[r - 1]);
                }
#pragma unroll
                for (int r = 0; r < DS; ++r) u[r] = col[r];
            }
            if constexpr (sizeof(F) == sizeof(double)) {
                __syncwarp();
                if (lane < DS) {
                    F &diagonal = S[(r0 + lane) * DLDS + r0 + lane];
                    const F root = sqrt(diagonal);
                    diagonal = root;
                    pivots[r0 + lane] = (F)1 / root;
                }
                __syncwarp();
#pragma unroll 4
                for (int r = 0; r < DS; ++r) {
                    F *const row = S + (r0 + r) * DLDS;
                    const F by = pivots[r0 + r];
                    if (lane != r0 + r) row[lane] *= by;
                    if (second && lane + 32 != r0 + r) row[lane + 32] *= by;
                }
            }
            if (lane == 0 && bad > FB) bad = worst;
        }
        __syncthreads();
        if (r0 == 0) break;
        // what is left: M[i][j] -= sum_k T[r0 + k][i] T[r0 + k][j], 4 x 4 entries per thread (the strict upper ones are not read)
        const int ti = (tid / 12) * 4, tj = (tid % 12) * 4;
        if (ti < r0 && tj <= ti) {
            F d[4][4];
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int y = 0; y < 4; ++y) d[x][y] = S[(ti + x) * DLDS + tj + y];
#pragma unroll 4
            for (int k = 0; k < DS; ++k) {
                F p[4], q[4];
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    p[x] = S[(r0 + k) * DLDS + ti + x];
                    q[x] = S[(r0 + k) * DLDS + tj + x];
                }
#pragma unroll
                for (int x = 0; x < 4; ++x)
#pragma unroll
                    for (int y = 0; y < 4; ++y) d[x][y] -= p[x] * q[y];
            }
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int y = 0; y < 4; ++y) S[(ti + x) * DLDS + tj + y] = d[x][y];
        }
        __syncthreads();
    }
    // the panel's CTAs, which need the inverse, take their places while it is formed
    let_the_next_launch_start();
    // inverses of the four diagonal blocks, one per warp, column c per lane: once an entry is known it is subtracted from those
    // below, which move up by one register
    if (warp < FB / DS) {
        const int r0 = warp * DS, c = lane & (DS - 1);
        F x[DS];
#pragma unroll
        for (int r = 0; r < DS; ++r) x[r] = r == c ? (F)1 : (F)0;
#pragma unroll 4
        for (int k = 0; k < DS; ++k) {
            F t[DS - 1];  // T below (r0 + k, r0 + k); past the block's end: read, never used
#pragma unroll
            for (int r = 0; r < DS - 1; ++r) t[r] = S[(r0 + k + 1 + r) * DLDS + r0 + k];
            const F xk = x[0] * pivots[r0 + k];
#pragma unroll
            for (int r = 0; r < DS - 1; ++r) x[r] = x[r + 1] - t[r] * xk;
            V[(r0 + k) * VLD + r0 + c] = xk;  // zero above the diagonal; both halves of the warp store the same
        }
    }
    __syncthreads();
    // doubling: X = -B^{-1} (C A^{-1}) completes pairs of finished blocks; 2 x 2 outputs per thread and round
#pragma unroll 1
    for (int b = DS; b < FB; b *= 2) {
        const int half = b / 2, pairs = FB / (2 * b), cells = pairs * half * half;
        for (int idx = tid; idx < cells; idx += DTH) {  // W = C A^{-1}, C = T[second half rows][first half columns]
            const int p = idx / (half * half), i = (idx / half) % half * 2, j = idx % half * 2, s0 = p * 2 * b, s1 = s0 + b;
            F w[2][2] = {{(F)0, (F)0}, {(F)0, (F)0}};
#pragma unroll 4
            for (int k = 0; k < b; k += 4) {  // the inverse has zeros above its diagonal
                F c0[4], c1[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    c0[e] = S[(s1 + i) * DLDS + s0 + k + e];
                    c1[e] = S[(s1 + i + 1) * DLDS + s0 + k + e];
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const F v0 = V[(s0 + k + e) * VLD + s0 + j], v1 = V[(s0 + k + e) * VLD + s0 + j + 1];
                    w[0][0] += c0[e] * v0; w[0][1] += c0[e] * v1;
                    w[1][0] += c1[e] * v0; w[1][1] += c1[e] * v1;
                }
            }
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int y = 0; y < 2; ++y) Wt[(p * b + i + x) * b + j + y] = w[x][y];
        }
        __syncthreads();
        for (int idx = tid; idx < cells; idx += DTH) {  // X = -B^{-1} W
            const int p = idx / (half * half), i = (idx / half) % half * 2, j = idx % half * 2, s0 = p * 2 * b, s1 = s0 + b;
            F x[2][2] = {{(F)0, (F)0}, {(F)0, (F)0}};
#pragma unroll 4
            for (int k = 0; k < b; k += 4) {
                F v0[4], v1[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    v0[e] = V[(s1 + i) * VLD + s1 + k + e];
                    v1[e] = V[(s1 + i + 1) * VLD + s1 + k + e];
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const F w0 = Wt[(p * b + k + e) * b + j], w1 = Wt[(p * b + k + e) * b + j + 1];
                    x[0][0] -= v0[e] * w0; x[0][1] -= v0[e] * w1;
                    x[1][0] -= v1[e] * w0; x[1][1] -= v1[e] * w1;
                }
            }
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int y = 0; y < 2; ++y) V[(s1 + i + e) * VLD + s0 + j + y] = x[e][y];
        }
        __syncthreads();
    }
    for (int idx = tid; idx < FB * FB; idx += DTH) {
        const int r = idx / FB, c = idx % FB;
        tinv[(int64_t)kb * FB * FB + idx] = (r < bs && c < bs && r >= c) ? V[r * VLD + c] : (F)0;
        if (r < bs && c < bs && r >= c) a[(o + r) * n + o + c] = S[r * DLDS + c];
    }
    if (tid == 0 && bad <= FB && flag) atomicCAS(flag, 0, (int)(o + bad));
}

// ---- step 1b: block row to the left of the diagonal block: T[kb, j] = T_kk^{-T} M'[kb, j] ----
template <typename F>
__global__ void __launch_bounds__(CTH) ldl_trsm_kernel(LdlBatch<F> B, int step_down) {
    after_the_launch_before();
    LDL_PROBLEM(blockIdx.y)
    const F *const tinv = Q.tinv;
    if ((int)blockIdx.x >= kb) return;
    __shared__ __align__(16) F As[chain_k<F> * CLD];
    __shared__ __align__(16) F Bs[chain_k<F> * CLD];
    const int j = blockIdx.x;  // column tile, j < kb
    const int64_t o = (int64_t)kb * FB, c0 = (int64_t)j * FB;
    const int bs = (int)min((int64_t)FB, n - o);
    const F *ti = tinv + (int64_t)kb * FB * FB;
    F acc[4][4] = {};
    // A(k, r) = Tinv[k][r], B(k, col) = M'[o + k][c0 + col]
    chain_product<F>(acc, bs, [&](int k, int r) { return ti[k * FB + r]; }, [&](int k, int col) { return a[(o + k) * n + c0 + col]; }, As, Bs);
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y)
            if (ty * 4 + x < bs) a[(o + ty * 4 + x) * n + c0 + tx * 4 + y] = acc[x][y];
    let_the_next_launch_start();
    if constexpr (std::is_same<F, float>::value) {
        const int kb_lo = kb / GROUP * GROUP;
        if (j >= kb_lo) {
            // the diagonal block of a block row of the group, which is factored one to three steps on: its own tile is all it takes
            F gram[4][4] = {};
            __syncthreads();
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int y = 0; y < 4; ++y) As[(ty * 4 + x) * CLD + tx * 4 + y] = acc[x][y];
            __syncthreads();
#pragma unroll 16
            for (int k = 0; k < FB; ++k) {
                F p[4], q[4];
#pragma unroll
                for (int x = 0; x < 4; ++x) p[x] = As[k * CLD + ty * 4 + x];
#pragma unroll
                for (int y = 0; y < 4; ++y) q[y] = As[k * CLD + tx * 4 + y];
#pragma unroll
                for (int x = 0; x < 4; ++x)
#pragma unroll
                    for (int y = 0; y < 4; ++y) gram[x][y] += p[x] * q[y];
            }
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int y = 0; y < 4; ++y)
                    if (tx * 4 + y <= ty * 4 + x) a[(c0 + ty * 4 + x) * n + c0 + tx * 4 + y] -= gram[x][y];
        }
        // tensor-core problems: the finished block row, transposed and split, is an operand of the group's trailing
        // update (columns left of the group only); rows beyond a ragged block are zero in acc already
        if (Q.tc && j < kb_lo) {
            const int pair = kb / (2 * GROUP);
            __half *hi = pair & 1 ? Q.pt_hi[1] : Q.pt_hi[0], *lo = pair & 1 ? Q.pt_lo[1] : Q.pt_lo[0];
            const int k0 = kb % (2 * GROUP) * FB;
            __syncthreads();
            F *const Ts = As;  // [column][k], row stride 65
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int y = 0; y < 4; ++y) Ts[(tx * 4 + y) * (FB + 1) + ty * 4 + x] = acc[x][y] * SYRK_PANEL_SCALE;
            __syncthreads();
#pragma unroll
            for (int t = 0; t < FB * FB / 8 / CTH; ++t) {
                const int idx = t * CTH + tid, c = idx >> 3, k = (idx & 7) * 8;
                __align__(16) __half h[8];
                __align__(16) __half l[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float v = Ts[c * (FB + 1) + k + e];
                    h[e] = __float2half_rn(v);
                    l[e] = __float2half_rn(v - __half2float(h[e]));
                }
                const int64_t at = (c0 + c) * SYRK_TC_K + k0 + k;
                *reinterpret_cast<uint4 *>(hi + at) = *reinterpret_cast<const uint4 *>(h);
                *reinterpret_cast<uint4 *>(lo + at) = *reinterpret_cast<const uint4 *>(l);
            }
        }
    }
}

// ---- step 1c (double): M'[TI, TJ] -= T[kb, TI]^T T[kb, TJ] for TJ <= TI < kb (lower triangle of tiles) ----
template <typename F>
__global__ void __launch_bounds__(CTH) ldl_syrk_kernel(LdlBatch<F> B, int step_down) {
    after_the_launch_before();
    LDL_PROBLEM(blockIdx.y)
    // tile pairs (TI, TJ), TJ <= TI < kb, in row order
    if ((int64_t)blockIdx.x >= (int64_t)kb * (kb + 1) / 2) return;
    __shared__ __align__(16) F As[chain_k<F> * CLD];
    __shared__ __align__(16) F Bs[chain_k<F> * CLD];
    const int64_t lin = blockIdx.x;
    int TI = (int)((sqrt(8.0 * (double)lin + 1.0) - 1.0) / 2.0);
    while ((int64_t)(TI + 1) * (TI + 2) / 2 <= lin) ++TI;
    while ((int64_t)TI * (TI + 1) / 2 > lin) --TI;
    const int TJ = (int)(lin - (int64_t)TI * (TI + 1) / 2);
    const int64_t o = (int64_t)kb * FB, r0 = (int64_t)TI * FB, c0 = (int64_t)TJ * FB;
    const int bs = (int)min((int64_t)FB, n - o);
    F acc[4][4] = {};
    chain_product<F>(acc, bs, [&](int k, int i) { return a[(o + k) * n + r0 + i]; }, [&](int k, int j) { return a[(o + k) * n + c0 + j]; }, As, Bs);
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        const int64_t r = r0 + ty * 4 + x;
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            const int64_t c = c0 + tx * 4 + y;
            if (c <= r) a[r * n + c] -= acc[x][y];
        }
    }
}

// ---- step 2: Lf = T^{-1} by doubling.  The 64 x 64 diagonal blocks of Lf are the inverted diagonal blocks of T.
// At level b (64, 128, ...) every aligned pair of finished b x b diagonal blocks [A^{-1} 0; . B^{-1}] is completed by
//     X = -B^{-1} (C A^{-1}),   C = T[second half rows, first half columns],
// as two batched tile products over all pairs: W = C A^{-1} into scratch, then X = -B^{-1} W into Lf.  Both inverses
// are lower triangular, which bounds the k range of every output tile. ----
template <typename F>
__global__ void __launch_bounds__(FTH) ldl_copy_diag_inverse_kernel(LdlBatch<F> B) {
    const LdlProblem<F> Q = blockIdx.y ? B.p[1] : B.p[0];
    const F *const tinv = Q.tinv;
    F *const out = Q.out;
    const int64_t n = Q.n;
    const int i = blockIdx.x;
    if ((int64_t)i * FB >= n) return;
    const int64_t r0 = (int64_t)i * FB;
    const int bs = (int)min((int64_t)FB, n - r0);
    for (int idx = threadIdx.x; idx < FB * FB; idx += FTH) {
        const int r = idx / FB, c = idx % FB;
        if (r < bs && c < bs) out[(r0 + r) * n + r0 + c] = tinv[(int64_t)i * FB * FB + idx];
    }
}

// second == false: W[pair block] = C A^{-1};  second == true: Lf[pair block] = -B^{-1} W
template <typename F>
__global__ void __launch_bounds__(FTH) ldl_trinv_level_kernel(LdlBatch<F> B, int64_t b, int pairs, bool second) {
    const LdlProblem<F> Q = (int)blockIdx.x >= pairs ? B.p[1] : B.p[0];
    const F *const a = Q.a;
    F *const w = Q.w, *const out = Q.out;
    const int64_t n = Q.n;
    __shared__ __align__(16) F As[FK * FLD];
    __shared__ __align__(16) F Bs[FK * FLD];
    const int64_t r0 = (int64_t)(blockIdx.x % pairs) * 2 * b, r1 = r0 + b;  // first half rows [r0, r1), second half rows [r1, r2)
    if (r1 >= n) return;
    const int64_t r2 = min(r0 + 2 * b, n);
    const int64_t ti = blockIdx.y, tj = blockIdx.z;  // output tile inside the b x b off-diagonal block
    const int64_t row0 = r1 + ti * FB, col0 = r0 + tj * FB;
    if (row0 >= r2) return;
    const int64_t rows = min((int64_t)FB, r2 - row0);
    F acc[8][8];
    zero_acc(acc);
    if (!second) {
        // W[i][j] = sum_{k >= j} C[i][k] A^{-1}[k][j]: k from the output tile's first column to the end of the first half
        const int64_t k_lo = col0, K = r1 - col0;
        tile_product<F>(acc, K, [&](int r, int64_t k) { return r < rows ? a[(row0 + r) * n + k_lo + k] : (F)0; },
                        [&](int64_t k, int c) { return out[(k_lo + k) * n + col0 + c]; }, As, Bs, true);
    } else {
        // X[i][j] = -sum_{k <= i} B^{-1}[i][k] W[k][j]: k from the start of the second half through the output tile's rows
        const int64_t k_lo = r1, K = min(row0 + FB, r2) - r1;
        tile_product<F>(acc, K, [&](int r, int64_t k) { return r < rows ? out[(row0 + r) * n + k_lo + k] : (F)0; },
                        [&](int64_t k, int c) { return w[(k_lo + k) * n + col0 + c]; }, As, Bs, true);
    }
    const int tid = threadIdx.x, ty = tid >> 3, tx = tid & 7;
    F *dst = second ? out : w;
#pragma unroll
    for (int x = 0; x < 8; ++x) {
        const int r = own8(ty, x);
#pragma unroll
        for (int y = 0; y < 8; ++y)
            if (r < rows) dst[(row0 + r) * n + col0 + own8(tx, y)] = second ? -acc[x][y] : acc[x][y];
    }
}

// ---- step 3: out = Lf D^{-1}.  Everything above the diagonal blocks is zero already (the output starts as zeros and
// only blocks on and below the diagonal are written), so the normalisation proper only sets the diagonal blocks to the
// identity: one thread per row ----
template <typename F>
__global__ void ldl_normalize_kernel(F *out, int64_t n, int size) {
    for (int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; row < n; row += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c0 = row / size * size;
        F *p = out + row * n + c0;
        for (int x = 0; x < size; ++x) p[x] = c0 + x == row ? (F)1 : (F)0;
    }
}

// The normalisation reads the diagonal blocks while other rows are rewritten, so the blocks are copied out first.
template <typename F>
__global__ void ldl_copy_diag_kernel(const F *out, int64_t n, int size, F *dblk, const F *scales) {
    const int64_t total = (n / size) * size * size;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t b = t / ((int64_t)size * size);
        const int r = (int)(t / size % size), c = (int)(t % size);
        dblk[t] = out[(b * size + r) * n + b * size + c] * (scales ? scales[b * size + r] : (F)1);
    }
}

// One CTA walks rows, its threads the column blocks left of the row's diagonal block (no index divisions per entry).  `scales`:
// the rows of an equilibrated problem are scaled back on the way (may be null).
template <typename F>
__global__ void ldl_scale_kernel(F *out, int64_t n, int size, const F *dblk, const F *scales) {
    for (int64_t row = blockIdx.x; row < n; row += gridDim.x) {
        const int64_t below = row / size;  // column blocks strictly left of the diagonal block
        const F scale = scales ? scales[row] : (F)1;
        if (size == 1) {
#pragma unroll 4
            for (int64_t b = threadIdx.x; b < below; b += blockDim.x) out[row * n + b] = out[row * n + b] * scale / dblk[b];
            continue;
        }
        for (int64_t b = threadIdx.x; b < below; b += blockDim.x) {
            F *p = out + row * n + b * size;
            const F *d = dblk + b * size * size;
            // x D = r with D lower triangular: back substitution from the last column of the block
            for (int x = size - 1; x >= 0; --x) {
                F acc = p[x] * scale;
                for (int x2 = x + 1; x2 < size; ++x2) acc -= p[x2] * d[x2 * size + x];
                p[x] = acc / d[x * size + x];
            }
        }
    }
}

// Streams for the look-ahead of the trailing updates: the chain of diagonal blocks and panels on one of the highest priority, the
// bulk of the updates on one of the lowest, so that a kernel of the chain takes the next SM that comes free instead of queueing
// behind a millisecond of update CTAs (on two streams of one priority the two ran one after the other).  Two
// factorizations that a caller runs concurrently on two streams take two lanes (see LaneChoice).  Created on first use per
// device and kept.  A call holds its lane's lock while it enqueues: two host threads whose streams share a lane (more than four
// streams, or one handle such as the per-thread default stream's) would otherwise record and wait for each other's events,
// and a chain could start before its own matrix is there.
struct SideLane {
    cudaStream_t stream = nullptr, chain = nullptr;
    cudaEvent_t panel[4] = {}, near[4] = {}, rest[4] = {}, fork = nullptr, join = nullptr;
    bool ready = false;
    std::mutex busy;
};
static bool build_side_lane(SideLane &l) {
    int least = 0, greatest = 0;
    if (cudaDeviceGetStreamPriorityRange(&least, &greatest) != cudaSuccess) return false;
    auto stream = [](cudaStream_t &s, int priority) { return s || cudaStreamCreateWithPriority(&s, cudaStreamNonBlocking, priority) == cudaSuccess; };
    auto event = [](cudaEvent_t &e) { return e || cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess; };
    bool ok = stream(l.stream, least) && stream(l.chain, greatest) && event(l.fork) && event(l.join);
    for (int k = 0; k < 4 && ok; ++k) ok = event(l.panel[k]) && event(l.near[k]) && event(l.rest[k]);
    return l.ready = ok;
}
// A lane of the current device with its lock held (through `held`), or null.
static SideLane *acquire_side_lane(cudaStream_t caller, std::unique_lock<std::mutex> &held) {
    static std::mutex choosing;
    static SideLane lanes[64][4];
    static LaneChoice choice[64];
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return nullptr;
    SideLane *lane;
    {
        std::lock_guard<std::mutex> lock(choosing);
        lane = &lanes[device][choice[device].pick(caller)];
    }
    held = std::unique_lock<std::mutex>(lane->busy);
    return lane->ready || build_side_lane(*lane) ? lane : nullptr;
}

// Workspace of one problem: inverted diagonal blocks, normalisation blocks, scratch of the doubling steps and, for float, the
// nine operand planes of the tensor-core triangular inverse, two pairs of transposed split panels and their scales.
inline int64_t plane_pitch(int64_t n) { return (n + 7) / 8 * 8; }  // rows of the 16-bit planes are 16-byte multiples (a TMA requirement)
struct LdlLayout {
    size_t tinv, dblk, w, planes, panels, scales, total;
};
static LdlLayout ldl_layout(size_t elem, int64_t n) {
    LdlLayout lay;
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t where = at; at += (bytes + 255) & ~(size_t)255; return where; };
    lay.tinv = take(elem * (size_t)ceil_div(n, (int64_t)FB) * FB * FB);  // [blocks][64][64]
    lay.dblk = take(elem * (size_t)n * FB);                              // [n / size][size][size]
    lay.w = take(elem * (size_t)n * n);                                  // [n][n]
    const bool tc = elem == 4;
    lay.planes = take(tc ? 9 * sizeof(__nv_bfloat16) * (size_t)n * plane_pitch(n) : 0);
    lay.panels = take(tc ? 4 * sizeof(__half) * (size_t)n * SYRK_TC_K : 0);
    lay.scales = take(tc ? sizeof(float) * (size_t)n : 0);
    lay.total = at;
    return lay;
}

// A kernel of the chain: on its stream behind the one before, as a programmatic dependent launch.
template <typename F>
static int launch_chain(void (*kernel)(LdlBatch<F>, int), dim3 grid, int threads, size_t smem, cudaStream_t stream, const LdlBatch<F> &B, int step) {
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = dim3((unsigned)threads);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    if (cudaLaunchKernelEx(&config, kernel, B, step) != cudaSuccess) return G2D_ERR_CUDA;
    return check_launch();
}

template <typename F>
int ldl_run(int count, const int64_t *ns, F *const *as, const int *sizes, F *const *outs, int *flags, void *const *workspaces, cudaStream_t caller) {
    LdlBatch<F> B;
    cudaStream_t st = caller;
    B.count = count;
    B.steps = 0;
    F *dblks[2] = {nullptr, nullptr};
    SyrkTcMaps pt_maps[2][2];
    int64_t n_max = 0;
    bool any_tc = false;
    Equilibration equilibrated{};
    float *scales[2] = {nullptr, nullptr};  // of the equilibrated problems
    int problems = 0;
    LdlLayout layout[2];
    for (int z = 0; z < count; ++z) {
        const int64_t n = ns[z];
        layout[z] = ldl_layout(sizeof(F), n);
        const LdlLayout &lay = layout[z];
        char *ws = (char *)workspaces[z];
        dblks[z] = (F *)(ws + lay.dblk);
        LdlProblem<F> &P = B.p[z];
        P = LdlProblem<F>{as[z], outs[z], (F *)(ws + lay.tinv), (F *)(ws + lay.w), n, flags ? flags + z : nullptr, 0, {nullptr, nullptr}, {nullptr, nullptr}};
        if (std::is_same<F, float>::value) {
            const size_t panel = sizeof(__half) * (size_t)n * SYRK_TC_K;
            for (int k = 0; k < 2; ++k) {
                P.pt_hi[k] = (__half *)(ws + lay.panels + (2 * k) * panel);
                P.pt_lo[k] = (__half *)(ws + lay.panels + (2 * k + 1) * panel);
                if (!syrk_tc_maps(&pt_maps[z][k], P.pt_hi[k], P.pt_lo[k], (float *)as[z], n)) return G2D_ERR_CUDA;
            }
            if (n > GROUP * FB) {  // more than one group: there are trailing updates on the tensor cores
                scales[z] = (float *)(ws + lay.scales);
                equilibrated.a[problems] = (float *)as[z];
                equilibrated.s[problems] = scales[z];
                equilibrated.n[problems++] = n;
            }
            P.tc = 1;
            any_tc = true;
        }
        const int padded = padded_block_rows(n);
        B.steps = padded > B.steps ? padded : B.steps;
        n_max = n > n_max ? n : n_max;
        if (cudaMemsetAsync(outs[z], 0, sizeof(F) * (size_t)n * n, st) != cudaSuccess) return G2D_ERR_CUDA;
    }
    if (problems > 0 && launch_equilibrate(problems, equilibrated, st) != G2D_OK) return G2D_ERR_CUDA;
    if (count == 1) B.p[1] = B.p[0];
    if (flags && cudaMemsetAsync(flags, 0, sizeof(int) * count, st) != cudaSuccess) return G2D_ERR_CUDA;
    // Each step factors one 64-row block row (last first): diagonal block, panel to its left, trailing update.  For double the
    // update of a step is a launch that reaches every row above.  For float (tensor-core problems) it is no launch of its own inside
    // the step's group of GROUP block rows: the panel's CTAs update the group's diagonal blocks, and a block row's other tiles are
    // brought up to date beside the factorization of its diagonal block; the rows above the group are updated from the tensor cores,
    // by two groups at a time (K = 512: an entry of the matrix is read and written half as often as with one, 106 -> 99 ms for the factors of
    // n = 28672 and 8192).  A problem's groups pair up as (p + 1, p), p even, whatever it is factored beside.  Look-ahead, so that the
    // latency-bound kernels of the next groups overlap the bulk of the updates:
    //   * group p + 1 updates only the rows of group p (K = 256), on the chain's stream;
    //   * group p then updates with both groups, in three launches: the rows of group p - 1 on the chain's stream, the rows of the
    //     groups p - 2 and p - 3 (near) and everything above (rest) on a side stream.
    // Group p - 1's own update shares its targets with near(p), which it follows; no other update on the chain meets one on the
    // side stream, so the order of the additions is fixed, hence the result.  A pair writes the panel planes that rest of the pair
    // two before it read, and waits for that.
    static PerDeviceOnce configured;
    if (configured.run([&] { return cudaFuncSetAttribute(ldl_diag_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize, diag_smem<F>) == cudaSuccess; }) != G2D_OK)
        return G2D_ERR_CUDA;
    // Updates on the side stream begin with the third group; without them (and for double) the chain stays on the caller's stream, which
    // saves the two hand-overs (64 x 64 and 64 x 64 in double: 166 us against 146).
    const bool beside = any_tc && B.steps > 2 * GROUP;
    std::unique_lock<std::mutex> held;  // until everything is enqueued
    SideLane *lane = beside ? acquire_side_lane(caller, held) : nullptr;
    if (beside) {
        if (!lane || cudaEventRecord(lane->fork, caller) != cudaSuccess || cudaStreamWaitEvent(lane->chain, lane->fork, 0) != cudaSuccess) return G2D_ERR_CUDA;
        st = lane->chain;
    }
    bool recorded[4] = {false, false, false, false};  // near and rest of the last four groups, where a problem closed a pair
    int newest = -1;                                  // the last group with an update on the side stream
    for (int s = B.steps - 1; s >= 0; --s) {  // block row of the largest problem; smaller problems are lined up by groups
        const int g = s / GROUP;
        // a pair that opens here writes the planes of the pair that closed three groups ago
        if (s % GROUP == GROUP - 1 && recorded[(g + 3) & 3] && cudaStreamWaitEvent(st, lane->rest[(g + 3) & 3], 0) != cudaSuccess) return G2D_ERR_CUDA;
        int64_t panel_tiles = 0, row_tiles = 0;  // row_tiles: of block rows with finished ones in their groups
        for (int z = 0; z < count; ++z) {
            const int kb = s - (B.steps - padded_block_rows(ns[z]));
            if (kb <= 0 || (int64_t)kb * FB >= ns[z]) continue;
            panel_tiles = kb > panel_tiles ? kb : panel_tiles;
            if (B.p[z].tc && kb % GROUP != GROUP - 1 && (int64_t)(kb + 1) * FB < ns[z] && kb > row_tiles) row_tiles = kb;
        }
        int status = launch_chain<F>(ldl_diag_kernel<F>, dim3((unsigned)(1 + row_tiles), count), DTH, diag_smem<F>, st, B, s);
        if (status != G2D_OK) return status;
        if (s == 0) break;
        if (panel_tiles > 0) {
            status = launch_chain<F>(ldl_trsm_kernel<F>, dim3((unsigned)panel_tiles, count), CTH, 0, st, B, s);
            if (status != G2D_OK) return status;
            if constexpr (!std::is_same<F, float>::value) status = launch_chain<F>(ldl_syrk_kernel<F>, dim3((unsigned)(panel_tiles * (panel_tiles + 1) / 2), count), CTH, 0, st, B, s);
            if (status != G2D_OK) return status;
        }
        if (s % GROUP != 0 || !any_tc) continue;
        // the group g is complete: the updates above it, for the tensor-core problems
        SyrkTcTarget next[2], near[2], rest[2];
        int targets = 0, closing = 0, rest_rows = 0;
        bool opens = false;
        for (int z = 0; z < count; ++z) {
            const int kb_lo = s - (B.steps - padded_block_rows(ns[z]));
            if (!B.p[z].tc || kb_lo <= 0) continue;
            constexpr int PER = GROUP * FB / 128;  // tile rows per group
            const int64_t o = (int64_t)kb_lo * FB;
            const int t_all = (int)(o / 128), t_next = t_all - PER, t_near = t_next > 2 * PER ? t_next - 2 * PER : 0;  // t_next >= 0: o is at least a group
            const bool closes = kb_lo / GROUP % 2 == 0;
            const int64_t most = closes ? 2 * GROUP * FB : GROUP * FB;
            SyrkTcTarget t{&pt_maps[z][kb_lo / (2 * GROUP) & 1], (float *)B.p[z].a, ns[z], o, t_next, t_all, closes ? 0 : GROUP * FB, (int)(ns[z] - o < most ? ns[z] - o : most), B.p[z].flag};
            next[targets++] = t;
            opens = opens || !closes;
            if (!closes || t_next == 0) continue;
            t.t_lo = t_near;
            t.t_hi = t_next;
            near[closing] = t;
            t.t_lo = 0;
            t.t_hi = t_near;
            rest[closing++] = t;
            rest_rows += t_near;
        }
        recorded[g & 3] = closing > 0;
        if (targets == 0) continue;
        if (closing > 0) {  // the panels are final
            if (cudaEventRecord(lane->panel[g & 3], st) != cudaSuccess || cudaStreamWaitEvent(lane->stream, lane->panel[g & 3], 0) != cudaSuccess)
                return G2D_ERR_CUDA;
            status = launch_syrk_tc(closing, near, lane->stream);
            if (status != G2D_OK) return status;
            if (cudaEventRecord(lane->near[g & 3], lane->stream) != cudaSuccess) return G2D_ERR_CUDA;
            if (rest_rows > 0) status = launch_syrk_tc(closing, rest, lane->stream);
            if (status != G2D_OK) return status;
            if (cudaEventRecord(lane->rest[g & 3], lane->stream) != cudaSuccess) return G2D_ERR_CUDA;
            newest = g;
        }
        if (opens && recorded[(g + 1) & 3] && cudaStreamWaitEvent(st, lane->near[(g + 1) & 3], 0) != cudaSuccess) return G2D_ERR_CUDA;
        status = launch_syrk_tc(targets, next, st);
        if (status != G2D_OK) return status;
    }
    // everything the side stream did joins the caller's stream before the inverse starts
    if (newest >= 0 && cudaStreamWaitEvent(caller, lane->rest[newest & 3], 0) != cudaSuccess) return G2D_ERR_CUDA;
    if (beside && (cudaEventRecord(lane->join, st) != cudaSuccess || cudaStreamWaitEvent(caller, lane->join, 0) != cudaSuccess)) return G2D_ERR_CUDA;
    st = caller;
    ldl_copy_diag_inverse_kernel<F><<<dim3(B.steps, count), FTH, 0, st>>>(B);
    if (check_launch() != G2D_OK) return G2D_ERR_CUDA;
    // The 64-level for everyone; from the 128-level on, float problems continue on the tensor cores.
    auto ffma_levels = [&](const LdlBatch<F> &batch, int problems, int64_t n_top, int64_t b_first, int64_t b_end) {
        for (int64_t b = b_first; b < n_top && b < b_end; b *= 2) {
            const int64_t pairs = ceil_div(n_top, 2 * b), tiles = b / FB;
            if (tiles > 65535) return (int)G2D_ERR_TOO_LARGE;
            dim3 grid((unsigned)(pairs * problems), (unsigned)tiles, (unsigned)tiles);
            ldl_trinv_level_kernel<F><<<grid, FTH, 0, st>>>(batch, b, (int)pairs, false);
            if (check_launch() != G2D_OK) return (int)G2D_ERR_CUDA;
            ldl_trinv_level_kernel<F><<<grid, FTH, 0, st>>>(batch, b, (int)pairs, true);
            if (check_launch() != G2D_OK) return (int)G2D_ERR_CUDA;
        }
        return (int)G2D_OK;
    };
    int status = ffma_levels(B, count, n_max, FB, any_tc ? 2 * FB : INT64_MAX);
    if (status != G2D_OK) return status;
    if (any_tc && n_max > 2 * FB) {
        FactorPlanes planes[2];
        for (int z = 0; z < count; ++z) {
            const int64_t n = ns[z], ld = plane_pitch(n);
            auto plane = [&](int k) { return (__nv_bfloat16 *)((char *)workspaces[z] + layout[z].planes) + (size_t)k * n * ld; };
            planes[z] = FactorPlanes{(const float *)as[z], (float *)outs[z], plane(0), plane(1), plane(2), plane(3), plane(4), plane(5), plane(6), plane(7), plane(8),
                                     n, ld, flags ? flags + z : nullptr};
        }
        status = launch_trinv_tc(count, planes, st);
        if (status != G2D_OK) return status;
    }
    for (int z = 0; z < count; ++z) {
        const int64_t n = ns[z];
        const int size = sizes[z];
        const int64_t blocks = n < 148 * 16 ? n : 148 * 16;  // rows are dealt out to CTAs
        ldl_copy_diag_kernel<F><<<(unsigned)(ceil_div(n * size, 256) < 148 * 64 ? ceil_div(n * size, 256) : 148 * 64), 256, 0, st>>>(outs[z], n, size, dblks[z], (const F *)scales[z]);
        if (check_launch() != G2D_OK) return G2D_ERR_CUDA;
        ldl_scale_kernel<F><<<(unsigned)blocks, 256, 0, st>>>(outs[z], n, size, dblks[z], (const F *)scales[z]);
        if (check_launch() != G2D_OK) return G2D_ERR_CUDA;
        ldl_normalize_kernel<F><<<(unsigned)ceil_div(n, (int64_t)256), 256, 0, st>>>(outs[z], n, size);
        if (check_launch() != G2D_OK) return G2D_ERR_CUDA;
    }
    return G2D_OK;
}

}  // namespace g2d

using namespace g2d;

static size_t ldl_bytes(int dtype, int64_t n) { return ldl_layout(dtype == G2D_F32 ? 4 : 8, n).total; }

extern "C" int g2d_ldl_workspace_bytes(int dtype, int64_t n, size_t *bytes) {
    if ((dtype != G2D_F32 && dtype != G2D_F64) || n < 0 || !bytes) return G2D_ERR_BAD_ARGUMENT;
    *bytes = ldl_bytes(dtype, n);
    return G2D_OK;
}

static int ldl_check(int dtype, int64_t n, int32_t size, const void *a, const void *out, const void *workspace, size_t workspace_bytes) {
    if ((dtype != G2D_F32 && dtype != G2D_F64) || n <= 0 || size <= 0) return G2D_ERR_BAD_ARGUMENT;
    if (n % size != 0 || size > FB) return size > FB ? G2D_ERR_TOO_LARGE : G2D_ERR_BAD_ARGUMENT;
    if (!a || !out) return G2D_ERR_BAD_ARGUMENT;
    if (!workspace || workspace_bytes < ldl_bytes(dtype, n)) return G2D_ERR_WORKSPACE;
    if (ceil_div(n, FB) > 46000) return G2D_ERR_TOO_LARGE;  // tile pairs of one launch must fit a 1-D grid
    return G2D_OK;
}

extern "C" int g2d_ldl_of_inverse(int dtype, int64_t n, void *a, int32_t size, void *out, int32_t *status_flag, void *workspace,
                                  size_t workspace_bytes, void *stream) {
    if (n == 0 && (dtype == G2D_F32 || dtype == G2D_F64) && size > 0) return G2D_OK;
    const int status = ldl_check(dtype, n, size, a, out, workspace, workspace_bytes);
    if (status != G2D_OK) return status;
    cudaStream_t st = (cudaStream_t)stream;
    const int sizes[1] = {size};
    void *const ws[1] = {workspace};
    if (dtype == G2D_F32) {
        float *as[1] = {(float *)a}, *outs[1] = {(float *)out};
        return ldl_run<float>(1, &n, as, sizes, outs, status_flag, ws, st);
    }
    double *as[1] = {(double *)a}, *outs[1] = {(double *)out};
    return ldl_run<double>(1, &n, as, sizes, outs, status_flag, ws, st);
}

extern "C" int g2d_ldl_of_inverse_pair(int dtype, int64_t n0, void *a0, int32_t size0, void *out0, void *workspace0, size_t workspace0_bytes,
                                       int64_t n1, void *a1, int32_t size1, void *out1, void *workspace1, size_t workspace1_bytes,
                                       int32_t *status_flags, void *stream) {
    int status = ldl_check(dtype, n0, size0, a0, out0, workspace0, workspace0_bytes);
    if (status != G2D_OK) return status;
    status = ldl_check(dtype, n1, size1, a1, out1, workspace1, workspace1_bytes);
    if (status != G2D_OK) return status;
    cudaStream_t st = (cudaStream_t)stream;
    const int64_t ns[2] = {n0, n1};
    const int sizes[2] = {size0, size1};
    void *const ws[2] = {workspace0, workspace1};
    if (dtype == G2D_F32) {
        float *as[2] = {(float *)a0, (float *)a1}, *outs[2] = {(float *)out0, (float *)out1};
        return ldl_run<float>(2, ns, as, sizes, outs, status_flags, ws, st);
    }
    double *as[2] = {(double *)a0, (double *)a1}, *outs[2] = {(double *)out0, (double *)out1};
    return ldl_run<double>(2, ns, as, sizes, outs, status_flags, ws, st);
}

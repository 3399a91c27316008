// The parts of the tile sweep (see g2d_tile_sweep.cu) that its two kernels share.
#pragma once
#include <type_traits>

#include "g2d_common.cuh"

namespace g2d {

// Push coefficients of a 16 x 16 diagonal block, one row per source p: entry [p][dd] is the coefficient that carries
// the value of source p to the receiver dd places further (L[p + dd][p] or U[p][p + dd]), zero for dd = 0 and past the
// block's end.  A lane fetches its row with four 16-byte loads; a row stride of 20 keeps eight lanes on distinct banks.
constexpr int DLD = SUB + 4;            // row stride
constexpr int ROLL = 4;                 // rounding stages per iteration of the stage loop
constexpr int DROWS = (2 * NSUB + 1) * SUB + SUB + 1;  // rows of all eight blocks with 16 zero rows before and 17 behind them
constexpr int SWEEPERS = NSUB;          // warps that sweep: one per sub-tile row
constexpr int HELPERS = NSUB;           // warps that feed them: one per sub-tile row
constexpr int TTH = (SWEEPERS + HELPERS) * 32;  // threads per CTA
// Quantizer parameters of the sub-tiles being swept, by entry, in two planes of pairs: (scale, its reciprocal), which every stage loads, and
// (zero point, result), so that stages without a zero point load half as much.  Both are there twice: the helpers prepare the next
// parameters and write the last results out while a sub-tile anti-diagonal is swept, and not between two.
constexpr int PLD = SUB + 2;            // entries per row of a sub-tile (the walk along an anti-diagonal moves 17 entries: no conflicts)
constexpr int PPLANE = NSUB * SUB * PLD * 2;  // values per plane
constexpr int PPAD = (SUB + 1) * PLD * 2;     // values behind a plane that lanes past their last entry may read (and ignore)

template <typename F>
__device__ __forceinline__ void load4(const F *p, F (&v)[4]);
template <>
__device__ __forceinline__ void load4<float>(const float *p, float (&v)[4]) {
    const float4 t = *reinterpret_cast<const float4 *>(p);
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
template <>
__device__ __forceinline__ void load4<double>(const double *p, double (&v)[4]) {
    const double2 a = *reinterpret_cast<const double2 *>(p), b = *reinterpret_cast<const double2 *>(p + 2);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
template <typename F>
__device__ __forceinline__ void store4(F *p, const F (&v)[4]);
template <>
__device__ __forceinline__ void store4<float>(float *p, const float (&v)[4]) {
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
template <>
__device__ __forceinline__ void store4<double>(double *p, const double (&v)[4]) {
    *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
    *reinterpret_cast<double2 *>(p + 2) = make_double2(v[2], v[3]);
}

// Sixteen bytes to shared memory without passing through registers: the first `bytes` from global memory, then zeros.
__device__ __forceinline__ void async16(void *dst, const void *src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint32_t shared_address(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
// Loads of the stage loop: volatile, so that they stay where they are written (one stage ahead of their use, behind the shuffle).
__device__ __forceinline__ void load4_here(uint32_t at, float (&v)[4]) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(at));
}
__device__ __forceinline__ void load4_here(uint32_t at, double (&v)[4]) {
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "r"(at));
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v[2]), "=d"(v[3]) : "r"(at + 16));
}
__device__ __forceinline__ void load2_here(uint32_t at, float &a, float &b) { asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(a), "=f"(b) : "r"(at)); }
__device__ __forceinline__ void load2_here(uint32_t at, double &a, double &b) { asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(a), "=d"(b) : "r"(at)); }
// A predicated store instead of a branch around a store
__device__ __forceinline__ void store_shared_if(uint32_t at, float v, bool on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.shared.f32 [%0], %1;\n\t}" ::"r"(at), "f"(v), "r"((uint32_t)on));
}
__device__ __forceinline__ void store_shared_if(uint32_t at, double v, bool on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.shared.f64 [%0], %1;\n\t}" ::"r"(at), "d"(v), "r"((uint32_t)on));
}

__device__ __forceinline__ void store16_if(void *at, uint4 v, bool on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\t@p st.global.v4.u32 [%0], {%1, %2, %3, %4};\n\t}" ::"l"(at), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"((uint32_t)on) : "memory");
}

// D += A B with 16 inner terms, all in shared memory with row stride LD; one warp.  The row and column counts of D are 16 x 16,
// 16 x 64 (WIDE) or 64 x 16 (TALL): the strips give a lane 4 x 8 or 8 x 4 outputs and need half the operand loads per
// multiply-add of the small block (2 x 4 outputs per lane), and shared-memory loads are what these products are short of.
enum Shape { SMALL, WIDE, TALL };
// Two neighbouring values, and multiply-adds of pairs: for float one instruction (each half rounded as on its own), which halves the
// instructions that a product issues.
template <typename F>
struct Pair;
template <>
struct Pair<float> {
    unsigned long long v;
    __device__ __forceinline__ static Pair both(float a) {
        Pair r;
        asm("mov.b64 %0, {%1, %1};" : "=l"(r.v) : "f"(a));
        return r;
    }
    __device__ __forceinline__ void add_product(Pair a, Pair b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v) : "l"(a.v), "l"(b.v)); }
};
template <>
struct Pair<double> {
    double v[2];
    __device__ __forceinline__ static Pair both(double a) { return {a, a}; }
    __device__ __forceinline__ void add_product(Pair a, Pair b) {
        v[0] += a.v[0] * b.v[0];
        v[1] += a.v[1] * b.v[1];
    }
};
__device__ __forceinline__ void load4(const float *p, Pair<float> (&v)[2]) {
    const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(p);
    v[0].v = t.x; v[1].v = t.y;
}
__device__ __forceinline__ void load4(const double *p, Pair<double> (&v)[2]) {
    load4(p, *reinterpret_cast<double(*)[4]>(&v));
}
__device__ __forceinline__ void store4(float *p, const Pair<float> (&v)[2]) { *reinterpret_cast<ulonglong2 *>(p) = make_ulonglong2(v[0].v, v[1].v); }
__device__ __forceinline__ void store4(double *p, const Pair<double> (&v)[2]) { store4(p, *reinterpret_cast<const double(*)[4]>(&v)); }

template <int SHAPE, typename F>
__device__ __forceinline__ void mm16(F *__restrict__ D, const F *__restrict__ A, const F *__restrict__ B, int lane) {
    constexpr int NR = SHAPE == SMALL ? 2 : SHAPE == WIDE ? 4 : 8, NC = SHAPE == WIDE ? 2 : 1;  // rows and groups of four columns per lane
    const int r = SHAPE == WIDE ? (lane >> 3) * 4 : SHAPE == TALL ? lane >> 2 : (lane >> 2) * 2, rs = SHAPE == TALL ? 8 : 1;
    const int c = SHAPE == WIDE ? (lane & 7) * 4 : (lane & 3) * 4;
    constexpr int CS = 32;  // distance of a lane's column groups
    Pair<F> d[NR][NC][2];
#pragma unroll
    for (int i = 0; i < NR; ++i)
#pragma unroll
        for (int g = 0; g < NC; ++g) load4(D + (r + i * rs) * LD + c + g * CS, d[i][g]);
    constexpr int KU = 4;  // inner terms per trip
    constexpr int UNROLL = SHAPE == SMALL ? SUB / KU : 2;  // steps per trip: the small product entirely unrolled
#pragma unroll UNROLL
    for (int k0 = 0; k0 < SUB; k0 += KU) {
        F a[NR][KU];
        Pair<F> b[KU][NC][2];
#pragma unroll
        for (int i = 0; i < NR; ++i) load4(A + (r + i * rs) * LD + k0, a[i]);
#pragma unroll
        for (int k = 0; k < KU; ++k)
#pragma unroll
            for (int g = 0; g < NC; ++g) load4(B + (k0 + k) * LD + c + g * CS, b[k][g]);
#pragma unroll
        for (int k = 0; k < KU; ++k)
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                const Pair<F> ai = Pair<F>::both(a[i][k]);
#pragma unroll
                for (int g = 0; g < NC; ++g)
#pragma unroll
                    for (int y = 0; y < 2; ++y) d[i][g][y].add_product(ai, b[k][g][y]);
            }
    }
#pragma unroll
    for (int i = 0; i < NR; ++i)
#pragma unroll
        for (int g = 0; g < NC; ++g) store4(D + (r + i * rs) * LD + c + g * CS, d[i][g]);
}

// What a sweeping warp needs to know of the sub-tile that it takes.
template <typename F>
struct SubTile {
    F *ys, *cs;              // its first entry in Ys and in Cs
    const F *dg_c, *dg_y;    // the first rows of the diagonal blocks of L and of U^T
    F *par;                  // its first entry's quantizer parameters (the second plane PPLANE values behind)
    int rows, cols;          // of the tile inside the matrix, from the sub-tile's first entry on
    F qmin, qmax;
    F *pre;                  // receives the values before rounding (may be null), rows of pre_ld
    int64_t pre_ld;
};
template <typename F, int KIND, int DIVIDE, bool RECORD>
__device__ __forceinline__ void sweep_sub_tile(const SubTile<F> tile, const int lane) {
    const int k = lane & 15, role = lane >> 4;
    // entries of this lane inside the matrix: the first `count` of its column or row
    const int along = role ? tile.cols : tile.rows, count = k < (role ? tile.rows : tile.cols) ? max(0, min(along, SUB)) : 0;
    const int step = role ? 1 : LD;
    F acc[SUB];
    {
        const F *const src = role ? tile.ys + k * LD : tile.cs + k;
#pragma unroll
        for (int r = 0; r < SUB; ++r) acc[r] = src[((r - k) & (SUB - 1)) * step];
    }
    F *const pre_ptr = tile.pre + k;
    const int partner0 = ((role ^ 1) << 4) - k;
    const F qmin = tile.qmin, qmax = tile.qmax;
    uint32_t dg = shared_address(role ? tile.dg_y : tile.dg_c) - (uint32_t)(k * DLD * (int)sizeof(F));
    uint32_t par = shared_address(tile.par) + (uint32_t)((role ? k * PLD - k : k - k * PLD) * 2 * (int)sizeof(F));
    const uint32_t par_bytes = (uint32_t)((role ? 1 : PLD) * 2 * (int)sizeof(F));
    uint32_t own = shared_address(role ? tile.cs + k * LD : tile.ys + k) - (uint32_t)(k * step * (int)sizeof(F));
    constexpr uint32_t second = PPLANE * (uint32_t)sizeof(F);
    F kc[SUB], pa[3];  // push coefficients; scale, reciprocal, zero point
    auto fetch = [&](uint32_t d, uint32_t q, F (&co)[SUB], F (&pq)[3]) {
        F unused;
        if (KIND != G2D_Q_ROUND) load2_here(q, pq[0], pq[1]);
        if (KIND == G2D_Q_AFFINE && DIVIDE != 4) load2_here(q + second, pq[2], unused);
#pragma unroll
        for (int v4 = 0; v4 < SUB; v4 += 4) {
            F t[4];
            load4_here(d + (uint32_t)(v4 * (int)sizeof(F)), t);
#pragma unroll
            for (int x = 0; x < 4; ++x) co[v4 + x] = t[x];
        }
    };
    fetch(dg, par, kc, pa);
    int p = -k;  // place of this lane's entry in its column or row
#pragma unroll 1
    for (int s_first = 0; s_first < 2 * SUB; s_first += ROLL) {
#pragma unroll
        for (int j = 0; j < ROLL; ++j) {
            const bool ok = (unsigned)p < (unsigned)count;
            const F other = __shfl_sync(0xffffffffu, acc[0], partner0 + s_first + j);
            F kc_next[SUB], pa_next[3];
            fetch(dg + (uint32_t)((j + 1) * DLD * (int)sizeof(F)), par + par_bytes, kc_next, pa_next);
            const F yv = acc[0] + other;
            F z, result;  // the rounded value, and what is stored of it: itself or what write_rounded forms it from
            if constexpr (KIND == G2D_Q_AFFINE && DIVIDE >= 3) {
                z = mul_rn(affine_steps_fast<DIVIDE == 4>(yv, pa[0], pa[2], pa[1], qmin, qmax, result), pa[0]);
            } else {
                if (KIND == G2D_Q_AFFINE) {
                    z = DIVIDE == 2 ? affine_value(yv, pa[0], pa[2], qmin, qmax) : affine_value_rcp(yv, pa[0], pa[2], pa[1], qmin, qmax);
                } else if (KIND == G2D_Q_FORCED) {
                    z = pa[0];
                } else {
                    z = rint_even(yv);
                }
                result = z;
            }
            // What is pushed: the error E of the float that is stored (column lanes), the completed C + E (row lanes), in the reference's order.  (Both
            // from the unrounded product of code and scale are one multiply-add where these are a product and two additions, 2 % of a small
            // sweep, but leave up to half an ulp of Z out of the feedback, and an infinite C is then no NaN in what goes to the right.)
            const F carried = (z - yv) + (role ? other : (F)0);
            const F v = ok ? carried : (F)0;     // lanes without an entry push zero
            // the push moves every accumulator down by one register on the way
            const F last = acc[0];
#pragma unroll
            for (int dd = 1; dd < SUB; ++dd) acc[dd - 1] = acc[dd] + kc[dd] * v;
            acc[SUB - 1] = last;
            store_shared_if(own, carried, ok);
            store_shared_if(par + second + (uint32_t)sizeof(F), result, ok);  // both lanes of an entry store the same value
            if (RECORD && ok && !role) pre_ptr[(int64_t)p * tile.pre_ld] = yv;
            own += (uint32_t)(step * (int)sizeof(F));
            par += par_bytes;
            ++p;
#pragma unroll
            for (int x = 0; x < SUB; ++x) kc[x] = kc_next[x];
#pragma unroll
            for (int x = 0; x < 3; ++x) pa[x] = pa_next[x];
        }
        dg += (uint32_t)(ROLL * DLD * (int)sizeof(F));
    }
}

// What the helpers need to know of the tile
template <typename F>
struct Tile {
    int64_t i0, j0, n, ld;               // first row and column; columns of the matrix; row stride of Y
    int rows, cols;                      // inside the matrix
    F *y;                                // of this batch
    const F *scale, *zero, *forced;
    int64_t srs, scs, zrs, zcs;
    bool unfinished;                     // the stages leave the last steps of a result to write_rounded, where scales allow their short form
    bool zvec;                           // rows of Y are vectors
};
// ---- quantizer parameters, prepared by the helper warps ----
// Helper warp h prepares the parameters of the sub-tile that sweeping warp h takes next, and writes out the results of the one that it took
// last: a lane has eight neighbouring entries of a row, 8 (lane % 2) on of row lane / 2.  Scale and zero point per row (column stride 0)
// are one load each, rows that are whole vectors two, anything else eight.  (Two rows apart, an entry at a time, the three
// functions below took a helper 2500 cycles of the 3700 that the shortest sweep lasts; cp.async of single values is worse still.)
// Scale, zero point and, for the affine quantizer, the reciprocal of the scale wait in shared memory by entry, with the
// warp-wide decisions whether every scale is in the range where the reciprocal form of the division is safe and every zero point +0.
constexpr int PR = SUB * SUB / 32;  // entries per helper lane
// Loads that stay where they are written: the compiler moves plain ones down to their use, half a sub-tile sweep later.
__device__ __forceinline__ float load_now(const float *p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double load_now(const double *p) {
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void load4_now(const float *p, float *v) { asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "l"(p)); }
__device__ __forceinline__ void load4_now(const double *p, double *v) {
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "l"(p));
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v[2]), "=d"(v[3]) : "l"(p + 2));
}
__device__ __forceinline__ bool is_positive_zero(float v) { return __float_as_uint(v) == 0u; }
__device__ __forceinline__ bool is_positive_zero(double v) { return __double_as_longlong(v) == 0ll; }
template <typename F>
struct Params {
    F scale[PR], zero[PR];  // forced values in scale
    bool one_scale, one_zero;  // for the whole row
};
template <typename F>
__device__ __forceinline__ void load_param_row(const F *base, int64_t row_stride, int64_t column_stride, int64_t row, int64_t column, int inside, bool one, F (&v)[PR]) {
    const F *at = base + row * row_stride + column * column_stride;
    if (one) {
        v[0] = load_now(at);
    } else if (column_stride == 1 && inside == PR && reinterpret_cast<uintptr_t>(at) % (4 * sizeof(F)) == 0) {
        load4_now(at, v);
        load4_now(at + 4, v + 4);
    } else {
#pragma unroll
        for (int x = 0; x < PR; ++x) v[x] = load_now(at + (x < inside ? x : 0) * column_stride);  // (entries outside the matrix: a value from inside it)
    }
}
// `inside`: how many of the lane's entries are inside the matrix
template <typename F>
__device__ __forceinline__ int params_inside(const Tile<F> &tile, int b, int helper, int lane) {
    const int r = helper * SUB + (lane >> 1), c = b * SUB + (lane & 1) * PR;
    return r < tile.rows ? max(0, min(PR, tile.cols - c)) : 0;
}
template <typename F, int KIND>
__device__ __forceinline__ void fetch_params(const Tile<F> &tile, int w_next, int helper, int lane, Params<F> &v) {
    const int b = w_next - helper;
    if (b < 0 || b >= NSUB || KIND == G2D_Q_ROUND) return;
    const int inside = params_inside(tile, b, helper, lane);
    const int64_t row = tile.i0 + helper * SUB + (lane >> 1), column = tile.j0 + b * SUB + (lane & 1) * PR;
    if (KIND == G2D_Q_AFFINE) {
        v.one_scale = tile.scs == 0;
        v.one_zero = tile.zcs == 0;
        if (inside == 0) return;
        load_param_row(tile.scale, tile.srs, tile.scs, row, column, inside, v.one_scale, v.scale);
        load_param_row(tile.zero, tile.zrs, tile.zcs, row, column, inside, v.one_zero, v.zero);
    } else {
        v.one_scale = false;
        if (inside != 0) load_param_row(tile.forced, tile.n, (int64_t)1, row, column, inside, false, v.scale);
    }
}
// Both without branches on what is the same for the whole call: behind them a warp that is alone waits for every operation by itself
// (950 and 850 cycles in place of 200).
template <typename F, int KIND>
__device__ __forceinline__ void finish_params(const Tile<F> &tile, F *params_at, unsigned *fast_at, int w_next, int helper, int lane, Params<F> &v) {
    const int b = w_next - helper;
    if (b < 0 || b >= NSUB || KIND == G2D_Q_ROUND) return;
    const int inside = params_inside(tile, b, helper, lane);
    F *dst = params_at + ((helper * SUB + (lane >> 1)) * PLD + (lane & 1) * PR) * 2;
    bool normal = true, zeros = true;
#pragma unroll
    for (int x = 0; x < PR; x += 2) {
        F first[4], second[4];
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            const bool in = x + y < inside;
            const F s = KIND == G2D_Q_AFFINE && v.one_scale ? v.scale[0] : v.scale[x + y], z = KIND == G2D_Q_AFFINE ? (v.one_zero ? v.zero[0] : v.zero[x + y]) : (F)0;
            first[2 * y] = in ? s : KIND == G2D_Q_AFFINE ? (F)1 : (F)0;
            second[2 * y] = in ? z : (F)0;
            if (KIND == G2D_Q_AFFINE) {
                normal = normal & reciprocal_is_safe(first[2 * y]);
                zeros = zeros & is_positive_zero(second[2 * y]);
            }
            first[2 * y + 1] = KIND == G2D_Q_AFFINE ? rounding_reciprocal(first[2 * y]) : (F)0;
            second[2 * y + 1] = (F)0;
        }
        store4(dst + x * 2, first);
        if (KIND == G2D_Q_AFFINE) store4(dst + PPLANE + x * 2, second);
    }
    const unsigned fast = (__all_sync(0xffffffffu, normal) ? 1u : 0u) | (__all_sync(0xffffffffu, zeros) ? 2u : 0u);
    if (lane == 0) *fast_at = fast;
}
// The rounded values of the sub-tiles of anti-diagonal w_swept: a helper warp writes out the block of its row.
template <typename F, int KIND>
__device__ __forceinline__ void write_rounded(const Tile<F> &tile, F *params_at, unsigned *fast_at, int w_swept, int helper, int lane) {
    const int b = w_swept - helper;
    if (b < 0 || b >= NSUB) return;
    const int inside = params_inside(tile, b, helper, lane);
    const unsigned how = *fast_at;
    const bool unfinished = tile.unfinished & (how & 1);
    const F *from = params_at + ((helper * SUB + (lane >> 1)) * PLD + (lane & 1) * PR) * 2;
    F *to = tile.y + (tile.i0 + helper * SUB + (lane >> 1)) * tile.ld + tile.j0 + b * SUB + (lane & 1) * PR;
    F v[PR];
#pragma unroll
    for (int x = 0; x < PR; x += 2) {
        F first[4], second[4];
        load4(from + x * 2, first);
        load4(from + PPLANE + x * 2, second);
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            v[x + y] = second[2 * y + 1];
            if constexpr (KIND == G2D_Q_AFFINE && sizeof(F) == sizeof(float)) {
                const F finished = affine_value_after(v[x + y], first[2 * y], second[2 * y], how & 2);
                v[x + y] = unfinished ? finished : v[x + y];
            }
        }
    }
    if (tile.zvec && inside == PR) {
        store4(to, *reinterpret_cast<F(*)[4]>(&v[0]));
        store4(to + 4, *reinterpret_cast<F(*)[4]>(&v[4]));
    } else {
#pragma unroll
        for (int x = 0; x < PR; ++x)
            if (x < inside) to[x] = v[x];
    }
    __syncwarp();  // the next parameters overwrite them
}

// ---- what leaves the tile ----
constexpr int LAST = NSUB - 1;  // row and column of the sub-tile that is swept last
// A block of Yns or Cns that is complete, from the warp that has completed it to the plane of the neighbour.  Rows and columns past the
// matrix are not stored; a row's last group of four may reach into its padding.
template <int ROWS, int COLS, typename F>
__device__ __forceinline__ void push_out(const F *from, F *to, int64_t ld, bool vectors, int rows_inside, int cols_inside, int lane) {
    __syncwarp();
    constexpr int COUNT = ROWS * COLS / 128, DOWN = 128 / COLS;  // vectors per lane, rows from one to the next
    const int r = lane / (COLS / 4), c = lane % (COLS / 4) * 4;
    from += r * LD + c;
    to += r * ld + c;
    if (vectors && rows_inside >= ROWS && cols_inside >= COLS) {
        F v[COUNT][4];
#pragma unroll
        for (int x = 0; x < COUNT; ++x) load4(from + x * DOWN * LD, v[x]);
#pragma unroll
        for (int x = 0; x < COUNT; ++x) store4(to + x * DOWN * ld, v[x]);
        return;
    }
#pragma unroll 1
    for (int x = 0; x < COUNT; ++x) {
        if (r + x * DOWN >= rows_inside || c >= cols_inside) continue;
        F v[4];
        load4(from + x * DOWN * LD, v);
        F *dst = to + x * DOWN * ld;
        if (vectors) store4(dst, v);
        else
            for (int y = 0; y < 4; ++y)
                if (c + y < cols_inside) dst[y] = v[y];
    }
}
// Eight floats, neighbours of a row (C) or of a column (E), times a power of two as fp16 pairs (zeros for a factor of zero, whatever they
// are); stored where `on`.  No branches: a warp that is alone has to overlap its own latencies.
template <bool COLUMN>
__device__ __forceinline__ void split8(const float *from, float by, __half *hi, __half *lo, bool on) {
    float v[8];
    if (COLUMN) {
#pragma unroll
        for (int x = 0; x < 8; ++x) v[x] = from[x * LD];
    } else {
        load4(from, *reinterpret_cast<float(*)[4]>(&v[0]));
        load4(from + 4, *reinterpret_cast<float(*)[4]>(&v[4]));
    }
    const bool zero = by == 0.f;
    __align__(16) __half2 h[4];
    __align__(16) __half2 l[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        const float a = zero ? 0.f : v[2 * x] * by, b = zero ? 0.f : v[2 * x + 1] * by;
        h[x] = __floats2half2_rn(a, b);
        const float2 back = __half22float2(h[x]);
        l[x] = __floats2half2_rn(a - back.x, b - back.y);
    }
    store16_if(hi, *reinterpret_cast<const uint4 *>(h), on);
    store16_if(lo, *reinterpret_cast<const uint4 *>(l), on);
}
// Largest values of rows, columns and the tile (entries outside the matrix are zero), of E in the lower and of C in the upper
// half of a word: the upper halves of floats are all that the scale and the comparison need.
__device__ __forceinline__ unsigned upper_halves(float e, float c) { return __byte_perm(__float_as_uint(e), __float_as_uint(c), 0x7632) & 0x7fff7fffu; }
__device__ __forceinline__ unsigned row_extreme(const float *e, const float *c, int count) {
    unsigned most = 0u;
#pragma unroll 4
    for (int x = 0; x < count; x += 4) {
        float ve[4], vc[4];
        load4(e + x, ve);
        load4(c + x, vc);
#pragma unroll
        for (int y = 0; y < 4; ++y) most = __vmaxu2(most, upper_halves(ve[y], vc[y]));
    }
    return most;
}
__device__ __forceinline__ unsigned column_extreme(const float *e, const float *c, int count) {
    unsigned most = 0u;
#pragma unroll 8
    for (int x = 0; x < count; ++x) most = __vmaxu2(most, upper_halves(e[x * LD], c[x * LD]));
    return most;
}
// `most`: two rows' largest values per lane; `least`: the smaller of these and of two columns', zeros apart.  row_max and column_max hold them
// without the last sub-tile (e and c), which is added here.
__device__ __forceinline__ void last_extremes(const float *e, const float *c, const unsigned *row_max, const unsigned *column_max, int lane, unsigned &most, unsigned &least) {
    // a lane has half a row and half a column: lanes 16 to 31 the second halves
    const int at = lane & 15, half = (lane >> 4) * 8;
    unsigned row = row_extreme(e + at * LD + half, c + at * LD + half, 8), column = column_extreme(e + half * LD + at, c + half * LD + at, 8);
    row = __vmaxu2(row, __shfl_xor_sync(0xffffffffu, row, 16));
    column = __vmaxu2(column, __shfl_xor_sync(0xffffffffu, column, 16));
    const unsigned r0 = row_max[lane], c0 = column_max[lane];
    unsigned r1 = row_max[32 + lane], c1 = column_max[32 + lane];  // lanes 16 to 31: the last sub-tile's
    if (lane >= 16) {
        r1 = __vmaxu2(r1, row);
        c1 = __vmaxu2(c1, column);
    }
    most = __vmaxu2(r0, r1);
    const auto zeros_apart = [](unsigned v) { return v | __vcmpeq2(v, 0u); };
    least = __vminu2(__vminu2(zeros_apart(r0), zeros_apart(r1)), __vminu2(zeros_apart(c0), zeros_apart(c1)));
}
// Barrier 1: the two warps that make the operand planes while the last sub-tile is swept.
__device__ __forceinline__ void early_planes_barrier() { asm volatile("bar.sync 1, 64;" ::: "memory"); }

// floats or doubles of a CTA's shared memory
template <typename F>
constexpr size_t tile_smem = sizeof(F) * (3 * TILE * LD + DROWS * DLD + 4 * PPLANE + (sizeof(F) == sizeof(float) ? 4 * TILE * LD : PPAD));

}  // namespace g2d

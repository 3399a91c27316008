// Shared definitions of the gptq2d_b200 kernels (sm_100a).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <functional>
#include <mutex>

#include "../../include/gptq2d_b200.h"

namespace g2d {

// Geometry of the fused sweep: the matrix is cut into TILE x TILE tiles that are
// swept one tile anti-diagonal at a time; inside a tile, SUB x SUB sub-tiles are
// swept by one warp each, again along anti-diagonals.
constexpr int TILE = 64;
constexpr int SUB = 16;
constexpr int NSUB = TILE / SUB;
constexpr int LD = TILE + 4;  // shared-memory row stride: LD + 1 odd keeps the diagonal walks conflict free

__host__ __device__ inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// IEEE round-to-nearest-even primitives that the compiler may not contract or approximate.
__device__ __forceinline__ float div_rn(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ double div_rn(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float rint_even(float a) { return rintf(a); }
__device__ __forceinline__ double rint_even(double a) { return rint(a); }

// (clamp(rint(y / scale + zp), qmin, qmax) - zp) * scale, every step rounded on its own
// (quantizer_int.py:81-83 / :204-205 of the reference).  Comparisons keep NaN like torch.clamp.
template <typename F>
__device__ __forceinline__ F affine_value(F y, F scale, F zp, F qmin, F qmax) {
    F t = rint_even(add_rn(div_rn(y, scale), zp));
    t = t < qmin ? qmin : t;
    t = t > qmax ? qmax : t;
    return mul_rn(sub_rn(t, zp), scale);
}

// The same value with the division done as a product with a precomputed reciprocal `rc` of the scale plus one
// residual correction: q = y rc, q += (y - q s) rc.  With rc within half an ulp of 1 / scale this is the IEEE
// quotient except, rarely, in its last bit, which can change the result only within one ulp of a rounding tie.
// Used inside the fused float sweep, where the exact division sits on the critical path of every stage.
__device__ __forceinline__ float affine_value_rcp(float y, float scale, float zp, float rc, float qmin, float qmax) {
    const float q0 = y * rc;
    const float q = fmaf(fmaf(-q0, scale, y), rc, q0);
    float t = rintf(__fadd_rn(q, zp));
    t = t < qmin ? qmin : t;
    t = t > qmax ? qmax : t;
    return __fmul_rn(__fsub_rn(t, zp), scale);
}
// The stage loop's form, for bounds that are integers below 2^22 in size: then clamping and rounding commute, and a clamped value is
// rounded half to even by adding and subtracting 1.5 * 2^23, eight cycles instead of the conversion unit's twenty-odd.
// NaN stays NaN as with the comparisons above.  Returns code - zp, whose product with the scale the chain goes on with, and in `clamped` what
// affine_value_after needs to form the value away from the chain: the difference code + 1.5 * 2^23 - 1.5 * 2^23 has lost the sign of a zero
// (a quotient of -0.3 rounds to -0).  ZERO: the zero point is +0, which leaves two additions out of the chain.
template <bool ZERO>
__device__ __forceinline__ float affine_steps_fast(float y, float scale, float zp, float rc, float qmin, float qmax, float &clamped) {
    const float q0 = y * rc;
    float t = fmaf(fmaf(-q0, scale, y), rc, q0);
    if (!ZERO) t = __fadd_rn(t, zp);
    asm("min.NaN.f32 %0, %0, %1;" : "+f"(t) : "f"(qmax));
    asm("max.NaN.f32 %0, %0, %1;" : "+f"(t) : "f"(qmin));
    clamped = t;
    const float code = __fsub_rn(__fadd_rn(t, 12582912.f), 12582912.f);
    return ZERO ? code : __fsub_rn(code, zp);
}
__device__ __forceinline__ float affine_value_after(float clamped, float scale, float zp, bool zero) {
    const float t = zero ? __fadd_rn(clamped, 0.f) : clamped;  // the addition that ZERO has left out: -0 + 0 = 0
    return __fmul_rn(__fsub_rn(copysignf(__fsub_rn(__fadd_rn(t, 12582912.f), 12582912.f), t), zp), scale);
}
// double: `rc` is the correctly rounded reciprocal; two residual corrections make the quotient correctly rounded (the
// first brings it within an ulp, and Markstein's theorem then gives RN(q + r rc) = RN(y / s)).  Same bits as
// affine_value, without the division's hundred-odd cycles on the critical path of every stage.  An infinite quotient (y infinite, or
// beyond the range of doubles in units of the scale) has no residual and stays, to be clamped.
__device__ __forceinline__ double affine_value_rcp(double y, double scale, double zp, double rc, double qmin, double qmax) {
    const double q0 = y * rc;
    double q = fma(fma(-q0, scale, y), rc, q0);
    q = fma(fma(-q, scale, y), rc, q);
    q = fabs(q0) <= 1.7976931348623157e308 ? q : q0;
    double t = rint(__dadd_rn(q, zp));
    t = t < qmin ? qmin : t;
    t = t > qmax ? qmax : t;
    return __dmul_rn(__dsub_rn(t, zp), scale);
}
// The reciprocal that affine_value_rcp takes, and the scales for which neither form leaves the range of normal numbers.
__device__ __forceinline__ float rounding_reciprocal(float s) {
    float v;
    asm("rcp.approx.f32 %0, %1;" : "=f"(v) : "f"(s));
    // one Newton-Raphson step: the correctly rounded reciprocal for every mantissa at the exponents from -100 to 125 that were tried,
    // those of reciprocal_is_safe (-60 to 59) among them; the intrinsic that rounds correctly by contract takes 4 % of a sweep more
    return fmaf(fmaf(-s, v, 1.f), v, v);
}
__device__ __forceinline__ double rounding_reciprocal(double s) { return __drcp_rn(s); }
__device__ __forceinline__ bool reciprocal_is_safe(float s) { return (fabsf(s) > 1e-18f) & (fabsf(s) < 1e18f); }
__device__ __forceinline__ bool reciprocal_is_safe(double s) { return (fabs(s) > 1e-150) & (fabs(s) < 1e150); }

// Largest value over a warp, in every lane.  Non-negative floats order like their bit patterns, so float takes one reduction
// instruction; NaN counts as the smallest, as fmax has it.
__device__ __forceinline__ float warp_max(float v) { return __uint_as_float(__reduce_max_sync(0xffffffffu, v == v ? __float_as_uint(v) : 0u)); }
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// float -> fp16 / bf16 -> float, round to nearest even (denormals kept).
__device__ __forceinline__ float round_to_half(float f, int half_kind) {
    return half_kind == G2D_BF16 ? __bfloat162float(__float2bfloat16_rn(f)) : __half2float(__float2half_rn(f));
}

// absmax / ((qmax - qmin) / 2) rounded to a 16-bit float through fp32, 0 -> 1 (quantizer_int.py:110-117, :357-363).
template <typename F>
__device__ __forceinline__ F absmax_scale_value(F absmax, F divisor, int half_kind) {
    F s = (F)round_to_half((float)div_rn(absmax, divisor), half_kind);
    return s == (F)0 ? (F)1 : s;
}

// Kernel launches made by this library in this process (read by g2d_launch_count); any host thread may launch.
extern std::atomic<unsigned long long> g_launches;
inline int check_launch() {
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaPeekAtLastError() == cudaSuccess ? G2D_OK : G2D_ERR_CUDA;
}

// One-time set-up per device (a kernel's opt-in to more than 48 KB of dynamic shared memory), safe when several host
// threads make their first call at the same time: `setup` runs once per device, under a lock, and must return true.
class PerDeviceOnce {
    std::mutex mutex_;
    bool done_[64] = {};

public:
    template <typename Setup>
    int run(Setup &&setup) {
        int device = 0;
        if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return G2D_ERR_CUDA;
        std::lock_guard<std::mutex> lock(mutex_);
        if (!done_[device]) {
            if (!setup()) return G2D_ERR_CUDA;
            done_[device] = true;
        }
        return G2D_OK;
    }
};

// ---- launchers implemented in the .cu files -------------------------------------------------

template <typename F>
struct SweepArgs {
    F *y, *c, *e;  // [batch, m, n] each: Y = X + right feedback (Z where done), C = down feedback, E = errors
    const F *l, *u;
    const int64_t *l_off, *u_off;
    const F *scale, *zero;
    const int64_t *scale_off, *zero_off;
    int64_t srs, scs, zrs, zcs;
    const F *forced;
    F *y_pre;
    F qmin, qmax;
    int small_integer_bounds = 0;  // qmin and qmax are integers of at most 2^22 in size
    int kind;
    int64_t batch, m, n;
    int nI, nJ;  // tiles per column / per row
    int64_t ld, ldl, ldu;      // row strides of Y, C, E and the float planes; of L; of U
    int64_t ldm = 0, ldn = 0;  // of E^T and of C among the operand planes
    // float, single matrix, tensor-core updates only (else null): scaled fp16 pairs of the finished tiles, E transposed (rows of
    // ldm values) and the completed C (rows of ldn), with the tiles' scales: operands of the updates (see TcPlanes)
    __half *et_hi = nullptr, *et_lo = nullptr, *c_hi = nullptr, *c_lo = nullptr;
    float *e_scale = nullptr, *c_scale = nullptr;
    int *wide_count = nullptr;
    // pipelined schedule only (else null / 0): planes that collect the far feedback apart from Y and C, added when a
    // tile is loaded
    const F *yf = nullptr, *cf = nullptr;
    // pipelined schedule only: the planes through which a tile hands the feedback for its lower and its right neighbour
    // on (the neighbour adds them when it loads); every entry that is read has been written one launch before
    F *yn = nullptr, *cn = nullptr;
};

// Float operands as fp16 pairs.  A value times a power of two, chosen so that the largest value it shares its scale with lies
// in [2^14, 2^15), is hi + lo with 11 significant bits each: relative error 2^-23 down to 2^-17 of the largest value (the same
// as a tf32 pair), an absolute error of 2^-40 of it below.  The three products hi hi + lo hi + hi lo then cost half of
// their tf32 counterparts in tensor cycles and operand bytes.  `range_exponent` is the power: x 2^-e in (2^14, 2^15].
__device__ __forceinline__ int range_exponent(float largest) {
    const int e = (int)((__float_as_uint(largest) >> 23) & 255) - 127;  // largest in [2^e, 2^(e + 1))
    return e == 128 ? 0 : (e < -100 ? -100 : e) - 14;                   // infinities and NaN stay what they are; zeros and tiny rows: any scale
}
__device__ __forceinline__ float power_of_two(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }  // -126 <= e <= 127
__device__ __forceinline__ void split_half(float scaled, __half &hi, __half &lo) {
    hi = __float2half_rn(scaled);
    lo = __float2half_rn(scaled - __half2float(hi));
}

// Operand planes of the tensor-core updates of the sweep (see g2d_macro_update_tc.cu): fp16 pairs, K-major, each 64 x 64 tile under
// a power of two of its own.  A slice of k is one tile wide, so the scales come out of a product slice by slice:
// `*_scale` holds what a product with the tile has to be multiplied by.
// Wide tiles.  What lies far below the tile's largest value loses bits (see split_half), which matters where whole rows or columns
// do: with rows in units of their own, L[i, k] grows as E[k, j] falls, and the rows of the small units consist of products of
// what is lost (rows apart by a factor of 2^12 alternately: 9 times the error of float32, by 2^20: three per cent of the
// values).  The tile sweep therefore compares the largest values of the rows and columns of E and of C; where one is
// 2^8 or more below the tile's (zeros apart), or not finite, the planes of that tile get zeros, its scale is stored with its sign
// set and its float values are stored too, and the products with it are formed from them in float32: by the near update itself, and by
// wide_update_kernel behind every far one.  Up to that ratio the error is that of an even tile.
constexpr unsigned WIDE_RATIO_BITS = 8u << 7;  // 2^8 in the upper halves of floats
struct TcPlanes {
    __half *et_hi, *et_lo, *c_hi, *c_lo;  // E^T [n][ldm] and the completed C [m][ldn], written by the tile sweep
    __half *l_hi, *l_lo, *ut_hi, *ut_lo;  // L [m][ldm] and U^T [n][ldn], below the diagonal tiles, written once per sweep
    float *e_scale, *c_scale;             // [nI][nJ]
    float *l_scale, *u_scale;             // [nI][nI], [nJ][nJ] (tile row of U^T, tile of k)
    int64_t ldm, ldn;                     // m and n rounded up to multiples of 8 (rows of 16-byte multiples, a TMA requirement)
    int *error_flag;                      // set when a bounded wait inside a kernel ran out
    const float *l, *u, *e, *c;           // the float values: rows of ldl, ldu and (E and C, of wide tiles only) ld
    int64_t ldl, ldu, ld;
    int *wide_count;                      // wide tiles of the sweep so far, E and C each
};
// Band updates between tiles on the tensor cores (pipelined schedule; see g2d_band_tc.cu): sources are the tiles of the
// anti-diagonal s, targets those of t0..t1 (t0 >= s + 2), feedback is added into the planes y (right) and c (down) of the maps.
// With outer_macro > 0 a target is left out when a far update on 128 x 128 macro tiles carries its source instead:
// when its macro anti-diagonal is lag_macro or more past the end of the source's group of outer_macro macro anti-diagonals.
struct BandTcMaps {
    alignas(64) unsigned char bytes[10 * 128];  // tensor maps of the eight operand planes and the two targets (opaque here)
    float *y, *c;                               // the targets
};
int band_tc_prepare(BandTcMaps *maps, const TcPlanes &planes, float *y, float *c, int64_t m, int64_t n, int64_t ld);
int launch_band_tc(const BandTcMaps *maps, const TcPlanes &planes, int64_t m, int64_t n, int s, int t0, int t1, int outer_macro, int lag_macro, cudaStream_t stream);
// l and u: rows of ldl and ldu values
int tc_prepare_operands(const float *l, int64_t ldl, const float *u, int64_t ldu, int64_t m, int64_t n, const TcPlanes &planes, cudaStream_t stream);
// The tiles of anti-diagonal S and the near update of s = S - 1 in one launch (see g2d_tile_sweep_step.cu)
int launch_sweep_step(const SweepArgs<float> &args, int S, const BandTcMaps *maps, const TcPlanes &planes, int s, int t0, int t1, int outer_macro, int lag_macro,
                      cudaStream_t stream);
struct MacroTcMaps {
    alignas(64) unsigned char bytes[10 * 128];  // tensor maps of the eight operand planes with 128-row boxes and of the two targets
    float *y, *c;                               // the targets
};
// y and c: the planes that receive the right and the down feedback, rows of ld values (a multiple of 4)
int macro_tc_prepare(MacroTcMaps *maps, const TcPlanes &planes, float *y, float *c, int64_t m, int64_t n, int64_t ld);
int launch_macro_update_tc(const MacroTcMaps *maps, const TcPlanes &planes, int64_t m, int64_t n, int s0, int s1, int s_end, cudaStream_t stream, int t_first = 0);

// One problem of the tensor-core triangular inverse of the factor preparation (see g2d_factors_tc.cu).
struct FactorPlanes {
    const float *a;            // [n][n], Cholesky factor T in its lower triangle
    float *out;                // [n][n], the inverse being built
    // every operand as three bf16 planes hi + mid + lo = the float32 value exactly, rows of ld values:
    __nv_bfloat16 *out_hi, *out_mid, *out_lo;      // the inverse
    __nv_bfloat16 *outt_hi, *outt_mid, *outt_lo;   // its transpose
    __nv_bfloat16 *tw_hi, *tw_mid, *tw_lo;         // lower triangle: T; upper triangle: the transposed intermediate product
    int64_t n, ld;
    int *flag;                 // receives -1 when a bounded wait inside a kernel ran out (may be null)
};
int launch_trinv_tc(int count, const FactorPlanes *problems, cudaStream_t stream);

// Tensor-core trailing update of the blocked Cholesky factorization (see g2d_factors_tc.cu).  pt planes are
// [n][SYRK_TC_K] fp16 pairs: pt[r][k] = SYRK_PANEL_SCALE a[o + k][r] for the two groups of block rows that start at row o.
constexpr int SYRK_TC_K = 512;
constexpr float SYRK_PANEL_SCALE = 8192.f;
struct SyrkTcMaps {
    alignas(64) unsigned char hi[128], lo[128], wide_hi[128], wide_lo[128], target[128];  // tensor maps of the planes and of the matrix (opaque here)
};
struct SyrkTcTarget {
    const SyrkTcMaps *maps;
    float *a;
    int64_t n, o;
    int t_lo, t_hi;  // target 128-row tile rows [t_lo, t_hi), tile columns up to the diagonal
    int k0, kw;      // first column of the planes, and how many of them; row o of the matrix belongs to k0
    int *flag;
};
struct Equilibration {
    float *a[2], *s[2];  // matrix and scales of its rows
    int64_t n[2];
};
int launch_equilibrate(int count, const Equilibration &q, cudaStream_t stream);
bool syrk_tc_maps(SyrkTcMaps *maps, const __half *pt_hi, const __half *pt_lo, float *a, int64_t n);
int launch_syrk_tc(int count, const SyrkTcTarget *targets, cudaStream_t stream);

// Trellis (Viterbi) search of `rows` sequences (see g2d_trellis.cu); `codes` optional packed paths, code bytes apart.
int64_t trellis_code_bytes(int T, int L, int K, int V, int tail_biting);
size_t trellis_scratch_bytes(int dtype, int64_t rows, int T, int L, int K, int V);
// An optional index of the code table: its distinct rows ([count, V], in the table's dtype) and, per state, the number of
// its row among them.  Tables with few distinct rows are searched from shared memory with it (same results).
struct TrellisIndex {
    const void *distinct;
    const uint16_t *ids;
    int count;
};
int launch_trellis(int dtype, int64_t rows, int T, const void *x, const void *table, int L, int K, int V, int tail, const void *scale,
                   void *out, int64_t *states, void *workspace, uint8_t *codes, cudaStream_t st, const TrellisIndex *index = nullptr);

template <typename F>
int launch_tile_sweep(const SweepArgs<F> &args, int S, cudaStream_t stream, int parity = 0);
bool load_tile_sweep();  // brings the kernel's code to the current device

enum BandMode { BAND_TILE = 0, BAND_PLAIN = 1, BAND_GENERAL = 2 };

template <typename F>
struct BandArgs {
    F *y, *c;
    const F *e, *l, *u;
    const int64_t *l_off, *u_off;
    int64_t batch, m, n;
    int P, Q;                 // stage(i, j) = i / P + j / Q
    int64_t s0, s1, s_end;    // sources s0..s1-1, targets s1..s_end-1
    int down_into_y;          // also add the down product into Y (the generic path keeps Y live)
    int mode;                 // BandMode
    int filter;               // tile mode only: 0 none, 1 sources with even tile row and column only, 2 targets with odd tile row and column only
    const int32_t *skew = nullptr;  // general mode only: batch b takes the stages s0 - skew[b], s1 - skew[b], s_end - skew[b]
};

template <typename F>
int launch_band_update(const BandArgs<F> &args, cudaStream_t stream);

// Feedback between tiles of TR x TC entries (see g2d_block_update.cu): sources the tile anti-diagonals s0..s1-1, targets
// t0..t1-1 (t0 >= s1); `y` and `c` receive the sums, `c_from` holds the completed C of the sources.
template <typename F>
struct BlockUpdateArgs {
    F *y, *c;
    const F *e, *c_from, *l, *u;
    const int64_t *l_off, *u_off;
    int64_t batch, m, n;
    int TR, TC;
    int s0, s1, t0, t1;
};
template <typename F>
int launch_block_update(const BlockUpdateArgs<F> &args, cudaStream_t stream);

// Which of four lanes of side streams a call takes: the one that the last call on the same stream took (the two run in order
// anyway), else the next in turn.  The GPU has few hardware queues (eight connections by default): a program that issues
// its calls on one or two streams then keeps to as many lanes, and its streams do not share a queue with one another.
struct LaneChoice {
    cudaStream_t last[4] = {};
    bool used[4] = {};
    unsigned next = 0;
    int pick(cudaStream_t caller) {  // under the owner's lock
        for (int k = 0; k < 4; ++k)
            if (used[k] && last[k] == caller) return k;
        const int k = (int)(next++ & 3);
        last[k] = caller;
        used[k] = true;
        return k;
    }
};

// Overlapped schedule: tile launches on the critical path, everything else beside them (see g2d_api.cu).
// tiles(s, stream) sweeps tile anti-diagonal s; update(s0, s1, t0, t1, far, stream) carries the sources s0..s1-1 into the
// targets t0..t1-1, into the far planes or into Y and C.  `pushes`: a tile hands the feedback for its two neighbours on itself.
typedef std::function<int(int, cudaStream_t)> TileLauncher;
typedef std::function<int(int, int, int, int, bool, cudaStream_t)> UpdateLauncher;
int sweep_overlapped(int waves, bool pushes, cudaStream_t caller, const TileLauncher &tiles, const UpdateLauncher &update);

// skew (device, one int per batch, may be null): batch b works at stage s - skew[b] (slabs of an N-factor sweep);
// z_stride: values of z per batch (0: exactly the stage's d p q)
template <typename F>
int launch_stage_push(const g2d_stage_desc &d, const F *z, int64_t s, int64_t s1, cudaStream_t stream, const int32_t *skew = nullptr,
                      int64_t z_stride = 0);
// Its first half alone: errors, completed C and rounded values of stage s.
template <typename F>
int launch_stage_commit(const g2d_stage_desc &d, const F *z, int64_t s, cudaStream_t stream, const int32_t *skew = nullptr, int64_t z_stride = 0);

// Launches that follow each other on one stream without a wait between them can be programmatic dependent launches: the CTAs of a launch
// start when those of the one before have all asked for it or ended, and SMs are free.  What a launch before writes is read, and
// anything is written, only behind the wait, which holds until that launch has ended.
__device__ __forceinline__ void after_the_launch_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_the_next_launch_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Clusters of CTAs: the CTA's number in its cluster, and a barrier of all threads of the cluster (by whole warps)
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() { asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory"); }

}  // namespace g2d

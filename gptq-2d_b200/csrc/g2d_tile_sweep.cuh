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
constexpr int PLD = SUB + 2;            // entries per row of a sub-tile's quantizer parameters (the walk along an anti-diagonal moves 17 entries: no conflicts)
constexpr int PPAD = (SUB + 1) * PLD;   // entries behind the parameters that lanes past their last entry may read (and ignore)

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

// Sixteen bytes from global to shared memory without passing through registers; zeros when `in` is false.
__device__ __forceinline__ void async16(void *dst, const void *src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
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
// A predicated store instead of a branch around a store
__device__ __forceinline__ void store_shared_if(uint32_t at, float v, bool on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.shared.f32 [%0], %1;\n\t}" ::"r"(at), "f"(v), "r"((uint32_t)on));
}
__device__ __forceinline__ void store_shared_if(uint32_t at, double v, bool on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.shared.f64 [%0], %1;\n\t}" ::"r"(at), "d"(v), "r"((uint32_t)on));
}

// D += A B with 16 inner terms, all in shared memory with row stride LD; one warp.  The row and column counts of D are 16 x 16,
// 16 x 64 (WIDE) or 64 x 16 (TALL): the strips give a lane 4 x 8 or 8 x 4 outputs and need half the operand loads per
// multiply-add of the small block (2 x 4 outputs per lane), and shared-memory loads are what these products are short of.
enum Shape { SMALL, WIDE, TALL };
template <int SHAPE, typename F>
__device__ __forceinline__ void mm16(F *__restrict__ D, const F *__restrict__ A, const F *__restrict__ B, int lane) {
    constexpr int NR = SHAPE == SMALL ? 2 : SHAPE == WIDE ? 4 : 8, NC = SHAPE == WIDE ? 2 : 1;  // rows and groups of four columns per lane
    const int r = SHAPE == WIDE ? (lane >> 3) * 4 : SHAPE == TALL ? lane >> 2 : (lane >> 2) * 2, rs = SHAPE == TALL ? 8 : 1;
    const int c = SHAPE == WIDE ? (lane & 7) * 4 : (lane & 3) * 4;
    constexpr int CS = 32;  // distance of a lane's column groups
    F d[NR][NC][4];
#pragma unroll
    for (int i = 0; i < NR; ++i)
#pragma unroll
        for (int g = 0; g < NC; ++g) load4(D + (r + i * rs) * LD + c + g * CS, d[i][g]);
    constexpr int KU = SHAPE == SMALL ? SUB : 4;  // inner terms per trip: the small product entirely unrolled, the strips in four trips
#pragma unroll 1
    for (int k0 = 0; k0 < SUB; k0 += KU) {
        F a[NR][KU], b[KU][NC][4];
#pragma unroll
        for (int k = 0; k < KU; k += 4) {
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                F t[4];
                load4(A + (r + i * rs) * LD + k0 + k, t);
#pragma unroll
                for (int x = 0; x < 4; ++x) a[i][k + x] = t[x];
            }
        }
#pragma unroll
        for (int k = 0; k < KU; ++k)
#pragma unroll
            for (int g = 0; g < NC; ++g) load4(B + (k0 + k) * LD + c + g * CS, b[k][g]);
#pragma unroll
        for (int k = 0; k < KU; ++k)
#pragma unroll
            for (int i = 0; i < NR; ++i)
#pragma unroll
                for (int g = 0; g < NC; ++g)
#pragma unroll
                    for (int y = 0; y < 4; ++y) d[i][g][y] += a[i][k] * b[k][g][y];
    }
#pragma unroll
    for (int i = 0; i < NR; ++i)
#pragma unroll
        for (int g = 0; g < NC; ++g) store4(D + (r + i * rs) * LD + c + g * CS, d[i][g]);
}

// A load that stays where it is written: the compiler moves a plain one down to its use, and the quantizer parameters are asked for
// a whole sub-tile sweep ahead (2048 x 2048 with a scale per entry: 3.28 ms when they had sunk, 2.17 now, as with a scale per row).
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

// floats or doubles of a CTA's shared memory
template <typename F>
constexpr size_t tile_smem = sizeof(F) * (3 * TILE * LD + DROWS * DLD + NSUB * SUB * PLD * 4 + (sizeof(F) == sizeof(float) ? 4 * TILE * LD : PPAD * 4));

}  // namespace g2d

// The two bulk products of the factor preparation on the tensor cores (float only): the trailing update of the
// blocked Cholesky factorization (second half of this file) and the triangular inverse.
//
// The inverse Lf = T^{-1} of the lower triangular Cholesky factor is built by doubling: at level b every aligned pair
// of finished b x b diagonal blocks [A^{-1} 0; . B^{-1}] of Lf is completed by X = -B^{-1} (C A^{-1}) with
// C = T[second half rows, first half columns].  From b = 128 on, both products of a level run here as tcgen05.mma
// kind::f16 GEMMs over output tiles of 128 x 128 (256 x 256 for two CTAs) on three bf16 planes per operand (six products per k step, see
// "Precision" below).  The MMA wants both operands K-major, so the first product is formed transposed,
//     W^T[j][i] = sum_k Lf^T[j][k] T[i][k]        (k from the tile's first row j0 to the end of the first half)
//     X[i][j]   = -sum_k Lf[i][k] W^T[j][k]       (k from the start of the second half through the tile's rows)
// and every operand is kept as ready-made hi / mid / lo planes: Lf and its transpose (both written by the second
// product's epilogue), and one plane triple whose lower triangle holds T and whose upper triangle receives W^T.
// Same pipeline as the macro updates of the sweep: one warp issues TMA loads into a two-stage ring of 96 KB stages, one
// warp issues the MMAs, four warps (eight in the kernel for two CTAs) read the accumulators and store; every wait is bounded.
#include <cstring>

#include "g2d_tc.cuh"

namespace g2d {

struct FactorMaps {
    CUtensorMap out[3], outt[3], tw[3];  // hi, mid, lo
};
struct TrinvJob {
    FactorMaps maps[2];
    FactorPlanes p[2];
    int pairs;   // pairs of diagonal blocks of the largest problem; blockIdx.x = problem * pairs + pair
    int tiles;   // b / 128
    int64_t b;
    int second;  // 0: W^T, 1: X
};

// Precision.  The inverse is where a badly conditioned factor shows: every level multiplies explicit inverse blocks, and
// the error of each product is amplified by the cancellation in -B^{-1} (C A^{-1}); with a two-plane split (2^-21 per
// product) the factors of a heavy-tailed, 1 %-damped 4096 x 4096 Gram came out 4e-5 from the float64 result where a float32
// LAPACK factorization is 1.5e-6 away.  So this kernel uses three planes per operand, a = hi + mid + lo exactly, and keeps the
// one large product (hi hi') in an accumulator of its own, so that the small ones are not truncated against it.  The planes
// are bf16 (8 + 8 + 8 bits, the exponent range of float): the six products leave out mid lo' and what is smaller, 2^-26 of a
// product, a quarter of what a float32 multiplication rounds off; they cost half of six tf32 products in tensor cycles and
// bytes, and the factors came closer (n = 4096: 1.3e-6 from float64, 2.8e-6 before).
// The second source of error is the tensor cores' accumulation: every add into the float accumulator truncates, and the sums
// here run over up to n / 2 terms.  So the k range is cut into slices of 256: each slice is accumulated in
// tensor memory, and the epilogue warps add the slices up in registers with round-to-nearest additions while the MMAs
// of the next slice run into a second pair of accumulators.
constexpr int TRINV_STAGES = 2;
constexpr int TRINV_STAGE_BYTES = 6 * HTILE_BYTES;         // A hi, mid, lo; B hi, mid, lo
constexpr int TRINV_SLICE = 4;                             // chunks per slice: k = 256
constexpr uint32_t TRINV_TMEM_COLS = 4 * MT;               // two alternating pairs of (main, correction) accumulators
constexpr uint32_t TRINV_DESC = idesc_16(MT, 1);           // bf16
// Two CTAs of a cluster per 256 x 256 tile (trinv_duo_kernel) where blocks are large and their tiles many.  Alone a CTA reads 256 rows of shared memory per
// MMA of 64 cycles and fills 768 per six of them, 1.5 times what the port gives meanwhile; two CTAs read 256 each (384 with the other's half) per MMA of 128
// cycles and fill 768 per six.  Tiles of the moment share their strips in L2: factors of 8192 and 28672 97 ms alone, 84.6 with two CTAs from blocks
// of 4096 on.  (256 x 128 tiles with half of the second operand each, three stages and alternating accumulators: 92 ms.)
// But a cluster takes a third longer for its tile than a CTA for one of the four, and a level with few tiles lasts as long as its longest.
// Whole preparations in ms, alone and with two CTAs at one level, by a factor's tiles of 256 x 256 there, one factor and two of that size:
// blocks of 4096, 16 tiles (n = 4352) 2.30 and 2.38, 2.70 and 2.76; 128 (6144) 3.41 and 3.47, 4.43 and 4.47; 192 (7168) 4.19 and 4.24, 5.71 and
// 5.70; 224 (7680) 4.58 and 4.63, 6.49 and 6.41; 256 (8192) 5.03 and 5.05, 7.30 and 7.13.  Blocks of 8192, 32 tiles (8300) 5.48 and 5.59; 128
// (9216) 6.11 and 6.13; 256 (10240) 7.43 and 7.44, 11.42 and 11.35; 512 (12288) 10.32 and 10.24, 17.53 and 17.26.  Of 16384, 64 (16640) 19.33
// and 19.34; 256 (17408) 21.86 and 21.72.  So from three tiles per cluster on.  (By a factor's own tiles, not those of a launch: a factor has the
// same bits alone and in a pair, and the two kernels differ in theirs.)  Blocks of 2048 do not gain: 16384 twice 33.74 and 33.81.
constexpr int DUO_BLOCK = 4096, DUO_TILES_EACH = 3;

// fp32 -> three bf16 values with a = hi + mid + lo exactly (8 significant bits each)
__device__ __forceinline__ void split_bf16_3(float a, __nv_bfloat16 &hi, __nv_bfloat16 &mid, __nv_bfloat16 &lo) {
    hi = __float2bfloat16_rn(a);
    const float r = a - __bfloat162float(hi);
    mid = __float2bfloat16_rn(r);
    lo = __float2bfloat16_rn(r - __bfloat162float(mid));
}

// A thread's row gi of a finished tile, columns n0 .. n0 + 127
__device__ __forceinline__ void trinv_write(const FactorPlanes &P, int second, int64_t gi, int64_t n0, int64_t r2, const float (&total)[MT]) {
    const int64_t n = P.n, ld = P.ld;
    const bool vec = n % 4 == 0;  // rows of the float matrix are 16-byte multiples; those of the planes always are
#pragma unroll
    for (int cb = 0; cb < MT / 8; ++cb) {
        const int64_t gj0 = n0 + cb * 8;
        __align__(16) __nv_bfloat16 h[8];
        __align__(16) __nv_bfloat16 c[8];
        __align__(16) __nv_bfloat16 l[8];
        if (!second) {
            // W^T[gi][gj]: gi is inside the first half (always a row of the matrix), gj is cut at r2; a group of eight that
            // reaches past it ends in the padding of its row (its extra products are zero)
            if (gj0 < r2) {
#pragma unroll
                for (int e = 0; e < 8; ++e) split_bf16_3(total[cb * 8 + e], h[e], c[e], l[e]);
                *reinterpret_cast<uint4 *>(P.tw_hi + gi * ld + gj0) = *reinterpret_cast<const uint4 *>(h);
                *reinterpret_cast<uint4 *>(P.tw_mid + gi * ld + gj0) = *reinterpret_cast<const uint4 *>(c);
                *reinterpret_cast<uint4 *>(P.tw_lo + gi * ld + gj0) = *reinterpret_cast<const uint4 *>(l);
            }
        } else if (gi < r2) {
            // X[gi][gj] = -acc (gj is inside the first half): the inverse itself, its split, and the split of its transpose
            // (coalesced across the lanes)
            float *dst = P.out + gi * n + gj0;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float v = -total[cb * 8 + e];
                split_bf16_3(v, h[e], c[e], l[e]);
                P.outt_hi[(gj0 + e) * ld + gi] = h[e];
                P.outt_mid[(gj0 + e) * ld + gi] = c[e];
                P.outt_lo[(gj0 + e) * ld + gi] = l[e];
                if (!vec) dst[e] = v;
            }
            if (vec) {
                *reinterpret_cast<float4 *>(dst) = make_float4(-total[cb * 8], -total[cb * 8 + 1], -total[cb * 8 + 2], -total[cb * 8 + 3]);
                *reinterpret_cast<float4 *>(dst + 4) = make_float4(-total[cb * 8 + 4], -total[cb * 8 + 5], -total[cb * 8 + 6], -total[cb * 8 + 7]);
            }
            *reinterpret_cast<uint4 *>(P.out_hi + gi * ld + gj0) = *reinterpret_cast<const uint4 *>(h);
            *reinterpret_cast<uint4 *>(P.out_mid + gi * ld + gj0) = *reinterpret_cast<const uint4 *>(c);
            *reinterpret_cast<uint4 *>(P.out_lo + gi * ld + gj0) = *reinterpret_cast<const uint4 *>(l);
        }
    }
}

__global__ void __launch_bounds__(TC_THREADS) trinv_tc_kernel(const __grid_constant__ TrinvJob job) {
    extern __shared__ unsigned char tc_smem_raw[];
    __shared__ __align__(8) TcRing ring;
    __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2];
    const int z = (int)blockIdx.x >= job.pairs ? 1 : 0;
    const int64_t pair = (int64_t)blockIdx.x - (int64_t)z * job.pairs;
    const FactorPlanes P = z ? job.p[1] : job.p[0];
    const FactorMaps *maps = z ? &job.maps[1] : &job.maps[0];
    const int64_t n = P.n, b = job.b;
    const int64_t r0 = pair * 2 * b, r1 = r0 + b;  // first half rows [r0, r1), second half rows [r1, r2)
    if (r1 >= n) return;
    const int64_t r2 = min(r0 + 2 * b, n);
    // output tile: rows m0.. of the A operand's matrix, columns n0.. of the B operand's
    int64_t m0, n0, k_lo, k_hi;
    const CUtensorMap *a_maps;
    if (!job.second) {
        m0 = r0 + (int64_t)blockIdx.z * MT;  // j: long k ranges (small j) are scheduled first
        n0 = r1 + (int64_t)blockIdx.y * MT;  // i
        if (n0 >= r2) return;
        k_lo = m0;
        k_hi = r1;
        a_maps = maps->outt;
    } else {
        m0 = r1 + (int64_t)(job.tiles - 1 - (int)blockIdx.y) * MT;  // i: long k ranges (large i) first
        if (m0 >= r2) return;
        n0 = r0 + (int64_t)blockIdx.z * MT;  // j
        k_lo = r1;
        k_hi = min(m0 + MT, r2);
        a_maps = maps->out;
    }
    const int chunks = (int)ceil_div(k_hi - k_lo, (int64_t)KH);  // a ragged tail reads zeros beyond the matrix
    const int slices = (chunks + TRINV_SLICE - 1) / TRINV_SLICE;

    const uint32_t smem_base = (smem_u32(tc_smem_raw) + 1023u) & ~1023u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s2 = 0; s2 < 2; ++s2) {
            mbar_init(&acc_full[s2], 1);
            mbar_init(&acc_empty[s2], 4);  // one arrival per epilogue warp
        }
    }
    const uint32_t tmem = tc_ring_setup(ring, TRINV_TMEM_COLS);  // fences the barrier initialisations and synchronises the CTA
    if (warp == 0) {
        if (lane == 0) {
            for (int ch = 0; ch < chunks; ++ch) {
                const int stage = ch % TRINV_STAGES, round = ch / TRINV_STAGES;
                if (round > 0 && !mbar_wait(&ring.empty[stage], (round - 1) & 1)) {
                    ring.failed = 1;
                    break;
                }
                const int k = (int)(k_lo + (int64_t)ch * KH);
                const uint32_t dst = smem_base + stage * TRINV_STAGE_BYTES;
                mbar_expect_tx(&ring.full[stage], TRINV_STAGE_BYTES);
                for (int part = 0; part < 3; ++part) {
                    tma_load_2d(dst + part * HTILE_BYTES, &a_maps[part], k, (int)m0, &ring.full[stage]);
                    tma_load_2d(dst + (3 + part) * HTILE_BYTES, &maps->tw[part], k, (int)n0, &ring.full[stage]);
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            for (int ch = 0; ch < chunks; ++ch) {
                const int stage = ch % TRINV_STAGES, round = ch / TRINV_STAGES;
                const int slice = ch / TRINV_SLICE, buf = slice & 1;
                const bool opens = ch % TRINV_SLICE == 0, closes = ch % TRINV_SLICE == TRINV_SLICE - 1 || ch == chunks - 1;
                // the accumulators must have been read out by the epilogue of the slice two before
                if (opens && slice >= 2 && !mbar_wait(&acc_empty[buf], ((slice >> 1) - 1) & 1)) {
                    ring.failed = 1;
                    break;
                }
                if (!mbar_wait(&ring.full[stage], round & 1)) {
                    ring.failed = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc_main = tmem + (uint32_t)(buf * 2 * MT), acc_small = acc_main + MT;
                const uint32_t base = smem_base + stage * TRINV_STAGE_BYTES;
                const uint32_t a_hi = base, a_mid = base + HTILE_BYTES, a_lo = base + 2 * HTILE_BYTES;
                const uint32_t b_hi = base + 3 * HTILE_BYTES, b_mid = base + 4 * HTILE_BYTES, b_lo = base + 5 * HTILE_BYTES;
#pragma unroll
                for (int ks = 0; ks < KH / 16; ++ks) {
                    const uint32_t off = ks * 32;  // 16 values = 32 bytes along the swizzled row
                    const uint32_t fresh = (opens && ks == 0) ? 0u : 1u;
                    umma_16(acc_main, umma_desc(a_hi + off), umma_desc(b_hi + off), TRINV_DESC, fresh);
                    umma_16(acc_small, umma_desc(a_hi + off), umma_desc(b_mid + off), TRINV_DESC, fresh);
                    umma_16(acc_small, umma_desc(a_mid + off), umma_desc(b_hi + off), TRINV_DESC, 1u);
                    umma_16(acc_small, umma_desc(a_mid + off), umma_desc(b_mid + off), TRINV_DESC, 1u);
                    umma_16(acc_small, umma_desc(a_hi + off), umma_desc(b_lo + off), TRINV_DESC, 1u);
                    umma_16(acc_small, umma_desc(a_lo + off), umma_desc(b_hi + off), TRINV_DESC, 1u);
                }
                umma_commit(&ring.empty[stage]);            // arrives when the MMAs above have read the stage
                if (closes) umma_commit(&acc_full[buf]);    // arrives when the slice is complete in tensor memory
            }
            umma_commit(&ring.accum);                       // arrives when every MMA issued so far has completed
        }
    } else {
        // epilogue warps: lanes 32 q .. 32 q + 31 of tensor memory, q = warp % 4; one accumulator row per thread, whose
        // 128 running sums stay in registers across the slices
        const int q = warp & 3;
        float total[MT];
#pragma unroll
        for (int x = 0; x < MT; ++x) total[x] = 0.f;
        bool go = true;
        for (int slice = 0; slice < slices && go; ++slice) {
            const int buf = slice & 1;
            const bool ok = mbar_wait(&acc_full[buf], (slice >> 1) & 1, 64);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (!ok) ring.failed = 1;
            go = __all_sync(0xffffffffu, ok && !ring.failed);  // warp-uniform: the tensor-memory loads are warp-wide
            if (!go) break;
#pragma unroll
            for (int cb = 0; cb < MT / 32; ++cb) {
                uint32_t v[32], w[32];
                tmem_load_32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * 2 * MT + cb * 32), v);
                tmem_load_32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * 2 * MT + MT + cb * 32), w);
#pragma unroll
                for (int x = 0; x < 32; ++x) total[cb * 32 + x] += __uint_as_float(v[x]) + __uint_as_float(w[x]);
            }
            // this warp has read the accumulators: hand them back to the MMA warp
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
        }
        if (go) {
            trinv_write(P, job.second, m0 + q * 32 + lane, n0, r2, total);
        }
    }
    const bool failed = tc_ring_teardown(ring, tmem, TRINV_TMEM_COLS);
    if (threadIdx.x == 0 && failed && P.flag) atomicExch(P.flag, -1);
}

// As trinv_tc_kernel, by two CTAs of a cluster on a tile of 256 x 256: each has 128 rows of the first operand and of the second.  The main and the
// correction accumulator fill tensor memory, so there is one pair of them: a chunk's large products come first, so that the reading warps take
// the main accumulator of a slice while its last small products are multiplied, and the small one under the first large products
// of the next.
struct TrinvDuoRing {
    uint64_t full[TRINV_STAGES], empty[TRINV_STAGES], acc_full[2], acc_empty[2];  // accumulators: main, correction
    uint64_t drained;  // as in PairRing
    uint32_t tmem;
    int failed;
};
constexpr int DUO_EDGE = 2 * MT, DUO_GROUP = 8;
static_assert(DUO_BLOCK % (DUO_EDGE * DUO_GROUP) == 0, "whole groups");
__global__ void __launch_bounds__(PAIR_THREADS, 1) trinv_duo_kernel(const __grid_constant__ TrinvJob job) {
    constexpr uint32_t DESC = idesc_16(DUO_EDGE, 1, DUO_EDGE), COLS = 2 * DUO_EDGE;  // bf16
    extern __shared__ unsigned char tc_smem_raw[];
    __shared__ __align__(8) TrinvDuoRing ring;
    const int rank = (int)cluster_rank();
    const int z = (int)blockIdx.y >= job.pairs ? 1 : 0;
    const int64_t pair = (int64_t)blockIdx.y - (int64_t)z * job.pairs;
    const FactorPlanes P = z ? job.p[1] : job.p[0];
    const FactorMaps *maps = z ? &job.maps[1] : &job.maps[0];
    const int64_t n = P.n, b = job.b;
    const int64_t r0 = pair * 2 * b, r1 = r0 + b;  // first half rows [r0, r1), second half rows [r1, r2)
    if (r1 >= n) return;
    const int64_t r2 = min(r0 + 2 * b, n);
    // Groups of eight tile rows, column after column, so that the clusters of the moment share 8 and 9 strips in L2; long k ranges first.
    const int64_t edge = b / DUO_EDGE, at = blockIdx.x >> 1, group = at / (DUO_GROUP * edge), within = at % (DUO_GROUP * edge);
    const int64_t row = group * DUO_GROUP + within % DUO_GROUP, column = within / DUO_GROUP;  // edge is a multiple of DUO_GROUP
    int64_t tile_m0, n0, k_lo, k_hi;
    const CUtensorMap *a_maps;
    if (!job.second) {
        tile_m0 = r0 + row * DUO_EDGE;  // j
        n0 = r1 + column * DUO_EDGE;    // i
        if (n0 >= r2) return;
        k_lo = tile_m0;
        k_hi = r1;
        a_maps = maps->outt;
    } else {
        tile_m0 = r1 + (edge - 1 - row) * DUO_EDGE;  // i
        if (tile_m0 >= r2) return;
        n0 = r0 + column * DUO_EDGE;  // j
        k_lo = r1;
        k_hi = min(tile_m0 + DUO_EDGE, r2);
        a_maps = maps->out;
    }
    const int64_t m0 = tile_m0 + rank * MT;
    const int chunks = (int)ceil_div(k_hi - k_lo, (int64_t)KH);  // a ragged tail reads zeros beyond the matrix
    // The ranges of k of the two CTAs' rows differ by 128: the first chunks of the first product belong to CTA 0's rows alone, the last ones of the
    // second to CTA 1's.  A slice boundary lies where they part (the first slice is half a slice), and the other CTA leaves that
    // slice out of its sums: zeros in place of its operand would carry NaN and infinities of the other operand into its rows.
    constexpr int APART = MT / KH;
    static_assert(TRINV_SLICE == 2 * APART && DUO_EDGE == TRINV_SLICE * KH, "a tile's ranges of k begin and end with half a slice");
    const int slices = (chunks + APART + TRINV_SLICE - 1) / TRINV_SLICE;
    const int not_mine = job.second ? (rank == 0 && k_hi > tile_m0 + MT ? slices - 1 : -1) : rank == 1 ? 0 : -1;

    const uint32_t smem_base = (smem_u32(tc_smem_raw) + 1023u) & ~1023u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < TRINV_STAGES; ++s) {
            mbar_init(&ring.full[s], 1);
            mbar_init(&ring.empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&ring.acc_full[s], 1);
            mbar_init(&ring.acc_empty[s], 16);  // one arrival per reading warp of both CTAs, at the leader's
        }
        mbar_init(&ring.drained, 1);
        ring.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc<true>(&ring.tmem, COLS);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    __syncwarp();
    cluster_sync();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = ring.tmem;
    if (warp == 0) {
        if (lane == 0) {
            int ch = 0;
            for (; ch < chunks; ++ch) {
                const int stage = ch % TRINV_STAGES, round = ch / TRINV_STAGES;
                if (round > 0 && !mbar_wait_cluster(&ring.empty[stage], (round - 1) & 1)) {
                    ring.failed = 1;
                    break;
                }
                const int k = (int)(k_lo + (int64_t)ch * KH);
                const uint32_t dst = smem_base + stage * TRINV_STAGE_BYTES, bar = leaders(&ring.full[stage]);
                // both CTAs' bytes count at the leader's barrier (they may do so before it expects them: the phase waits for its arrival)
                if (rank == 0) mbar_expect_tx(&ring.full[stage], 2 * TRINV_STAGE_BYTES);
                for (int part = 0; part < 3; ++part) {
                    tma_load_2d_duo(dst + part * HTILE_BYTES, &a_maps[part], k, (int)m0, bar);
                    tma_load_2d_duo(dst + (3 + part) * HTILE_BYTES, &maps->tw[part], k, (int)n0 + rank * MT, bar);
                }
            }
            // both CTAs' last loads have landed, or had their time to, before their shared memory is given back, whatever became of the MMAs
            if (rank == 0)
                for (int k = max(ch - TRINV_STAGES, 0); k < ch; ++k) mbar_wait_cluster(&ring.full[k % TRINV_STAGES], (k / TRINV_STAGES) & 1);
            // the leader's commits arrive here as well: none may be under way when this CTA ends (those of the accumulators are awaited below)
            for (int k = max(chunks - TRINV_STAGES, 0); k < chunks && !ring.failed; ++k)
                if (!mbar_wait_cluster(&ring.empty[k % TRINV_STAGES], (k / TRINV_STAGES) & 1)) ring.failed = 1;
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            const uint32_t acc_main = tmem, acc_small = tmem + DUO_EDGE;
            int slice = 0;
            for (int ch = 0; ch < chunks; ++ch) {
                const int stage = ch % TRINV_STAGES, round = ch / TRINV_STAGES;
                const bool opens = ch == 0 || ch % TRINV_SLICE == APART, closes = ch % TRINV_SLICE == APART - 1 || ch == chunks - 1;
                if (!mbar_wait_cluster(&ring.full[stage], round & 1)) { ring.failed = 1; break; }
                // the accumulators must have been read out for the slice before
                if (opens && slice > 0 && !mbar_wait_cluster(&ring.acc_empty[0], (slice - 1) & 1)) { ring.failed = 1; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a_hi = smem_base + stage * TRINV_STAGE_BYTES, a_mid = a_hi + HTILE_BYTES, a_lo = a_hi + 2 * HTILE_BYTES;
                const uint32_t b_hi = a_hi + 3 * HTILE_BYTES, b_mid = b_hi + HTILE_BYTES, b_lo = b_mid + HTILE_BYTES;
#pragma unroll
                for (int ks = 0; ks < KH / 16; ++ks) mma<true>(acc_main, a_hi + ks * 32, b_hi + ks * 32, DESC, (opens && ks == 0) ? 0u : 1u);
                if (closes) commit<true>(&ring.acc_full[0]);
                if (opens && slice > 0) {
                    if (!mbar_wait_cluster(&ring.acc_empty[1], (slice - 1) & 1)) { ring.failed = 1; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                }
#pragma unroll
                for (int ks = 0; ks < KH / 16; ++ks) {
                    const uint32_t off = ks * 32;  // 16 values = 32 bytes along the swizzled row
                    mma<true>(acc_small, a_hi + off, b_mid + off, DESC, (opens && ks == 0) ? 0u : 1u);
                    mma<true>(acc_small, a_mid + off, b_hi + off, DESC, 1u);
                    mma<true>(acc_small, a_mid + off, b_mid + off, DESC, 1u);
                    mma<true>(acc_small, a_hi + off, b_lo + off, DESC, 1u);
                    mma<true>(acc_small, a_lo + off, b_hi + off, DESC, 1u);
                }
                commit<true>(&ring.empty[stage]);  // arrives when the MMAs above have read the stage
                if (closes) {
                    commit<true>(&ring.acc_full[1]);
                    ++slice;
                }
            }
            // every MMA that was issued completes, or has its time to, as in pair_gemm
            if (ring.failed) {
                commit<true>(&ring.drained);
                mbar_wait_cluster(&ring.drained, 0);
            } else {
                mbar_wait_cluster(&ring.acc_full[1], (slice - 1) & 1);
            }
        }
    } else {
        // reading warps: lanes 32 q .. 32 q + 31 of tensor memory, q = warp % 4, and half of the columns; 128 running sums in registers
        const int q = warp & 3, c0 = ((warp - 2) >> 2) * MT;
        float total[MT];
#pragma unroll
        for (int x = 0; x < MT; ++x) total[x] = 0.f;
        bool go = true;
        for (int s = 0; s < 2 * slices && go; ++s) {
            const int which = s & 1;
            const bool ok = mbar_wait_cluster(&ring.acc_full[which], (s >> 1) & 1, 64);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (!ok) ring.failed = 1;
            go = __all_sync(0xffffffffu, ok && !ring.failed);  // warp-uniform: the tensor-memory loads are warp-wide
            if (!go) break;
            if (s >> 1 != not_mine) {
#pragma unroll
                for (int cb = 0; cb < MT / 16; ++cb) {  // 16 at a time, as in pair_gemm
                    uint32_t v[16];
                    tmem_load_16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(which * DUO_EDGE + c0 + cb * 16), v);
#pragma unroll
                    for (int x = 0; x < 16; ++x) total[cb * 16 + x] += __uint_as_float(v[x]);
                }
            }
            // this warp has read the accumulator: hand it back to the MMA warp
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_at(leaders(&ring.acc_empty[which]));
        }
        if (go) trinv_write(P, job.second, m0 + q * 32 + lane, n0 + c0, r2, total);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    // neither CTA leaves while the other's MMAs may read its shared memory or arrive at its barriers
    if (threadIdx.x == 0 && ring.failed) let_it_land();
    __syncwarp();
    cluster_sync();
    if (warp == 1) tmem_free<true>(tmem, COLS);
    if (threadIdx.x == 0 && ring.failed && P.flag) atomicExch(P.flag, -1);
}

// Operand planes after the 64-level of the doubling: T strictly below the diagonal into the lower triangle of tw, and the
// finished 128 x 128 diagonal blocks of Lf (lower triangular) into out / outt with explicit zeros in their other halves.
// One block per row, eight entries per thread; HBM bound (4 bytes in and 6 out per entry of the lower triangle).
__global__ void __launch_bounds__(256) trinv_split_kernel(FactorPlanes p0, FactorPlanes p1) {
    const FactorPlanes P = blockIdx.y ? p1 : p0;
    const int64_t n = P.n, ld = P.ld;
    const bool vec = n % 4 == 0;
    for (int64_t r = blockIdx.x; r < n; r += gridDim.x) {
        const int64_t d0 = r / MT * MT;
        for (int64_t c = (int64_t)threadIdx.x * 8; c < r; c += (int64_t)blockDim.x * 8) {
            __align__(16) __nv_bfloat16 h[8];
            __align__(16) __nv_bfloat16 m[8];
            __align__(16) __nv_bfloat16 l[8];
            float v[8];
            const float *src = P.a + r * n + c;
            if (vec && c + 8 <= r) {
                const float4 x = *reinterpret_cast<const float4 *>(src), y = *reinterpret_cast<const float4 *>(src + 4);
                v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] = c + e < r ? src[e] : 0.f;
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) split_bf16_3(v[e], h[e], m[e], l[e]);
            *reinterpret_cast<uint4 *>(P.tw_hi + r * ld + c) = *reinterpret_cast<const uint4 *>(h);
            *reinterpret_cast<uint4 *>(P.tw_mid + r * ld + c) = *reinterpret_cast<const uint4 *>(m);
            *reinterpret_cast<uint4 *>(P.tw_lo + r * ld + c) = *reinterpret_cast<const uint4 *>(l);
        }
        if (threadIdx.x < MT) {
            const int64_t c = d0 + threadIdx.x;
            if (c < n) {
                split_bf16_3(c <= r ? P.out[r * n + c] : 0.f, P.out_hi[r * ld + c], P.out_mid[r * ld + c], P.out_lo[r * ld + c]);
                split_bf16_3(c >= r ? P.out[c * n + r] : 0.f, P.outt_hi[r * ld + c], P.outt_mid[r * ld + c], P.outt_lo[r * ld + c]);
            }
        }
    }
}

static bool factor_maps(FactorMaps *maps, const FactorPlanes &p) {
    __nv_bfloat16 *const out[3] = {p.out_hi, p.out_mid, p.out_lo}, *const outt[3] = {p.outt_hi, p.outt_mid, p.outt_lo},
                  *const tw[3] = {p.tw_hi, p.tw_mid, p.tw_lo};
    bool ok = true;
    for (int part = 0; part < 3; ++part)
        ok = ok && make_map_16(&maps->out[part], out[part], p.n, p.n, MT, true, p.ld) && make_map_16(&maps->outt[part], outt[part], p.n, p.n, MT, true, p.ld) &&
             make_map_16(&maps->tw[part], tw[part], p.n, p.n, MT, true, p.ld);
    return ok;
}

// Whether a factor's products of the level b go to two CTAs per tile, by its tiles there: a pair's second half may end with the matrix, or be missing.
static bool two_ctas_pay(int64_t n, int64_t b) {
    if (b < DUO_BLOCK) return false;
    int64_t tiles = 0;
    for (int64_t r1 = b; r1 < n; r1 += 2 * b) tiles += b / DUO_EDGE * ceil_div(n - r1 < b ? n - r1 : b, (int64_t)DUO_EDGE);
    return tiles >= DUO_TILES_EACH * 74;
}

// Levels b = 128, 256, ... of the doubling for one or two problems whose 128 x 128 diagonal blocks are finished.
int launch_trinv_tc(int count, const FactorPlanes *problems, cudaStream_t stream) {
    static PerDeviceOnce configured;
    const size_t smem = (size_t)TRINV_STAGES * TRINV_STAGE_BYTES + 1024;
    if (configured.run([&] {
            return cudaFuncSetAttribute(trinv_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess &&
                   cudaFuncSetAttribute(trinv_duo_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess;
        }) != G2D_OK)
        return G2D_ERR_CUDA;
    TrinvJob all;
    int64_t n_max = 0;
    for (int z = 0; z < 2; ++z) {
        all.p[z] = problems[z < count ? z : 0];
        if (!factor_maps(&all.maps[z], all.p[z])) return G2D_ERR_CUDA;
        n_max = all.p[z].n > n_max ? all.p[z].n : n_max;
    }
    trinv_split_kernel<<<dim3((unsigned)(n_max < 148 * 16 ? n_max : 148 * 16), count), 256, 0, stream>>>(all.p[0], all.p[1]);
    if (check_launch() != G2D_OK) return G2D_ERR_CUDA;
    for (int64_t b = MT; b < n_max; b *= 2) {
        const int64_t tiles = b / MT, edge = b / DUO_EDGE;
        if (tiles > 65535) return G2D_ERR_TOO_LARGE;
        for (const bool two_ctas : {true, false}) {  // together what goes to the same kernel
            TrinvJob job = all;
            int mine = 0;
            int64_t largest = 0;
            for (int z = 0; z < count; ++z) {
                if (all.p[z].n <= b || two_ctas_pay(all.p[z].n, b) != two_ctas) continue;
                job.p[mine] = all.p[z];
                job.maps[mine] = all.maps[z];
                largest = all.p[z].n > largest ? all.p[z].n : largest;
                ++mine;
            }
            if (mine == 0) continue;
            const int64_t pairs = ceil_div(largest, 2 * b);
            if (pairs * mine > 0x7fffffff) return G2D_ERR_TOO_LARGE;
            job.pairs = (int)pairs;
            job.tiles = (int)tiles;
            job.b = b;
            for (int second = 0; second < 2; ++second) {
                job.second = second;
                if (two_ctas) {
                    if (launch_duo(trinv_duo_kernel, dim3((unsigned)(2 * edge * edge), (unsigned)(pairs * mine)), PAIR_THREADS, smem, stream, job) != G2D_OK) return G2D_ERR_CUDA;
                } else {
                    trinv_tc_kernel<<<dim3((unsigned)(pairs * mine), (unsigned)tiles, (unsigned)tiles), TC_THREADS, smem, stream>>>(job);
                    if (check_launch() != G2D_OK) return G2D_ERR_CUDA;
                }
            }
        }
    }
    return G2D_OK;
}

// ---- trailing update of the blocked Cholesky factorization ----
// After a group of four 64-row block rows [o, o + kw) is factored, everything above it receives
//     a[r][c] -= sum_{k < kw} a[o + k][r] a[o + k][c],      c <= r < o,
// a few tiles per CTA.  Both operands are the same K-major fp16 pairs pt[r][k] = 2^13 a[o + k][r], which the panel kernel writes
// as it finishes a block row.  M is equilibrated first (rows and columns scaled by powers of two, exactly, to diagonal
// entries in [1, 4)): the squares of T[., r] add up to M[r][r], so every entry of a panel is below 2 and one scale serves all
// of them.  One CTA owns each target entry and no other kernel touches the targets meanwhile, so the result does not depend on
// scheduling.
// Accuracy.  The tensor cores add each product into the float accumulator with truncation, which biases long sums of
// one sign by about 1e-8 of the sum per term, and the diagonal of this update is a sum of squares, subtracted from pivots
// that a damped, badly conditioned Gram leaves one or two orders of magnitude smaller than the sum.  Two measures keep the
// factors at the accuracy of a float32 LAPACK factorization: the k range is cut into slices of 128 (added up in registers, round
// to nearest), and the diagonal entries are left out and updated with a float64 sum of the float panel by CTAs of their own
// (the first ones of the launch, one per 128 rows).
// Bound: HBM for factors beyond L2 (8 bytes per entry and pair of groups, 512 rows: 61 GB at n = 28672, 10 ms), shared-memory port
// below (see pair_gemm).  n = 28672 and 8192 together: 73 ms with 128 x 128 tf32 tiles, 36 ms with a group at a time, 28 ms now.
constexpr int SYRK_SLICE_CHUNKS = 2;  // k = 128 per slice: as many additions into one accumulator as 64 take in tf32
static_assert(SYRK_TC_K % (2 * KH) == 0, "whole chunks per group");

struct SyrkJob {
    CUtensorMap a_hi[2], a_lo[2], b_hi[2], b_lo[2];  // the same planes in boxes of 128 and of NT rows
    CUtensorMap target[2];                           // the matrix itself in boxes of 16 x 32 (n a multiple of 4: its rows 16-byte multiples)
    float *a[2];
    int64_t n[2], o[2];    // size, first row of the group
    int t_lo[2], t_hi[2];  // target tile rows [t_lo, t_hi), with every tile column up to the diagonal
    int k0[2], kw[2];
    int tiles_per_cta;
    int *flag[2];
};
template <int NT>
constexpr int syrk_stages = NT == 256 ? 2 : 3;

template <int NT>
__global__ void __launch_bounds__(PAIR_THREADS, 1) syrk_tc_kernel(const __grid_constant__ SyrkJob job) {
    constexpr int MINE = NT / 2;
    extern __shared__ unsigned char tc_smem_raw[];
    __shared__ __align__(8) PairRing<syrk_stages<NT>> ring;
    const int z = blockIdx.y;
    const int t_lo = z ? job.t_lo[1] : job.t_lo[0], t_hi = z ? job.t_hi[1] : job.t_hi[0];
    float *const a = z ? job.a[1] : job.a[0];
    const int64_t n = z ? job.n[1] : job.n[0], o = z ? job.o[1] : job.o[0];
    const int k0 = z ? job.k0[1] : job.k0[0], kw = z ? job.kw[1] : job.kw[0];
    const int diagonals = t_hi - t_lo;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if ((int)blockIdx.x < diagonals) {
        // a[r][r] -= sum_k a[o + k][r]^2 for 128 rows r, lanes along r, warps along k
        double (*const part)[MT] = reinterpret_cast<double (*)[MT]>(tc_smem_raw);
        const int64_t r0 = (int64_t)(t_lo + (int)blockIdx.x) * MT + lane;
        double sum[4] = {0., 0., 0., 0.};
#pragma unroll 4
        for (int k = warp; k < kw; k += PAIR_THREADS / 32) {
            const float *src = a + (o + k) * n + r0;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const double v = (double)src[e * 32];
                sum[e] += v * v;
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) part[warp][e * 32 + lane] = sum[e];
        __syncthreads();
        if (threadIdx.x < MT) {
            double all = 0.;
            for (int w = 0; w < PAIR_THREADS / 32; ++w) all += part[w][threadIdx.x];
            const int64_t r = (int64_t)(t_lo + (int)blockIdx.x) * MT + threadIdx.x;
            a[r * n + r] = (float)((double)a[r * n + r] - all);
        }
        return;
    }
    const int64_t first = lower_tiles<NT>(t_lo) + ((int64_t)blockIdx.x - diagonals) * job.tiles_per_cta, last = lower_tiles<NT>(t_hi);
    if (first >= last) return;
    const CUtensorMap *a_hi = z ? &job.a_hi[1] : &job.a_hi[0], *a_lo = z ? &job.a_lo[1] : &job.a_lo[0];
    const CUtensorMap *b_hi = z ? &job.b_hi[1] : &job.b_hi[0], *b_lo = z ? &job.b_lo[1] : &job.b_lo[0];
    const bool vec = n % 4 == 0;
    const uint32_t smem_base = (smem_u32(tc_smem_raw) + 1023u) & ~1023u;
    int I_first, J_first;
    lower_tile<NT>(first, I_first, J_first);
    auto next = [&](int it, PairTile &t) {
        if (it >= job.tiles_per_cta || first + it >= last) return false;
        int I2 = I_first, J2 = J_first + it;
        for (int row; J2 >= (row = NT == 256 ? I2 / 2 + 1 : I2 + 1); ++I2) J2 -= row;
        t = PairTile{I2 * MT, J2 * NT, (kw + KH - 1) / KH, k0};
        return true;
    };
    auto load = [&](const PairTile &t, int ch, uint32_t dst, uint64_t *bar) {
        const int k = t.k0 + ch * KH;
        tma_load_2d(dst, a_hi, k, t.i0, bar);
        tma_load_2d(dst + HTILE_BYTES, a_lo, k, t.i0, bar);
        tma_load_2d(dst + 2 * HTILE_BYTES, b_hi, k, t.j0, bar);
        tma_load_2d(dst + 2 * HTILE_BYTES + NT * KH * 2, b_lo, k, t.j0, bar);
    };
    constexpr float UNSCALE = -1.f / (SYRK_PANEL_SCALE * SYRK_PANEL_SCALE);
    const CUtensorMap *target = z ? &job.target[1] : &job.target[0];
    auto finish = [&](const PairTile &t, int q, int ln, int c0, float (&total)[MINE], uint32_t box) {
        const int i0 = t.i0 + q * 32, gi = i0 + ln;  // always a row of the matrix: the targets lie above the group
        if (vec) {
#pragma unroll
            for (int cb = 0; cb < MINE / 32; ++cb) {
                const int gj0 = t.j0 + c0 + cb * 32;
                if (gj0 > i0 + 31) continue;  // warp-uniform
                if (gj0 + 31 >= i0) {
                    // the diagonal entries are updated above; what lies right of the diagonal is never read: both get zeros
#pragma unroll
                    for (int x = 0; x < 32; ++x) total[cb * 32 + x] = gj0 + x < gi ? total[cb * 32 + x] : 0.f;
                }
                add_block<false>(target, box, ln, total + cb * 32, UNSCALE, gj0, i0, true, (int)n);
            }
            return;
        }
#pragma unroll
        for (int x = 0; x < MINE; ++x) {
            const int gj = t.j0 + c0 + x;
            if (gj < gi) asm volatile("red.global.add.f32 [%0], %1;" ::"l"(a + (int64_t)gi * n + gj), "f"(UNSCALE * total[x]) : "memory");
        }
    };
    const bool failed = pair_gemm<NT, syrk_stages<NT>, SYRK_SLICE_CHUNKS>(ring, smem_base, next, load, finish);
    int *const flag = z ? job.flag[1] : job.flag[0];
    if (threadIdx.x == 0 && failed && flag) atomicExch(flag, -1);
}

bool syrk_tc_maps(SyrkTcMaps *maps, const __half *pt_hi, const __half *pt_lo, float *a, int64_t n) {
    static_assert(sizeof(maps->hi) == sizeof(CUtensorMap), "opaque tensor-map storage has the wrong size");
    if (n % 4 == 0 && !make_map(reinterpret_cast<CUtensorMap *>(maps->target), a, n, n, HALF_BOX_ROWS)) return false;
    return make_map_16(reinterpret_cast<CUtensorMap *>(maps->hi), pt_hi, n, SYRK_TC_K, MT) &&
           make_map_16(reinterpret_cast<CUtensorMap *>(maps->lo), pt_lo, n, SYRK_TC_K, MT) &&
           make_map_16(reinterpret_cast<CUtensorMap *>(maps->wide_hi), pt_hi, n, SYRK_TC_K, 256) &&
           make_map_16(reinterpret_cast<CUtensorMap *>(maps->wide_lo), pt_lo, n, SYRK_TC_K, 256);
}

template <int NT>
static int launch_syrk_tiles(int count, const SyrkJob &job, int64_t blocks, cudaStream_t stream) {
    static PerDeviceOnce configured;
    constexpr size_t smem = (size_t)syrk_stages<NT> * pair_stage_bytes<NT> + PAIR_BOXES + 1024;
    if (configured.run([&] { return cudaFuncSetAttribute(syrk_tc_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess; }) != G2D_OK)
        return G2D_ERR_CUDA;
    syrk_tc_kernel<NT><<<dim3((unsigned)blocks, count), PAIR_THREADS, smem, stream>>>(job);
    return check_launch();
}

int launch_syrk_tc(int count, const SyrkTcTarget *targets, cudaStream_t stream) {
    SyrkJob job;
    int64_t wide = 0, square = 0;
    for (int z = 0; z < count; ++z) {
        wide += lower_tiles<256>(targets[z].t_hi) - lower_tiles<256>(targets[z].t_lo);
        square += lower_tiles<128>(targets[z].t_hi) - lower_tiles<128>(targets[z].t_lo);
    }
    if (square <= 0) return G2D_OK;
    const bool use_wide = tiles_that_pay(square, wide) == WIDE_TILES;
    // Several tiles per CTA once there are more than two waves of them, but few enough that an SM comes free every other
    // moment: the diagonal blocks and panels of the next group, on a stream of higher priority, wait for one.
    const int64_t tiles = use_wide ? wide : square;
    job.tiles_per_cta = (int)(tiles / (2 * 148) < 1 ? 1 : tiles / (2 * 148) > 6 ? 6 : tiles / (2 * 148));
    int64_t blocks = 0;
    for (int z = 0; z < count; ++z) {
        const SyrkTcTarget &t = targets[z];
        const int64_t mine = use_wide ? lower_tiles<256>(t.t_hi) - lower_tiles<256>(t.t_lo) : lower_tiles<128>(t.t_hi) - lower_tiles<128>(t.t_lo);
        const int64_t need = ceil_div(mine, (int64_t)job.tiles_per_cta) + t.t_hi - t.t_lo;
        blocks = need > blocks ? need : blocks;
    }
    if (blocks > 0x7fffffff) return G2D_ERR_TOO_LARGE;
    for (int z = 0; z < 2; ++z) {
        const SyrkTcTarget &t = targets[z < count ? z : 0];
        memcpy(&job.a_hi[z], t.maps->hi, sizeof(CUtensorMap));
        memcpy(&job.a_lo[z], t.maps->lo, sizeof(CUtensorMap));
        memcpy(&job.b_hi[z], use_wide ? t.maps->wide_hi : t.maps->hi, sizeof(CUtensorMap));
        memcpy(&job.b_lo[z], use_wide ? t.maps->wide_lo : t.maps->lo, sizeof(CUtensorMap));
        memcpy(&job.target[z], t.maps->target, sizeof(CUtensorMap));
        job.a[z] = t.a;
        job.n[z] = t.n;
        job.o[z] = t.o;
        job.t_lo[z] = t.t_lo;
        job.t_hi[z] = t.t_hi;
        job.k0[z] = t.k0;
        job.kw[z] = t.kw;
        job.flag[z] = t.flag;
    }
    return use_wide ? launch_syrk_tiles<256>(count, job, blocks, stream) : launch_syrk_tiles<128>(count, job, blocks, stream);
}

// Equilibration: s[r] = 2^-e with sqrt(M[r][r]) in [2^e, 2^(e + 1)), M[r][c] *= s[r] s[c].  Exact short of the ends of the
// range of floats; the factor of the scaled matrix is T diag(s), and the rows of its inverse are scaled back at the end.
__global__ void equilibrate_scale_kernel(Equilibration q) {
    const int z = blockIdx.y;
    const int64_t n = q.n[z];
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float root = sqrtf(q.a[z][i * n + i]);
        const int e = (int)((__float_as_uint(root) >> 23) & 255) - 127;
        q.s[z][i] = root > 0.f && e < 128 ? power_of_two(-e) : 1.f;  // not a positive definite matrix: the pivots will tell
    }
}
__global__ void __launch_bounds__(256) equilibrate_kernel(Equilibration q) {
    const int z = blockIdx.y;
    const int64_t n = q.n[z];
    const float *s = q.s[z];
    for (int64_t r = blockIdx.x; r < n; r += gridDim.x) {
        float *row = q.a[z] + r * n;
        const float sr = s[r];
        if (n % 4 == 0) {
            for (int64_t c = (int64_t)threadIdx.x * 4; c <= r; c += (int64_t)blockDim.x * 4) {  // a group may reach past the diagonal: never read there
                float4 v = *reinterpret_cast<const float4 *>(row + c);
                const float4 sc = *reinterpret_cast<const float4 *>(s + c);
                v.x = v.x * sr * sc.x; v.y = v.y * sr * sc.y; v.z = v.z * sr * sc.z; v.w = v.w * sr * sc.w;
                *reinterpret_cast<float4 *>(row + c) = v;
            }
        } else {
            for (int64_t c = threadIdx.x; c <= r; c += blockDim.x) row[c] = row[c] * sr * s[c];
        }
    }
}
int launch_equilibrate(int count, const Equilibration &q, cudaStream_t stream) {
    const int64_t most = count > 1 && q.n[1] > q.n[0] ? q.n[1] : q.n[0];
    equilibrate_scale_kernel<<<dim3((unsigned)(ceil_div(most, (int64_t)128) < 592 ? ceil_div(most, (int64_t)128) : 592), count), 128, 0, stream>>>(q);
    if (check_launch() != G2D_OK) return G2D_ERR_CUDA;
    equilibrate_kernel<<<dim3((unsigned)(most < 148 * 16 ? most : 148 * 16), count), 256, 0, stream>>>(q);
    return check_launch();
}

}  // namespace g2d

// Hessian-factor accumulation on the tensor cores (float only): H += alpha X^T X for a batch of activations
// X [k samples, n channels], the step before ldl_of_inverse in a quantization pipeline.  The reference takes its
// Hessian factors from the caller (demo.ipynb:103-106 forms them with a plain matrix product), so this entry has no
// counterpart there.
//
// X^T is first written as K-major fp16 pairs [n][k], every channel scaled by a power of two of its own (the channel is the
// index that is not summed over, so the scale comes out of the product again), then every 256 x 256 tile that touches the
// lower triangle of H is that of a cluster of two CTAs (one CTA per SM; smaller tiles where those fill their waves better, see
// tiles_that_pay): TMA into a three-stage ring of 64 KB in each, tcgen05.mma kind::f16 with three products per k step into tensor memory, eight warps that add the accumulators up in registers slice of k by slice of k, and at the end
// write H and its mirror image.  Every entry of H has one owner, so the result does not depend on scheduling.
//
// Bound: tensor pipe.  A 128 x 256 x 16 MMA of one CTA reads 12 KB of operands in 128 cycles and a chunk's 96 KB arrive in the 1536 cycles
// of its MMAs: 160 of the port's 128 bytes per cycle, so 80 % of the tensor rate.  Two CTAs with half of B each read 8 KB and
// fill 64 KB: 107 bytes per cycle.  8192 samples of 8192 channels, calls one after the other: 4.61 ms with 128 x 128 tf32 tiles (60 % of half the
// rate, every slice added to H in global memory), 1.69 ms with 128 x 256, 1.54 ms now; with H cleared and the L2 emptied between calls 1.79 and
// 1.70.  2048 samples of 4096 channels 153 and 152 us.
#include "g2d_tc.cuh"

namespace g2d {

constexpr int GRAM_STAGES = 2, GRAM_DUO_STAGES = 3;
constexpr size_t GRAM_DUO_BYTES = 4 * HTILE_BYTES;  // 128 rows of A and of B, two planes each
// Slices of the k range (see pair_gemm): the diagonal of a Gram matrix is a sum of squares, which one accumulator over
// k = 8192 truncates to 9e-5 relative.
constexpr int GRAM_SLICE = 2;  // chunks per slice: 128 samples

// four neighbouring channels of a sample; `vec`: 16-byte aligned (n is a multiple of 4, the array itself may start anywhere)
__device__ __forceinline__ float4 four_channels(const float *p, bool vec) {
    return vec ? *reinterpret_cast<const float4 *>(p) : make_float4(p[0], p[1], p[2], p[3]);
}

// largest |x| of every channel, as the bits of a non-negative float
__global__ void gram_range_kernel(const float *__restrict__ x, int64_t k, int64_t n, int64_t rows_per_block, bool vec, unsigned *__restrict__ largest) {
    const int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (c >= n) return;
    const int64_t s0 = blockIdx.y * rows_per_block, s1 = min(k, s0 + rows_per_block);
    unsigned m[4] = {0u, 0u, 0u, 0u};
#pragma unroll 8
    for (int64_t s = s0; s < s1; ++s) {
        const float4 v = four_channels(x + s * n + c, vec);
        m[0] = max(m[0], __float_as_uint(v.x) & 0x7fffffffu);
        m[1] = max(m[1], __float_as_uint(v.y) & 0x7fffffffu);
        m[2] = max(m[2], __float_as_uint(v.z) & 0x7fffffffu);
        m[3] = max(m[3], __float_as_uint(v.w) & 0x7fffffffu);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) atomicMax(largest + c + e, m[e]);
}

// X [k][n] -> scaled pairs [n][kp], kp = k rounded up to a multiple of 8 (a TMA stride must be a multiple of 16 bytes); the
// padding columns are zero.  64 x 64 blocks through shared memory, 16-byte loads and stores.
// OWN_RANGE: the block finds its channels' largest values itself, from all of their samples.  For small inputs only, where
// a launch less (and the clearing of the array) is worth more than reading the samples once per block.
template <bool OWN_RANGE>
__global__ void __launch_bounds__(256) gram_split_transposed_kernel(const float *__restrict__ x, int64_t k, int64_t n, int64_t kp, bool vec,
                                                                    unsigned *__restrict__ largest, __half *__restrict__ hi, __half *__restrict__ lo) {
    __shared__ float tile[64][65];
    __shared__ unsigned range[64];
    const int tid = threadIdx.x;
    const int64_t j0 = (int64_t)blockIdx.x * 64, s0 = (int64_t)blockIdx.y * 64;
    if (OWN_RANGE) {
        if (tid < 64) range[tid] = 0u;
        __syncthreads();
        const int c = (tid & 15) * 4;
        unsigned m[4] = {0u, 0u, 0u, 0u};
        if (j0 + c < n) {
#pragma unroll 8
            for (int64_t s = tid >> 4; s < k; s += 16) {
                const float4 v = four_channels(x + s * n + j0 + c, vec);
                m[0] = max(m[0], __float_as_uint(v.x) & 0x7fffffffu);
                m[1] = max(m[1], __float_as_uint(v.y) & 0x7fffffffu);
                m[2] = max(m[2], __float_as_uint(v.z) & 0x7fffffffu);
                m[3] = max(m[3], __float_as_uint(v.w) & 0x7fffffffu);
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) atomicMax(&range[c + e], m[e]);
        __syncthreads();
        if (blockIdx.y == 0 && tid < 64 && j0 + tid < n) largest[j0 + tid] = range[tid];
    } else if (tid < 64 && j0 + tid < n) {
        range[tid] = largest[j0 + tid];
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const int idx = t * 256 + tid, r = idx >> 4, c = (idx & 15) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (s0 + r < k && j0 + c < n) v = four_channels(x + (s0 + r) * n + j0 + c, vec);
        tile[r][c] = v.x; tile[r][c + 1] = v.y; tile[r][c + 2] = v.z; tile[r][c + 3] = v.w;
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int idx = t * 256 + tid, j = idx >> 3, s = (idx & 7) * 8;
        if (j0 + j >= n || s0 + s >= kp) continue;
        const float scale = power_of_two(-range_exponent(__uint_as_float(range[j])));
        __align__(16) __half h[8];
        __align__(16) __half l[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) split_half(tile[s + e][j] * scale, h[e], l[e]);
        *reinterpret_cast<uint4 *>(hi + (j0 + j) * kp + s0 + s) = *reinterpret_cast<const uint4 *>(h);
        *reinterpret_cast<uint4 *>(lo + (j0 + j) * kp + s0 + s) = *reinterpret_cast<const uint4 *>(l);
    }
}

struct GramJob {
    CUtensorMap a_hi, a_lo, b_hi, b_lo;  // the same planes in boxes of 128 and of NT rows
    float *h;
    const unsigned *largest;
    int64_t n, tiles;
    int chunks;
    float alpha;
    int *flag;
    long long wait_cycles;  // limit of the waits
};

template <int NT, bool DUO>
__global__ void __launch_bounds__(PAIR_THREADS, 1) gram_tc_kernel(const __grid_constant__ GramJob job) {
    constexpr int MINE = NT / 2;  // columns per reading warp
    extern __shared__ unsigned char tc_smem_raw[];
    constexpr int NSTAGE = DUO ? GRAM_DUO_STAGES : GRAM_STAGES, B_ROWS = DUO ? NT / 2 : NT;
    __shared__ __align__(8) PairRing<NSTAGE> ring;
    const int rank = DUO ? (int)cluster_rank() : 0;
    const int64_t n = job.n;
    const uint32_t smem_base = (smem_u32(tc_smem_raw) + 1023u) & ~1023u;
    auto next = [&](int it, PairTile &t) {
        const int64_t lin = (blockIdx.x + (int64_t)it * gridDim.x) / (DUO ? 2 : 1);
        if (lin >= job.tiles) return false;
        int I2, J2;
        if (DUO) {
            lower_tile<128>(lin, I2, J2);
            I2 = 2 * I2 + rank;
        } else {
            lower_tile<NT>(lin, I2, J2);
        }
        t = PairTile{I2 * MT, J2 * NT, job.chunks};
        return true;
    };
    auto load = [&](const PairTile &t, int ch, uint32_t dst, uint64_t *bar) {
        const auto bring = [&](uint32_t to, const CUtensorMap *map, int row) {
            if (DUO) tma_load_2d_duo(to, map, ch * KH, row, leaders(bar));
            else tma_load_2d(to, map, ch * KH, row, bar);
        };
        bring(dst, &job.a_hi, t.i0);
        bring(dst + HTILE_BYTES, &job.a_lo, t.i0);
        bring(dst + 2 * HTILE_BYTES, &job.b_hi, t.j0 + rank * B_ROWS);
        bring(dst + 2 * HTILE_BYTES + B_ROWS * KH * 2, &job.b_lo, t.j0 + rank * B_ROWS);
    };
    auto finish = [&](const PairTile &t, int q, int lane, int c0, float (&total)[MINE], uint32_t) {
        const int64_t gi = (int64_t)t.i0 + q * 32 + lane;
        if (gi >= n) return;
        constexpr int GROUP = 16;
        const float row_scale = power_of_two(range_exponent(__uint_as_float(job.largest[gi])));
#pragma unroll
        for (int x0 = 0; x0 < MINE; x0 += GROUP) {
            const int64_t gj0 = (int64_t)t.j0 + c0 + x0;
            if (gj0 > gi) continue;  // the upper triangle is the mirror image of the lower one
            float *const dst = job.h + gi * n + gj0;
            // the old values of sixteen columns travel together, before the first is used
            const bool whole = gj0 + GROUP - 1 <= gi;
            float old[GROUP];
            if (whole) {
#pragma unroll
                for (int x = 0; x < GROUP; x += 4) {
                    const float4 v = *reinterpret_cast<const float4 *>(dst + x);
                    old[x] = v.x; old[x + 1] = v.y; old[x + 2] = v.z; old[x + 3] = v.w;
                }
            } else {
#pragma unroll
                for (int x = 0; x < GROUP; ++x) old[x] = gj0 + x <= gi ? dst[x] : 0.f;
            }
#pragma unroll
            for (int x = 0; x < GROUP; ++x) {
                const int64_t at = min(gj0 + x, n - 1);
                const float column_scale = power_of_two(range_exponent(__uint_as_float(job.largest[at])));
                // the smaller scale first: the other order could leave the range of floats on the way
                old[x] += job.alpha * (total[x0 + x] * fminf(row_scale, column_scale) * fmaxf(row_scale, column_scale));
            }
            if (whole) {
#pragma unroll
                for (int x = 0; x < GROUP; x += 4) *reinterpret_cast<float4 *>(dst + x) = make_float4(old[x], old[x + 1], old[x + 2], old[x + 3]);
            }
#pragma unroll
            for (int x = 0; x < GROUP; ++x) {
                if (!whole && gj0 + x <= gi) dst[x] = old[x];
                if (gj0 + x < gi) job.h[(gj0 + x) * n + gi] = old[x];  // consecutive lanes write consecutive columns
            }
        }
    };
    const bool failed = pair_gemm<NT, NSTAGE, GRAM_SLICE, DUO>(ring, smem_base, next, load, finish, PairNoScale(), job.wait_cycles);
    if (threadIdx.x == 0 && failed && job.flag) atomicExch(job.flag, -1);
}

template <int NT, bool DUO>
static int launch_gram(GramJob &job, const __half *hi, const __half *lo, int64_t kp, int64_t tiles, cudaStream_t st) {
    static PerDeviceOnce configured;
    constexpr size_t smem = (DUO ? GRAM_DUO_STAGES * GRAM_DUO_BYTES : (size_t)GRAM_STAGES * pair_stage_bytes<NT>) + 1024;
    constexpr int B_ROWS = DUO ? NT / 2 : NT;
    if (configured.run([&] { return cudaFuncSetAttribute(gram_tc_kernel<NT, DUO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess; }) != G2D_OK)
        return G2D_ERR_CUDA;
    if (!make_map_16(&job.a_hi, hi, job.n, kp, MT) || !make_map_16(&job.a_lo, lo, job.n, kp, MT) || !make_map_16(&job.b_hi, hi, job.n, kp, B_ROWS) ||
        !make_map_16(&job.b_lo, lo, job.n, kp, B_ROWS))
        return G2D_ERR_CUDA;
    job.tiles = tiles;
    if (DUO) return launch_duo(gram_tc_kernel<NT, DUO>, dim3(2 * (unsigned)(tiles < 74 ? tiles : 74)), PAIR_THREADS, smem, st, job);
    gram_tc_kernel<NT, DUO><<<(unsigned)(tiles < 148 ? tiles : 148), PAIR_THREADS, smem, st>>>(job);
    return check_launch();
}

}  // namespace g2d

using namespace g2d;

// samples rounded up to a multiple of 8 (16-byte strides), at least one k chunk
static int64_t gram_padded(int64_t k) { return k < KH ? KH : (k + 7) / 8 * 8; }

static size_t gram_plane(int64_t n, int64_t k) { return (2 * (size_t)n * (size_t)gram_padded(k) + 255) & ~(size_t)255; }
static size_t gram_bytes(int64_t n, int64_t k) { return 2 * gram_plane(n, k) + ((sizeof(unsigned) * (size_t)n + 255) & ~(size_t)255); }

extern "C" int g2d_gram_workspace_bytes(int64_t n, int64_t k, size_t *bytes) {
    if (n < 0 || k < 0 || !bytes) return G2D_ERR_BAD_ARGUMENT;
    *bytes = gram_bytes(n, k);
    return G2D_OK;
}

static int accumulate(int64_t n, int64_t k, const float *x, float alpha, float *h, int32_t *status_flag, void *workspace, size_t workspace_bytes, long long wait_cycles,
                      void *stream) {
    if (n < 0 || k < 0) return G2D_ERR_BAD_ARGUMENT;
    if (n == 0 || k == 0) return G2D_OK;
    if (!x || !h || n % 4 != 0 || ((uintptr_t)h & 15) != 0 || ((uintptr_t)x & 3) != 0) return G2D_ERR_BAD_ARGUMENT;
    if (!workspace || workspace_bytes < gram_bytes(n, k) || ((uintptr_t)workspace & 255) != 0) return G2D_ERR_WORKSPACE;
    const int64_t kp = gram_padded(k), rows = ceil_div(n, (int64_t)MT);
    if (rows * (rows + 1) / 2 > 0x7fffffff || kp > 0x3fffffff || ceil_div(kp, (int64_t)64) > 65535) return G2D_ERR_TOO_LARGE;
    cudaStream_t st = (cudaStream_t)stream;
    __half *hi = (__half *)workspace, *lo = (__half *)((char *)workspace + gram_plane(n, k));
    unsigned *largest = (unsigned *)((char *)workspace + 2 * gram_plane(n, k));
    const bool vec = ((uintptr_t)x & 15) == 0;
    const dim3 split_grid((unsigned)ceil_div(n, (int64_t)64), (unsigned)ceil_div(kp, (int64_t)64));
    // Both sides of the line, in us: 512 samples of 2048 channels 54 with the channels' ranges found in the same launch, 513 samples 62
    // with a launch of their own; 512 samples of 2052 channels 68.
    if (k <= 512 && n <= 2048) {
        gram_split_transposed_kernel<true><<<split_grid, 256, 0, st>>>(x, k, n, kp, vec, largest, hi, lo);
    } else {
        if (cudaMemsetAsync(largest, 0, sizeof(unsigned) * (size_t)n, st) != cudaSuccess) return G2D_ERR_CUDA;
        const int64_t across = ceil_div(n / 4, (int64_t)128);
        int64_t parts = ceil_div((int64_t)148 * 8, across);  // about eight blocks per SM, at least 32 samples each
        if (parts > ceil_div(k, (int64_t)32)) parts = ceil_div(k, (int64_t)32);
        const int64_t per = ceil_div(k, parts);
        gram_range_kernel<<<dim3((unsigned)across, (unsigned)ceil_div(k, per)), 128, 0, st>>>(x, k, n, per, vec, largest);
        if (check_launch() != G2D_OK) return G2D_ERR_CUDA;
        gram_split_transposed_kernel<false><<<split_grid, 256, 0, st>>>(x, k, n, kp, vec, largest, hi, lo);
    }
    if (check_launch() != G2D_OK) return G2D_ERR_CUDA;
    GramJob job;
    job.h = h;
    job.largest = largest;
    job.n = n;
    job.chunks = (int)ceil_div(kp, (int64_t)KH);
    job.alpha = alpha;
    job.flag = status_flag;
    job.wait_cycles = wait_cycles;
    const int64_t square = lower_tiles<128>(rows), wide = lower_tiles<256>(rows), duo = duo_tiles(ceil_div(rows, (int64_t)2));
    const TileChoice choice = tiles_that_pay(square, wide, duo);
    if (choice == DUO_TILES) return launch_gram<256, true>(job, hi, lo, kp, duo, st);
    if (choice == WIDE_TILES) return launch_gram<256, false>(job, hi, lo, kp, wide, st);
    return launch_gram<128, false>(job, hi, lo, kp, square, st);
}

extern "C" int g2d_gram_accumulate(int64_t n, int64_t k, const float *x, float alpha, float *h, int32_t *status_flag, void *workspace,
                                   size_t workspace_bytes, void *stream) {
    return accumulate(n, k, x, alpha, h, status_flag, workspace, workspace_bytes, WAIT_CYCLES, stream);
}

// For tests: with a limit of its own on the waits inside the kernel.  One that runs out sets *status_flag to -1 and leaves H incomplete.
extern "C" int g2d_gram_accumulate_limited(int64_t n, int64_t k, const float *x, float alpha, float *h, int32_t *status_flag, void *workspace,
                                           size_t workspace_bytes, int64_t wait_cycles, void *stream) {
    if (wait_cycles < 0 || wait_cycles > WAIT_CYCLES) return G2D_ERR_BAD_ARGUMENT;
    return accumulate(n, k, x, alpha, h, status_flag, workspace, workspace_bytes, wait_cycles, stream);
}

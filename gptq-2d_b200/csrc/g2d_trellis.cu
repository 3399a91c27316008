// Bitshift-trellis (QTIP) quantizer: Viterbi search as a shared-memory dynamic program.
//
// Replaces _viterbi_step_kernel / _viterbi_final_kernel / _viterbi_backtrack_kernel of the reference
// (quantizer_trellis.py:146-268) and reproduces _trellis_quantize_torch (:121-143) bit for bit: costs are
// (table - x)^2 summed over the V <= 2 values without fused multiply-adds, the running cost is added last,
// and every minimum takes the first index among equals.
//
// A state is an L-bit window; a step shifts in KV = K*V bits, so state s has the predecessors
// h * G + (s >> KV), h < 2^KV, G = 2^(L-KV).  All 2^KV states that share (s >> KV)... equivalently, the cost of a
// state is the minimum over its group of predecessors plus its own local cost, so only the G group minima
// of every step are kept:  B_t[g] = min_h (B_{t-1}[(h G + g) >> KV] + local_t[h G + g]).
// One CTA runs R sequences at once: B_t and B_{t-1} of each live in shared memory (2 R G values), every
// table entry is loaded once per step for all R sequences, and one barrier separates the steps.  The
// arg-min h of every (step, group) goes to global scratch (one byte each) for the walk back.
//
// Packed paths.  A path is also emitted as its bit string, the storage format of a trellis code (T K bits per sequence
// when tail-biting; the reference only notes that "the T K-bit code can be recovered", quantizer_trellis.py:11-14).
// The string is the sequence of the K V bits that every step shifts into the state, most significant bit first,
// preceded, when the path is not tail-biting, by the L - K V upper bits of the first state (tail-biting paths need no
// header: their first state continues the end of the string).  State t is then the L bits of the string that end
// with step t's symbol, read circularly for a tail-biting path.  Bit i of the string is bit i % 8 of byte i / 8.
#include "g2d_common.cuh"

namespace g2d {

constexpr int VT = 512;  // threads per CTA

template <typename F>
__device__ __forceinline__ F local_cost(const F *__restrict__ table, int64_t s, int V, F x0, F x1) {
    const F d0 = sub_rn(table[s * V], x0);
    F c = mul_rn(d0, d0);
    if (V == 2) {
        const F d1 = sub_rn(table[s * V + 1], x1);
        c = add_rn(c, mul_rn(d1, d1));
    }
    return c;
}

template <typename F>
__device__ __forceinline__ F pos_inf() { return (F)INFINITY; }

// the two values of a table entry in one load (V = 2: entries are pairs, naturally aligned)
__device__ __forceinline__ void load_pair(const float *p, float &a, float &b) {
    const float2 t = *reinterpret_cast<const float2 *>(p);
    a = t.x; b = t.y;
}
__device__ __forceinline__ void load_pair(const double *p, double &a, double &b) {
    const double2 t = *reinterpret_cast<const double2 *>(p);
    a = t.x; b = t.y;
}

template <typename F, int R>
__global__ void __launch_bounds__(VT) viterbi_kernel(int64_t rows, int T, const F *__restrict__ x, const F *__restrict__ table,
                                                     int Lbits, int shift, int V, int tail_biting, const F *__restrict__ scale,
                                                     F *__restrict__ out, int64_t *__restrict__ states, uint8_t *__restrict__ choices,
                                                     uint8_t *__restrict__ codes, int64_t code_bytes) {
    extern __shared__ __align__(16) unsigned char g2d_vsmem[];
    const int64_t S = (int64_t)1 << Lbits, G = S >> shift;
    const int H = 1 << shift;
    const int steps = T / V;
    F *B = reinterpret_cast<F *>(g2d_vsmem);  // [2][R][G]
    __shared__ F red_val[VT / 32][R];
    __shared__ long long red_arg[VT / 32][R];
    __shared__ long long seq_state[R];    // state at the step the walk back starts from / stops at
    __shared__ long long seq_overlap[R];  // tail-biting overlap bits, -1 when unconstrained
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t slots = steps > 1 ? steps - 1 : 1;

    for (int64_t row0 = (int64_t)blockIdx.x * R; row0 < rows; row0 += (int64_t)gridDim.x * R) {
        if (tid < R) seq_overlap[tid] = -1;
        __syncthreads();
        for (int pass = tail_biting ? 0 : 1; pass < 2; ++pass) {
            const int half = steps / 2;
            const int roll = pass == 0 ? steps - half : 0;
            const int stop = pass == 0 ? half : 0;
            // ---- forward: group minima of the steps 0 .. steps-2 ----
            for (int t = 0; t + 1 < steps; ++t) {
                const F *prev = B + (size_t)((t + 1) & 1) * R * G;
                F *next = B + (size_t)(t & 1) * R * G;
                F x0[R], x1[R];
                long long ov[R];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int64_t row = row0 + r < rows ? row0 + r : rows - 1;
                    const F *xt = x + row * T + (int64_t)((t + roll) % steps) * V;
                    x0[r] = xt[0];
                    x1[r] = V == 2 ? xt[1] : (F)0;
                    ov[r] = seq_overlap[r];
                }
                const int Gi = (int)G;  // the states fit 32-bit arithmetic (L <= 24)
                int ovi[R];
#pragma unroll
                for (int r = 0; r < R; ++r) ovi[r] = (int)ov[r];
                // The common shape (sixteen predecessors, pairs of values, not the first step) has a path of its own:
                // everything that the generic loop below derives per predecessor is a constant stride here.
                const bool fast = H == 16 && V == 2 && t > 0 && (Gi & 15) == 0;
                for (int g = tid; fast && g < Gi; g += VT) {
                    const F *entry = table + 2 * g;            // predecessor h: + h * 2 Gi
                    const F *before = prev + (g >> 4);         // its group minimum: + h * (Gi >> 4), + r * Gi
                    const int table_stride = 2 * Gi, low_stride = Gi >> 4;
                    F best[R];
                    int arg[R];
#pragma unroll
                    for (int half_h = 0; half_h < 2; ++half_h) {
                        F tt0[8], tt1[8];
#pragma unroll
                        for (int q = 0; q < 8; ++q) load_pair(entry + (half_h * 8 + q) * table_stride, tt0[q], tt1[q]);
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            const int h = half_h * 8 + q;
#pragma unroll
                            for (int r = 0; r < R; ++r) {
                                const F d0 = sub_rn(tt0[q], x0[r]), d1 = sub_rn(tt1[q], x1[r]);
                                const F c = add_rn(before[r * Gi + h * low_stride], add_rn(mul_rn(d0, d0), mul_rn(d1, d1)));
                                if (h == 0 || c < best[r]) { best[r] = c; arg[r] = h; }
                            }
                        }
                    }
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        next[r * Gi + g] = best[r];
                        if (row0 + r < rows) choices[((row0 + r) * slots + t) * G + g] = (uint8_t)arg[r];
                    }
                }
                for (int g = tid; !fast && g < Gi; g += VT) {
                    F best[R];
                    int arg[R];
#pragma unroll
                    for (int r = 0; r < R; ++r) { best[r] = pos_inf<F>(); arg[r] = 0; }
                    // the table entries of eight predecessors are fetched before any of them is used: a thread's loads
                    // (L2 hits: the table is larger than L1) overlap instead of queueing behind the running minimum
                    constexpr int HB = 8;
                    for (int h0 = 0; h0 < H; h0 += HB) {
                        F tt0[HB], tt1[HB];
#pragma unroll
                        for (int q = 0; q < HB; ++q) {
                            const int s = (h0 + q < H ? h0 + q : H - 1) * Gi + g;
                            if (V == 2) {
                                load_pair(table + 2 * s, tt0[q], tt1[q]);
                            } else {
                                tt0[q] = table[s];
                                tt1[q] = (F)0;
                            }
                        }
#pragma unroll
                        for (int q = 0; q < HB; ++q) {
                            const int h = h0 + q;
                            if (h >= H) break;
                            const int low = (h * Gi + g) >> shift;
                            const F t0 = tt0[q], t1 = tt1[q];
#pragma unroll
                            for (int r = 0; r < R; ++r) {
                                const F d0 = sub_rn(t0, x0[r]);
                                F c = mul_rn(d0, d0);
                                if (V == 2) {
                                    const F d1 = sub_rn(t1, x1[r]);
                                    c = add_rn(c, mul_rn(d1, d1));
                                }
                                if (t == 0) {
                                    if (ovi[r] >= 0 && low != ovi[r]) c = pos_inf<F>();
                                } else {
                                    c = add_rn(prev[r * Gi + low], c);
                                }
                                if (h == 0 || c < best[r]) { best[r] = c; arg[r] = h; }
                            }
                        }
                    }
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        next[(size_t)r * G + g] = best[r];
                        if (row0 + r < rows) choices[((row0 + r) * slots + t) * G + g] = (uint8_t)arg[r];
                    }
                }
                __syncthreads();
            }
            // ---- last step: first arg-min over all states, with the final mask ----
            {
                const int t = steps - 1;
                const F *prev = B + (size_t)((t + 1) & 1) * R * G;
                F best[R];
                long long arg[R];
#pragma unroll
                for (int r = 0; r < R; ++r) { best[r] = pos_inf<F>(); arg[r] = S; }
                F x0[R], x1[R];
                long long ov[R];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int64_t row = row0 + r < rows ? row0 + r : rows - 1;
                    const F *xt = x + row * T + (int64_t)((t + roll) % steps) * V;
                    x0[r] = xt[0];
                    x1[r] = V == 2 ? xt[1] : (F)0;
                    ov[r] = seq_overlap[r];
                }
                for (int64_t s = tid; s < S; s += VT) {
                    const F t0 = table[s * V], t1 = V == 2 ? table[s * V + 1] : (F)0;
                    const int64_t low = s >> shift;
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const F d0 = sub_rn(t0, x0[r]);
                        F c = mul_rn(d0, d0);
                        if (V == 2) {
                            const F d1 = sub_rn(t1, x1[r]);
                            c = add_rn(c, mul_rn(d1, d1));
                        }
                        if (t == 0) {
                            if (ov[r] >= 0 && low != ov[r]) c = pos_inf<F>();
                        } else {
                            c = add_rn(prev[(size_t)r * G + low], c);
                        }
                        if (ov[r] >= 0 && (s & (G - 1)) != ov[r]) c = pos_inf<F>();
                        // ascending s within a thread: strict < keeps the first minimum
                        if (arg[r] == S || c < best[r]) { best[r] = c; arg[r] = s; }
                    }
                }
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    F b = best[r];
                    long long a = arg[r];
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        const F ob = __shfl_xor_sync(0xffffffffu, b, o);
                        const long long oa = __shfl_xor_sync(0xffffffffu, a, o);
                        if (oa < S && (a >= S || ob < b || (ob == b && oa < a))) { b = ob; a = oa; }
                    }
                    if (lane == 0) { red_val[warp][r] = b; red_arg[warp][r] = a; }
                }
                __syncthreads();
                if (tid < R) {
                    F b = red_val[0][tid];
                    long long a = red_arg[0][tid];
                    for (int w = 1; w < VT / 32; ++w) {
                        const F ob = red_val[w][tid];
                        const long long oa = red_arg[w][tid];
                        if (oa < S && (a >= S || ob < b || (ob == b && oa < a))) { b = ob; a = oa; }
                    }
                    seq_state[tid] = a;
                }
                __syncthreads();
            }
            // ---- walk back: thread r follows sequence r ----
            if (tid < R && row0 + tid < rows) {
                const int64_t row = row0 + tid;
                long long state = seq_state[tid];
                const F sc = scale ? scale[row] : (F)1;
                uint8_t *code = (pass == 1 && codes) ? codes + row * code_bytes : nullptr;
                const int header = tail_biting ? 0 : Lbits - shift;
                if (code)
                    for (int64_t b = 0; b < code_bytes; ++b) code[b] = 0;
                for (int t = steps - 1; t >= stop; --t) {
                    if (pass == 1) {
                        for (int v = 0; v < V; ++v) out[row * T + (int64_t)t * V + v] = mul_rn(table[state * V + v], sc);
                        if (states) states[row * steps + t] = state;
                        if (code) {
                            // this step's symbol, most significant bit first; the first state's upper bits when a header is kept
                            for (int b = 0; b < shift; ++b) {
                                const int64_t at = header + (int64_t)t * shift + b;
                                if ((state >> (shift - 1 - b)) & 1) code[at >> 3] |= (uint8_t)(1u << (at & 7));
                            }
                            if (t == 0)
                                for (int b = 0; b < header; ++b)
                                    if ((state >> (Lbits - 1 - b)) & 1) code[b >> 3] |= (uint8_t)(1u << (b & 7));
                        }
                    }
                    if (t > stop) {
                        const long long low = state >> shift;
                        state = (long long)choices[(row * slots + (t - 1)) * G + low] * G + low;
                    }
                }
                if (pass == 0) seq_overlap[tid] = state >> shift;
            }
            __syncthreads();
        }
    }
}

// The same search for a code table with few distinct rows.  The shipped codes map 2^16 states onto about a thousand
// distinct value tuples (HYB: 2^9 lookup rows times a sign; 1MAD: a sum of four bytes), and the local cost of a state
// depends on its tuple only.  With the states' tuple numbers (`ids`, 16 bits each, the whole array in shared memory) and
// the distinct tuples, a step first forms the D local costs of every sequence (the same subtractions, products and sum
// as above, so the same bits), then every state costs one shared-memory lookup and one addition instead of a table load
// from L2 and five arithmetic instructions.  A thread takes eight neighbouring groups at a time: their tuple numbers are
// one 16-byte load and they share their predecessors' group minimum.  Results are bit for bit those of viterbi_kernel.
template <typename F, int R>
__global__ void __launch_bounds__(VT) viterbi_indexed_kernel(int64_t rows, int T, const F *__restrict__ x, const F *__restrict__ table,
                                                             const F *__restrict__ distinct, int D, const uint16_t *__restrict__ ids,
                                                             int Lbits, int shift, int V, int tail_biting, const F *__restrict__ scale,
                                                             F *__restrict__ out, int64_t *__restrict__ states, uint8_t *__restrict__ choices,
                                                             uint8_t *__restrict__ codes, int64_t code_bytes) {
    extern __shared__ __align__(16) unsigned char g2d_vsmem[];
    const int S = 1 << Lbits, G = S >> shift, H = 1 << shift;
    const int steps = T / V;
    uint16_t *id_s = reinterpret_cast<uint16_t *>(g2d_vsmem);                        // [S]
    F *B = reinterpret_cast<F *>(g2d_vsmem + (size_t)S * sizeof(uint16_t));          // [2][R][G]
    F *dist = B + (size_t)2 * R * G;                                                 // [R][D]
    __shared__ F red_val[VT / 32][R];
    __shared__ int red_arg[VT / 32][R];
    __shared__ int seq_state[R], seq_overlap[R];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t slots = steps > 1 ? steps - 1 : 1;
    for (int i = tid; i < S / 8; i += VT) reinterpret_cast<uint4 *>(id_s)[i] = reinterpret_cast<const uint4 *>(ids)[i];

    for (int64_t row0 = (int64_t)blockIdx.x * R; row0 < rows; row0 += (int64_t)gridDim.x * R) {
        if (tid < R) seq_overlap[tid] = -1;
        __syncthreads();
        for (int pass = tail_biting ? 0 : 1; pass < 2; ++pass) {
            const int half = steps / 2;
            const int roll = pass == 0 ? steps - half : 0;
            const int stop = pass == 0 ? half : 0;
            for (int t = 0; t < steps; ++t) {
                const bool last = t == steps - 1;
                const F *prev = B + (size_t)((t + 1) & 1) * R * G;
                F *next = B + (size_t)(t & 1) * R * G;
                F x0[R], x1[R];
                int ov[R];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int64_t row = row0 + r < rows ? row0 + r : rows - 1;
                    const F *xt = x + row * T + (int64_t)((t + roll) % steps) * V;
                    x0[r] = xt[0];
                    x1[r] = V == 2 ? xt[1] : (F)0;
                    ov[r] = seq_overlap[r];
                }
                // the local cost of every distinct tuple, for every sequence of the CTA
                for (int d = tid; d < D; d += VT) {
                    const F t0 = distinct[(int64_t)d * V], t1 = V == 2 ? distinct[(int64_t)d * V + 1] : (F)0;
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const F d0 = sub_rn(t0, x0[r]);
                        F c = mul_rn(d0, d0);
                        if (V == 2) {
                            const F d1 = sub_rn(t1, x1[r]);
                            c = add_rn(c, mul_rn(d1, d1));
                        }
                        dist[r * D + d] = c;
                    }
                }
                __syncthreads();
                if (!last) {
                    // group minima of this step: eight neighbouring groups per thread and round
                    for (int g0 = tid * 8; g0 < G; g0 += VT * 8) {
                        F best[R][8];
                        int arg[R][8];
                        for (int h = 0; h < H; ++h) {
                            const uint4 packed = *reinterpret_cast<const uint4 *>(id_s + (size_t)h * G + g0);
                            const uint32_t word[4] = {packed.x, packed.y, packed.z, packed.w};
                            const int low = (h * G + g0) >> shift;  // shared by the eight groups when shift >= 3
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                const int id = (word[e >> 1] >> ((e & 1) * 16)) & 0xFFFF;
                                const int low_e = shift >= 3 ? low : (h * G + g0 + e) >> shift;
#pragma unroll
                                for (int r = 0; r < R; ++r) {
                                    F c = dist[r * D + id];
                                    if (t == 0) {
                                        if (ov[r] >= 0 && low_e != ov[r]) c = pos_inf<F>();
                                    } else {
                                        c = add_rn(prev[r * G + low_e], c);
                                    }
                                    if (h == 0 || c < best[r][e]) { best[r][e] = c; arg[r][e] = h; }
                                }
                            }
                        }
#pragma unroll
                        for (int r = 0; r < R; ++r)
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                next[r * G + g0 + e] = best[r][e];
                                if (row0 + r < rows) choices[((row0 + r) * slots + t) * G + g0 + e] = (uint8_t)arg[r][e];
                            }
                    }
                    __syncthreads();
                } else {
                    // last step: first arg-min over all states, with the final mask
                    F best[R];
                    int arg[R];
#pragma unroll
                    for (int r = 0; r < R; ++r) { best[r] = pos_inf<F>(); arg[r] = S; }
                    for (int s = tid; s < S; s += VT) {
                        const int id = id_s[s], low = s >> shift;
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            F c = dist[r * D + id];
                            if (t == 0) {
                                if (ov[r] >= 0 && low != ov[r]) c = pos_inf<F>();
                            } else {
                                c = add_rn(prev[r * G + low], c);
                            }
                            if (ov[r] >= 0 && (s & (G - 1)) != ov[r]) c = pos_inf<F>();
                            if (arg[r] == S || c < best[r]) { best[r] = c; arg[r] = s; }  // ascending s: strict < keeps the first minimum
                        }
                    }
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        F b = best[r];
                        int a = arg[r];
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) {
                            const F ob = __shfl_xor_sync(0xffffffffu, b, o);
                            const int oa = __shfl_xor_sync(0xffffffffu, a, o);
                            if (oa < S && (a >= S || ob < b || (ob == b && oa < a))) { b = ob; a = oa; }
                        }
                        if (lane == 0) { red_val[warp][r] = b; red_arg[warp][r] = a; }
                    }
                    __syncthreads();
                    if (tid < R) {
                        F b = red_val[0][tid];
                        int a = red_arg[0][tid];
                        for (int w = 1; w < VT / 32; ++w) {
                            const F ob = red_val[w][tid];
                            const int oa = red_arg[w][tid];
                            if (oa < S && (a >= S || ob < b || (ob == b && oa < a))) { b = ob; a = oa; }
                        }
                        seq_state[tid] = a;
                    }
                    __syncthreads();
                }
            }
            // ---- walk back: thread r follows sequence r ----
            if (tid < R && row0 + tid < rows) {
                const int64_t row = row0 + tid;
                long long state = seq_state[tid];
                const F sc = scale ? scale[row] : (F)1;
                uint8_t *code = (pass == 1 && codes) ? codes + row * code_bytes : nullptr;
                const int header = tail_biting ? 0 : Lbits - shift;
                if (code)
                    for (int64_t b = 0; b < code_bytes; ++b) code[b] = 0;
                for (int t = steps - 1; t >= stop; --t) {
                    if (pass == 1) {
                        for (int v = 0; v < V; ++v) out[row * T + (int64_t)t * V + v] = mul_rn(table[state * V + v], sc);
                        if (states) states[row * steps + t] = state;
                        if (code) {
                            for (int b = 0; b < shift; ++b) {
                                const int64_t at = header + (int64_t)t * shift + b;
                                if ((state >> (shift - 1 - b)) & 1) code[at >> 3] |= (uint8_t)(1u << (at & 7));
                            }
                            if (t == 0)
                                for (int b = 0; b < header; ++b)
                                    if ((state >> (Lbits - 1 - b)) & 1) code[b >> 3] |= (uint8_t)(1u << (b & 7));
                        }
                    }
                    if (t > stop) {
                        const long long low = state >> shift;
                        state = (long long)choices[(row * slots + (t - 1)) * G + low] * G + low;
                    }
                }
                if (pass == 0) seq_overlap[tid] = (int)(state >> shift);
            }
            __syncthreads();
        }
    }
}

// The search for 2^16 states in float, one sequence per cluster of four CTAs: every thread owns 32 states for good and
// keeps their table values in registers.
//
// A step of the search is 2^16 times (table - x)^2 summed, plus the group minimum of the predecessors, compared: nine
// operations per state with nothing to load but the minima (one per predecessor and up to 16 groups), 900 cycles on four
// SMs, against a table read or a look-up of the local cost per state in the kernels above (11 k cycles on one SM, bound by
// shared memory).  Four CTAs are what it takes to hold 2^16 value pairs in registers, and a coarse stage of a sweep
// rarely has more sequences than the GPU has clusters of four.  What a step adds is the exchange: the group minimum of
// g is needed by the CTA that owns the groups (g mod G / H) H .. + H - 1 and goes straight into its shared memory, counted in
// by an mbarrier there (650 cycles from one step to the next; a cluster barrier behind plain remote stores takes 1560).
// HYB, T = 256, 32 sequences (one coarse stage of a sweep): 1.47 ms on one SM each, 0.40 ms with the cluster barrier, 0.29 ms now.
//
// Mapping.  G = 2^16 / H groups, Gc = G / 4 per CTA.  A thread has NG neighbouring groups and NH = 32 / NG predecessors of
// each; with more than 32 predecessors per group, H / 32 neighbouring lanes share a group and settle its minimum by shuffle.
// The arg-mins of a thread's groups are packed into one unit of one or two bytes per step, kept in shared memory where
// they fit and in the global scratch otherwise.  The walk back is one warp's: its lanes fetch the units of the next
// steps for every choice that could lead there (1 + H + H^2 lanes), so that one round of latency settles several steps.
// Costs, sums and tie rules are those of viterbi_kernel: same values, same states.
constexpr int CT = 512;  // threads
constexpr int CCL = 4;   // CTAs per cluster
constexpr int CSTATES = 32;

__device__ __forceinline__ uint32_t remote(const void *p, uint32_t rank) {  // the same variable in another CTA of the cluster
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
// Stores that count towards the transaction count of an mbarrier of the same CTA as the destination
__device__ __forceinline__ void async_store(uint32_t at, float v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(at), "f"(v), "r"(bar) : "memory");
}
__device__ __forceinline__ void async_store(uint32_t at, float a, float b, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(at), "f"(a), "f"(b), "r"(bar) : "memory");
}
__device__ __forceinline__ void async_store(uint32_t at, float a, float b, float c, float d, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(at), "f"(a), "f"(b), "f"(c), "f"(d), "r"(bar)
                 : "memory");
}
// Bounded wait for a phase of this CTA's barrier; false when it ran out.
constexpr unsigned SEARCH_WAIT_CYCLES = 2000000000u;  // about a second
constexpr unsigned SEARCH_DRAIN_CYCLES = 1 << 20;      // half a millisecond: a store to another CTA is on its way for a few hundred cycles
__device__ __forceinline__ bool cluster_wait(uint32_t bar, uint32_t parity, unsigned limit) {
    if (limit == 0) return false;  // a test's wait: it runs out whether the phase is complete or not
    const unsigned start = (unsigned)clock();
    for (;;) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
        if ((unsigned)clock() - start > limit) return false;
    }
}
// Two floats in one register pair: the packed additions and products round each half on its own, so a pair of states costs one
// issue slot per operation and the same bits.
typedef unsigned long long pair32;
__device__ __forceinline__ pair32 pack2(float a, float b) { pair32 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void unpack2(pair32 v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ pair32 add2(pair32 a, pair32 b) { pair32 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ pair32 mul2(pair32 a, pair32 b) { pair32 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ void remote_store(uint32_t at, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory"); }
__device__ __forceinline__ void remote_store(uint32_t at, int v) { asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(at), "r"(v) : "memory"); }
__device__ __forceinline__ uint32_t remote_load_unit(uint32_t at, int bytes) {
    uint32_t v;
    if (bytes == 1) asm volatile("ld.shared::cluster.u8 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
    else asm volatile("ld.shared::cluster.u16 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
    return v;
}

// Set to -1 by a search whose bounded wait ran out; never cleared by a kernel (see g2d_search_status).
__device__ int search_status;

// Waits.  The four CTAs of a cluster are resident together, so a step's minima arrive unless the GPU is broken.  A wait that runs
// out all the same ends the CTA's steps one step later, so the others run out of minima as well; every wait between two
// cluster barriers being bounded, so are the barriers.  At the barrier that ends the pass the CTAs learn of one
// another's failure, the first of them overwrites the rows of the cluster from this one on with what no search returns (NaN,
// states of -1, codes of zeros) and sets the status word, and all of them stay until the stores on their way have landed.
template <int V, int LOG_NG>
__global__ void __launch_bounds__(CT, 1) viterbi_cluster_kernel(int64_t rows, int T, const float *__restrict__ x, const float *__restrict__ table, int shift,
                                                                int tail_biting, const float *__restrict__ scale, float *__restrict__ out,
                                                                int64_t *__restrict__ states, uint8_t *__restrict__ scratch, int64_t scratch_row,
                                                                int choices_in_smem, uint8_t *__restrict__ codes, int64_t code_bytes, unsigned wait_limit) {
    constexpr int NG = 1 << LOG_NG, NH = CSTATES / NG;
    extern __shared__ __align__(16) unsigned char g2d_vsmem[];
    const int H = 1 << shift, G = (1 << 16) >> shift, Gc = G / CCL, parts = H / NH;
    const int steps = T / V, slots = steps > 1 ? steps - 1 : 1;
    const int PW = Gc >= H ? Gc >> shift : 1;          // minima per predecessor number that this CTA's groups need
    const int period = G >> shift;                     // G / H
    const int minima = H * PW;
    const int units = CT / parts, unit_bytes = NG * shift > 8 ? 2 : 1;
    float *const prev = reinterpret_cast<float *>(g2d_vsmem);        // [2][H][PW]
    float *const xs = prev + 2 * minima;                             // [T]
    int *const path = reinterpret_cast<int *>(xs + T);               // [steps]
    uint8_t *const kept = reinterpret_cast<uint8_t *>(path + steps); // [slots][units] units
    __shared__ float red_val[CT / 32];
    __shared__ int red_arg[CT / 32];
    __shared__ float all_val[CCL];
    __shared__ int all_arg[CCL];
    __shared__ int overlap;
    __shared__ int late;    // a wait of this CTA ran out
    __shared__ int failed;  // a wait of one of the four CTAs did; read behind a cluster barrier
    __shared__ __align__(8) uint64_t arrived[2];  // the minima of a step have arrived in prev[0] / prev[1]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t rank = cluster_rank();
    const uint32_t bar0 = (uint32_t)__cvta_generic_to_shared(arrived);
    uint32_t phases = 0;  // bit b: parity of the next wait on arrived[b]
    if (tid == 0) {
        late = failed = 0;
        for (int b = 0; b < 2; ++b) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8 * b) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const int unit = tid / parts, part = tid % parts, gl0 = unit * NG, h0 = part * NH, g0 = (int)rank * Gc + gl0;

    // states in pairs: of neighbouring groups, or of neighbouring predecessors where a thread has one group
    pair32 tv[CSTATES / 2][V];
#pragma unroll
    for (int e = 0; e < CSTATES; e += 2) {
        const int s0 = (h0 + e / NG) * G + g0 + e % NG, s1 = (h0 + (e + 1) / NG) * G + g0 + (e + 1) % NG;
#pragma unroll
        for (int v = 0; v < V; ++v) tv[e / 2][v] = pack2(table[s0 * V + v], table[s1 * V + v]);
    }
    // where the minima of this thread's groups go: neighbouring groups are neighbours there too (PW is a multiple of NG)
    const int within = g0 & (period - 1);
    const uint32_t to_rank = Gc >= H ? (uint32_t)(within / PW) : 0u;
    const uint32_t to = remote(prev + (Gc >= H ? (g0 / period) * PW + (within & (PW - 1)) : g0), to_rank), to_bar = remote(arrived, to_rank);
    const int64_t clusters = gridDim.x / CCL;
    for (int64_t row = blockIdx.x / CCL; row < rows; row += clusters) {
        for (int i = tid; i < T; i += CT) xs[i] = x[row * T + i];
        if (tid == 0) overlap = -1;
        uint8_t *const far = scratch + row * scratch_row + (int64_t)rank * units * unit_bytes;  // + slot * CCL * units * unit_bytes
        __syncthreads();
        for (int pass = tail_biting ? 0 : 1; pass < 2; ++pass) {
            const int half = steps / 2, roll = pass == 0 ? steps - half : 0, stop = pass == 0 ? half : 0;
            const int ov = overlap;
            // "minima before the first step": nothing, or the tail-biting constraint on the predecessors
            for (int i = tid; i < minima; i += CT) {
                const int low = (i / PW) * period + (Gc >= H ? (int)rank * PW + i % PW : 0);
                prev[minima + i] = ov >= 0 && low != ov ? INFINITY : 0.f;
            }
            cluster_sync();  // every CTA is done with the last pass (and has its barriers initialised)
            float best[NG];
            int arg[NG];
            for (int t = 0; t < steps; ++t) {
                const float *const before = prev + ((t + 1) & 1) * minima + h0 * PW + (gl0 >> shift);
                int at = t + roll;
                if (at >= steps) at -= steps;
                const float x0 = xs[at * V], x1 = V == 2 ? xs[at * V + 1] : 0.f;
                const pair32 nx0 = pack2(-x0, -x0), nx1 = pack2(-x1, -x1);
                auto local = [&](int e) {  // the local costs of the pair e
                    const pair32 d0 = add2(tv[e][0], nx0);
                    pair32 c = mul2(d0, d0);
                    if constexpr (V == 2) {
                        const pair32 d1 = add2(tv[e][V - 1], nx1);
                        c = add2(c, mul2(d1, d1));
                    }
                    return c;
                };
                if constexpr (NG == 1) {
#pragma unroll
                    for (int hh = 0; hh < NH; hh += 2) {
                        float c0, c1;
                        unpack2(add2(pack2(before[hh * PW], before[(hh + 1) * PW]), local(hh / 2)), c0, c1);
                        if (hh == 0 || c0 < best[0]) { best[0] = c0; arg[0] = h0 + hh; }
                        if (c1 < best[0]) { best[0] = c1; arg[0] = h0 + hh + 1; }
                    }
                } else {
#pragma unroll
                    for (int hh = 0; hh < NH; ++hh) {
                        float pv = 0.f;
#pragma unroll
                        for (int q = 0; q < NG; q += 2) {
                            // neighbouring groups share their predecessor's minimum, as far as there are predecessors per group
                            if (q % NH == 0) pv = before[hh * PW + q / NH];
                            float c0, c1;
                            unpack2(add2(pack2(pv, pv), local((hh * NG + q) / 2)), c0, c1);
                            if (hh == 0 || c0 < best[q]) { best[q] = c0; arg[q] = h0 + hh; }
                            if (hh == 0 || c1 < best[q + 1]) { best[q + 1] = c1; arg[q + 1] = h0 + hh; }
                        }
                    }
                }
                if constexpr (NG == 1) {
                    for (int o = 1; o < parts; o <<= 1) {  // the lanes that share a group: smaller cost, then smaller number
                        const float ob = __shfl_xor_sync(0xffffffffu, best[0], o);
                        const int oa = __shfl_xor_sync(0xffffffffu, arg[0], o);
                        if (ob < best[0] || (ob == best[0] && oa < arg[0])) { best[0] = ob; arg[0] = oa; }
                    }
                }
                if (t + 1 < steps) {
                    const int buf = t & 1;
                    const uint32_t bar = bar0 + 8 * buf;
                    if (tid == 0) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(minima * (int)sizeof(float)) : "memory");
                    // Every thread of this CTA has read the minima of step t - 1 when the first of step t leaves.  A CTA overwrites
                    // a buffer two steps later, after it has received minima of the step between from every CTA of the
                    // cluster (each sends to all four), so it never overwrites what is still being read.
                    __syncthreads();
                    // Whether a wait of step t - 1 ran out.  The answer is used behind this step's own wait, so that the load is on its
                    // way meanwhile: the barrier that the next step would arm is the one whose phase is not complete.
                    const bool stop_here = late;
                    if (part == 0) {
                        const uint32_t at_buf = to + (uint32_t)(buf * minima * (int)sizeof(float)), at_bar = to_bar + 8 * buf;
                        if constexpr (NG == 1) {
                            if (Gc >= H) async_store(at_buf, best[0], at_bar);
                            else
                                for (uint32_t r = 0; r < CCL; ++r)
                                    async_store(remote(prev + g0, r) + (uint32_t)(buf * minima * (int)sizeof(float)), best[0], remote(arrived, r) + 8 * buf);
                        } else if constexpr (NG == 2) {
                            async_store(at_buf, best[0], best[1], at_bar);
                        } else {
#pragma unroll
                            for (int q = 0; q < NG; q += 4) async_store(at_buf + q * 4, best[q], best[q + 1], best[q + 2], best[q + 3], at_bar);
                        }
                        uint32_t packed = 0;
#pragma unroll
                        for (int q = 0; q < NG; ++q) packed |= (uint32_t)arg[q] << (q * shift);
                        uint8_t *const u = choices_in_smem ? kept + ((size_t)t * units + unit) * unit_bytes : far + ((int64_t)t * CCL * units + unit) * unit_bytes;
                        if (unit_bytes == 1) *u = (uint8_t)packed;
                        else *reinterpret_cast<uint16_t *>(u) = (uint16_t)packed;
                    }
                    if (!cluster_wait(bar, (phases >> buf) & 1, wait_limit)) late = 1;
                    phases ^= 1u << buf;
                    if (stop_here) break;
                }
            }
            // ---- first arg-min over all states of the last step, with the final mask ----
            float b = INFINITY;
            int a = 1 << 16;
#pragma unroll
            for (int q = 0; q < NG; ++q) {
                const float c = ov >= 0 && g0 + q != ov ? INFINITY : best[q];
                // a masked group offers its first state, as a masked search over its states would
                const int s = (ov >= 0 && g0 + q != ov ? 0 : arg[q]) * G + g0 + q;
                if (a == 1 << 16 || c < b || (c == b && s < a)) { b = c; a = s; }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ob = __shfl_xor_sync(0xffffffffu, b, o);
                const int oa = __shfl_xor_sync(0xffffffffu, a, o);
                if (ob < b || (ob == b && oa < a)) { b = ob; a = oa; }
            }
            if (lane == 0) { red_val[warp] = b; red_arg[warp] = a; }
            __syncthreads();
            if (late && tid < CCL) remote_store(remote(&failed, tid), 1);
            if (tid == 0) {
                for (int w = 1; w < CT / 32; ++w)
                    if (red_val[w] < b || (red_val[w] == b && red_arg[w] < a)) { b = red_val[w]; a = red_arg[w]; }
                remote_store(remote(all_val + rank, 0), b);
                remote_store(remote(all_arg + rank, 0), a);
            }
            if (!choices_in_smem) __threadfence();  // the walk back reads other CTAs' units
            cluster_sync();
            if (failed) break;
            // ---- walk back ----
            if (rank == 0 && warp == 0) {
                b = all_val[0];
                a = all_arg[0];
                for (int r = 1; r < CCL; ++r)
                    if (all_val[r] < b || (all_val[r] == b && all_arg[r] < a)) { b = all_val[r]; a = all_arg[r]; }
                const int levels = 1 + H + H * H <= 32 ? 3 : 1 + H <= 32 ? 2 : 1;
                // this lane's place: level 0 is the next step, level l the step reached through l choices
                int level = 0, combo = 0;
                if (lane >= 1 + H && levels >= 3) { level = 2; combo = lane - 1 - H; }
                else if (lane >= 1 && levels >= 2) { level = 1; combo = lane - 1; }
                const bool used = level == 0 ? lane == 0 : level == 1 ? combo < H : combo < H * H;
                int state = a;
                if (lane == 0) path[steps - 1] = state;
                for (int t = steps - 1; t > stop; t -= levels) {
                    int low = state >> shift;
                    if (level == 1) low = combo * period + (low >> shift);
                    if (level == 2) low = (combo & (H - 1)) * period + (((combo >> shift) * period + (low >> shift)) >> shift);
                    int choice = 0;
                    const int slot = t - 1 - level;
                    if (used && slot >= stop) {
                        const int owner = low / Gc, gl = low & (Gc - 1), u = gl >> LOG_NG;
                        const uint32_t packed =
                            choices_in_smem ? remote_load_unit(remote(kept + ((size_t)slot * units + u) * unit_bytes, (uint32_t)owner), unit_bytes)
                            : unit_bytes == 1 ? (uint32_t)__ldcg(scratch + row * scratch_row + ((int64_t)slot * CCL + owner) * units + u)
                                              : (uint32_t)__ldcg(reinterpret_cast<const uint16_t *>(scratch + row * scratch_row) + ((int64_t)slot * CCL + owner) * units + u);
                        choice = (int)(packed >> ((gl & (NG - 1)) * shift)) & (H - 1);
                    }
                    int from = 0;
                    for (int l = 0; l < levels && t - 1 - l >= stop; ++l) {
                        const int c = __shfl_sync(0xffffffffu, choice, l == 0 ? 0 : l == 1 ? 1 + from : 1 + H + from);
                        state = c * G + (state >> shift);
                        if (lane == 0) path[t - 1 - l] = state;
                        from = from * H + c;
                    }
                }
                if (lane == 0 && pass == 0)
                    for (int r = 0; r < CCL; ++r) remote_store(remote(&overlap, r), state >> shift);
            }
            cluster_sync();
        }
        if (failed) {
            if (rank == 0) {
                for (; row < rows; row += clusters) {
                    for (int t = tid; t < T; t += CT) out[row * T + t] = __int_as_float(0x7fc00000);
                    for (int t = tid; states && t < steps; t += CT) states[row * steps + t] = -1;
                    for (int64_t byte = tid; codes && byte < code_bytes; byte += CT) codes[row * code_bytes + byte] = 0;
                }
                if (tid == 0) atomicExch(&search_status, -1);
            }
            for (const unsigned start = (unsigned)clock(); (unsigned)clock() - start < SEARCH_DRAIN_CYCLES;) __nanosleep(1000);
            __syncthreads();
            cluster_sync();
            return;
        }
        if (rank == 0) {
            const float sc = scale ? scale[row] : 1.f;
            for (int t = tid; t < steps; t += CT) {
                const int state = path[t];
#pragma unroll
                for (int v = 0; v < V; ++v) out[row * T + (int64_t)t * V + v] = mul_rn(table[state * V + v], sc);
                if (states) states[row * steps + t] = state;
            }
            if (codes) {
                const int header = tail_biting ? 0 : 16 - shift;
                for (int64_t byte = tid; byte < code_bytes; byte += CT) {
                    uint32_t v = 0;
                    for (int k = 0; k < 8; ++k) {
                        const int64_t at = byte * 8 + k;
                        int bit = 0;
                        if (at < header) bit = path[0] >> (15 - (int)at) & 1;
                        else if (at - header < (int64_t)steps * shift) bit = path[(at - header) / shift] >> (shift - 1 - (int)((at - header) % shift)) & 1;
                        v |= (uint32_t)bit << k;
                    }
                    codes[row * code_bytes + byte] = (uint8_t)v;
                }
            }
        }
        __syncthreads();  // the next row reuses the buffers (other CTAs' ones are guarded by the first cluster_sync of its passes)
    }
}

template <int V, int LOG_NG>
static int launch_viterbi_cluster(int64_t rows, int T, const void *x, const void *table, int shift, int tail, const void *scale, void *out, int64_t *states,
                                  void *workspace, uint8_t *codes, int64_t code_bytes, unsigned wait_limit, cudaStream_t st) {
    static PerDeviceOnce configured;
    constexpr int NG = 1 << LOG_NG, NH = CSTATES / NG, LIMIT = 200 * 1024;
    const int H = 1 << shift, G = (1 << 16) >> shift, Gc = G / CCL, parts = H / NH, steps = T / V, slots = steps > 1 ? steps - 1 : 1;
    const int minima = Gc >= H ? Gc : H, unit_bytes = NG * shift > 8 ? 2 : 1;
    const size_t base = sizeof(float) * (2 * (size_t)minima + T) + sizeof(int) * (size_t)steps, kept = (size_t)slots * (CT / parts) * unit_bytes;
    const int in_smem = base + kept <= LIMIT;
    const size_t smem = base + (in_smem ? kept : 0);
    if (smem > LIMIT) return G2D_ERR_UNSUPPORTED;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(CCL);
    config.blockDim = dim3(CT);
    config.dynamicSmemBytes = LIMIT;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeClusterDimension;
    attribute.val.clusterDim.x = CCL;
    attribute.val.clusterDim.y = attribute.val.clusterDim.z = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    // Clusters that are resident together: fewer than SMs / 4, since a cluster lies within one of the GPU's partitions.  A grid of
    // more would deal sequences out to clusters that start when the others are done (148 sequences: 2.26 ms against 1.5).
    static int resident[64];
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || configured.run([&] {
            return cudaFuncSetAttribute(viterbi_cluster_kernel<V, LOG_NG>, cudaFuncAttributeMaxDynamicSharedMemorySize, LIMIT) == cudaSuccess &&
                   cudaOccupancyMaxActiveClusters(&resident[device], viterbi_cluster_kernel<V, LOG_NG>, &config) == cudaSuccess && resident[device] > 0;
        }) != G2D_OK)
        return G2D_ERR_CUDA;
    const int64_t clusters = rows < resident[device] ? rows : resident[device];
    config.gridDim = dim3((unsigned)(clusters * CCL));
    config.dynamicSmemBytes = smem;
    config.stream = st;
    const int64_t scratch_row = (int64_t)slots * G;  // what the scratch holds per row; the units take no more
    if (cudaLaunchKernelEx(&config, viterbi_cluster_kernel<V, LOG_NG>, rows, T, (const float *)x, (const float *)table, shift, tail, (const float *)scale,
                           (float *)out, states, (uint8_t *)workspace, scratch_row, in_smem, codes, code_bytes, wait_limit) != cudaSuccess)
        return G2D_ERR_CUDA;
    return check_launch();
}

// Float searches over 2^16 states with 4 to 256 predecessors per state, the path short enough for shared memory, choices that may
// be stored two bytes at a time; the others go to the kernels above.
static bool cluster_search_serves(int dtype, int T, int L, int shift, int V, const void *workspace) {
    return dtype == G2D_F32 && L == 16 && shift >= 2 && T >= 2 * V && T <= 8192 && ((uintptr_t)workspace & 1) == 0;
}
// Whether the cluster search is the faster one.  It takes 33 to 36 sequences at a time, each in a quarter of the time of the kernels
// above or less; those take 148, 296 (two per SM) or 592 (four) at a time.  Up to 148 sequences the cluster search wins throughout;
// beyond, `pair` and `four` are the rounds of it that take as long as one round of 296 and of 592 sequences.  Measured, in
// us at T = 64, cluster search and the other: V = 2, 4 bits per step: 296 sequences 695 / 695, 592: 1355 / 1166, 593: 1356 / 2269,
// 1184: 2663 / 2292; V = 1, 2 bits: 592: 4253 / 7895; V = 1, 8 bits: 148: 1831 / 2156, 224: 2545 / 2531, 592: 6474 / 3310.
static bool cluster_search_pays(int64_t rows, int shift, int V) {
    static const int pair[2][9] = {{0, 0, 16, 13, 14, 12, 11, 7, 7}, {0, 0, 15, 0, 9, 0, 11, 0, 7}};
    static const int four[2][9] = {{0, 0, 33, 27, 19, 16, 14, 10, 9}, {0, 0, 30, 0, 15, 0, 15, 0, 9}};
    const int64_t rounds = ceil_div(rows, (int64_t)33);
    return rows <= 148 || rounds <= (rows <= 296 ? pair[V - 1][shift] : four[V - 1][shift] * ceil_div(rows, (int64_t)592));
}
template <int V>
static int cluster_search(int64_t rows, int T, const void *x, const void *table, int shift, int tail, const void *scale, void *out, int64_t *states,
                          void *workspace, uint8_t *codes, int64_t code_bytes, unsigned wait_limit, cudaStream_t st) {
    switch (shift) {
    case 2: return launch_viterbi_cluster<V, 3>(rows, T, x, table, shift, tail, scale, out, states, workspace, codes, code_bytes, wait_limit, st);
    case 3: return launch_viterbi_cluster<V, 2>(rows, T, x, table, shift, tail, scale, out, states, workspace, codes, code_bytes, wait_limit, st);
    case 4: return launch_viterbi_cluster<V, 1>(rows, T, x, table, shift, tail, scale, out, states, workspace, codes, code_bytes, wait_limit, st);
    default: return launch_viterbi_cluster<V, 0>(rows, T, x, table, shift, tail, scale, out, states, workspace, codes, code_bytes, wait_limit, st);
    }
}

// Values (and optionally states) of stored bit strings: one thread per (sequence, step) rebuilds the state from the L
// bits of the string that end with the step's symbol.
template <typename F>
__global__ void trellis_decode_kernel(int64_t rows, int T, const uint8_t *__restrict__ codes, int64_t code_bytes, const F *__restrict__ table,
                                      int Lbits, int shift, int V, int tail_biting, const F *__restrict__ scale, F *__restrict__ out,
                                      int64_t *__restrict__ states) {
    const int steps = T / V;
    const int header = tail_biting ? 0 : Lbits - shift;
    const int64_t bits = header + (int64_t)steps * shift, total = rows * steps;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t row = idx / steps;
        const int t = (int)(idx % steps);
        const uint8_t *code = codes + row * code_bytes;
        const int64_t end = header + (int64_t)(t + 1) * shift;  // one past the last bit of the state
        long long state = 0;
        for (int b = 0; b < Lbits; ++b) {
            int64_t at = end - Lbits + b;
            if (at < 0) at += bits;  // tail-biting only: a string with a header always reaches back far enough
            state = (state << 1) | ((code[at >> 3] >> (at & 7)) & 1);
        }
        const F sc = scale ? scale[row] : (F)1;
        for (int v = 0; v < V; ++v) out[row * T + (int64_t)t * V + v] = mul_rn(table[state * V + v], sc);
        if (states) states[row * steps + t] = state;
    }
}

template <typename F, int R>
static int launch_viterbi(int64_t rows, int T, const void *x, const void *table, int L, int K, int V, int tail, const void *scale,
                          void *out, int64_t *states, void *workspace, uint8_t *codes, int64_t code_bytes, cudaStream_t st) {
    static PerDeviceOnce configured;
    const int64_t G = ((int64_t)1 << L) >> (K * V);
    const size_t smem = sizeof(F) * 2 * R * (size_t)G;
    if (configured.run([&] { return cudaFuncSetAttribute(viterbi_kernel<F, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) == cudaSuccess; }) != G2D_OK)
        return G2D_ERR_CUDA;
    int64_t blocks = ceil_div(rows, R);
    if (blocks > 148 * 8) blocks = 148 * 8;
    viterbi_kernel<F, R><<<(unsigned)blocks, VT, smem, st>>>(rows, T, (const F *)x, (const F *)table, L, K * V, V, tail, (const F *)scale,
                                                             (F *)out, states, (uint8_t *)workspace, codes, code_bytes);
    return check_launch();
}

template <typename F>
static int trellis_dispatch(int64_t rows, int T, const void *x, const void *table, int L, int K, int V, int tail, const void *scale,
                            void *out, int64_t *states, void *workspace, uint8_t *codes, int64_t code_bytes, cudaStream_t st) {
    const int64_t G = ((int64_t)1 << L) >> (K * V);
    const size_t per_seq = sizeof(F) * 2 * (size_t)G;
    const size_t budget = 200 * 1024;
    if (per_seq > budget) return G2D_ERR_TOO_LARGE;
    // More sequences per CTA share each table read and its address arithmetic, fewer finish a short coarse anti-diagonal
    // sooner.  Measured on B200 (HYB, L = 16, T = 256) one wave of CTAs with 1 / 2 / 4 sequences each takes 1.6 / 2.4 /
    // 4.3 ms, so the fewest sequences per CTA that still fit one wave of SMs win, and four per CTA beyond that.
    int R = 1;
    if (rows > 148 && 2 * per_seq <= budget) R = 2;
    if (rows > 2 * 148 && 4 * per_seq <= budget) R = 4;
    switch (R) {
    case 4: return launch_viterbi<F, 4>(rows, T, x, table, L, K, V, tail, scale, out, states, workspace, codes, code_bytes, st);
    case 2: return launch_viterbi<F, 2>(rows, T, x, table, L, K, V, tail, scale, out, states, workspace, codes, code_bytes, st);
    default: return launch_viterbi<F, 1>(rows, T, x, table, L, K, V, tail, scale, out, states, workspace, codes, code_bytes, st);
    }
}

int64_t trellis_code_bytes(int T, int L, int K, int V, int tail_biting) {
    const int64_t bits = (tail_biting ? 0 : L - K * V) + (int64_t)(T / V) * K * V;
    return (bits + 7) / 8;
}

size_t trellis_scratch_bytes(int dtype, int64_t rows, int T, int L, int K, int V) {
    const int64_t steps = T / V, slots = steps > 1 ? steps - 1 : 1, G = ((int64_t)1 << L) >> (K * V);
    (void)dtype;
    return ((size_t)rows * slots * G + 255) & ~(size_t)255;
}

template <typename F, int R>
static int launch_viterbi_indexed(int64_t rows, int T, const void *x, const void *table, const TrellisIndex &index, int L, int K, int V, int tail,
                                  const void *scale, void *out, int64_t *states, void *workspace, uint8_t *codes, int64_t code_bytes, cudaStream_t st) {
    static PerDeviceOnce configured;
    const int64_t S = (int64_t)1 << L, G = S >> (K * V);
    const size_t smem = (size_t)S * sizeof(uint16_t) + sizeof(F) * (2 * R * (size_t)G + (size_t)R * index.count);
    if (configured.run([&] { return cudaFuncSetAttribute(viterbi_indexed_kernel<F, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024) == cudaSuccess; }) != G2D_OK)
        return G2D_ERR_CUDA;
    int64_t blocks = ceil_div(rows, R);
    if (blocks > 148 * 8) blocks = 148 * 8;
    viterbi_indexed_kernel<F, R><<<(unsigned)blocks, VT, smem, st>>>(rows, T, (const F *)x, (const F *)table, (const F *)index.distinct, index.count,
                                                                     index.ids, L, K * V, V, tail, (const F *)scale, (F *)out, states,
                                                                     (uint8_t *)workspace, codes, code_bytes);
    return check_launch();
}

// The indexed search serves tables of up to 2^16 states whose distinct rows fit shared memory beside the group minima, and
// only calls of at most one sequence per SM.  Measured on B200 (HYB, L = 16, T = 256): 148 sequences take 1.58 ms against
// 1.87 ms for the search that reads the table from L2, but with two sequences per CTA the random look-ups of the local
// costs collide in the shared-memory banks (256 sequences: 3.6 ms against 2.6 ms; 4096: 49 ms against 30 ms), so larger
// calls keep the other kernel.
template <typename F>
static int indexed_sequences_per_cta(const TrellisIndex *index, int64_t rows, int L, int K, int V) {
    if (index == nullptr || index->ids == nullptr || index->distinct == nullptr || index->count <= 0) return 0;
    const int64_t S = (int64_t)1 << L, G = S >> (K * V);
    if (L > 16 || G < 8 || S < 8 || rows > 148) return 0;
    const size_t bytes = (size_t)S * 2 + sizeof(F) * (2 * (size_t)G + (size_t)index->count);
    return bytes <= 216 * 1024 ? 1 : 0;
}

int launch_trellis(int dtype, int64_t rows, int T, const void *x, const void *table, int L, int K, int V, int tail, const void *scale,
                   void *out, int64_t *states, void *workspace, uint8_t *codes, cudaStream_t st, const TrellisIndex *index) {
    const int64_t code_bytes = trellis_code_bytes(T, L, K, V, tail);
    if (cluster_search_serves(dtype, T, L, K * V, V, workspace) && cluster_search_pays(rows, K * V, V)) {
        if (V == 2) return cluster_search<2>(rows, T, x, table, K * V, tail, scale, out, states, workspace, codes, code_bytes, SEARCH_WAIT_CYCLES, st);
        return cluster_search<1>(rows, T, x, table, K * V, tail, scale, out, states, workspace, codes, code_bytes, SEARCH_WAIT_CYCLES, st);
    }
    const int R = dtype == G2D_F32 ? indexed_sequences_per_cta<float>(index, rows, L, K, V) : indexed_sequences_per_cta<double>(index, rows, L, K, V);
    if (R == 1 && dtype == G2D_F32) return launch_viterbi_indexed<float, 1>(rows, T, x, table, *index, L, K, V, tail, scale, out, states, workspace, codes, code_bytes, st);
    if (R == 1) return launch_viterbi_indexed<double, 1>(rows, T, x, table, *index, L, K, V, tail, scale, out, states, workspace, codes, code_bytes, st);
    return dtype == G2D_F32 ? trellis_dispatch<float>(rows, T, x, table, L, K, V, tail, scale, out, states, workspace, codes, code_bytes, st)
                            : trellis_dispatch<double>(rows, T, x, table, L, K, V, tail, scale, out, states, workspace, codes, code_bytes, st);
}

}  // namespace g2d

using namespace g2d;

static int trellis_check(int dtype, int64_t rows, int32_t T, int32_t L, int32_t K, int32_t V) {
    if (dtype != G2D_F32 && dtype != G2D_F64) return G2D_ERR_BAD_ARGUMENT;
    if (rows < 0 || T <= 0 || V < 1 || V > 2 || K < 1 || K * V > 8 || L < K * V || L > 24 || T % V != 0) return G2D_ERR_BAD_ARGUMENT;
    return G2D_OK;
}

extern "C" int g2d_trellis_workspace_bytes(int dtype, int64_t rows, int32_t T, int32_t L, int32_t K, int32_t V, size_t *bytes) {
    const int status = trellis_check(dtype, rows, T, L, K, V);
    if (status != G2D_OK || !bytes) return status != G2D_OK ? status : G2D_ERR_BAD_ARGUMENT;
    *bytes = trellis_scratch_bytes(dtype, rows, T, L, K, V);
    return G2D_OK;
}

extern "C" int g2d_trellis_quantize(int dtype, int64_t rows, int32_t T, const void *x, const void *table, int32_t L, int32_t K,
                                    int32_t V, int32_t tail_biting, const void *scale, void *out, int64_t *states,
                                    void *workspace, size_t workspace_bytes, void *stream) {
    const int status = trellis_check(dtype, rows, T, L, K, V);
    if (status != G2D_OK) return status;
    if (rows == 0) return G2D_OK;
    if (!x || !table || !out) return G2D_ERR_BAD_ARGUMENT;
    size_t need = 0;
    g2d_trellis_workspace_bytes(dtype, rows, T, L, K, V, &need);
    if (!workspace || workspace_bytes < need) return G2D_ERR_WORKSPACE;
    return launch_trellis(dtype, rows, T, x, table, L, K, V, tail_biting, scale, out, states, workspace, nullptr, (cudaStream_t)stream);
}

extern "C" int g2d_trellis_code_bytes(int32_t T, int32_t L, int32_t K, int32_t V, int32_t tail_biting, int64_t *bytes) {
    const int status = trellis_check(G2D_F32, 0, T, L, K, V);
    if (status != G2D_OK || !bytes) return status != G2D_OK ? status : G2D_ERR_BAD_ARGUMENT;
    *bytes = trellis_code_bytes(T, L, K, V, tail_biting);
    return G2D_OK;
}

extern "C" int g2d_trellis_quantize_packed(int dtype, int64_t rows, int32_t T, const void *x, const void *table, int32_t L, int32_t K,
                                           int32_t V, int32_t tail_biting, const void *scale, void *out, uint8_t *codes,
                                           void *workspace, size_t workspace_bytes, void *stream) {
    const int status = trellis_check(dtype, rows, T, L, K, V);
    if (status != G2D_OK) return status;
    if (rows == 0) return G2D_OK;
    if (!x || !table || !out || !codes) return G2D_ERR_BAD_ARGUMENT;
    if (!tail_biting && (int64_t)(T / V) * K * V + L - K * V < L) return G2D_ERR_BAD_ARGUMENT;
    if (!workspace || workspace_bytes < trellis_scratch_bytes(dtype, rows, T, L, K, V)) return G2D_ERR_WORKSPACE;
    return launch_trellis(dtype, rows, T, x, table, L, K, V, tail_biting, scale, out, nullptr, workspace, codes, (cudaStream_t)stream);
}

extern "C" int g2d_trellis_quantize_indexed(int dtype, int64_t rows, int32_t T, const void *x, const void *table, int32_t L, int32_t K,
                                            int32_t V, int32_t tail_biting, const void *scale, void *out, int64_t *states, uint8_t *codes,
                                            const void *distinct, int32_t distinct_count, const uint16_t *ids, void *workspace,
                                            size_t workspace_bytes, void *stream) {
    const int status = trellis_check(dtype, rows, T, L, K, V);
    if (status != G2D_OK) return status;
    if (rows == 0) return G2D_OK;
    if (!x || !table || !out || !distinct || !ids || distinct_count <= 0 || distinct_count > 65536) return G2D_ERR_BAD_ARGUMENT;
    if (((uintptr_t)ids & 15) != 0) return G2D_ERR_BAD_ARGUMENT;
    if (!workspace || workspace_bytes < trellis_scratch_bytes(dtype, rows, T, L, K, V)) return G2D_ERR_WORKSPACE;
    const TrellisIndex index{distinct, ids, distinct_count};
    return launch_trellis(dtype, rows, T, x, table, L, K, V, tail_biting, scale, out, states, workspace, codes, (cudaStream_t)stream, &index);
}

extern "C" int g2d_trellis_quantize_limited(int64_t rows, int32_t T, const void *x, const void *table, int32_t K, int32_t V, int32_t tail_biting,
                                            void *out, int64_t *states, uint8_t *codes, void *workspace, size_t workspace_bytes, int64_t wait_cycles,
                                            void *stream) {
    const int status = trellis_check(G2D_F32, rows, T, 16, K, V);
    if (status != G2D_OK) return status;
    if (rows == 0) return G2D_OK;
    if (!x || !table || !out || wait_cycles < 0 || wait_cycles > SEARCH_WAIT_CYCLES) return G2D_ERR_BAD_ARGUMENT;
    if (!workspace || workspace_bytes < trellis_scratch_bytes(G2D_F32, rows, T, 16, K, V)) return G2D_ERR_WORKSPACE;
    if (!cluster_search_serves(G2D_F32, T, 16, K * V, V, workspace)) return G2D_ERR_UNSUPPORTED;
    const int64_t code_bytes = trellis_code_bytes(T, 16, K, V, tail_biting);
    const auto search = V == 2 ? cluster_search<2> : cluster_search<1>;
    return search(rows, T, x, table, K * V, tail_biting, nullptr, out, states, workspace, codes, code_bytes, (unsigned)wait_cycles, (cudaStream_t)stream);
}

extern "C" int g2d_search_status(int32_t *status) {
    if (!status) return G2D_ERR_BAD_ARGUMENT;
    *status = 0;
    if (cudaDeviceSynchronize() != cudaSuccess || cudaMemcpyFromSymbol(status, search_status, sizeof(int)) != cudaSuccess) return G2D_ERR_CUDA;
    const int none = 0;
    if (*status != 0 && cudaMemcpyToSymbol(search_status, &none, sizeof(int)) != cudaSuccess) return G2D_ERR_CUDA;
    return G2D_OK;
}

extern "C" int g2d_trellis_decode(int dtype, int64_t rows, int32_t T, const uint8_t *codes, const void *table, int32_t L, int32_t K,
                                  int32_t V, int32_t tail_biting, const void *scale, void *out, int64_t *states, void *stream) {
    const int status = trellis_check(dtype, rows, T, L, K, V);
    if (status != G2D_OK) return status;
    if (rows == 0) return G2D_OK;
    if (!codes || !table || !out) return G2D_ERR_BAD_ARGUMENT;
    if (tail_biting && (int64_t)(T / V) * K * V < L) return G2D_ERR_UNSUPPORTED;  // a string shorter than one state does not determine it
    const int64_t bytes = trellis_code_bytes(T, L, K, V, tail_biting), total = rows * (T / V);
    int64_t blocks = ceil_div(total, 256);
    if (blocks > 148 * 32) blocks = 148 * 32;
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == G2D_F32)
        trellis_decode_kernel<float><<<(unsigned)blocks, 256, 0, st>>>(rows, T, codes, bytes, (const float *)table, L, K * V, V, tail_biting,
                                                                      (const float *)scale, (float *)out, states);
    else
        trellis_decode_kernel<double><<<(unsigned)blocks, 256, 0, st>>>(rows, T, codes, bytes, (const double *)table, L, K * V, V, tail_biting,
                                                                       (const double *)scale, (double *)out, states);
    return check_launch();
}

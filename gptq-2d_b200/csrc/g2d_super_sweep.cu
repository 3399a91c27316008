// Super-entry and N-factor sweeps with the quantizer inside the library.
//
// The reference drives a super-entry sweep from Python: per coarse anti-diagonal it calls the quantizer (for the trellis
// code 2 x 129 kernel launches, quantizer_trellis.py:271-341) and the two super-entry push kernels
// (gptq_2d.py:428-601), and flushes at block ends (gptq_2d.py:1342-1374).  Here the whole loop runs inside one C call:
// per coarse stage a quantizer kernel of this library (round, affine, dynamic abs-max, trellis), the commit-and-push
// kernels and, at block ends, the band update.  Nothing returns to the host between stages, so a sweep is one
// asynchronous enqueue and can be captured.
//
// N-factor sweeps (Algorithm 4, gptq_2d_reference.py:269-294) run on the same loop.  A tensor [n_1, ..., n_D] with one
// unit lower triangular factor per mode is taken as a batch of n_1 ... n_{D-2} slabs [n_{D-1}, n_D]; slab b with the
// leading multi-index (i_1, ..., i_{D-2}) is a two-sided sweep under (L_{D-1}, L_D^T) whose input is
//     X_b + sum_k sum_{i' < i_k} L_k[i_k, i'] F_k[b with i_k -> i'],        F_k = Z - X - (the folds of the modes 0..k),
// because folding the errors of a finished slab through every remaining mode gives exactly Z - (its input): the
// leading modes couple the slabs by plain scaled additions of those residuals, entry by entry, and are never expanded
// into a Kronecker product.  An entry of slab b needs the same entry of the slabs before it in every leading mode,
// so slab b runs sigma_b = i_1 + ... + i_{D-2} stages behind slab 0: global stage g holds the hyper-anti-diagonal
// i_1 + ... + i_D = g, as in the reference, 1 + sum_d (n_d - 1) stages in all.
#include "g2d_common.cuh"

#include <vector>

namespace g2d {

namespace {

constexpr int MAX_LEAD = 4;

struct LeadModes {
    int count;
    int64_t size[MAX_LEAD], stride[MAX_LEAD];  // stride: batches per step of the mode's index
    const void *factor[MAX_LEAD];
};

template <typename F>
struct SuperArgs {
    F *y, *z;
    const F *scale, *zero;
    const int64_t *scale_off, *zero_off;
    int64_t srs, scs, zrs, zcs;
    F qmin, qmax, divisor;
    int half;
    const int32_t *skew;
    int64_t batch, m, n, stage, dmax;  // dmax: super-entries per batch that z holds at this stage
    int p, q;
    F *xs, *row_scale;                 // trellis: gathered sequences and their scales
    LeadModes lead;
    F *fold;                           // lead.count planes [batch, m, n]
    F *c, *e;
    const F *l, *u;
    const int64_t *l_off, *u_off;
    int64_t s0;                        // first stage of the inner block: pushes of the stages s0 .. stage - 1 are pending
    int pull_room, pull_stages;        // stage_pull_staged_kernel: (source stage, entry) pairs and source stages that its shared memory has room for
};

// Entry (k, a, b) of the stage of `batch`: false when the batch has no such entry at this global stage.
template <typename F>
__device__ __forceinline__ bool locate(const SuperArgs<F> &A, int64_t batch, int64_t k, int a, int b, int64_t &i, int64_t &j) {
    const int64_t mbar = A.m / A.p, nbar = A.n / A.q;
    const int64_t s = A.stage - (A.skew ? A.skew[batch] : 0);
    if (s < 0 || s >= mbar + nbar - 1) return false;
    const int64_t i_lo = max((int64_t)0, s - nbar + 1), i_hi = min(s + 1, mbar);
    if (k >= i_hi - i_lo) return false;
    i = (i_lo + k) * A.p + a;
    j = (s - i_lo - k) * A.q + b;
    return true;
}

// One thread per entry of the stage: the leading modes' feedback is added to live Y, and the running fold planes are
// brought up to "minus the input of this entry's sub-problem at level k" (they started as -X).
template <typename F>
__global__ void fold_kernel(SuperArgs<F> A) {
    const int64_t pq = (int64_t)A.p * A.q, per = A.dmax * pq, total = per * A.batch, plane = A.batch * A.m * A.n;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t batch = t / per, rest = t % per;
        int64_t i, j;
        if (!locate(A, batch, rest / pq, (int)(rest % pq) / A.q, (int)(rest % pq) % A.q, i, j)) continue;
        const int64_t pos = i * A.n + j, at = batch * A.m * A.n + pos;
        F sum = (F)0;
        for (int k = 0; k < A.lead.count; ++k) {
            const int64_t size = A.lead.size[k], stride = A.lead.stride[k];
            const int64_t ik = batch / stride % size;
            const F *factor = (const F *)A.lead.factor[k] + ik * size;
            const F *residual = A.fold + (int64_t)k * plane + (batch - ik * stride) * A.m * A.n + pos;  // index 0 of mode k
            F fold = (F)0;
            for (int64_t ip = 0; ip < ik; ++ip) fold += factor[ip] * residual[ip * stride * A.m * A.n];
            sum += fold;
            A.fold[(int64_t)k * plane + at] -= sum;
        }
        A.y[at] += sum;
    }
}

// After the stage is rounded: F_k = Z - (input of the level-k sub-problem).
template <typename F>
__global__ void fold_commit_kernel(SuperArgs<F> A) {
    const int64_t pq = (int64_t)A.p * A.q, per = A.dmax * pq, total = per * A.batch, plane = A.batch * A.m * A.n;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t batch = t / per, rest = t % per;
        int64_t i, j;
        if (!locate(A, batch, rest / pq, (int)(rest % pq) / A.q, (int)(rest % pq) % A.q, i, j)) continue;
        const int64_t at = batch * A.m * A.n + i * A.n + j;
        const F zv = A.z[t];
        for (int k = 0; k < A.lead.count; ++k) A.fold[(int64_t)k * plane + at] += zv;
    }
}

template <typename F>
__global__ void negate_into_planes_kernel(const F *__restrict__ x, F *__restrict__ planes, int64_t count, int copies) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < count; t += (int64_t)gridDim.x * blockDim.x) {
        const F v = -x[t];
        for (int k = 0; k < copies; ++k) planes[(int64_t)k * count + t] = v;
    }
}

__global__ void skew_kernel(int32_t *skew, int64_t batch, LeadModes lead) {
    for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < batch; b += (int64_t)gridDim.x * blockDim.x) {
        int64_t sum = 0;
        for (int k = 0; k < lead.count; ++k) sum += b / lead.stride[k] % lead.size[k];
        skew[b] = (int32_t)sum;
    }
}

// Elementwise quantizers of one stage (round, affine) and the gather of the trellis sequences: one thread per entry.
template <typename F, int KIND>
__global__ void quantize_entries_kernel(SuperArgs<F> A) {
    const int64_t pq = (int64_t)A.p * A.q, per = A.dmax * pq, total = per * A.batch;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t batch = t / per, rest = t % per;
        int64_t i, j;
        const bool on = locate(A, batch, rest / pq, (int)(rest % pq) / A.q, (int)(rest % pq) % A.q, i, j);
        if (KIND == G2D_Q_TRELLIS) {
            // sequences of super-entries that do not exist at this stage are searched along with the others (their result
            // is never read): give them zeros
            const F sc = A.scale[A.scale_off ? A.scale_off[batch] : 0];
            A.xs[t] = on ? div_rn(A.y[batch * A.m * A.n + i * A.n + j], sc) : (F)0;
            if (rest % pq == 0) A.row_scale[t / pq] = sc;
            continue;
        }
        if (!on) continue;
        const F yv = A.y[batch * A.m * A.n + i * A.n + j];
        if (KIND == G2D_Q_ROUND) {
            A.z[t] = rint_even(yv);
        } else {
            const F sc = A.scale[(A.scale_off ? A.scale_off[batch] : 0) + i * A.srs + j * A.scs];
            const F zp = A.zero[(A.zero_off ? A.zero_off[batch] : 0) + i * A.zrs + j * A.zcs];
            A.z[t] = affine_value(yv, sc, zp, A.qmin, A.qmax);
        }
    }
}

// Dynamic abs-max rounding (quantizer_int.py:120-134, :407-439): one warp per row of a super-entry.
template <typename F>
__global__ void quantize_absmax_kernel(SuperArgs<F> A) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5, rows = A.batch * A.dmax * A.p;
    for (int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < rows; row += warps) {
        const int64_t batch = row / (A.dmax * A.p), k = row / A.p % A.dmax;
        const int a = (int)(row % A.p);
        int64_t i, j;
        if (!locate(A, batch, k, a, 0, i, j)) continue;
        const F *src = A.y + batch * A.m * A.n + i * A.n + j;
        F top = (F)0;
        for (int c = lane; c < A.q; c += 32) top = fmax(top, fabs(src[c]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
        const F s = absmax_scale_value(top, A.divisor, A.half);
        for (int c = lane; c < A.q; c += 32) {
            F t = rint_even(div_rn(src[c], s));
            t = t < A.qmin ? A.qmin : t;
            t = t > A.qmax ? A.qmax : t;
            A.z[row * A.q + c] = mul_rn(t, s);
        }
    }
}

constexpr int PTH = 256;       // threads of a CTA of the pull kernel
constexpr int PULL_ROOM = 2048;  // (source stage, entry) pairs whose sums wait in shared memory
constexpr int Q_PULL_ONLY = -1;  // KIND: only bring Y and C up to date

// Loads that stay where they are written: the compiler moved plain ones down to their uses in some of the kernels below (512 x 512
// as 16 x 16 under the round quantizer: 1349 us against 940).
__device__ __forceinline__ float load_here(const float *p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ double load_here(const double *p) {
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
template <int BATCH, typename F>
__device__ __forceinline__ void dot_batches(F &sum, int &x, const F *a, const F *b, int64_t ld, int count) {
    for (; x + BATCH <= count; x += BATCH) {
        F av[BATCH], bv[BATCH];
#pragma unroll
        for (int e = 0; e < BATCH; ++e) {
            av[e] = load_here(a + x + e);
            bv[e] = load_here(b + (x + e) * ld);
        }
#pragma unroll
        for (int e = 0; e < BATCH; ++e) sum += av[e] * bv[e];
    }
}
// sum over x of a[x] b[x ld], ascending; the loads of eight terms travel together (double: of sixteen, whose sums take longer)
template <typename F>
__device__ __forceinline__ F dot(const F *a, const F *b, int64_t ld, int count) {
    F sum = (F)0;
    int x = 0;
    if (sizeof(F) == sizeof(double)) dot_batches<16>(sum, x, a, b, ld, count);
    dot_batches<8>(sum, x, a, b, ld, count);
    for (; x < count; ++x) sum += a[x] * b[x * ld];
    return sum;
}

// A rounded entry's values, or what the quantizer of a later launch takes: Y and C with all feedback are y and c, s the row's scale.
template <typename F, int KIND>
__device__ __forceinline__ void finish_entry(const SuperArgs<F> &A, int64_t batch, int64_t seq, int64_t i, int64_t j, int entry, F y, F c, F s) {
    const int64_t at = i * A.n + j, plane = batch * A.m * A.n;
    F *const yg = A.y + plane, *const cg = A.c + plane, *const eg = A.e + plane;
    if (KIND == Q_PULL_ONLY) {
        yg[at] = y;
        cg[at] = c;
    } else if (KIND == G2D_Q_TRELLIS) {
        yg[at] = y;
        cg[at] = c;
        A.xs[seq * A.p * A.q + entry] = div_rn(y, s);
    } else {
        F z;
        if (KIND == G2D_Q_ROUND) {
            z = rint_even(y);
        } else if (KIND == G2D_Q_AFFINE) {
            const F sc = A.scale[(A.scale_off ? A.scale_off[batch] : 0) + i * A.srs + j * A.scs];
            const F zp = A.zero[(A.zero_off ? A.zero_off[batch] : 0) + i * A.zrs + j * A.zcs];
            z = affine_value(y, sc, zp, A.qmin, A.qmax);
        } else {
            F t = rint_even(div_rn(y, s));
            t = t < A.qmin ? A.qmin : t;
            t = t > A.qmax ? A.qmax : t;
            z = mul_rn(t, s);
        }
        const F ev = z - y;
        eg[at] = ev;
        cg[at] = c + ev;
        yg[at] = z;
    }
}

// Sweeps whose blocks are short enough (see pull_pays).  One CTA per super-entry of the stage: first what the earlier stages of the
// inner block owe it, then its quantizer, then its error, completed C and rounded values.  One launch per stage where the sources used to push (error, push and quantizer
// kernels, 3 launches), because a super-entry that fetches its own feedback when its turn comes needs no launch for it.
// Bound by launch latency and the chain of one stage: the sums of all source stages are formed side by side, each in the
// order and from the start that the push had, and added in the order of the stages, so the values are bit for bit the same.
// Stage kernels follow each other with programmatic dependent launch: a CTA of the next stage is resident when this one ends.
template <typename F, int KIND>
__global__ void __launch_bounds__(PTH) stage_pull_kernel(SuperArgs<F> A) {
    __shared__ F down_s[PULL_ROOM], right_s[PULL_ROOM];
    let_the_next_launch_start();
    after_the_launch_before();
    const int p = A.p, q = A.q, pq = p * q;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t m = A.m, n = A.n;
    for (int64_t batch = blockIdx.y; batch < A.batch; batch += gridDim.y) {
        int64_t i0, j0;
        if (!locate(A, batch, (int64_t)blockIdx.x, 0, 0, i0, j0)) continue;
        F *yg = A.y + batch * m * n, *cg = A.c + batch * m * n, *eg = A.e + batch * m * n;
        const F *lg = A.l + (A.l_off ? A.l_off[batch] : 0), *ug = A.u + (A.u_off ? A.u_off[batch] : 0);
        const int64_t ib = i0 / p, jb = j0 / q;
        const int pulls = (int)min(A.stage - A.s0, max(ib, jb));  // source stages, dd = pulls .. 1 before this one
        const int64_t seq = batch * A.dmax + blockIdx.x;
        auto sums = [&](int dd, int a, int b, F &down, F &right) {
            const int64_t i = i0 + a, j = j0 + b;
            down = right = (F)0;
            if (ib - dd >= 0) {
                down = dot(lg + i * m + (ib - dd) * p, eg + (ib - dd) * p * n + j, n, p);
            }
            if (jb - dd >= 0) {
                right = dot(cg + i * n + (jb - dd) * q, ug + (jb - dd) * q * n + j, n, q);
            }
        };
        for (int t = tid; t < pulls * pq; t += PTH) {  // at most PULL_ROOM (see pull_pays)
            const int at = t % pq;
            sums(pulls - t / pq, at / q, at % q, down_s[t], right_s[t]);
        }
        __syncthreads();
        // a warp per row of the super-entry
        for (int a = warp; a < p; a += PTH / 32) {
            constexpr int KEEP = 4;  // values of a row that stay in a lane's registers
            F yv[KEEP], cv[KEEP], top = (F)0;
            auto update = [&](int b, F &y, F &c) {  // entry (a, b) with all pending feedback
                const int64_t at = (i0 + a) * n + j0 + b;
                y = yg[at];
                c = cg[at];
                for (int x = 0; x < pulls; ++x) {
                    const int dd = pulls - x;
                    const F down = down_s[x * pq + a * q + b], right = right_s[x * pq + a * q + b];
                    if (ib - dd >= 0) c += down;
                    if (ib - dd >= 0 || jb - dd >= 0) y += down + right;
                }
            };
            auto finish = [&](int b, F y, F c, F s) { finish_entry<F, KIND>(A, batch, seq, i0 + a, j0 + b, a * q + b, y, c, s); };
            F s = (F)1;
            if (KIND == G2D_Q_TRELLIS) {
                s = A.scale[A.scale_off ? A.scale_off[batch] : 0];
                if (a == 0 && lane == 0) A.row_scale[seq] = s;
            }
            if (q <= 32 * KEEP) {
#pragma unroll
                for (int x = 0; x < KEEP; ++x)
                    if (lane + 32 * x < q) {
                        update(lane + 32 * x, yv[x], cv[x]);
                        top = fmax(top, fabs(yv[x]));
                    }
                if (KIND == G2D_Q_ABSMAX_DYNAMIC) s = absmax_scale_value(warp_max(top), A.divisor, A.half);
#pragma unroll
                for (int x = 0; x < KEEP; ++x)
                    if (lane + 32 * x < q) finish(lane + 32 * x, yv[x], cv[x], s);
            } else if (KIND == G2D_Q_ABSMAX_DYNAMIC) {
                for (int b = lane; b < q; b += 32) {
                    const int64_t at = (i0 + a) * n + j0 + b;
                    F y, c;
                    update(b, y, c);
                    yg[at] = y;
                    cg[at] = c;
                    top = fmax(top, fabs(y));
                }
                s = absmax_scale_value(warp_max(top), A.divisor, A.half);
                for (int b = lane; b < q; b += 32) {
                    const int64_t at = (i0 + a) * n + j0 + b;
                    finish(b, yg[at], cg[at], s);  // this lane's own stores
                }
            } else {
                for (int b = lane; b < q; b += 32) {
                    F y, c;
                    update(b, y, c);
                    finish(b, y, c, s);
                }
            }
        }
        __syncthreads();  // the next batch reuses the staged sums
    }
}

// The same where the blocks of the factors that a super-entry needs are small (see PULL_FACTORS).  The CTAs are resident long before the stage
// before them ends and bring those blocks to shared memory ahead of the wait; behind it they fetch the errors and C of all source
// stages and their own Y and C in one round trip.  The same sums in the same order.  A stage of 512 x 2048 as 1 x 32 takes 2.5 us, 3.6 with the
// kernel above.  (A stage that lets the next one start behind its wait, so that the next could form the sums of all but the last stage ahead
// of its own: 4.5 us, the start of a launch is longer than what it hides.)
template <typename F, int KIND>
__global__ void __launch_bounds__(PTH) stage_pull_staged_kernel(SuperArgs<F> A) {
    extern __shared__ __align__(16) unsigned char pull_smem[];
    let_the_next_launch_start();
    const int p = A.p, q = A.q, pq = p * q;
    F *const down_s = reinterpret_cast<F *>(pull_smem), *const right_s = down_s + A.pull_room;    // sums by source stage and entry
    F *const e_src = right_s + A.pull_room, *const c_src = e_src + A.pull_room;                   // the stages' E above and C to the left
    F *const y_s = c_src + A.pull_room, *const c_s = y_s + pq;                                    // Y and C of the super-entry
    F *const l_s = c_s + pq, *const u_s = l_s + (A.pull_stages) * p * p;                          // blocks of L and U
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t m = A.m, n = A.n;
    bool waited = false;
    for (int64_t batch = blockIdx.y; batch < A.batch; batch += gridDim.y) {
        int64_t i0, j0;
        if (!locate(A, batch, (int64_t)blockIdx.x, 0, 0, i0, j0)) continue;
        F *yg = A.y + batch * m * n, *cg = A.c + batch * m * n, *eg = A.e + batch * m * n;
        const F *lg = A.l + (A.l_off ? A.l_off[batch] : 0), *ug = A.u + (A.u_off ? A.u_off[batch] : 0);
        const int64_t ib = i0 / p, jb = j0 / q;
        const int pulls = (int)min(A.stage - A.s0, max(ib, jb));  // source stages, dd = pulls .. 1 before this one, in this order below
        const int64_t seq = batch * A.dmax + blockIdx.x;
        for (int t = tid; t < pulls * p * p; t += PTH) {
            const int x = t / (p * p), r = t % (p * p);
            if (ib - (pulls - x) >= 0) l_s[t] = lg[(i0 + r / p) * m + (ib - (pulls - x)) * p + r % p];
        }
        for (int t = tid; t < pulls * q * q; t += PTH) {
            const int x = t / (q * q), r = t % (q * q);
            if (jb - (pulls - x) >= 0) u_s[t] = ug[((jb - (pulls - x)) * q + r / q) * n + j0 + r % q];
        }
        if (!waited) after_the_launch_before();
        waited = true;
        for (int t = tid; t < (pulls + 1) * pq; t += PTH) {
            const int x = t / pq, at = t % pq, a = at / q, b = at % q, dd = pulls - x;
            if (x < pulls) {
                e_src[t] = ib - dd >= 0 ? load_here(eg + (i0 - dd * p + a) * n + j0 + b) : (F)0;
                c_src[t] = jb - dd >= 0 ? load_here(cg + (i0 + a) * n + j0 - dd * q + b) : (F)0;
            } else {
                y_s[at] = load_here(yg + (i0 + a) * n + j0 + b);
                c_s[at] = load_here(cg + (i0 + a) * n + j0 + b);
            }
        }
        __syncthreads();
        for (int t = tid; t < pulls * pq; t += PTH) {
            const int x = t / pq, at = t % pq, a = at / q, b = at % q, dd = pulls - x;
            const F *const e = e_src + x * pq + b, *const c = c_src + x * pq + a * q;
            F down = (F)0, right = (F)0;
            if (ib - dd >= 0) {
                const F *const l = l_s + x * p * p + a * p;
                for (int k = 0; k < p; ++k) down += l[k] * e[k * q];
            }
            if (jb - dd >= 0) {
                const F *const u = u_s + x * q * q + b;
#pragma unroll 8
                for (int k = 0; k < q; ++k) right += c[k] * u[k * q];
            }
            down_s[t] = down;
            right_s[t] = right;
        }
        __syncthreads();
        for (int t = tid; t < pq; t += PTH) {
            F y = y_s[t], c = c_s[t];
            for (int x = 0; x < pulls; ++x) {
                const int dd = pulls - x;
                const F down = down_s[x * pq + t], right = right_s[x * pq + t];
                if (ib - dd >= 0) c += down;
                if (ib - dd >= 0 || jb - dd >= 0) y += down + right;
            }
            y_s[t] = y;
            c_s[t] = c;
        }
        __syncthreads();
        // a warp per row of the super-entry
        for (int a = warp; a < p; a += PTH / 32) {
            F s = (F)1;
            if (KIND == G2D_Q_TRELLIS) {
                s = A.scale[A.scale_off ? A.scale_off[batch] : 0];
                if (a == 0 && lane == 0) A.row_scale[seq] = s;
            }
            if (KIND == G2D_Q_ABSMAX_DYNAMIC) {
                F top = (F)0;
                for (int b = lane; b < q; b += 32) top = fmax(top, fabs(y_s[a * q + b]));
                s = absmax_scale_value(warp_max(top), A.divisor, A.half);
            }
            for (int b = lane; b < q; b += 32) {
                finish_entry<F, KIND>(A, batch, seq, i0 + a, j0 + b, a * q + b, y_s[a * q + b], c_s[a * q + b], s);
            }
        }
        __syncthreads();  // the next batch reuses the shared memory
    }
    after_the_launch_before();  // a launch's end implies the ends of all before it, also through CTAs without a super-entry
}

// Whether a sweep pulls.  A CTA forms stages p q sums of p + q products with 256 threads, where a push spreads them over the whole
// GPU: from about 600 products per thread on, the push is the faster one, and beyond PULL_ROOM sums there is no room for
// them.  Measured, push and pull in us: 256 x 1024 as 1 x 32, blocks of 64 stages (264 products per thread) 4437 / 3151;
// 64 x 2048 as 1 x 128, 8 stages (516) 2265 / 2053, 16 stages (1032) 2028 / 2716; 512 x 512 as 32 x 32, 2 stages (512) 866 / 764;
// 512 x 1024 as 4 x 128, 4 stages (1056) 3835 / 4005; 2048 x 64 as 512 x 1, 1 stage (1026) 5925 / 8467.  With leading modes a pull
// is a launch of its own, which blocks of one or two stages do not repay (8 x 64 x 128 as 1 x 2, one stage: 4149 / 4429).
bool pull_pays(int64_t stages, int p, int q, bool leading) {
    const double sums = (double)stages * p * q;
    return sums <= PULL_ROOM && sums * (p + q) <= 600.0 * PTH && (!leading || stages > 2);
}

// Where a stage's blocks of the factors wait in shared memory: up to 32 KB of floats (7 blocks of 32 x 32).  In us, with loads where they are used
// and staged, blocks of 8 stages: 512 x 2048 as 1 x 16 5250 and 4710, as 1 x 32 5870 and 4970, as 1 x 64 (115 KB) 7870 and 8670; 256 x 1024 as
// 4 x 32 880 and 770.
constexpr int PULL_FACTORS = 8192;

template <typename F, int KIND>
int launch_stage_pull(const SuperArgs<F> &A, cudaStream_t st) {
    cudaLaunchConfig_t config{};
    config.gridDim = dim3((unsigned)A.dmax, (unsigned)(A.batch < 65535 ? A.batch : 65535));
    config.blockDim = dim3(PTH);
    config.stream = st;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    if (A.pull_stages > 0) {
        constexpr size_t most = sizeof(F) * (size_t)(6 * PULL_ROOM + PULL_FACTORS);
        static PerDeviceOnce configured;
        if (configured.run([&] { return cudaFuncSetAttribute(stage_pull_staged_kernel<F, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) == cudaSuccess; }) != G2D_OK)
            return G2D_ERR_CUDA;
        config.dynamicSmemBytes = sizeof(F) * (size_t)(4 * A.pull_room + 2 * A.p * A.q + A.pull_stages * (A.p * A.p + A.q * A.q));
        if (cudaLaunchKernelEx(&config, stage_pull_staged_kernel<F, KIND>, A) != cudaSuccess) return G2D_ERR_CUDA;
    } else if (cudaLaunchKernelEx(&config, stage_pull_kernel<F, KIND>, A) != cudaSuccess) {
        return G2D_ERR_CUDA;
    }
    return check_launch();
}

// Packed trellis paths of one stage into the matrix-level array [batch, m / p, n / q, bytes].
template <typename F>
__global__ void scatter_codes_kernel(SuperArgs<F> A, const uint8_t *__restrict__ stage_codes, uint8_t *__restrict__ codes, int64_t bytes) {
    const int64_t per = A.dmax * bytes, total = per * A.batch, nbar = A.n / A.q, mbar = A.m / A.p;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t batch = t / per, k = t % per / bytes, byte = t % bytes;
        int64_t i, j;
        if (!locate(A, batch, k, 0, 0, i, j)) continue;
        codes[((batch * mbar + i / A.p) * nbar + j / A.q) * bytes + byte] = stage_codes[t];
    }
}

inline unsigned blocks_for(int64_t work, int threads) {
    int64_t blocks = ceil_div(work, threads);
    if (blocks < 1) blocks = 1;
    if (blocks > 148 * 16) blocks = 148 * 16;
    return (unsigned)blocks;
}

inline size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

struct Plan {
    size_t c, e, z, skew, fold, xs, row_scale, stage_codes, viterbi, total;
    int64_t lanes, stages2d, lead_total;
    int64_t code_bytes;
};

int make_plan(const g2d_super_desc *d, Plan *plan) {
    const size_t elem = d->dtype == G2D_F32 ? 4 : 8;
    const int64_t mbar = d->m / d->p, nbar = d->n / d->q;
    plan->lanes = mbar < nbar ? mbar : nbar;
    plan->stages2d = mbar + nbar - 1;
    plan->lead_total = 0;
    for (int k = 0; k < d->lead_count; ++k) plan->lead_total += d->lead_size[k] - 1;
    const size_t matrix = align256(elem * (size_t)(d->batch * d->m * d->n));
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t where = at; at += align256(bytes); return where; };
    plan->c = take(matrix);
    plan->e = take(matrix);
    plan->z = take(elem * (size_t)(d->batch * plan->lanes * d->p * d->q));
    plan->skew = take(d->lead_count > 0 ? sizeof(int32_t) * (size_t)d->batch : 0);
    plan->fold = take((size_t)d->lead_count * matrix);
    plan->xs = plan->row_scale = plan->stage_codes = plan->viterbi = at;
    plan->code_bytes = 0;
    if (d->quant_kind == G2D_Q_TRELLIS) {
        const int64_t rows = d->batch * plan->lanes;
        const int T = d->p * d->q;
        plan->xs = take(elem * (size_t)(rows * T));
        plan->row_scale = take(elem * (size_t)rows);
        plan->code_bytes = trellis_code_bytes(T, d->trellis_L, d->trellis_K, d->trellis_V, d->tail_biting);
        plan->stage_codes = take(d->codes ? (size_t)(rows * plan->code_bytes) : 0);
        plan->viterbi = take(trellis_scratch_bytes(d->dtype, rows, T, d->trellis_L, d->trellis_K, d->trellis_V));
    }
    plan->total = at;
    return G2D_OK;
}

int check_super(const g2d_super_desc *d) {
    if (!d) return G2D_ERR_BAD_ARGUMENT;
    if (d->dtype != G2D_F32 && d->dtype != G2D_F64) return G2D_ERR_BAD_ARGUMENT;
    if (d->batch < 0 || d->m < 0 || d->n < 0 || d->p <= 0 || d->q <= 0) return G2D_ERR_BAD_ARGUMENT;
    if (d->m % d->p || d->n % d->q) return G2D_ERR_BAD_ARGUMENT;
    if (d->lead_count < 0 || d->lead_count > MAX_LEAD) return G2D_ERR_BAD_ARGUMENT;
    int64_t slabs = 1;
    for (int k = 0; k < d->lead_count; ++k) {
        if (d->lead_size[k] <= 0) return G2D_ERR_BAD_ARGUMENT;
        slabs *= d->lead_size[k];
    }
    if (d->lead_count > 0 && slabs != d->batch) return G2D_ERR_BAD_ARGUMENT;
    switch (d->quant_kind) {
    case G2D_Q_ROUND: break;
    case G2D_Q_AFFINE:
    case G2D_Q_ABSMAX_DYNAMIC:
        if (!(d->qmin < d->qmax)) return G2D_ERR_BAD_ARGUMENT;
        break;
    case G2D_Q_TRELLIS: {
        const int V = d->trellis_V, K = d->trellis_K, L = d->trellis_L, T = d->p * d->q;
        if (V < 1 || V > 2 || K < 1 || K * V > 8 || L < K * V || L > 24 || T % V != 0) return G2D_ERR_BAD_ARGUMENT;
        if (d->codes && d->tail_biting && (int64_t)(T / V) * K * V < L) return G2D_ERR_UNSUPPORTED;
        break;
    }
    default: return G2D_ERR_UNSUPPORTED;
    }
    return G2D_OK;
}

template <typename F>
int sweep_super(const g2d_super_desc *d, const Plan &plan, cudaStream_t st) {
    char *ws = (char *)d->workspace;
    const int64_t count = d->batch * d->m * d->n;
    F *c = (F *)(ws + plan.c), *e = (F *)(ws + plan.e), *z = (F *)(ws + plan.z);
    int32_t *skew = d->lead_count > 0 ? (int32_t *)(ws + plan.skew) : nullptr;
    if (cudaMemsetAsync(c, 0, sizeof(F) * (size_t)count, st) != cudaSuccess) return G2D_ERR_CUDA;

    SuperArgs<F> A{};
    A.y = (F *)d->y; A.z = z;
    A.scale = (const F *)d->scale; A.zero = (const F *)d->zero;
    A.scale_off = d->scale_offsets; A.zero_off = d->zero_offsets;
    A.srs = d->scale_row_stride; A.scs = d->scale_col_stride; A.zrs = d->zero_row_stride; A.zcs = d->zero_col_stride;
    A.qmin = (F)d->qmin; A.qmax = (F)d->qmax;
    A.divisor = (F)((d->qmax - d->qmin) / 2);
    A.half = d->half;
    A.skew = skew;
    A.batch = d->batch; A.m = d->m; A.n = d->n; A.p = d->p; A.q = d->q;
    A.xs = (F *)(ws + plan.xs); A.row_scale = (F *)(ws + plan.row_scale);
    A.fold = (F *)(ws + plan.fold);
    A.c = c; A.e = e;
    A.l = (const F *)d->l; A.u = (const F *)d->u; A.l_off = d->l_offsets; A.u_off = d->u_offsets;
    A.lead.count = d->lead_count;
    int64_t stride = d->batch;
    for (int k = 0; k < d->lead_count; ++k) {
        stride /= d->lead_size[k];
        A.lead.size[k] = d->lead_size[k];
        A.lead.stride[k] = stride;
        A.lead.factor[k] = d->lead_factor[k];
    }
    if (d->lead_count > 0) {
        skew_kernel<<<blocks_for(d->batch, 256), 256, 0, st>>>(skew, d->batch, A.lead);
        if (check_launch() != G2D_OK) return G2D_ERR_CUDA;
        negate_into_planes_kernel<F><<<blocks_for(count, 256), 256, 0, st>>>((const F *)d->y, A.fold, count, d->lead_count);
        if (check_launch() != G2D_OK) return G2D_ERR_CUDA;
    }

    g2d_stage_desc sd{};
    sd.dtype = d->dtype; sd.p = d->p; sd.q = d->q;
    sd.batch = d->batch; sd.m = d->m; sd.n = d->n;
    sd.y = d->y; sd.c = c; sd.e = e;
    sd.l = d->l; sd.l_offsets = d->l_offsets; sd.u = d->u; sd.u_offsets = d->u_offsets;
    BandArgs<F> b;
    b.y = (F *)d->y; b.c = c; b.e = e; b.l = (const F *)d->l; b.u = (const F *)d->u; b.l_off = d->l_offsets; b.u_off = d->u_offsets;
    b.batch = d->batch; b.m = d->m; b.n = d->n; b.P = d->p; b.Q = d->q; b.down_into_y = 1; b.filter = 0;
    b.mode = (d->p == 1 && d->q == 1 && skew == nullptr) ? BAND_PLAIN : BAND_GENERAL;
    b.skew = skew;

    const int64_t mbar = d->m / d->p, nbar = d->n / d->q, pq = (int64_t)d->p * d->q;
    const int64_t stages = plan.stages2d + plan.lead_total;
    // super-entries on the local anti-diagonal t of a slab, and the most that any slab holds at the global stage g
    auto on_stage = [&](int64_t t) -> int64_t {
        if (t < 0 || t >= plan.stages2d) return 0;
        const int64_t lo = t - nbar + 1 > 0 ? t - nbar + 1 : 0, hi = t + 1 < mbar ? t + 1 : mbar;
        return hi - lo;
    };
    // the reference's clamping rules (gptq_2d.py:1327-1329)
    const int64_t inner = d->inner_block > 0 && d->inner_block <= stages ? d->inner_block : stages;
    const int64_t outer = d->outer_block > inner && d->outer_block < stages ? d->outer_block : inner;
    const int T = d->p * d->q;
    const bool pull = pull_pays(inner, d->p, d->q, d->lead_count > 0);
    if (pull) {
        A.pull_room = (int)((inner - 1) * pq);
        A.pull_stages = (inner - 1) * ((int64_t)d->p * d->p + (int64_t)d->q * d->q) <= PULL_FACTORS ? (int)(inner - 1) : 0;
    }
    for (int64_t outer_start = 0; outer_start < stages; outer_start += outer) {
        const int64_t outer_stop = outer_start + outer < stages ? outer_start + outer : stages;
        for (int64_t s0 = outer_start; s0 < outer_stop; s0 += inner) {
            const int64_t s1 = s0 + inner < outer_stop ? s0 + inner : outer_stop;
            for (int64_t s = s0; s < s1; ++s) {
                int64_t dmax = 0;
                for (int64_t behind = 0; behind <= plan.lead_total; ++behind) dmax = on_stage(s - behind) > dmax ? on_stage(s - behind) : dmax;
                if (dmax == 0) continue;
                A.stage = s; A.dmax = dmax; A.s0 = s0;
                const int64_t work = d->batch * dmax * pq;
                if (pull && d->lead_count == 0) {
                    int status;
                    switch (d->quant_kind) {
                    case G2D_Q_ROUND: status = launch_stage_pull<F, G2D_Q_ROUND>(A, st); break;
                    case G2D_Q_AFFINE: status = launch_stage_pull<F, G2D_Q_AFFINE>(A, st); break;
                    case G2D_Q_ABSMAX_DYNAMIC: status = launch_stage_pull<F, G2D_Q_ABSMAX_DYNAMIC>(A, st); break;
                    default: status = launch_stage_pull<F, G2D_Q_TRELLIS>(A, st); break;
                    }
                    if (status != G2D_OK) return status;
                    if (d->quant_kind != G2D_Q_TRELLIS) continue;
                } else {
                    // the leading modes' feedback comes between the pending pushes and the quantizer
                    if (pull) {
                        const int status = launch_stage_pull<F, Q_PULL_ONLY>(A, st);
                        if (status != G2D_OK) return status;
                    }
                    if (d->lead_count > 0) {
                        fold_kernel<F><<<blocks_for(work, 128), 128, 0, st>>>(A);
                        if (check_launch() != G2D_OK) return G2D_ERR_CUDA;
                    }
                    switch (d->quant_kind) {
                    case G2D_Q_ROUND: quantize_entries_kernel<F, G2D_Q_ROUND><<<blocks_for(work, 128), 128, 0, st>>>(A); break;
                    case G2D_Q_AFFINE: quantize_entries_kernel<F, G2D_Q_AFFINE><<<blocks_for(work, 128), 128, 0, st>>>(A); break;
                    case G2D_Q_ABSMAX_DYNAMIC: quantize_absmax_kernel<F><<<blocks_for(d->batch * dmax * d->p * 32, 128), 128, 0, st>>>(A); break;
                    default: quantize_entries_kernel<F, G2D_Q_TRELLIS><<<blocks_for(work, 128), 128, 0, st>>>(A); break;
                    }
                    if (check_launch() != G2D_OK) return G2D_ERR_CUDA;
                }
                if (d->quant_kind == G2D_Q_TRELLIS) {
                    uint8_t *stage_codes = d->codes ? (uint8_t *)(ws + plan.stage_codes) : nullptr;
                    const TrellisIndex index{d->table_distinct, d->table_ids, d->table_distinct_count};
                    const int status = launch_trellis(d->dtype, d->batch * dmax, T, A.xs, d->table, d->trellis_L, d->trellis_K, d->trellis_V,
                                                      d->tail_biting, A.row_scale, z, nullptr, ws + plan.viterbi, stage_codes, st,
                                                      d->table_ids != nullptr ? &index : nullptr);
                    if (status != G2D_OK) return status;
                    if (stage_codes) {
                        scatter_codes_kernel<F><<<blocks_for(d->batch * dmax * plan.code_bytes, 256), 256, 0, st>>>(A, stage_codes, d->codes, plan.code_bytes);
                        if (check_launch() != G2D_OK) return G2D_ERR_CUDA;
                    }
                }
                if (d->lead_count > 0) {
                    fold_commit_kernel<F><<<blocks_for(work, 128), 128, 0, st>>>(A);
                    if (check_launch() != G2D_OK) return G2D_ERR_CUDA;
                }
                const int status = pull ? launch_stage_commit<F>(sd, z, s, st, skew, dmax * pq) : launch_stage_push<F>(sd, z, s, s1, st, skew, dmax * pq);
                if (status != G2D_OK) return status;
            }
            if (s1 < outer_stop) {
                b.s0 = s0; b.s1 = s1; b.s_end = outer_stop;
                const int status = launch_band_update<F>(b, st);
                if (status != G2D_OK) return status;
            }
        }
        if (outer_stop < stages) {
            b.s0 = outer_start; b.s1 = outer_stop; b.s_end = stages;
            const int status = launch_band_update<F>(b, st);
            if (status != G2D_OK) return status;
        }
    }
    return G2D_OK;
}

}  // namespace

}  // namespace g2d

using namespace g2d;

extern "C" int g2d_super_workspace_bytes(const g2d_super_desc *desc, size_t *bytes) {
    const int status = check_super(desc);
    if (status != G2D_OK || !bytes) return status != G2D_OK ? status : G2D_ERR_BAD_ARGUMENT;
    Plan plan;
    make_plan(desc, &plan);
    *bytes = plan.total;
    return G2D_OK;
}

extern "C" int g2d_sweep_super_entry(const g2d_super_desc *desc, void *stream) {
    const int status = check_super(desc);
    if (status != G2D_OK) return status;
    if (desc->batch == 0 || desc->m == 0 || desc->n == 0) return G2D_OK;
    if (!desc->y || !desc->l || !desc->u) return G2D_ERR_BAD_ARGUMENT;
    if (desc->quant_kind == G2D_Q_AFFINE && (!desc->scale || !desc->zero)) return G2D_ERR_BAD_ARGUMENT;
    if (desc->quant_kind == G2D_Q_TRELLIS && (!desc->scale || !desc->table)) return G2D_ERR_BAD_ARGUMENT;
    if (desc->table_ids != nullptr && (!desc->table_distinct || desc->table_distinct_count <= 0 || ((uintptr_t)desc->table_ids & 15) != 0))
        return G2D_ERR_BAD_ARGUMENT;
    if (desc->quant_kind == G2D_Q_ABSMAX_DYNAMIC && desc->half != G2D_FP16 && desc->half != G2D_BF16) return G2D_ERR_BAD_ARGUMENT;
    for (int k = 0; k < desc->lead_count; ++k)
        if (!desc->lead_factor[k]) return G2D_ERR_BAD_ARGUMENT;
    if (desc->m / desc->p + desc->n / desc->q > (int64_t)1 << 30) return G2D_ERR_TOO_LARGE;
    Plan plan;
    make_plan(desc, &plan);
    if (!desc->workspace || desc->workspace_bytes < plan.total || ((uintptr_t)desc->workspace & 255) != 0) return G2D_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    return desc->dtype == G2D_F32 ? sweep_super<float>(desc, plan, st) : sweep_super<double>(desc, plan, st);
}

// The body of the tile sweep's kernels, taken in as text: extracted into a function, the same statements compiled to tiles 2 % slower.
// G2D_JOINT: the launch may have started before the one before it has ended (see g2d_tile_sweep_step.cu).
    F *Ys = reinterpret_cast<F *>(g2d_smem);  // X + right feedback; the errors E once a sub-tile is swept
    F *Cs = Ys + TILE * LD;                   // down feedback; the completed C once a sub-tile is swept
    F *LUs = Cs + TILE * LD;                  // strict lower part: L[I, I]; strict upper part: U[J, J]
    F *Dg = LUs + TILE * LD;                  // zero-padded diagonal blocks L[a, a] and U[b, b]^T, strictly lower, between rows of zeros
    F *Par = Dg + DROWS * DLD;                // [NSUB][SUB][PLD][4]: scale, zero point, reciprocal, rounded value of the entries of the sub-tiles being swept
    F *Ubs = Par + NSUB * SUB * PLD * 4;      // float only, pipelined schedule: U[J, J + 1], the right neighbour's coupling block
    F *Lbs = Ubs + TILE * LD;                 // the same: L[I + 1, I], the lower neighbour's
    F *Yns = Lbs + TILE * LD;                 // the same: the feedback for the right neighbour, C[I, J] U[J, J + 1], growing sub-tile by sub-tile
    F *Cns = Yns + TILE * LD;                 // and for the lower one, L[I + 1, I] E[I, J]
    __shared__ unsigned row_max[TILE];
    __shared__ __align__(16) unsigned column_max[TTH / 32][TILE];
    __shared__ unsigned fast_div[NSUB];       // every scale of the sub-tile allows the division by reciprocal

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int k = lane & 15, role = lane >> 4;
    const int I = i_first + i_step * (int)blockIdx.x, J = S - I;  // tiles of the anti-diagonal S, every one or every second
    const int64_t i0 = (int64_t)I * TILE, j0 = (int64_t)J * TILE;
    const int64_t m = P.m, n = P.n;
    const bool full = i0 + TILE <= m && j0 + TILE <= n;
    // Warps w and w + 4 share one of the SM's four schedulers.  The sweeping warps take two of them (rows 0 and 2, rows 1 and 3)
    // and the helpers the other two: a helper's product beside it costs a sweeping warp more than its neighbour does.
    static_assert(SWEEPERS == 4 && HELPERS == 4, "warps are dealt out to the schedulers in twos");
    const bool sweeper = (warp & 2) == 0;
    const int number = (warp & 1) + (warp >> 2) * 2;  // of the warp among those of its kind
    const int helper = number;                        // the sub-tile row whose parameters a helper prepares
    const int rows_in = (int)(m - i0 < TILE ? m - i0 : TILE), cols_in = (int)(n - j0 < TILE ? n - j0 : TILE);  // of this tile

    for (int64_t batch = blockIdx.y; batch < P.batch; batch += gridDim.y) {
        // Y, C, E and the planes have rows of ld values (n, or n rounded up to a multiple of 4), L and U rows of ldl and ldu
        const int64_t ld = P.ld, ldl = P.ldl, ldu = P.ldu;
        F *yg = P.y + batch * m * ld, *cg = P.c + batch * m * ld, *eg = P.e + batch * m * ld;
        const F *lg = P.l + (P.l_off ? P.l_off[batch] : 0);
        const F *ug = P.u + (P.u_off ? P.u_off[batch] : 0);
        const F *sg = KIND == G2D_Q_AFFINE ? P.scale + (P.scale_off ? P.scale_off[batch] : 0) : nullptr;
        const F *zg = KIND == G2D_Q_AFFINE ? P.zero + (P.zero_off ? P.zero_off[batch] : 0) : nullptr;
        const F *fg = KIND == G2D_Q_FORCED ? P.forced + batch * m * n : nullptr;
        F *pre = P.y_pre ? P.y_pre + batch * m * n : nullptr;
        const F *yfg = P.yf ? P.yf + batch * m * ld : nullptr, *cfg = P.yf ? P.cf + batch * m * ld : nullptr;
        // neighbour push (pipelined schedule): what this tile receives and what it owes
        F *yng = P.yn ? P.yn + batch * m * ld : nullptr, *cng = P.yn ? P.cn + batch * m * ld : nullptr;
        const bool gets_right = yng != nullptr && J > 0, gets_down = yng != nullptr && I > 0;
        const bool owes_right = yng != nullptr && J + 1 < P.nJ, owes_down = yng != nullptr && I + 1 < P.nI;

        // ---- quantizer parameters, prepared by the helper warps ----
        // Helper warp h prepares the parameters of the sub-tile that sweeping warp h takes next: a lane has the entries
        // (2 x + lane / 16, lane % 16).  Scale, zero point and, for the affine quantizer, the reciprocal of the scale wait
        // in shared memory by entry, with the warp-wide decision whether every scale is in the range where the reciprocal
        // form of the division is safe.  The loads are issued one sub-tile anti-diagonal ahead and travel while the helper
        // does its other work.
        constexpr int PR = SUB * SUB / 32;  // entries per helper lane
        F sc[PR], zp[PR], rc[PR];
        bool pfast = true;
        unsigned pvalid = 0;  // entries inside the matrix
        auto fetch_params = [&](int w_next) {
            const int b = w_next - helper;
            if (b < 0 || b >= NSUB || KIND == G2D_Q_ROUND) return;
            const int r = helper * SUB + role, c = b * SUB + k;  // first entry; the others follow two rows apart
            // entries outside the matrix load a value from inside it (no select waits on the load here) and get their
            // neutral parameters in finish_params
            const int rc_ = min(r, rows_in - 1), cc = min(c, cols_in - 1);
            pvalid = 0;
#pragma unroll
            for (int x = 0; x < PR; ++x) pvalid |= (r + 2 * x < rows_in && c < cols_in) ? (1u << x) : 0u;
            if (KIND == G2D_Q_AFFINE) {
                const F *ps = sg + (i0 + rc_) * P.srs + (j0 + cc) * P.scs, *pz = zg + (i0 + rc_) * P.zrs + (j0 + cc) * P.zcs;
                const int64_t ss = 2 * P.srs, zs = 2 * P.zrs;
#pragma unroll
                for (int x = 0; x < PR; ++x) {
                    sc[x] = load_now(ps);
                    zp[x] = load_now(pz);
                    if (r + 2 * x + 2 < rows_in) {
                        ps += ss;
                        pz += zs;
                    }
                }
            } else {
                const F *pf = fg + (i0 + rc_) * n + j0 + cc;
#pragma unroll
                for (int x = 0; x < PR; ++x) {
                    sc[x] = load_now(pf);
                    if (r + 2 * x + 2 < rows_in) pf += 2 * n;
                }
            }
        };
        auto finish_params = [&](int w_next) {
            if (w_next - helper < 0 || w_next - helper >= NSUB) return;
            bool normal = true;
#pragma unroll
            for (int x = 0; x < PR; ++x) {
                const bool in = (pvalid >> x) & 1u;
                if (KIND == G2D_Q_AFFINE) {
                    sc[x] = in ? sc[x] : (F)1;
                    zp[x] = in ? zp[x] : (F)0;
                    normal = normal && reciprocal_is_safe(sc[x]);
                    rc[x] = rounding_reciprocal(sc[x]);
                } else if (KIND == G2D_Q_FORCED) {
                    sc[x] = in ? sc[x] : (F)0;
                }
            }
            pfast = __all_sync(0xffffffffu, normal);
        };
        auto store_params = [&](int w_next) {
            if (w_next - helper < 0 || w_next - helper >= NSUB) return;
            F *dst = Par + ((helper * SUB + role) * PLD + k) * 4;
#pragma unroll
            for (int x = 0; x < PR; ++x) {
                if (KIND == G2D_Q_AFFINE) {
                    const F v[4] = {sc[x], zp[x], rc[x], (F)0};
                    store4(dst + 2 * x * PLD * 4, v);
                } else if (KIND == G2D_Q_FORCED) {
                    dst[2 * x * PLD * 4] = sc[x];
                }
            }
            if (lane == 0) fast_div[helper] = pfast ? 1u : 0u;
        };
        if (!sweeper) fetch_params(0);
        constexpr bool PUSH = sizeof(F) == sizeof(float);  // the neighbour push exists for float (pipelined schedule) only

        // ---- load the tile ----
        const bool vec = full && ((ld | ldl | ldu) % 4 == 0) &&
                         ((reinterpret_cast<uintptr_t>(yg) | reinterpret_cast<uintptr_t>(cg) | reinterpret_cast<uintptr_t>(eg) |
                           reinterpret_cast<uintptr_t>(lg) | reinterpret_cast<uintptr_t>(ug)) % (4 * sizeof(F)) == 0);
        bool have_diagonal = false;
        if constexpr (PUSH) {
            if (owes_right || owes_down)
                for (int idx = tid; idx < 2 * TILE * LD / 4; idx += TTH) {
                    const F zero[4] = {(F)0, (F)0, (F)0, (F)0};
                    store4(Yns + idx * 4, zero);
                }
            if (vec) {
                // One wait on global memory: the off-diagonal blocks of L[I, I] and U[J, J] and the two coupling blocks
                // travel to shared memory on their own (cp.async), the diagonal blocks and the six planes that make up Y and
                // C through registers, and all of them are issued before the first is used.
                have_diagonal = true;
                for (int c = tid; c < 12 * SUB * 4; c += TTH) {
                    const int blk = c / (SUB * 4), ba = blk / 3, bb = blk % 3 + (blk % 3 >= ba ? 1 : 0), row = ba * SUB + c / 4 % SUB, col = bb * SUB + c % 4 * 4;
                    async16(LUs + row * LD + col, ba > bb ? lg + (i0 + row) * ldl + i0 + col : ug + (j0 + row) * ldu + j0 + col, true);
                }
                if (owes_right)
                    for (int c = tid; c < TILE * TILE / 4; c += TTH) {
                        const int row = c / (TILE / 4), col = c % (TILE / 4) * 4;
                        // n is not always a multiple of 4, the row stride is.  The tail of a padded copy is not defined: what is formed
                        // with it goes to columns from n on, which are not stored, or stored to padding that nothing reads.
                        const bool in = j0 + TILE + col < n;
                        async16(Ubs + row * LD + col, ug + (j0 + row) * ldu + (in ? j0 + TILE + col : 0), in);
                    }
                if (owes_down)
                    for (int c = tid; c < TILE * TILE / 4; c += TTH) {
                        const int row = c / (TILE / 4), col = c % (TILE / 4) * 4;
                        const bool in = i0 + TILE + row < m;
                        async16(Lbs + row * LD + col, lg + (in ? i0 + TILE + row : 0) * ldl + i0 + col, in);
                    }
                asm volatile("cp.async.commit_group;" ::: "memory");
                constexpr int PER = TILE * TILE / 4 / TTH;  // vectors per thread and array
                F vy[PER][4], vc[PER][4], fy[PER][4], fc[PER][4], ny[PER][4], nc[PER][4], dv[2][4];
#if G2D_JOINT  // the factors ahead of the wait
#pragma unroll
                for (int t = 0; t < 2; ++t) {  // the eight diagonal blocks, 64 vectors each
                    const int idx = t * TTH + tid, blk = idx / 64, r = idx / 4 % SUB, c = idx % 4 * 4, o = (blk % NSUB) * SUB;
                    load4(blk < NSUB ? lg + (i0 + o + r) * ldl + i0 + o + c : ug + (j0 + o + r) * ldu + j0 + o + c, dv[t]);
                }
                for (int idx = tid; idx < DROWS * DLD / 4; idx += TTH) {
                    const F zero[4] = {(F)0, (F)0, (F)0, (F)0};
                    store4(Dg + idx * 4, zero);
                }
                after_the_launch_before();
#endif
#pragma unroll
                for (int t = 0; t < PER; ++t) {
                    const int idx = t * TTH + tid, r = idx / (TILE / 4), c = (idx % (TILE / 4)) * 4;
                    const int64_t at = (i0 + r) * ld + j0 + c;
                    load4(yg + at, vy[t]);
                    load4(cg + at, vc[t]);
#pragma unroll
                    for (int x = 0; x < 4; ++x) fy[t][x] = fc[t][x] = ny[t][x] = nc[t][x] = (F)0;
                    if (yfg != nullptr) {
                        load4(yfg + at, fy[t]);
                        load4(cfg + at, fc[t]);
                    }
                    if (gets_right) load4(yng + at, ny[t]);
                    if (gets_down) load4(cng + at, nc[t]);
                }
#if !G2D_JOINT
#pragma unroll
                for (int t = 0; t < 2; ++t) {  // the eight diagonal blocks, 64 vectors each
                    const int idx = t * TTH + tid, blk = idx / 64, r = idx / 4 % SUB, c = idx % 4 * 4, o = (blk % NSUB) * SUB;
                    load4(blk < NSUB ? lg + (i0 + o + r) * ldl + i0 + o + c : ug + (j0 + o + r) * ldu + j0 + o + c, dv[t]);
                }
                for (int idx = tid; idx < DROWS * DLD / 4; idx += TTH) {
                    const F zero[4] = {(F)0, (F)0, (F)0, (F)0};
                    store4(Dg + idx * 4, zero);
                }
#endif
                __syncthreads();
#pragma unroll
                for (int t = 0; t < PER; ++t) {
                    const int idx = t * TTH + tid, r = idx / (TILE / 4), c = (idx % (TILE / 4)) * 4;
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        // the two feedbacks first, which are smaller: one rounding at the size of Y (error of 777 x 1333 from float64
                        // 1.568e-7 with two, 1.556e-7 with one, 1.548e-7 for float32 products throughout)
                        vy[t][x] += fy[t][x] + ny[t][x];
                        vc[t][x] += fc[t][x] + nc[t][x];
                    }
                    store4(Ys + r * LD + c, vy[t]);
                    store4(Cs + r * LD + c, vc[t]);
                }
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    const int idx = t * TTH + tid, blk = idx / 64, r = idx / 4 % SUB, c = idx % 4 * 4;
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        const int p = blk < NSUB ? c + x : r, q = blk < NSUB ? r : c + x;  // source and receiver
                        if (q > p) Dg[(SUB + blk * SUB + p) * DLD + q - p] = dv[t][x];
                    }
                }
                asm volatile("cp.async.wait_all;" ::: "memory");
            }
        }
#if G2D_JOINT
        after_the_launch_before();
#endif
        if (!have_diagonal) {
            constexpr int UN = 8;
            for (int base = 0; base < TILE * TILE; base += TTH * UN) {
                F vy[UN], vc[UN], vl[UN];
#pragma unroll
                for (int t = 0; t < UN; ++t) {
                    const int idx = base + t * TTH + tid, r = idx / TILE, c = idx % TILE;
                    const int64_t gi = i0 + r, gj = j0 + c;
                    const bool in = gi < m && gj < n;
                    vy[t] = in ? yg[gi * ld + gj] : (F)0;
                    vc[t] = in ? cg[gi * ld + gj] : (F)0;
                    if (in && yfg != nullptr) {
                        vy[t] += yfg[gi * ld + gj] + (gets_right ? yng[gi * ld + gj] : (F)0);
                        vc[t] += cfg[gi * ld + gj] + (gets_down ? cng[gi * ld + gj] : (F)0);
                    }
                    vl[t] = (F)0;
                    if (r > c) {
                        if (gi < m) vl[t] = lg[gi * ldl + i0 + c];
                    } else if (r < c) {
                        if (gj < n) vl[t] = ug[(j0 + r) * ldu + gj];
                    }
                }
#pragma unroll
                for (int t = 0; t < UN; ++t) {
                    const int idx = base + t * TTH + tid, r = idx / TILE, c = idx % TILE;
                    Ys[r * LD + c] = vy[t];
                    Cs[r * LD + c] = vc[t];
                    LUs[r * LD + c] = vl[t];
                }
            }
            if constexpr (PUSH) {
                if (owes_right)
                    for (int idx = tid; idx < TILE * TILE; idx += TTH) {
                        const int r = idx / TILE, c = idx % TILE;
                        Ubs[r * LD + c] = (j0 + r < n && j0 + TILE + c < n) ? ug[(j0 + r) * ldu + j0 + TILE + c] : (F)0;
                    }
                if (owes_down)
                    for (int idx = tid; idx < TILE * TILE; idx += TTH) {
                        const int r = idx / TILE, c = idx % TILE;
                        Lbs[r * LD + c] = (i0 + TILE + r < m && i0 + c < m) ? lg[(i0 + TILE + r) * ldl + i0 + c] : (F)0;
                    }
            }
            __syncthreads();
            for (int idx = tid; idx < DROWS * DLD; idx += TTH) {
                const int row = idx / DLD - SUB, dd = idx % DLD, blk = row / SUB, p = row % SUB;
                F v = (F)0;
                if (row >= 0 && blk < 2 * NSUB && dd >= 1 && dd < SUB && p + dd < SUB) {
                    const int at = (blk % NSUB) * SUB + p;
                    v = blk < NSUB ? LUs[(at + dd) * LD + at] : LUs[at * LD + at + dd];
                }
                Dg[idx] = v;
            }
        }
        if (!sweeper) {
            finish_params(0);
            store_params(0);
        }
        __syncthreads();
        // Sweep of the sub-tiles: sweeping warp a takes the sub-tiles of row a, one per sub-tile anti-diagonal.  Lane k of the
        // warp's first half owns column k of the sub-tile (down feedback, "C"), lane k of the second half row k (right
        // feedback, "Y"), both skewed so that the entry of stage s sits in register 0 when the stage comes.  At stage s the
        // column lane k and the row lane p = s - k hold the two summands of entry (p, k): one shuffle exchanges them and
        // both lanes round the entry (the sum commutes, so they get the same bits).  The column lane pushes the error down,
        // the row lane, which received the C accumulator with the same shuffle, the completed C to the right: one shuffle
        // and fifteen multiply-adds per lane and stage.  (Half a warp per sub-tile with both feedbacks in one lane takes
        // two shuffles and thirty multiply-adds: 208 cycles per stage against about 100.)
        // What bounds a stage is the chain from one rounding to the next (multiply-add, shuffle, the quantizer's dozen dependent
        // operations: about 95 cycles); everything else has to fit into its gaps.  So every address of a stage is a lane's base
        // plus a constant stride (lanes before their first or past their last entry read zero rows or values that they
        // ignore, and store nothing), the operands of a stage are loaded one stage ahead, and there is no branch inside the
        // four unrolled stages (one branch per stage costs 40 cycles): about 120 cycles per stage for one warp on its
        // scheduler, 150 for two, against 168 with wrapped addresses and selects.
        // The two roles run the same sequence of barriers from loops of their own, so that neither holds the other's registers.
        if (sweeper) {
            const int sub_a = number, r0 = sub_a * SUB;
            const int par0 = (sub_a * SUB * PLD + (role ? k * PLD - k : k - k * PLD)) * 4, par_step = (role ? 1 : PLD) * 4;
            for (int w = 0; w < 2 * NSUB - 1; ++w) {
                const int b = w - sub_a;
                if (b >= 0 && b < NSUB) {
                    const int c0 = b * SUB;
                    // entries of this lane inside the matrix: the first `count` of its column or row
                    const int rows_left = rows_in - r0, cols_left = cols_in - c0;
                    const int along = role ? cols_left : rows_left, count = k < (role ? rows_left : cols_left) ? max(0, min(along, SUB)) : 0;
                    const int step = role ? 1 : LD;
                    F acc[SUB];
                    {
                        const F *const src = role ? Ys + (r0 + k) * LD + c0 : Cs + r0 * LD + c0 + k;
#pragma unroll
                        for (int r = 0; r < SUB; ++r) acc[r] = src[((r - k) & (SUB - 1)) * step];
                    }
                    F *const pre_ptr = pre + (i0 + r0) * n + j0 + c0 + k;  // the caller's array: rows of n
                    const int partner0 = ((role ^ 1) << 4) - k;
                    auto stages = [&](auto divide_tag, auto record_tag) {
                        constexpr int DIVIDE = decltype(divide_tag)::value;
                        constexpr bool RECORD = decltype(record_tag)::value;
                        uint32_t dg = shared_address(Dg) + (uint32_t)((SUB + ((role ? NSUB + b : sub_a)) * SUB - k) * DLD * (int)sizeof(F));
                        uint32_t par = shared_address(Par) + (uint32_t)(par0 * (int)sizeof(F));
                        const uint32_t par_bytes = (uint32_t)(par_step * (int)sizeof(F));
                        uint32_t own = shared_address(role ? Cs + (r0 + k) * LD + c0 : Ys + r0 * LD + c0 + k) - (uint32_t)(k * step * (int)sizeof(F));
                        F kc[SUB], pa[4];
                        auto fetch = [&](uint32_t d, uint32_t q, F (&co)[SUB], F (&pq)[4]) {
                            if (KIND != G2D_Q_ROUND) load4_here(q, pq);
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
                                F kc_next[SUB], pa_next[4];
                                fetch(dg + (uint32_t)((j + 1) * DLD * (int)sizeof(F)), par + par_bytes, kc_next, pa_next);
                                const F carry = role ? other : (F)0;
                                const F yv = acc[0] + other;
                                F z, z_out;  // what is stored: z, with the sign of a zero
                                if (KIND == G2D_Q_AFFINE && DIVIDE == 0) {
                                    z = affine_value_fast(yv, pa[0], pa[1], pa[2], P.qmin, P.qmax, z_out);
                                } else if (KIND == G2D_Q_AFFINE) {
                                    z = DIVIDE == 2 ? affine_value(yv, pa[0], pa[1], P.qmin, P.qmax) : affine_value_rcp(yv, pa[0], pa[1], pa[2], P.qmin, P.qmax);
                                } else if (KIND == G2D_Q_FORCED) {
                                    z = pa[0];
                                } else {
                                    z = rint_even(yv);
                                }
                                if (KIND != G2D_Q_AFFINE || DIVIDE != 0) z_out = z;
                                const F carried = (z - yv) + carry;  // completed C (row lanes) or error (column lanes)
                                const F v = ok ? carried : (F)0;     // lanes without an entry push zero
#pragma unroll
                                // the push moves every accumulator down by one register on the way
                                const F last = acc[0];
#pragma unroll
                                for (int dd = 1; dd < SUB; ++dd) acc[dd - 1] = acc[dd] + kc[dd] * v;
                                acc[SUB - 1] = last;
                                store_shared_if(own, carried, ok);
                                store_shared_if(par + 3 * (uint32_t)sizeof(F), z_out, ok);  // both lanes of an entry store the same value
                                if (RECORD && ok && !role) pre_ptr[(int64_t)p * n] = yv;
                                own += (uint32_t)(step * (int)sizeof(F));
                                par += par_bytes;
                                ++p;
#pragma unroll
                                for (int x = 0; x < SUB; ++x) kc[x] = kc_next[x];
#pragma unroll
                                for (int x = 0; x < 4; ++x) pa[x] = pa_next[x];
                            }
                            dg += (uint32_t)(ROLL * DLD * (int)sizeof(F));
                        }
                    };
                    using std::integral_constant;
                    // 0 and 1 for the common case, without a branch in the stages; recording the pre-rounding values is a matter of tests
                    const bool exact = !fast_div[sub_a];
                    if (pre != nullptr) {
                        if (exact) stages(integral_constant<int, 2>{}, std::true_type{});
                        else stages(integral_constant<int, 1>{}, std::true_type{});
                    } else if (exact) stages(integral_constant<int, 2>{}, std::false_type{});
                    else if (sizeof(F) != sizeof(float) || !P.small_integer_bounds) stages(integral_constant<int, 1>{}, std::false_type{});
                    else stages(integral_constant<int, 0>{}, std::false_type{});
                }
                __syncthreads();
                if (w + 1 < 2 * NSUB - 1) {
                    // the anti-diagonal just swept, carried into the next one: the right product here, the down product by the helper
                    const int bn = w + 1 - sub_a;
                    if (bn >= 1 && bn < NSUB)
                        mm16<SMALL>(Ys + r0 * LD + bn * SUB, Cs + r0 * LD + (bn - 1) * SUB, LUs + (bn - 1) * SUB * LD + bn * SUB, lane);
                    __syncthreads();
                }
            }
        } else {
            for (int w = 0; w < 2 * NSUB - 1; ++w) {
                const bool more = w + 1 < 2 * NSUB - 1;
                const int ap = helper;
                if (more) fetch_params(w + 1);
                // While sub-tile anti-diagonal w is swept: the products of the sub-tiles (a, b) swept one anti-diagonal ago, i.e.
                // the row strip of each in the push to the right neighbour, the column strip in the push to the lower one
                // (dealt out to the helpers in turn), and the feedback to the sub-tiles two or more places down (helpers 0
                // and 1) and to the right (2 and 3).  All these products have targets of their own, none of them on w.
                const int a_lo = max(0, w - NSUB), a_hi = min(NSUB, w);
#pragma unroll 1
                for (int a = a_lo; a < a_hi; ++a) {
                    const int b = w - 1 - a, to = helper < 2 ? a + 2 + helper : b + helper;
                    if (to >= NSUB) continue;
                    if (helper < 2) mm16<SMALL>(Cs + to * SUB * LD + b * SUB, LUs + to * SUB * LD + a * SUB, Ys + a * SUB * LD + b * SUB, lane);
                    else mm16<SMALL>(Ys + a * SUB * LD + to * SUB, Cs + a * SUB * LD + b * SUB, LUs + b * SUB * LD + to * SUB, lane);
                }
                if constexpr (PUSH) {
#pragma unroll 1
                    for (int job = helper; job < 2 * (a_hi - a_lo); job += HELPERS) {
                        const int a = a_lo + (job >> 1), b = w - 1 - a;
                        if (job & 1) {
                            if (owes_down) mm16<TALL>(Cns + b * SUB, Lbs + a * SUB, Ys + a * SUB * LD + b * SUB, lane);
                        } else {
                            if (owes_right) mm16<WIDE>(Yns + a * SUB * LD, Cs + a * SUB * LD + b * SUB, Ubs + b * SUB * LD, lane);
                        }
                    }
                }
                if (more) finish_params(w + 1);
                __syncthreads();
                {   // the rounded values of the sub-tiles just swept: helper warp ap writes out the block of its row
                    const int bz = w - ap;
                    if (bz >= 0 && bz < NSUB) {
                        const bool zvec = ld % 4 == 0 && reinterpret_cast<uintptr_t>(yg) % (4 * sizeof(F)) == 0;
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            const int e = lane * 2 + q, row = e >> 2, c4 = (e & 3) * 4;
                            const int64_t gi = i0 + ap * SUB + row, gj = j0 + bz * SUB + c4;
                            F v[4];
#pragma unroll
                            for (int x = 0; x < 4; ++x) v[x] = Par[((ap * SUB + row) * PLD + c4 + x) * 4 + 3];
                            if (gi < m) {
                                if (zvec) {
                                    if (gj < n) store4(yg + gi * ld + gj, v);
                                } else {
#pragma unroll
                                    for (int x = 0; x < 4; ++x)
                                        if (gj + x < n) yg[gi * ld + gj + x] = v[x];
                                }
                            }
                        }
                        __syncwarp();  // the next parameters overwrite them
                    }
                }
                // ---- between two sweeps: the anti-diagonal just swept, carried into the next one; the next parameters ----
                if (more) {
                    store_params(w + 1);
                    const int bn = w + 1 - ap;
                    if (ap >= 1 && bn >= 0 && bn < NSUB)  // the right product is the sweeping warp's
                        mm16<SMALL>(Cs + ap * SUB * LD + bn * SUB, LUs + ap * SUB * LD + (ap - 1) * SUB, Ys + (ap - 1) * SUB * LD + bn * SUB, lane);
                    __syncthreads();
                }
            }
        }
#if G2D_JOINT
        let_the_next_launch_start();
#endif
        // ---- neighbour push: the last sub-tile's terms, one product per warp, then out to the planes of the neighbours ----
        if constexpr (PUSH) {
            if (owes_right || owes_down) {
                constexpr int last = NSUB - 1;
                const int x = warp & 3;
                F *const D = warp < 4 ? Yns + last * SUB * LD + x * SUB : Cns + x * SUB * LD + last * SUB;
                const F *const A = warp < 4 ? Cs + last * SUB * LD + last * SUB : Lbs + x * SUB * LD + last * SUB;
                const F *const B = warp < 4 ? Ubs + last * SUB * LD + x * SUB : Ys + last * SUB * LD + last * SUB;
                if (warp < 4 ? owes_right : owes_down) mm16<SMALL>(D, A, B, lane);
                __syncthreads();
                // rows and columns past the matrix are not stored; a row's last group of four may reach into its padding
                const bool pvec = ld % 4 == 0 && reinterpret_cast<uintptr_t>(yng) % (4 * sizeof(F)) == 0;
                for (int idx = tid; idx < TILE * TILE / 4; idx += TTH) {
                    const int r = idx / (TILE / 4), c = (idx % (TILE / 4)) * 4;
                    F v[4];
                    if (owes_right && i0 + r < m && j0 + TILE + c < n) {
                        load4(Yns + r * LD + c, v);
                        F *dst = yng + (i0 + r) * ld + j0 + TILE + c;
                        if (pvec) store4(dst, v);
                        else
                            for (int x4 = 0; x4 < 4; ++x4)
                                if (j0 + TILE + c + x4 < n) dst[x4] = v[x4];
                    }
                    if (owes_down && i0 + TILE + r < m && j0 + c < n) {
                        load4(Cns + r * LD + c, v);
                        F *dst = cng + (i0 + TILE + r) * ld + j0 + c;
                        if (pvec) store4(dst, v);
                        else
                            for (int x4 = 0; x4 < 4; ++x4)
                                if (j0 + c + x4 < n) dst[x4] = v[x4];
                    }
                }
            }
        }
        // ---- operands of the tensor-core updates: fp16 pairs of E (transposed) and of the completed C under the tile's scales ----
        bool wide_e = false, wide_c = false;
        if constexpr (sizeof(F) == sizeof(float)) {
            if (P.c_hi != nullptr) {
                // Largest values of the rows, the columns and the tile (entries outside the matrix are zero), of E in the lower and of C in
                // the upper half of a word: the upper halves of floats are all that the scale and the comparison need.
                unsigned column[4] = {0u, 0u, 0u, 0u};
#pragma unroll
                for (int t = 0; t < TILE * TILE / 4 / TTH; ++t) {  // a thread's vectors lie in the same four columns
                    const int idx = t * TTH + tid, r = idx / (TILE / 4), c = (idx % (TILE / 4)) * 4;
                    F ve[4], vc[4];
                    load4(Ys + r * LD + c, ve);
                    load4(Cs + r * LD + c, vc);
                    unsigned row = 0u;
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        const unsigned both = __byte_perm(__float_as_uint((float)ve[x]), __float_as_uint((float)vc[x]), 0x7632) & 0x7fff7fffu;
                        row = __vmaxu2(row, both);
                        column[x] = __vmaxu2(column[x], both);
                    }
#pragma unroll
                    for (int o = 1; o < TILE / 4; o <<= 1) row = __vmaxu2(row, __shfl_xor_sync(0xffffffffu, row, o));
                    if ((lane & 15) == 0) row_max[r] = row;
                }
#pragma unroll
                for (int x = 0; x < 4; ++x) column[x] = __vmaxu2(column[x], __shfl_xor_sync(0xffffffffu, column[x], 16));
                if (lane < 16) *reinterpret_cast<uint4 *>(&column_max[warp][lane * 4]) = make_uint4(column[0], column[1], column[2], column[3]);
                __syncthreads();
                unsigned most = 0u, least = 0xffffffffu;  // every warp for itself: two rows and two columns per lane
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    unsigned col = column_max[0][h * 32 + lane];
#pragma unroll
                    for (int w2 = 1; w2 < TTH / 32; ++w2) col = __vmaxu2(col, column_max[w2][h * 32 + lane]);
                    const unsigned row = row_max[h * 32 + lane];
                    most = __vmaxu2(most, row);
                    least = __vminu2(least, __vminu2(row | __vcmpeq2(row, 0u), col | __vcmpeq2(col, 0u)));  // zeros apart
                }
                const unsigned most_e = __reduce_max_sync(0xffffffffu, most & 0xffffu), most_c = __reduce_max_sync(0xffffffffu, most >> 16);
                const unsigned least_e = __reduce_min_sync(0xffffffffu, least & 0xffffu), least_c = __reduce_min_sync(0xffffffffu, least >> 16);
                wide_e = most_e >= 0x7f80u || least_e + WIDE_RATIO_BITS <= most_e;
                wide_c = most_c >= 0x7f80u || least_c + WIDE_RATIO_BITS <= most_c;
                const int ee = range_exponent(__uint_as_float(most_e << 16)), ec = range_exponent(__uint_as_float(most_c << 16));
                if (tid == 0) {
                    P.e_scale[(int64_t)I * P.nJ + J] = wide_e ? -1.f : power_of_two(ee);
                    P.c_scale[(int64_t)I * P.nJ + J] = wide_c ? -1.f : power_of_two(ec);
                    if (wide_e || wide_c) atomicAdd(P.wide_count, wide_e + wide_c);
                }
                const float e_by = power_of_two(-ee), c_by = power_of_two(-ec);
                // eight entries per thread and store.  C along its rows; E transposed: a thread gathers eight rows of one column
                // (consecutive threads take consecutive columns, so the shared-memory reads do not collide) and writes them as
                // one vector of a row of E^T.  A row's last vector may reach into its padding.
                for (int idx = tid; idx < TILE * TILE / 8; idx += TTH) {
                    __align__(16) __half h[8];
                    __align__(16) __half l[8];
                    {
                        const int r = idx / (TILE / 8), c = (idx % (TILE / 8)) * 8;
                        if (r < rows_in && c < cols_in) {
#pragma unroll
                            for (int x = 0; x < 8; ++x) split_half(wide_c ? 0.f : (float)Cs[r * LD + c + x] * c_by, h[x], l[x]);
                            const int64_t at = (i0 + r) * P.ldn + j0 + c;
                            *reinterpret_cast<uint4 *>(P.c_hi + at) = *reinterpret_cast<const uint4 *>(h);
                            *reinterpret_cast<uint4 *>(P.c_lo + at) = *reinterpret_cast<const uint4 *>(l);
                        }
                    }
                    {
                        const int c = idx % TILE, r = (idx / TILE) * 8;
                        if (r < rows_in && c < cols_in) {
#pragma unroll
                            for (int x = 0; x < 8; ++x) split_half(wide_e ? 0.f : (float)Ys[(r + x) * LD + c] * e_by, h[x], l[x]);
                            const int64_t at = (j0 + c) * P.ldm + i0 + r;
                            *reinterpret_cast<uint4 *>(P.et_hi + at) = *reinterpret_cast<const uint4 *>(h);
                            *reinterpret_cast<uint4 *>(P.et_lo + at) = *reinterpret_cast<const uint4 *>(l);
                        }
                    }
                }
            }
        }
        // ---- store the errors and the completed C of the tile, unless only their operand planes are read from here on ----
        const bool planes_only = P.c_hi != nullptr && yng != nullptr;
        const bool keep_e = !planes_only || wide_e, keep_c = !planes_only || wide_c;
        if (!keep_e && !keep_c) {
        } else if (vec) {
            for (int idx = tid; idx < TILE * TILE / 4; idx += TTH) {
                const int r = idx / (TILE / 4), c = (idx % (TILE / 4)) * 4;
                F ve[4], vc[4];
                load4(Ys + r * LD + c, ve);
                load4(Cs + r * LD + c, vc);
                if (keep_e) store4(eg + (i0 + r) * ld + j0 + c, ve);
                if (keep_c) store4(cg + (i0 + r) * ld + j0 + c, vc);
            }
        } else {
            for (int r = warp; r < rows_in; r += TTH / 32)
                for (int c = lane; c < cols_in; c += 32) {
                    if (keep_e) eg[(i0 + r) * ld + j0 + c] = Ys[r * LD + c];
                    if (keep_c) cg[(i0 + r) * ld + j0 + c] = Cs[r * LD + c];
                }
        }
        __syncthreads();
    }

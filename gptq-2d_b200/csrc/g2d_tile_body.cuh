// The body of the tile sweep's kernels, taken in as text: extracted into a function, the same statements compiled to tiles 2 % slower.
// G2D_JOINT: the launch may have started before the one before it has ended (see g2d_tile_sweep_step.cu).
    F *Ys = reinterpret_cast<F *>(g2d_smem);  // X + right feedback; the errors E once a sub-tile is swept
    F *Cs = Ys + TILE * LD;                   // down feedback; the completed C once a sub-tile is swept
    F *LUs = Cs + TILE * LD;                  // strict lower part: L[I, I]; strict upper part: U[J, J]
    F *Dg = LUs + TILE * LD;                  // zero-padded diagonal blocks L[a, a] and U[b, b]^T, strictly lower, between rows of zeros
    F *Par = Dg + DROWS * DLD;                // twice (by turns) two planes [NSUB][SUB][PLD][2]: scale and reciprocal, zero point and result of the entries of the sub-tiles being swept
    F *Ubs = Par + 4 * PPLANE;                // float only, pipelined schedule: U[J, J + 1], the right neighbour's coupling block
    F *Lbs = Ubs + TILE * LD;                 // the same: L[I + 1, I], the lower neighbour's
    F *Yns = Lbs + TILE * LD;                 // the same: the feedback for the right neighbour, C[I, J] U[J, J + 1], growing sub-tile by sub-tile
    F *Cns = Yns + TILE * LD;                 // and for the lower one, L[I + 1, I] E[I, J]
    __shared__ unsigned row_max[TILE], column_max[TILE];  // see last_extremes
    __shared__ int early_exponent[2];         // of E and C without the sub-tile that is swept last
    __shared__ unsigned fast_div[2][NSUB];       // bit 0: every scale of the sub-tile allows the division by reciprocal; bit 1: its zero points are +0

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
        // where the feedback for the neighbours belongs, and how much of it is inside the matrix
        F *const yn_out = yng + i0 * ld + j0 + TILE, *const cn_out = cng + (i0 + TILE) * ld + j0;
        const bool push_vec = ld % 4 == 0 && reinterpret_cast<uintptr_t>(yng) % (4 * sizeof(F)) == 0;
        const int cols_right = (int)min((int64_t)TILE, n - j0 - TILE), rows_below = (int)min((int64_t)TILE, m - i0 - TILE);
        const bool owes_right = yng != nullptr && J + 1 < P.nJ, owes_down = yng != nullptr && I + 1 < P.nI;

        Tile<F> tile;
        tile.i0 = i0; tile.j0 = j0; tile.n = n; tile.ld = ld; tile.rows = rows_in; tile.cols = cols_in;
        tile.y = yg; tile.scale = sg; tile.zero = zg; tile.forced = fg;
        tile.srs = P.srs; tile.scs = P.scs; tile.zrs = P.zrs; tile.zcs = P.zcs;
        tile.unfinished = pre == nullptr && P.small_integer_bounds;
        tile.zvec = ld % 4 == 0 && reinterpret_cast<uintptr_t>(yg) % (4 * sizeof(F)) == 0;
        const auto params_of = [&](int w) { return Par + (w & 1) * 2 * PPLANE; };
        Params<F> params;
        if (!sweeper) fetch_params<F, KIND>(tile, 0, helper, lane, params);
        constexpr bool PUSH = sizeof(F) == sizeof(float);  // the neighbour push exists for float (pipelined schedule) only

        // ---- load the tile ----
        // rows as vectors: of a tile at the matrix's edge too, which then loads from inside the matrix and puts zeros outside (a value at a time
        // took 5 us more, on nearly every launch of a matrix that is no multiple of 64)
        const bool row_vectors = ((ld | ldl | ldu) % 4 == 0) &&
                                 ((reinterpret_cast<uintptr_t>(yg) | reinterpret_cast<uintptr_t>(cg) | reinterpret_cast<uintptr_t>(eg) |
                                   reinterpret_cast<uintptr_t>(lg) | reinterpret_cast<uintptr_t>(ug)) % (4 * sizeof(F)) == 0);
        const bool vec = full && row_vectors;
        bool have_diagonal = false;
        if constexpr (PUSH) {
            if (owes_right || owes_down)
                for (int idx = tid; idx < 2 * TILE * LD / 4; idx += TTH) {
                    const F zero[4] = {(F)0, (F)0, (F)0, (F)0};
                    store4(Yns + idx * 4, zero);
                }
            if (row_vectors) {
                // One wait on global memory: the off-diagonal blocks of L[I, I] and U[J, J] and the two coupling blocks
                // travel to shared memory on their own (cp.async), the diagonal blocks and the six planes that make up Y and
                // C through registers, and all of them are issued before the first is used.
                have_diagonal = true;
                for (int c = tid; c < 12 * SUB * 4; c += TTH) {
                    const int blk = c / (SUB * 4), ba = blk / 3, bb = blk % 3 + (blk % 3 >= ba ? 1 : 0), row = ba * SUB + c / 4 % SUB, col = bb * SUB + c % 4 * 4;
                    const int inside = ba > bb ? rows_in : cols_in, there = row < inside ? min(4, max(0, inside - col)) : 0;  // values of the vector
                    const F *src = ba > bb ? lg + (i0 + row) * ldl + i0 + col : ug + (j0 + row) * ldu + j0 + col;
                    async16(LUs + row * LD + col, there ? src : lg, there * (int)sizeof(F));
                }
                if (owes_right)
                    for (int c = tid; c < TILE * TILE / 4; c += TTH) {
                        const int row = c / (TILE / 4), col = c % (TILE / 4) * 4;
                        // n is not always a multiple of 4, the row stride is.  The tail of a padded copy is not defined: what is formed
                        // with it goes to columns from n on, which are not stored, or stored to padding that nothing reads.
                        const bool in = j0 + TILE + col < n;
                        async16(Ubs + row * LD + col, ug + (j0 + row) * ldu + (in ? j0 + TILE + col : 0), in ? 16 : 0);
                    }
                if (owes_down)
                    for (int c = tid; c < TILE * TILE / 4; c += TTH) {
                        const int row = c / (TILE / 4), col = c % (TILE / 4) * 4;
                        const bool in = i0 + TILE + row < m;
                        async16(Lbs + row * LD + col, lg + (in ? i0 + TILE + row : 0) * ldl + i0 + col, in ? 16 : 0);
                    }
                asm volatile("cp.async.commit_group;" ::: "memory");
                constexpr int PER = TILE * TILE / 4 / TTH;  // vectors per thread and array
                F vy[PER][4], vc[PER][4], fy[PER][4], fc[PER][4], ny[PER][4], nc[PER][4], dv[2][4];
#if G2D_JOINT  // the factors ahead of the wait
#pragma unroll
                for (int t = 0; t < 2; ++t) {  // the eight diagonal blocks, 64 vectors each
                    const int idx = t * TTH + tid, blk = idx / 64, o = (blk % NSUB) * SUB, inside = blk < NSUB ? rows_in : cols_in;
                    const int r = min(o + idx / 4 % SUB, inside - 1), c = o + idx % 4 * 4 < inside ? o + idx % 4 * 4 : 0;
                    load4(blk < NSUB ? lg + (i0 + r) * ldl + i0 + c : ug + (j0 + r) * ldu + j0 + c, dv[t]);
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
                    const int64_t at = (i0 + min(r, rows_in - 1)) * ld + j0 + (c < cols_in ? c : 0);
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
                    const int idx = t * TTH + tid, blk = idx / 64, o = (blk % NSUB) * SUB, inside = blk < NSUB ? rows_in : cols_in;
                    const int r = min(o + idx / 4 % SUB, inside - 1), c = o + idx % 4 * 4 < inside ? o + idx % 4 * 4 : 0;
                    load4(blk < NSUB ? lg + (i0 + r) * ldl + i0 + c : ug + (j0 + r) * ldu + j0 + c, dv[t]);
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
                    if (!full)
#pragma unroll
                        for (int x = 0; x < 4; ++x)
                            if (r >= rows_in || c + x >= cols_in) vy[t][x] = vc[t][x] = (F)0;
                    store4(Ys + r * LD + c, vy[t]);
                    store4(Cs + r * LD + c, vc[t]);
                }
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    const int idx = t * TTH + tid, blk = idx / 64, r = idx / 4 % SUB, c = idx % 4 * 4;
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        const int p = blk < NSUB ? c + x : r, q = blk < NSUB ? r : c + x;  // source and receiver
                        const int inside = (blk < NSUB ? rows_in : cols_in) - (blk % NSUB) * SUB;
                        if (q > p) Dg[(SUB + blk * SUB + p) * DLD + q - p] = q < inside ? dv[t][x] : (F)0;
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
            finish_params<F, KIND>(tile, params_of(0), &fast_div[0][helper], 0, helper, lane, params);
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
        // What bounds a stage is the chain from one rounding to the next (multiply-add, shuffle of 26 cycles, the quantizer's
        // dependent operations at 4.5 to 5.4 cycles each: about 82 cycles, 92 with a zero point, 95 before affine_steps_fast); everything else has to fit into its
        // gaps.  So every address of a stage is a lane's base plus a constant stride (lanes before their first or past their last entry
        // read zero rows or values that they ignore, and store nothing), the operands of a stage are loaded one stage ahead, and there is
        // no branch inside the four unrolled stages (one branch per stage costs 40 cycles): with the other warps' work beside it 123 to 143 cycles
        // per stage where one or two sub-tiles are swept and 180 where four are.
        // The two roles run the same sequence of barriers from loops of their own, so that neither holds the other's registers.
        // Operands of the tensor-core updates: fp16 pairs of E (transposed) and of the completed C under the tile's scales, eight entries
        // per thread and store.  C along its rows; E transposed: a thread gathers eight rows of one column (consecutive threads take
        // consecutive columns, so the shared-memory reads do not collide) and writes them as one vector of a row of E^T.  A
        // row's last vector may reach into its padding.  Zeros where the factor is.
        auto split_c = [&](int r, int c, float by) {
            if constexpr (PUSH) {
                const int64_t at = (i0 + r) * P.ldn + j0 + c;
                split8<false>(Cs + r * LD + c, by, P.c_hi + at, P.c_lo + at, r < rows_in && c < cols_in);
            }
        };
        auto split_e = [&](int r, int c, float by) {
            if constexpr (PUSH) {
                const int64_t at = (j0 + c) * P.ldm + i0 + r;
                split8<true>(Ys + r * LD + c, by, P.et_hi + at, P.et_lo + at, r < rows_in && c < cols_in);
            }
        };
        if (sweeper) {
            const int sub_a = number, r0 = sub_a * SUB;
#pragma unroll 1
            for (int w = 0; w < 2 * NSUB - 1; ++w) {
                const int b = w - sub_a;
                if (b >= 0 && b < NSUB) {
                    SubTile<F> t;
                    t.ys = Ys + r0 * LD + b * SUB;
                    t.cs = Cs + r0 * LD + b * SUB;
                    t.dg_c = Dg + (SUB + sub_a * SUB) * DLD;
                    t.dg_y = Dg + (SUB + (NSUB + b) * SUB) * DLD;
                    t.par = Par + (w & 1) * 2 * PPLANE + sub_a * SUB * PLD * 2;
                    t.rows = rows_in - r0;
                    t.cols = cols_in - b * SUB;
                    t.qmin = P.qmin;
                    t.qmax = P.qmax;
                    t.pre = pre != nullptr ? pre + (i0 + r0) * n + j0 + b * SUB : nullptr;  // the caller's array: rows of n
                    t.pre_ld = n;
                    // 3 and 4 (float) and 1 (double) for the common case, without a branch in the stages; recording the pre-rounding
                    // values is a matter of tests.  The zero points of symmetric codes are zeros.  Cycles per stage with 4, 3 and 1, where one
                    // sub-tile is swept and where four are: 134 and 180, 155 and 198, 164 and 217 (256 x 256).
                    const unsigned how = fast_div[w & 1][sub_a];
                    const bool exact = !(how & 1);
                    if (pre != nullptr) {
                        if (exact) sweep_sub_tile<F, KIND, 2, true>(t, lane);
                        else sweep_sub_tile<F, KIND, 1, true>(t, lane);
                    } else if (exact) sweep_sub_tile<F, KIND, 2, false>(t, lane);
                    else if constexpr (sizeof(F) == sizeof(float)) {
                        if (!P.small_integer_bounds) sweep_sub_tile<F, KIND, 1, false>(t, lane);
                        else if (how & 2) sweep_sub_tile<F, KIND, 4, false>(t, lane);
                        else sweep_sub_tile<F, KIND, 3, false>(t, lane);
                    } else sweep_sub_tile<F, KIND, 1, false>(t, lane);
                }
                if constexpr (PUSH) {
                    // While the last sub-tile is swept, the warps of rows 0 and 2 make the operand planes of everything else, under the scales that
                    // follow from everything else: the last sub-tile seldom changes them.  (They share a scheduler; row 1 shares one with
                    // the sweep, which took 180 cycles a stage beside it in place of 120.)
                    if (w == 2 * NSUB - 2 && (number & 1) == 0 && P.c_hi != nullptr) {
                        const int at = (number >> 1) * 32 + lane;  // row, then column
                        row_max[at] = row_extreme(Ys + at * LD, Cs + at * LD, at < LAST * SUB ? TILE : LAST * SUB);
                        early_planes_barrier();
                        const unsigned all = __vmaxu2(row_max[lane], row_max[32 + lane]);
                        const int ee = range_exponent(__uint_as_float(__reduce_max_sync(0xffffffffu, all & 0xffffu) << 16));
                        const int ec = range_exponent(__uint_as_float(__reduce_max_sync(0xffffffffu, all >> 16) << 16));
                        if (at == 0) {
                            early_exponent[0] = ee;
                            early_exponent[1] = ec;
                        }
                        const float e_by = power_of_two(-ee), c_by = power_of_two(-ec);
#pragma unroll 2
                        for (int r = 0; r < TILE; r += 8) {  // (the last sub-tile as it is at the moment; it is done again)
                            split_e(r, at, e_by);
                            split_c(r + at / 8, at % 8 * 8, c_by);
                        }
                    }
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
#pragma unroll 1
            for (int w = 0; w < 2 * NSUB - 1; ++w) {
                const bool more = w + 1 < 2 * NSUB - 1;
                const int ap = helper;
                write_rounded<F, KIND>(tile, params_of(w - 1), &fast_div[(w - 1) & 1][helper], w - 1, helper, lane);
                if (more) fetch_params<F, KIND>(tile, w + 1, helper, lane, params);
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
                            if (!owes_down) continue;
                            mm16<TALL>(Cns + b * SUB, Lbs + a * SUB, Ys + a * SUB * LD + b * SUB, lane);
                            if (a == LAST) push_out<TILE, SUB>(Cns + b * SUB, cn_out + b * SUB, ld, push_vec, rows_below, cols_in - b * SUB, lane);
                        } else {
                            if (!owes_right) continue;
                            mm16<WIDE>(Yns + a * SUB * LD, Cs + a * SUB * LD + b * SUB, Ubs + b * SUB * LD, lane);
                            if (b == LAST) push_out<SUB, TILE>(Yns + a * SUB * LD, yn_out + a * SUB * ld, ld, push_vec, rows_in - a * SUB, cols_right, lane);
                        }
                    }
                }
                if constexpr (PUSH) {
                    if (!more && helper < 2 && P.c_hi != nullptr) {
                        const int column = helper * 32 + lane;
                        column_max[column] = column_extreme(Ys + column, Cs + column, column < LAST * SUB ? TILE : LAST * SUB);
                    }
                }
                if (more) {
                    finish_params<F, KIND>(tile, params_of(w + 1), &fast_div[(w + 1) & 1][helper], w + 1, helper, lane, params);
                }
                __syncthreads();
                // ---- between two sweeps: the anti-diagonal just swept, carried into the next one ----
                if (more) {
                    const int bn = w + 1 - ap;
                    if (ap >= 1 && bn >= 0 && bn < NSUB)  // the right product is the sweeping warp's
                        mm16<SMALL>(Cs + ap * SUB * LD + bn * SUB, LUs + ap * SUB * LD + (ap - 1) * SUB, Ys + (ap - 1) * SUB * LD + bn * SUB, lane);
                    __syncthreads();
                }
            }
            write_rounded<F, KIND>(tile, params_of(2 * NSUB - 2), &fast_div[(2 * NSUB - 2) & 1][helper], 2 * NSUB - 2, helper, lane);
        }
#if G2D_JOINT
        let_the_next_launch_start();
#endif
        // ---- neighbour push: the last sub-tile's terms, one product per warp ----
        if constexpr (PUSH) {
            const int x = warp & 3;
            if (warp < 4) {
                if (owes_right) {
                    F *const D = Yns + LAST * SUB * LD + x * SUB;
                    mm16<SMALL>(D, Cs + LAST * SUB * LD + LAST * SUB, Ubs + LAST * SUB * LD + x * SUB, lane);
                    push_out<SUB, SUB>(D, yn_out + LAST * SUB * ld + x * SUB, ld, push_vec, rows_in - LAST * SUB, cols_right - x * SUB, lane);
                }
            } else if (owes_down) {
                F *const D = Cns + x * SUB * LD + LAST * SUB;
                mm16<SMALL>(D, Lbs + x * SUB * LD + LAST * SUB, Ys + LAST * SUB * LD + LAST * SUB, lane);
                push_out<SUB, SUB>(D, cn_out + x * SUB * ld + LAST * SUB, ld, push_vec, rows_below - x * SUB, cols_in - LAST * SUB, lane);
            }
        }
        // ---- operands of the tensor-core updates: what the last sub-tile changes, and what it adds ----
        const bool planes_only = P.c_hi != nullptr && yng != nullptr;  // the errors and the completed C are read from their operand planes alone
        bool keep_e = !planes_only, keep_c = !planes_only;
        if constexpr (PUSH) {
            if (P.c_hi != nullptr) {
                // Every warp for itself: the largest values of the rows and columns of the last sub-tile, on top of the others'
                unsigned most, least;
                last_extremes(Ys + LAST * SUB * LD + LAST * SUB, Cs + LAST * SUB * LD + LAST * SUB, row_max, column_max, lane, most, least);
                const unsigned most_e = __reduce_max_sync(0xffffffffu, most & 0xffffu), most_c = __reduce_max_sync(0xffffffffu, most >> 16);
                const unsigned least_e = __reduce_min_sync(0xffffffffu, least & 0xffffu), least_c = __reduce_min_sync(0xffffffffu, least >> 16);
                const bool wide_e = most_e >= 0x7f80u || least_e + WIDE_RATIO_BITS <= most_e;
                const bool wide_c = most_c >= 0x7f80u || least_c + WIDE_RATIO_BITS <= most_c;
                const int ee = range_exponent(__uint_as_float(most_e << 16)), ec = range_exponent(__uint_as_float(most_c << 16));
                if (tid == 0) {
                    P.e_scale[(int64_t)I * P.nJ + J] = wide_e ? -1.f : power_of_two(ee);
                    P.c_scale[(int64_t)I * P.nJ + J] = wide_c ? -1.f : power_of_two(ec);
                    if (wide_e || wide_c) atomicAdd(P.wide_count, wide_e + wide_c);
                }
                const float e_by = wide_e ? 0.f : power_of_two(-ee), c_by = wide_c ? 0.f : power_of_two(-ec);
                const bool as_foreseen = !wide_e && !wide_c && ee == early_exponent[0] && ec == early_exponent[1];
                if (as_foreseen) {
                    if (warp == 0) split_c(LAST * SUB + lane / 2, LAST * SUB + lane % 2 * 8, c_by);
                    if (warp == 1) split_e(LAST * SUB + lane / SUB * 8, LAST * SUB + lane % SUB, e_by);
                } else {
#pragma unroll 1
                    for (int idx = tid; idx < TILE * TILE / 8; idx += TTH) {
                        split_c(idx / (TILE / 8), idx % (TILE / 8) * 8, c_by);
                        split_e(idx / TILE * 8, idx % TILE, e_by);
                    }
                }
                keep_e = keep_e || wide_e;
                keep_c = keep_c || wide_c;
            }
        }
        // ---- store the errors and the completed C of the tile, unless only their operand planes are read from here on ----
        if (!keep_e && !keep_c) {
        } else if (vec) {
#pragma unroll 1
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

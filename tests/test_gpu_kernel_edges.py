"""The CUDA kernels at the sizes where they can go wrong: edges of tiles, remainders, the smallest and largest of a variant's range.

Bounds are worst-case rounding bounds: a sum of k products is off by at most (k + 2) u of the sum of their magnitudes
(u = 2^-24 for float32, 2^-53 for float64), whatever the order of its additions.
"""
import ctypes
import functools

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


# Float matrices: 64 x 64 tiles, macro tiles of 128, rows that need padding (m or n no multiple of 4), near updates from three tile
# anti-diagonals on, far updates from six macro anti-diagonals on; (7001, 7107): 2 x 2 macro tiles per CTA with ragged
# edges on both sides; outer_tiles = 16: far updates of rank 1024.  Batches and float64: the overlapped schedule.
@pytest.mark.parametrize("batch, m, n, dtype, outer", [
    (1, 1, 1, "float32", 0), (1, 1, 300, "float32", 0), (1, 63, 65, "float32", 0), (1, 129, 64, "float32", 0), (1, 131, 258, "float32", 0),
    (1, 257, 190, "float32", 0), (1, 705, 962, "float32", 0), (1, 1500, 1703, "float32", 0), (1, 2050, 1153, "float32", 16), (1, 7001, 7107, "float32", 0),
    (3, 65, 130, "float32", 0), (2, 577, 643, "float32", 0), (1, 65, 63, "float64", 0), (2, 129, 200, "float64", 0), (1, 641, 515, "float64", 0)])
def test_sweep_identity(batch, m, n, dtype, outer):
    """Z - X = (L + I) E (U + I) with E = Z - Y_pre, the defining identity of the sweep, entry by entry."""
    import _abi
    import gptq_2d as G

    dtype = getattr(torch, dtype)
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    rand = lambda *shape: torch.randn(*shape, generator=gen, device="cuda", dtype=dtype)
    w = 3 * rand(batch, m, n)
    l, u = torch.tril(rand(batch, m, m) * (0.3 / m ** .5), -1), torch.triu(rand(batch, n, n) * (0.3 / n ** .5), 1)
    if batch == 1:
        w, l, u = w[0], l[0], u[0]
    y, _, _, batch_shape = G._prepare_output(w, l, u, False)
    y_pre = torch.empty_like(y)
    G._sweep_fused(y, l, u, batch_shape, dict(kind=_abi.Q_ROUND), (), y_pre=y_pre, outer_tiles=outer)
    assert torch.equal(y, torch.round(y_pre))
    unit = 2.0 ** (-24 if dtype == torch.float32 else -53)
    wide = torch.float64
    e, full_l, full_u = (y - y_pre).to(wide), l.to(wide) + torch.eye(m, device="cuda", dtype=wide), u.to(wide) + torch.eye(n, device="cuda", dtype=wide)
    residual = (y.to(wide) - w.to(wide)) - full_l @ e @ full_u
    magnitude = full_l.abs() @ e.abs() @ full_u.abs() + y.to(wide).abs() + w.to(wide).abs()
    # an entry: up to 64 products per tile, then one addition per tile along its column and its row; a product of the tensor cores'
    # 16-bit pairs is off by 2 u; the completed C enters the right products with an error of its own; the identity is
    # evaluated in float64, whose sums of m + n products have an error too
    terms = 2 * (64 + 2 + (m + n) / 64) + (0 if dtype == torch.float32 else 2 * (m + n))
    assert ((residual.abs() - terms * unit * magnitude).max() <= 0).item(), (residual.abs() / (unit * magnitude)).max().item()
    again = w.clone()
    G._sweep_fused(again, l, u, batch_shape, dict(kind=_abi.Q_ROUND), (), outer_tiles=outer)
    assert torch.equal(again, y)


# tiles and near updates in one launch: two tiles and three along a side, one tile across the other, ragged last tiles, more jobs than stages per
# updating CTA, with far updates beside; and both sides of the limit of 128 tiles
@pytest.mark.parametrize("m, n", [(65, 130), (129, 192), (64, 640), (641, 63), (1000, 1028), (640, 8190), (8192, 8180), (8193, 8256)])
def test_sweep_identity_where_a_launch_updates_and_sweeps(m, n):
    test_sweep_identity(1, m, n, "float32", 0)


# from 1.5e8 entries on: far updates of rank 1024 by default, near updates in launches of their own
def test_sweep_identity_of_a_matrix_bound_by_far_updates():
    test_sweep_identity(1, 12250, 12301, "float32", 0)


# p * q entries per super-entry: rows and column groups that end inside a flush, one and several column groups per CTA, more columns
# than a CTA has threads for (q > 128), a single row, more stages than one flush collects
@pytest.mark.parametrize("m, n, p, q", [(1, 64, 1, 16), (13, 96, 1, 32), (70, 640, 1, 64), (20, 768, 4, 32), (9, 768, 1, 192), (150, 2048, 1, 16), (64, 4096, 4, 128)])
def test_absmax_super_entries_match_the_generic_engine(m, n, p, q):
    """The fused sweep against the engine that calls the quantizer once per stage, in float64: no entry may differ but by rounding."""
    import gptq_2d as G
    import quantizer_int as Q

    rng = np.random.default_rng(m + n)
    w = cuda(0.02 * rng.standard_normal((m, n)))
    l, u = cuda(np.tril(rng.standard_normal((m, m)) * (0.3 / m ** .5), -1)), cuda(np.triu(rng.standard_normal((n, n)) * (0.3 / n ** .5), 1))
    quantizer = functools.partial(Q.int_abs_max_quantizer_cuda, qmin=-8, qmax=7, dtype=torch.float16)
    fused = G.gptq_2d_super_entry(w, l, u, quantizer=quantizer, super_entry_shape=(p, q))
    generic = G.gptq_2d_super_entry(w, l, u, quantizer=lambda *a, **k: quantizer(*a, **k), super_entry_shape=(p, q))
    # a rounded value is a code times an fp16 scale: equal decisions give equal values up to the last bits
    assert (fused - generic).abs().max().item() <= 1e-12 * w.abs().max().item()


# 2^16 states: the cluster search from 2 to 8 bits per step; few steps and many, with the choices in shared memory and beyond it,
# more sequences than clusters run at a time, with and without the wrap-around
@pytest.mark.parametrize("rows, T, K, V, tail", [(1, 2, 2, 1, False), (3, 32, 2, 1, True), (2, 24, 3, 1, True), (3, 16, 4, 2, True), (2, 40, 1, 2, False),
                                                 (1, 16, 8, 1, True), (90, 8, 2, 2, False), (1, 256, 2, 1, True), (1, 1500, 2, 2, False)])
def test_cluster_search_matches_the_oracle(oracle, rows, T, K, V, tail):
    import quantizer_trellis as Q

    rng = np.random.default_rng(rows + T + K)
    table = rng.standard_normal((1 << 16, V)).astype(np.float32)
    x = rng.standard_normal((rows, T)).astype(np.float32)
    values, path = oracle.trellis_quantize(x, table, K, tail)
    out, states = torch.empty(rows, T, device="cuda"), torch.empty(rows, T // V, dtype=torch.int64, device="cuda")
    Q._trellis_quantize_triton(cuda(x), cuda(table), K, tail, out=out, scale=torch.ones(rows, device="cuda"), states=states)
    assert torch.equal(states.cpu(), torch.from_numpy(path)) and torch.equal(out.cpu(), torch.from_numpy(values))


# k and n around the 64-wide chunks and the 128- and 256-wide tiles; k = 512 and n = 2048 end the range in which the split kernel
# finds the channels' ranges itself; x that starts off a 16-byte boundary
@pytest.mark.parametrize("k, n, offset", [(1, 4, 0), (63, 132, 0), (65, 252, 1), (512, 2048, 0), (513, 2048, 0), (512, 2052, 0), (300, 1004, 1), (2000, 4100, 0)])
def test_gram_at_edges(k, n, offset):
    import kron_factors as K

    gen = torch.Generator(device="cuda").manual_seed(k + n)
    x = torch.randn(offset + k * n, generator=gen, device="cuda")[offset:].view(k, n)
    x *= torch.exp(2 * torch.randn(n, generator=gen, device="cuda"))
    x[:, n // 2] = 0
    h0 = torch.randn(n, n, generator=gen, device="cuda")
    h0 = h0 + h0.T
    h = K.accumulate_gram(h0.clone(), x, alpha=0.5)
    wide = x.double()
    want = h0.double() + 0.5 * wide.T @ wide
    # k products of 16-bit pairs (2 u each, and 2^-40 of the channels' largest products), added in float
    magnitude = 0.5 * wide.abs().T @ wide.abs() + h0.double().abs()
    largest = wide.abs().amax(0)
    bound = (k + 6) * 2.0 ** -24 * magnitude + k * 2.0 ** -38 * largest[:, None] * largest[None, :]
    assert ((h.double() - want).abs() <= bound).all() and torch.equal(h, h.T)


# two CTAs per 256 x 256 tile: a second tile row of four channels or none, fewer chunks than stages and more, one tile per cluster and several,
# and one CTA per 128 x 256 tile beside them (n = 2944)
@pytest.mark.parametrize("k, n", [(64, 2180), (130, 2052), (600, 2816), (1030, 3072), (700, 2944), (449, 5000)])
def test_gram_of_two_ctas_per_tile(k, n):
    test_gram_at_edges(k, n, 0)


# block rows of 64, groups of four and pairs of groups: one group, one pair, a pair cut short on either side, a last block row
# that is nearly empty, and pairs whose sizes start in different halves of a pair
@pytest.mark.parametrize("n, other", [(257, 64), (320, 1025), (513, 258), (769, 2049), (1025, 513), (1281, 1283), (3001, 700)])
def test_float_factors_at_group_edges(n, other):
    import kron_factors as K

    def gram(size):
        gen = torch.Generator(device="cuda").manual_seed(size)
        x = torch.randn(2 * size, size, generator=gen, device="cuda", dtype=torch.float64)
        x *= torch.exp(0.5 * torch.randn(size, generator=gen, device="cuda", dtype=torch.float64))
        h = x.T @ x / (2 * size)
        h.diagonal().add_(0.01 * h.diagonal().mean())
        return h

    g, h = gram(n), gram(other)
    l, u = K.feedback_factors_from_grams(g.float(), h.float())
    for got, m in ((l, g), (u.T, h)):
        exact = K.ldl_of_inverse(m)
        # the factor of a float Gram: its condition number (below 1e3 with this damping) times u
        assert (got.double() - exact).abs().max().item() < 2e-5 * max(1.0, exact.abs().max().item())
        assert torch.equal(got, K.ldl_of_inverse(m.float()))  # two problems in one pass equal two passes


# block rows brought up to date beside the factorization of their diagonal block: groups with one to four block rows, ragged last ones, two
# problems whose groups end at different block rows
@pytest.mark.parametrize("n, other", [(64, 65), (127, 256), (255, 449), (448, 2047), (511, 512)])
def test_float_factors_of_short_groups(n, other):
    test_float_factors_at_group_edges(n, other)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n, k", [(1, 0), (64, 5), (64, 16), (64, 60), (130, 122), (400, 85), (1000, 3)])
def test_the_failing_pivot_is_named(n, k, dtype):
    """Pivots are eliminated from the last to the first, 16 rows of a block of 64 at a time."""
    import kron_factors as K

    x = torch.randn(2 * n, n, generator=torch.Generator(device="cuda").manual_seed(n), device="cuda", dtype=dtype)
    h = x.T @ x / (2 * n) + torch.eye(n, device="cuda", dtype=dtype)
    h[k, k] = -1
    with pytest.raises(torch.linalg.LinAlgError, match=rf"pivot {k + 1} "):
        K.ldl_of_inverse(h)


@pytest.mark.parametrize("before", [0, 127, 128, 200])
def test_flags_of_a_long_unchecked_run(before):
    """A matrix that is not positive definite is reported by one of the next 256 calls; the calls around it stay settled or pending."""
    import kron_factors as K

    K.check_pending()
    good = 2 * torch.eye(64, device="cuda")
    bad = good.clone()
    bad[5, 5] = -1
    for _ in range(before):
        K.feedback_factors_from_grams(good, good)
    K.feedback_factors_from_grams(good, bad)
    with pytest.raises(torch.linalg.LinAlgError, match="H is not positive definite"):
        for _ in range(256):
            K.feedback_factors_from_grams(good, good)
    K.check_pending()


@pytest.mark.parametrize("bits", range(1, 9))
def test_pack_out_of_the_fast_range(oracle, bits):
    """Scales and quotients beyond the reciprocal form's range, a field far from zero, a ragged last group, ties to even."""
    import packed_codes as P

    rng = np.random.default_rng(bits)
    m, n = 6, 1029
    top = 2 ** bits - 1
    for qmin in (0, -3, -(1 << 22)):
        scale = np.ones((m, n), dtype=np.float32)
        zero = np.zeros((m, n), dtype=np.float32)
        z = (rng.integers(2 * qmin - 4, 2 * (qmin + top) + 4, (m, n)) / 2).astype(np.float32)  # halves: ties
        scale[1], z[1] = 1e-35, np.where(z[1] < qmin + top / 2, -1e-20, 1e-20)
        scale[2], z[2] = 1e32, 1e30
        z[3, ::7] = np.where(np.arange(n)[::7] % 2, 3e38, -3e38)
        zero[4] = rng.integers(-4, 4, n)
        packed = P.pack_codes(cuda(z), cuda(scale), cuda(zero), qmin=qmin, bits=bits)
        assert np.array_equal(packed.cpu().numpy(), oracle.pack_codes(z, scale, zero, qmin, bits))
        back = P.unpack_codes(packed, cuda(scale), cuda(zero), qmin=qmin, bits=bits, n=n)
        assert np.array_equal(back.cpu().numpy(), oracle.unpack_codes(packed.cpu().numpy(), scale, zero, qmin, bits, n))


# both sides of each line at which a search over 2^16 states changes kernels: 148 sequences, 296, 592, and those between where the
# cluster search stops being the faster one; and choices that may only be stored byte by byte
@pytest.mark.parametrize("rows, K, V, offset", [(148, 8, 1, 0), (149, 8, 1, 0), (231, 8, 1, 0), (232, 8, 1, 0), (297, 4, 2, 0), (298, 4, 2, 0), (495, 2, 2, 0),
                                                (496, 2, 2, 0), (593, 2, 2, 0), (5, 2, 2, 1)])
def test_searches_on_both_sides_of_the_dispatch(oracle, rows, K, V, offset):
    import _abi

    T = 8 * V
    rng = np.random.default_rng(rows + K)
    table = rng.standard_normal((1 << 16, V)).astype(np.float32)
    x = rng.standard_normal((rows, T)).astype(np.float32)
    values, path = oracle.trellis_quantize(x, table, K, True)
    out, states = torch.empty(rows, T, device="cuda"), torch.empty(rows, T // V, dtype=torch.int64, device="cuda")
    size = ctypes.c_size_t()
    _abi.check(_abi.library().g2d_trellis_workspace_bytes(_abi.F32, rows, T, 16, K, V, ctypes.byref(size)), "g2d_trellis_workspace_bytes")
    workspace, xs, ts = torch.empty(size.value + 16, dtype=torch.uint8, device="cuda"), cuda(x), cuda(table)
    _abi.check(_abi.library().g2d_trellis_quantize(_abi.F32, rows, T, xs.data_ptr(), ts.data_ptr(), 16, K, V, 1, None, out.data_ptr(), states.data_ptr(),
                                                   workspace.data_ptr() + offset, size.value, _abi.stream_of(xs)), "g2d_trellis_quantize")
    assert torch.equal(states.cpu(), torch.from_numpy(path)) and torch.equal(out.cpu(), torch.from_numpy(values))


# sums per stage on both sides of the shared-memory room (2048) and of the work (600 products per thread) up to which a super-entry
# fetches its feedback itself; a single block (0); leading modes with short blocks
@pytest.mark.parametrize("m, n, p, q, inner, outer", [(40, 96, 1, 16, 128, 0), (40, 96, 1, 16, 129, 0), (96, 96, 16, 16, 8, 64), (96, 96, 16, 16, 9, 64), (96, 96, 32, 32, 2, 0),
                                                      (128, 128, 64, 64, 8, 64), (12, 1024, 1, 128, 9, 64), (12, 1024, 1, 128, 10, 64), (60, 120, 2, 4, 0, 0)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_blocks_on_both_sides_of_the_pull(m, n, p, q, inner, outer, dtype):
    """The two ways to bring feedback to a stage add the same sums in the same order: the fused sweep equals the engine that calls the
    quantizer once per stage, bit for bit."""
    import gptq_2d as G
    import quantizer_int as Q

    gen = torch.Generator(device="cuda").manual_seed(m + n + inner)
    rand = lambda *shape: torch.randn(*shape, generator=gen, device="cuda", dtype=dtype)
    w, l, u = 0.02 * rand(m, n), torch.tril(rand(m, m) * (0.3 / m ** .5), -1), torch.triu(rand(n, n) * (0.3 / n ** .5), 1)
    quantizer = functools.partial(Q.int_abs_max_quantizer_cuda, qmin=-8, qmax=7, dtype=torch.float16)
    options = dict(super_entry_shape=(p, q), inner_block_size=inner, outer_block_size=outer)
    fused = G.gptq_2d_super_entry(w, l, u, quantizer=quantizer, **options)
    generic = G.gptq_2d_super_entry(w, l, u, quantizer=lambda *a, **k: quantizer(*a, **k), **options)
    assert torch.equal(fused, generic)


@pytest.mark.parametrize("inner", [1, 2, 3, 0])
def test_leading_modes_on_both_sides_of_the_pull(inner):
    import kron_factors as K

    gen = torch.Generator(device="cuda").manual_seed(inner)
    x = 3 * torch.randn(3, 12, 16, generator=gen, device="cuda", dtype=torch.float64)
    factors = []
    for k, block in zip(x.shape, (1, 2, 2)):  # identity diagonal blocks, which the two routes share
        index = torch.arange(k, device="cuda") // block
        f = 0.2 * torch.randn(k, k, generator=gen, device="cuda", dtype=torch.float64)
        factors.append(f.masked_fill(index[:, None] <= index[None, :], 0) + torch.eye(k, device="cuda", dtype=torch.float64))
    want = K.gptq_d_sided(x, factors, super_entry_shape=(2, 2), dense_row_factor=True)
    assert torch.equal(K.gptq_d_sided(x, factors, super_entry_shape=(2, 2), inner_block_size=inner, outer_block_size=0), want)


# the longest sequences whose choices stay in the 200 KB of shared memory, and the next: 2 bits per step as 1024 bytes of choices per
# step beside 32 KB of minima, 4 bits as 512 beside 8 KB
@pytest.mark.parametrize("T, K, V", [(167, 2, 1), (168, 2, 1), (752, 2, 2), (754, 2, 2)])
@pytest.mark.parametrize("tail", [False, True])
def test_cluster_search_where_the_choices_leave_shared_memory(oracle, T, K, V, tail):
    import quantizer_trellis as Q

    shift, steps = K * V, T // V
    minima, unit = (1 << 16 >> shift) // 4, 2 if K * V == 2 else 1
    need = lambda n: 4 * (2 * minima + n * V + n) + (n - 1) * 512 * unit
    assert (need(steps) <= 200 * 1024) == (T in (167, 752))
    rng = np.random.default_rng(T)
    table = rng.standard_normal((1 << 16, V)).astype(np.float32)
    x = rng.standard_normal((1, T)).astype(np.float32)
    values, path = oracle.trellis_quantize(x, table, K, tail)
    out, states = torch.empty(1, T, device="cuda"), torch.empty(1, steps, dtype=torch.int64, device="cuda")
    Q._trellis_quantize_triton(cuda(x), cuda(table), K, tail, out=out, scale=torch.ones(1, device="cuda"), states=states)
    assert torch.equal(states.cpu(), torch.from_numpy(path)) and torch.equal(out.cpu(), torch.from_numpy(values))

"""Quantizer parameters of the tile sweep: the layouts that are loaded in different ways, and the stages that they choose between."""
import functools

import pytest
import torch

pytestmark = pytest.mark.gpu

# one tile, ragged tiles with rows of vectors and without, several tiles (rows of vectors at the edge, padded copies)
SIZES = [(64, 64), (61, 68), (130, 190), (77, 333), (1, 5), (200, 1)]


def layouts(full):
    """Views of the same m x n values; the last two have a column stride other than 1 and rows that are not aligned to vectors."""
    m, n = full.shape
    apart = torch.full((m, n + 3), float("nan"), device="cuda", dtype=full.dtype)
    apart[:, 1:n + 1] = full
    return {"whole": full.contiguous(), "columns first": full.T.contiguous().T, "rows apart": apart[:, 1:n + 1]}


def quantize(w, l, u, scale, zero):
    import gptq_2d as G
    import quantizer_int as Q

    return G.gptq_2d(w, l, u, quantizer=functools.partial(Q.affine_quantizer_cuda, qmin=-8, qmax=7), quantizer_inputs=(scale, zero))


@pytest.mark.parametrize("m, n", SIZES)
@pytest.mark.parametrize("batch", [0, 2])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_layouts_of_scales_and_zero_points(m, n, batch, dtype):
    """Broadcast, whole and strided parameters of the same values: the same bits."""
    gen = torch.Generator(device="cuda").manual_seed(3 * m + n)
    rand = lambda *shape: torch.randn(*shape, generator=gen, device="cuda", dtype=dtype)
    lead = (batch,) if batch else ()
    w, l, u = rand(*lead, m, n), torch.tril(rand(m, m) * 0.1, -1), torch.triu(rand(*lead, n, n) * 0.1, 1)
    for shape in ((1, 1), (m, 1), (1, n), (m, n)):
        scale = 0.1 + 0.05 * rand(*shape).abs()
        zero = torch.randint(-1, 2, shape, generator=gen, device="cuda").to(dtype)
        want = None
        for name, s in {"broadcast": scale.expand(m, n), **layouts(scale.expand(m, n))}.items():
            for other, z in {"broadcast": zero.expand(m, n), **layouts(zero.expand(m, n))}.items():
                got = quantize(w, l, u, s.expand(w.shape), z.expand(w.shape))
                want = got if want is None else want
                assert torch.equal(got, want), (shape, name, other)
    assert not want.isnan().any()


@pytest.mark.parametrize("m, n", SIZES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_stages_chosen_by_sub_tile(m, n, dtype):
    """Sub-tiles of 16 x 16 with zero points of +0, of -0 and others, and with scales too small for a reciprocal, side by side.  No factor, so
    the input is rounded as it is; quotients are sixteenths, exact in any form of the division."""
    gen = torch.Generator(device="cuda").manual_seed(m * n)
    kind = torch.randint(0, 4, ((m + 15) // 16, (n + 15) // 16), generator=gen, device="cuda").repeat_interleave(16, 0).repeat_interleave(16, 1)[:m, :n]
    scale = torch.where(kind == 3, torch.full((), 2.0 ** -100, device="cuda", dtype=dtype), torch.full((), 0.125, device="cuda", dtype=dtype))
    if dtype == torch.float64:
        scale = torch.where(kind == 3, torch.full((), 2.0 ** -600, device="cuda", dtype=dtype), scale)
    zero = torch.where(kind == 1, torch.full((), -0.0, device="cuda", dtype=dtype), torch.zeros((), device="cuda", dtype=dtype))
    zero = torch.where(kind == 2, torch.randint(0, 3, (m, n), generator=gen, device="cuda").to(dtype), zero)
    y = torch.randint(-200, 201, (m, n), generator=gen, device="cuda").to(dtype) / 16 * scale
    eye = lambda k: torch.eye(k, device="cuda", dtype=dtype)
    got = quantize(y, eye(m), eye(n), scale, zero)
    want = (torch.clamp(torch.round(y / scale + zero), -8, 7) - zero) * scale
    assert torch.equal(got, want) and torch.equal(torch.signbit(got), torch.signbit(want))


@pytest.mark.parametrize("m, n", [(64, 64), (130, 190), (77, 333), (520, 901)])
@pytest.mark.parametrize("offset", [0, 2 ** 18])
def test_feedback_of_the_values_that_are_stored(m, n, offset):
    """Scales in full precision, sub-tiles with zero points and without, factors that couple all entries: an ordinary sweep (short stages) commits
    what a sweep that records its values before rounding does (long stages), those follow from the recorded values, and Z - X = L E U with
    the errors of the stored floats.  Large zero points make half an ulp of Z a sixty-fourth of a code."""
    import _abi
    import gptq_2d as G

    gen = torch.Generator(device="cuda").manual_seed(m + n)
    rand = lambda *shape: torch.randn(*shape, generator=gen, device="cuda")
    l, u = torch.tril(rand(m, m) * 0.3 / m ** 0.5, -1), torch.triu(rand(n, n) * 0.3 / n ** 0.5, 1)
    scale = 0.1 + 0.05 * torch.rand(m, n, generator=gen, device="cuda")
    some = torch.randint(0, 2, ((m + 15) // 16, (n + 15) // 16), generator=gen, device="cuda").repeat_interleave(16, 0).repeat_interleave(16, 1)[:m, :n]
    zero = some * (offset + torch.randint(1, 8, (m, n), generator=gen, device="cuda")).float()
    w = (4 * rand(m, n) - zero) * scale
    ordinary = quantize(w, l, u, scale, zero)
    y, _, _, batch_shape = G._prepare_output(w, l, u, False)
    pre = torch.empty_like(y)
    G._sweep_fused(y, l, u, batch_shape, dict(kind=_abi.Q_AFFINE, qmin=-8, qmax=7), (scale, zero), y_pre=pre)
    assert torch.equal(ordinary, y)
    assert torch.equal(y, (torch.clamp(torch.round(pre / scale + zero), -8, 7) - zero) * scale)
    wide = torch.float64
    e, lower, upper = y.to(wide) - pre.to(wide), l.to(wide) + torch.eye(m, device="cuda", dtype=wide), u.to(wide) + torch.eye(n, device="cuda", dtype=wide)
    # m + n products and additions per entry, each rounded at the size of the sums that it joins
    magnitude = lower.abs() @ e.abs() @ upper.abs() + w.abs()
    assert ((y.to(wide) - w.to(wide) - lower @ e @ upper).abs() <= (m + n) * 2.0 ** -24 * magnitude).all()


@pytest.mark.parametrize("raised", [0.0, 3.0, 40.0])
def test_last_sub_tile_sets_the_scale(raised, monkeypatch):
    """Operand planes are made before the last sub-tile of a tile is swept, under the scale of the others: where that sub-tile has the largest
    errors and sums they are made again.  Later tiles then see the feedback that the schedule without planes gives them."""
    import _abi
    import gptq_2d as G

    gen = torch.Generator(device="cuda").manual_seed(5)
    rand = lambda *shape: torch.randn(*shape, generator=gen, device="cuda")
    m = n = 320
    w, l, u = 3 * rand(m, n), torch.tril(rand(m, m) * 0.02, -1), torch.triu(rand(n, n) * 0.02, 1)
    last = (torch.arange(m, device="cuda") % 64 >= 48)[:, None] & (torch.arange(n, device="cuda") % 64 >= 48)[None, :]
    decisions = torch.round(w) + raised * last  # errors of about a half elsewhere; below 2^8 apart, so no tile is a wide one
    y, _, _, batch_shape = G._prepare_output(w, l, u, False)
    pre = {}
    for schedule in (0, 1):
        monkeypatch.setattr(G, "SWEEP_SCHEDULE", schedule)
        pre[schedule] = torch.empty_like(w)
        G._sweep_fused(w.clone(), l, u, batch_shape, dict(kind=_abi.Q_FORCED), (), forced_z=decisions, y_pre=pre[schedule])
    # the two sum at most m + n products per entry in orders of their own, each product off by 2 u beside the sums' own u
    e = (decisions - pre[1]).abs()
    magnitude = (l.abs() + torch.eye(m, device="cuda")) @ e @ (u.abs() + torch.eye(n, device="cuda")) + w.abs()
    assert ((pre[0] - pre[1]).abs() <= 2 * (m + n) * 2.0 ** -24 * magnitude).all()

"""Float sweeps whose rows or columns are of very different size, or not all finite: the 16-bit operand planes of the tensor-core
updates share a scale per 64 x 64 tile, and what a scale cannot serve is formed in float32."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _problem(m, n, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda *shape: torch.randn(*shape, generator=gen, device="cuda")
    return 0.02 * rand(m, n), torch.tril(rand(m, m) * (0.3 / m ** .5), -1), torch.triu(rand(n, n) * (0.3 / n ** .5), 1)


def _sweep(w, l, u, step):
    """Rounded values and the values before rounding, 4 bits with the given steps."""
    import _abi
    import gptq_2d as G

    y, _, _, batch_shape = G._prepare_output(w, l, u, False)
    y_pre = torch.empty_like(y)
    G._sweep_fused(y, l, u, batch_shape, dict(kind=_abi.Q_AFFINE, qmin=-8, qmax=7), (step.expand(w.shape), torch.zeros(1, 1, device="cuda").expand(w.shape)), y_pre=y_pre)
    return y, y_pre


def _check_identity(w, l, u, z, y_pre):
    """Z - X = (L + I) E (U + I) with E = Z - Y_pre, entry by entry; the bound of test_sweep_identity."""
    (m, n), wide = w.shape, torch.float64
    e, full_l, full_u = (z.to(wide) - y_pre.to(wide)), l.to(wide) + torch.eye(m, device="cuda", dtype=wide), u.to(wide) + torch.eye(n, device="cuda", dtype=wide)
    residual = (z.to(wide) - w.to(wide)) - full_l @ e @ full_u
    magnitude = full_l.abs() @ e.abs() @ full_u.abs() + z.to(wide).abs() + w.to(wide).abs()
    terms = 2 * (64 + 2 + (m + n) / 64)
    assert ((residual.abs() - terms * 2.0 ** -24 * magnitude).max() <= 0).item(), (residual.abs() / (2.0 ** -24 * magnitude)).max().item()


# the units of every second row or column, or of one row in sixty; no updates but near ones (300), far ones with one macro tile per CTA
# (1030) and with 2 x 2 (3900 x 4100); ratios on both sides of 2^8 where a tile counts as wide
@pytest.mark.parametrize("m, n", [(300, 450), (1030, 901), (3900, 4100)])
@pytest.mark.parametrize("power", [7, 8, 9, 12, 20, 40])
@pytest.mark.parametrize("what", ["rows", "columns", "one row"])
def test_units_of_their_own(m, n, power, what):
    """The defining identity in the units of each row and column, with the bound of an even matrix."""
    if m > 3000 and power not in (8, 20):
        pytest.skip("the large size with two ratios")
    w, l, u = _problem(m, n, m + power)
    small = 2.0 ** -power
    rows, columns = torch.ones(m, 1, device="cuda"), torch.ones(1, n, device="cuda")
    if what == "rows":
        rows[1::2] = small
    elif what == "columns":
        columns[:, 1::2] = small
    else:
        rows[7::60] = small
    step = (w.abs().amax(1, keepdim=True) / 7.5) * rows * columns
    w, l, u = w * rows * columns, l * rows / rows.T, u / columns.T * columns
    z, y_pre = _sweep(w, l, u, step)
    _check_identity(w, l, u, z, y_pre)
    again, _ = _sweep(w, l, u, step)
    assert torch.equal(again, z)


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf"), 1e30])
@pytest.mark.parametrize("m, n, r, c", [(300, 450, 70, 130), (1030, 901, 200, 3), (3900, 4100, 1000, 900)])
def test_values_that_are_not_finite_stay_below_and_to_the_right(m, n, r, c, bad):
    """An entry feeds the entries below and to the right of it alone: the others stay as accurate as without it."""
    if m > 3000 and bad != float("inf"):
        pytest.skip("the large size with one value")
    w, l, u = _problem(m, n, m)
    w *= 2.0 ** -14
    step = w.abs().amax(1, keepdim=True) / 7.5
    w[r, c] = bad
    z, y_pre = _sweep(w, l, u, step)
    _check_identity(w[:r], l[:r, :r], u, z[:r], y_pre[:r])
    _check_identity(w[:, :c], l, u[:c, :c], z[:, :c], y_pre[:, :c])


@pytest.mark.parametrize("m, n", [(777, 1333), (1001, 1503)])
def test_error_beside_the_float32_schedule(m, n):
    """Root mean square error of the values before rounding, from float64: the updates on the tensor cores add at most one per cent to
    that of the tile schedule, whose products are float32 throughout (a hundred thousand entries: the figure itself is good to 0.3 %)."""
    import gptq_2d as G

    w, l, u = _problem(m, n, m)
    step = w.abs().amax(1, keepdim=True) / 7.5
    z = torch.round(w / step) * step
    wide = torch.float64
    lower, upper = l.to(wide) + torch.eye(m, device="cuda", dtype=wide), u.to(wide) + torch.eye(n, device="cuda", dtype=wide)
    e = torch.linalg.solve_triangular(lower, z.to(wide) - w.to(wide), upper=False, unitriangular=True)
    want = z.to(wide) - torch.linalg.solve_triangular(upper, e, upper=True, left=False, unitriangular=True)
    errors = []
    for schedule in (0, 1):
        G.SWEEP_SCHEDULE = schedule
        try:
            errors.append((G.gptq_2d_forced(w, l, u, z)[1].to(wide) - want).norm().item())
        finally:
            G.SWEEP_SCHEDULE = 0
    assert errors[0] <= 1.01 * errors[1], errors[0] / errors[1]


# near updates inside the tile launches and in launches of their own: a target gets the same additions in the same order.  One tile across,
# ragged last tiles, far updates of rank 512 and 1024 beside; every product wide, some of them, none; every quantizer
@pytest.mark.parametrize("m, n, outer", [(64, 650, 0), (300, 450, 0), (777, 1333, 0), (1030, 901, 16), (2050, 1153, 0)])
@pytest.mark.parametrize("what", ["rows", "columns", "one row", "not finite", "affine", "round", "forced"])
def test_both_places_of_the_near_updates(m, n, outer, what):
    import _abi
    import gptq_2d as G

    w, l, u = _problem(m, n, m + outer)
    rows, columns = torch.ones(m, 1, device="cuda"), torch.ones(1, n, device="cuda")
    if what in ("rows", "columns"):
        (rows if what == "rows" else columns.T)[1::2] = 2.0 ** -20
    elif what == "one row":
        rows[7::60] = 2.0 ** -20
    step = (w.abs().amax(1, keepdim=True) / 7.5) * rows * columns
    w, l, u = w * rows * columns, l * rows / rows.T, u / columns.T * columns
    if what == "not finite":
        w[m // 3, n // 4] = float("inf")
    kind, inputs, forced = _abi.Q_AFFINE, (step.expand(w.shape), torch.zeros(1, 1, device="cuda").expand(w.shape)), None
    if what == "round":
        kind, inputs, w = _abi.Q_ROUND, (), 150 * w
    elif what == "forced":
        kind, inputs, forced = _abi.Q_FORCED, (), torch.round(w / step) * step
    results = []
    for schedule in (0, 4):
        y, _, _, batch_shape = G._prepare_output(w, l, u, False)
        y_pre = torch.empty_like(y)
        G.SWEEP_SCHEDULE = schedule
        try:
            G._sweep_fused(y, l, u, batch_shape, dict(kind=kind, qmin=-8, qmax=7), inputs, forced_z=forced, y_pre=y_pre, outer_tiles=outer)
        finally:
            G.SWEEP_SCHEDULE = 0
        results.append((y, y_pre))
    for inside, apart in zip(*results):
        assert ((inside == apart) | (inside.isnan() & apart.isnan())).all()
    if what != "not finite":
        _check_identity(w, l, u, *results[1])


def test_near_updates_of_their_own_in_a_graph():
    import functools

    import gptq_2d as G
    import quantizer_int as Q

    w, l, u = _problem(456, 328, 5)
    w[1::2] *= 2.0 ** -20
    l[1::2] *= 2.0 ** -20
    l[:, 1::2] *= 2.0 ** 20
    scale = (w.abs().amax(1, keepdim=True) / 7.5).expand(w.shape).contiguous()
    options = dict(quantizer=functools.partial(Q.affine_quantizer_cuda, qmin=-8, qmax=7), quantizer_inputs=(scale, torch.zeros_like(scale)))
    want = [G.gptq_2d(x, l, u, **options) for x in (w, 1.01 * w)]
    G.SWEEP_SCHEDULE = 4
    try:
        replay = G.capture_gptq_2d(w, l, u, **options)
        for x, z in ((w, want[0]), (1.01 * w, want[1]), (w, want[0])):
            assert torch.equal(replay(x, l, u, *options["quantizer_inputs"]), z)
    finally:
        G.SWEEP_SCHEDULE = 0

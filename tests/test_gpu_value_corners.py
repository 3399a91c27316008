"""Values at the edges of what the kernels' short forms of the quantizer serve: signs of zero, infinities, NaN."""
import functools

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value, scale", [(float("inf"), 0.1), (-float("inf"), 0.1), (1e300, 1e-100), (-1e300, 1e-100), (1.7e308, 0.5), (float("nan"), 0.1), (1e300, 0.1)])
def test_double_quotients_beyond_the_range(value, scale):
    """The fused float64 sweep against the engine whose quantizer divides: an infinite quotient is clamped, NaN stays NaN."""
    import gptq_2d as G
    import quantizer_int as Q

    gen = torch.Generator(device="cuda").manual_seed(3)
    rand = lambda *shape: torch.randn(*shape, generator=gen, device="cuda", dtype=torch.float64)
    m, n = 20, 70
    w, l, u = rand(m, n), torch.tril(rand(m, m) * 0.1, -1), torch.triu(rand(n, n) * 0.1, 1)
    w[4, 9] = value
    inputs = (torch.full((m, n), scale, device="cuda", dtype=torch.float64), torch.zeros(m, n, device="cuda", dtype=torch.float64))
    quantizer = functools.partial(Q.affine_quantizer_cuda, qmin=-8, qmax=7)
    fused = G.gptq_2d(w, l, u, quantizer=quantizer, quantizer_inputs=inputs)
    generic = G.gptq_2d(w, l, u, quantizer=lambda *a, **k: quantizer(*a, **k), quantizer_inputs=inputs)
    assert torch.equal(fused[4, 9].isnan(), generic[4, 9].isnan())
    if not generic[4, 9].isnan():
        assert fused[4, 9] == generic[4, 9]
    fed = torch.zeros(m, n, dtype=torch.bool, device="cuda")
    fed[4:, 9:] = True
    assert torch.equal(fused[~fed], generic[~fed])


@pytest.mark.parametrize("m, n", [(16, 16), (40, 50), (130, 190)])
@pytest.mark.parametrize("kind", ["forced", "divided"])
def test_infinite_feedback_from_above(m, n, kind, oracle):
    """Below an infinite value the completed C, (Z - Y) + C, is NaN, and so is what the entries to the right receive, as in the oracle: with values
    committed as they are, and under scales that take the exact division (a clamped infinity is finite)."""
    import _abi
    import gptq_2d as G

    rng = np.random.default_rng(m)
    w, l, u = (rng.standard_normal(s).astype(np.float32) for s in ((m, n), (m, m), (n, n)))
    l, u = np.tril(0.1 * l, -1), np.triu(0.1 * u, 1)
    z, small = np.rint(w), np.float32(2.0 ** -70)
    w[4, 9] = np.inf
    cuda = lambda a: torch.from_numpy(a).cuda()
    if kind == "forced":
        want = oracle.sweep(w, l, u, kind=oracle.Q_FORCED, forced_z=z, return_y_pre=True)[1]
        got = G.gptq_2d_forced(cuda(w), cuda(l), cuda(u), cuda(z))[1]
    else:
        scale, zero = np.full((m, n), small), np.zeros((m, n), np.float32)
        want = oracle.sweep(w * small, l, u, kind=oracle.Q_AFFINE, scale=scale, zero_point=zero, qmin=-8, qmax=7, return_y_pre=True)[1]
        y, _, _, batch_shape = G._prepare_output(cuda(w * small), cuda(l), cuda(u), False)
        got = torch.empty_like(y)
        G._sweep_fused(y, cuda(l), cuda(u), batch_shape, dict(kind=_abi.Q_AFFINE, qmin=-8, qmax=7), (cuda(scale), cuda(zero)), y_pre=got)
    assert np.isnan(want[5:, 10:]).all() and got[5:, 10:].isnan().all()


@pytest.mark.parametrize("qmin, qmax, zero", [(-8, 7, 0.0), (0, 15, 0.0), (-15, 0, 0.0), (0, 15, 8.0), (-8, 7, -0.0), (-8, 7, 3.0)])
@pytest.mark.parametrize("m, n", [(64, 64), (100, 71), (200, 333)])
@pytest.mark.parametrize("scale_sign", [1, -1])
def test_signs_of_zeros(qmin, qmax, zero, m, n, scale_sign):
    """Rounded values bit for bit as (clamp(round(y / scale + zero)) - zero) * scale gives them, zeros included.  No factor, so y is the
    input; the quotients are sixteenths of powers of two, exact in any form of the division."""
    import gptq_2d as G
    import quantizer_int as Q

    gen = torch.Generator(device="cuda").manual_seed(m + n)
    scale = torch.full((m, n), 0.125 * scale_sign, device="cuda")
    y = torch.randint(-200, 201, (m, n), generator=gen, device="cuda") / 16 * scale
    zeros = torch.full((m, n), zero, device="cuda")
    z = G.gptq_2d(y, torch.eye(m, device="cuda"), torch.eye(n, device="cuda"), quantizer=functools.partial(Q.affine_quantizer_cuda, qmin=qmin, qmax=qmax),
                  quantizer_inputs=(scale, zeros))
    want = (torch.clamp(torch.round(y / scale + zeros), qmin, qmax) - zeros) * scale
    assert torch.equal(z, want)
    assert torch.equal(torch.signbit(z), torch.signbit(want))


@pytest.mark.parametrize("m, n, q", [(64, 1024, 16), (96, 512, 32)])
def test_infinite_coupling_of_groups(m, n, q, oracle):
    """An infinite entry of U makes its receivers infinite and their groups' scales with them, so whole groups are NaN from there on, as in the oracle: a
    flush forms no zero times infinity for sources outside a row's stages, which would leave NaN that a group's largest value passes over."""
    import gptq_2d as G
    import quantizer_int as Q

    rng = np.random.default_rng(n)
    w, l, u = (0.02 * rng.standard_normal(s).astype(np.float32) for s in ((m, n), (m, m), (n, n)))
    block = np.arange(n) // q
    l, u = np.tril(l, -1) + np.eye(m, dtype=np.float32), np.where(block[:, None] < block[None, :], u, np.float32(0)) + np.eye(n, dtype=np.float32)
    u[n // 4, n // 2 + 3] = np.inf
    want = oracle.sweep(w, l, u, kind=oracle.Q_ABSMAX, super_entry_shape=(1, q), qmin=-8, qmax=7, half=oracle.FP16)
    cuda = lambda a: torch.from_numpy(a).cuda()
    quantizer = functools.partial(Q.int_abs_max_quantizer_cuda, qmin=-8, qmax=7, dtype=torch.float16)
    got = G.gptq_2d_super_entry(cuda(w), cuda(l), cuda(u), quantizer=quantizer, super_entry_shape=(1, q)).cpu().numpy()
    assert np.isnan(want[:, n // 2:]).all() and np.array_equal(np.isnan(got), np.isnan(want))


@pytest.mark.parametrize("n", [8, 9, 32])
def test_packing_under_a_zero_point_that_is_nan(n):
    """Converts to 0 before it is clamped, in whole groups of eight as in ragged ones."""
    import packed_codes as P

    z, scale, zero = torch.zeros(2, n, device="cuda"), torch.ones(2, n, device="cuda"), torch.zeros(2, n, device="cuda")
    zero[1, n - 1] = float("nan")
    for zeros, at in ((zero, (1, n - 1)), (torch.full((2, 1), float("nan"), device="cuda"), None)):
        codes = P.pack_codes(z, scale, zeros, qmin=-8, bits=8).cpu().numpy()
        assert np.array_equal(codes, np.full_like(codes, 8))

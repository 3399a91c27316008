"""Waits inside kernels that run out: nothing that they leave passes for a result, the status says so, and the GPU stays usable."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# NG = 8, 4, 2 and 1 groups per thread (2, 3, 4 and more bits per step), minima sent to one CTA and to all four (8 bits), more
# sequences than clusters, choices in shared memory and in the scratch
@pytest.mark.parametrize("rows, T, K, V, tail", [(1, 64, 2, 1, True), (3, 4, 3, 1, False), (2, 64, 4, 1, True), (2, 60, 3, 2, True), (1, 16, 8, 1, True),
                                                 (90, 32, 1, 2, False), (1, 1024, 2, 1, True)])
def test_search_whose_waits_run_out(rows, T, K, V, tail):
    import _abi

    lib = _abi.library()
    gen = torch.Generator(device="cuda").manual_seed(T)
    table, x = torch.randn(1 << 16, V, generator=gen, device="cuda"), torch.randn(rows, T, generator=gen, device="cuda")
    size, code_bytes = ctypes.c_size_t(), ctypes.c_int64()
    _abi.check(lib.g2d_trellis_workspace_bytes(_abi.F32, rows, T, 16, K, V, ctypes.byref(size)), "g2d_trellis_workspace_bytes")
    _abi.check(lib.g2d_trellis_code_bytes(T, 16, K, V, int(tail), ctypes.byref(code_bytes)), "g2d_trellis_code_bytes")
    workspace = torch.empty(size.value, dtype=torch.uint8, device="cuda")

    def search(wait_cycles):
        out, states = torch.zeros(rows, T, device="cuda"), torch.zeros(rows, T // V, dtype=torch.int64, device="cuda")
        codes = torch.full((rows, code_bytes.value), 255, dtype=torch.uint8, device="cuda")
        _abi.check(lib.g2d_trellis_quantize_limited(rows, T, x.data_ptr(), table.data_ptr(), K, V, int(tail), out.data_ptr(), states.data_ptr(), codes.data_ptr(),
                                                    workspace.data_ptr(), size.value, wait_cycles, _abi.stream_of(x)), "g2d_trellis_quantize_limited")
        return out, states, codes

    device = torch.device("cuda", torch.cuda.current_device())
    _abi.check_status(device)
    before = search(2_000_000_000)
    _abi.check_status(device)
    out, states, codes = search(0)
    assert out.isnan().all() and (states == -1).all() and (codes == 0).all()
    with pytest.raises(RuntimeError, match="bounded wait"):
        _abi.check_status(device)
    _abi.check_status(device)  # reported once
    after = search(2_000_000_000)
    assert all(torch.equal(a, b) for a, b in zip(before, after)) and np.isfinite(before[0].cpu().numpy()).all()
    _abi.check_status(device)


# tiles of one CTA and of two; fewer tiles than CTAs and more
@pytest.mark.parametrize("n, k", [(128, 512), (2944, 300), (3072, 300), (4096, 1000)])
def test_gram_whose_waits_run_out(n, k):
    """Loads, products and their commits come to their end before a CTA leaves: the next call, into the same shared and tensor memory, is right."""
    import _abi

    lib = _abi.library()
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(k, n, generator=gen, device="cuda")
    size = ctypes.c_size_t()
    _abi.check(lib.g2d_gram_workspace_bytes(n, k, ctypes.byref(size)), "g2d_gram_workspace_bytes")
    workspace, status = torch.empty(size.value, dtype=torch.uint8, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")

    def accumulate(wait_cycles):
        h = torch.zeros(n, n, device="cuda")
        status.zero_()
        _abi.check(lib.g2d_gram_accumulate_limited(n, k, x.data_ptr(), 1.0, h.data_ptr(), status.data_ptr(), workspace.data_ptr(), size.value, wait_cycles,
                                                   _abi.stream_of(x)), "g2d_gram_accumulate_limited")
        return h

    before = accumulate(2_000_000_000)
    assert status.item() == 0
    accumulate(0)
    after = accumulate(2_000_000_000)  # enqueued behind it at once
    assert status.item() == 0 and torch.equal(before, after)
    accumulate(0)
    assert status.item() == -1
    assert lib.g2d_gram_accumulate_limited(n, k, x.data_ptr(), 1.0, before.data_ptr(), status.data_ptr(), workspace.data_ptr(), size.value, -1, _abi.stream_of(x)) == -1

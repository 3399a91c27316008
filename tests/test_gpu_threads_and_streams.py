"""Calls from several host threads and streams at once: the same results as one after the other."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def in_threads(count, work):
    """work(k) in a thread of its own for every k; the first exception is raised here."""
    failures = []

    def run(k):
        try:
            work(k)
        except BaseException as failure:  # noqa: BLE001 - handed to the caller
            failures.append(failure)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(count)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if failures:
        raise failures[0]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_factors_from_more_threads_than_lanes(dtype):
    """Ten threads with a stream each share the library's four lanes; every Gram arrives on the caller's stream right before its
    call, behind work that takes longer than the enqueueing."""
    import kron_factors as K

    count, rounds, n = 10, 6, 320
    gen = torch.Generator(device="cuda").manual_seed(1)
    x = [torch.randn(2 * n, n, generator=gen, device="cuda", dtype=dtype) for _ in range(count)]
    eye = torch.eye(n, device="cuda", dtype=dtype)
    grams = [a.T @ a / (2 * n) + eye for a in x]
    want = [K.ldl_of_inverse(g) for g in grams]
    torch.cuda.synchronize()
    results = [[] for _ in range(count)]

    def work(k):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            heavy = torch.randn(2048, 2048, device="cuda")
            for _ in range(rounds):
                h = torch.full_like(grams[k], float("nan"))
                heavy = heavy @ heavy / 2048  # a few hundred microseconds ahead of the Gram
                h.copy_(grams[k])
                results[k].append(K.ldl_of_inverse(h, check=False))
        stream.synchronize()

    in_threads(count, work)
    K.check_pending()
    for k in range(count):
        for got in results[k]:
            assert torch.equal(got, want[k])


@pytest.mark.parametrize("single", [True, False])
def test_pending_flags_of_another_stream(single):
    """A matrix that is not positive definite, prepared on a stream that the current one does not wait for."""
    import kron_factors as K

    K.check_pending()
    good = 2 * torch.eye(64, device="cuda")
    bad = good.clone()
    bad[7, 7] = -1
    K.ldl_of_inverse(good)  # the library is loaded and its lanes exist
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        heavy = torch.randn(8192, 8192, device="cuda")
        for _ in range(10):
            heavy = heavy @ heavy / 8192  # some ten milliseconds ahead of the factors
        if single:
            K.ldl_of_inverse(bad, check=False)
        else:
            K.feedback_factors_from_grams(good, bad)
    with pytest.raises(torch.linalg.LinAlgError, match="pivot 8 "):
        K.check_pending()
    K.check_pending()
    torch.cuda.synchronize()


def test_unchecked_calls_do_not_pile_up():
    import kron_factors as K

    K.check_pending()
    good = 2 * torch.eye(8, device="cuda")
    for _ in range(3 * K._PENDING_LIMIT):
        K.ldl_of_inverse(good, check=False)
    assert len(K._PENDING) <= K._PENDING_LIMIT
    K.check_pending()
    assert not K._PENDING

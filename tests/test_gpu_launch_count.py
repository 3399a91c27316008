"""The library's launch counter against the kernels that a captured call holds."""
import functools

import pytest
import torch

pytestmark = pytest.mark.gpu


def library_kernels(graph):
    from cuda.bindings import driver, runtime

    def ok(result):
        assert int(result[0]) == 0, result[0]
        return result[1] if len(result) == 2 else result[1:]

    handle = driver.CUgraph(graph.raw_cuda_graph())
    count = ok(driver.cuGraphGetNodes(handle))[1]
    names = []
    for node in ok(driver.cuGraphGetNodes(handle, count))[0]:
        if ok(driver.cuGraphNodeGetType(node)) == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            params = ok(driver.cuGraphKernelNodeGetParams(node))
            names.append(ok(driver.cuFuncGetName(params.func) if int(params.func) else driver.cuKernelGetName(params.kern)))
    return sum(b"g2d" in name for name in names)  # the namespace, or a file of the library before a namespace without a name


# factors with and without products of two CTAs, of one size and of two; a Gram on tiles of one CTA and of two; sweeps of one tile and of many
@pytest.mark.parametrize("what, m, n", [("factors", 300, 700), ("factors", 300, 4300), ("factors", 4200, 8300), ("gram", 256, 512), ("gram", 300, 3072),
                                        ("sweep", 64, 64), ("sweep", 300, 450)])
def test_every_launch_is_counted_once(what, m, n):
    import _abi
    import gptq_2d as G
    import kron_factors as K
    import quantizer_int as Q

    eye = lambda k: torch.eye(k, device="cuda")
    w, h, x = torch.randn(m, n, device="cuda"), torch.zeros(n, n, device="cuda"), torch.randn(m, n, device="cuda")
    inputs = (torch.full((1, 1), 0.1, device="cuda").expand(m, n), torch.zeros(1, 1, device="cuda").expand(m, n))
    quantizer = functools.partial(Q.affine_quantizer_cuda, qmin=-8, qmax=7)
    call = {"factors": lambda: K.feedback_factors_from_grams(eye(m), eye(n)), "gram": lambda: K.accumulate_gram(h, x),
            "sweep": lambda: G.gptq_2d(w, eye(m), eye(n), quantizer=quantizer, quantizer_inputs=inputs)}[what]
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    before = _abi.library().g2d_launch_count()
    with torch.cuda.graph(graph):
        call()
    counted = _abi.library().g2d_launch_count() - before
    assert counted == library_kernels(graph) > 0

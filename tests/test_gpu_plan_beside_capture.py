"""A plan made while a stream of the caller's records a graph (relaxed mode, a
stream that does not wait for the default one): neither fails the other, and
both give what they give alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_plan_created_during_a_capture(femg, oracle, cuda):
    torch = cuda
    first, second = (femg.Problem(femg.config_c2(m=m, order=2)) for m in (3, 4))
    plan = first.plan()
    plan.bind_terms()
    v = torch.zeros(first.nnz, dtype=torch.complex128, device="cuda")
    r = torch.zeros(int(first.sys.n_rows), dtype=torch.complex128, device="cuda")
    s = torch.cuda.Stream()

    def call():
        femg.check(femg.lib().fg_assemble_fp64_static(plan.ptr, None, v.data_ptr(), r.data_ptr(), s.cuda_stream))

    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s, capture_error_mode="relaxed"):
        call()
        other = second.plan()
        call()
    v.zero_()
    graph.replay()
    torch.cuda.synchronize()
    for prob, values in ((first, v.cpu().numpy()), (second, other.assemble("fp64")[0])):
        want, _ = oracle.assemble(prob.arrays(), *prob.terms())
        assert np.linalg.norm(values - want) <= 1e-12 * np.linalg.norm(want)

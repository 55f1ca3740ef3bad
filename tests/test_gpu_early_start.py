"""Kernels that start beside the one before them (programmatic dependent
launch): calls on plans of different sizes and paths follow each other on one
stream without a wait and give what each gives alone, bit for bit; a stream
capture records plain dependencies and replays to the same values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def problems(F):
    return {"tri_small": F.config(dim=2, m=5, mesh_order=1, gauss=2, dirichlet=1, dirichlet_value=1.5, source=1),
            "tet_p2": F.config_c2(m=4, order=2), "tet_p3": F.config_c3(m=6), "tet_p4": F.config_c2(m=2, order=4),
            "navier": F.config_c5(m=3)}


def test_calls_in_a_row(femg, cuda):
    torch = cuda
    runs = []
    for name, cfg in problems(femg).items():
        prob = femg.Problem(cfg)
        for path in ("fp64", "factored", "mixed"):
            if path == "factored" and name == "navier":
                continue
            plan = prob.plan()
            if path == "factored":
                plan.set_fp64_method(femg.FG_FP64_FACTORED)
            plan.bind_terms()
            v = torch.zeros(prob.nnz, dtype=torch.complex128, device="cuda")
            r = torch.zeros(int(prob.sys.n_rows), dtype=torch.complex128, device="cuda")
            call = lambda plan=plan, path=path, v=v, r=r: plan.assemble(  # noqa: E731
                "mixed" if path == "mixed" else "fp64", values=v.data_ptr(), rhs=r.data_ptr(), bound=True)
            torch.cuda.synchronize()
            call()
            torch.cuda.synchronize()
            runs.append((call, v, r, v.clone(), r.clone()))
    order = np.random.default_rng(1).integers(0, len(runs), 300)
    for _, v, r, _, _ in runs:
        v.fill_(7.0)
        r.fill_(7.0)
    for k in order:
        runs[k][0]()
    for k in range(len(runs)):
        runs[k][0]()
    torch.cuda.synchronize()
    for _, v, r, v0, r0 in runs:
        assert torch.equal(v, v0) and torch.equal(r, r0)


def test_capture(femg, cuda):
    torch = cuda
    prob = femg.Problem(problems(femg)["tet_p2"])
    plan = prob.plan()
    plan.bind_terms()
    v = torch.zeros(prob.nnz, dtype=torch.complex128, device="cuda")
    r = torch.zeros(int(prob.sys.n_rows), dtype=torch.complex128, device="cuda")
    s = torch.cuda.Stream()

    def call():
        femg.check(femg.lib().fg_assemble_fp64_static(plan.ptr, None, v.data_ptr(), r.data_ptr(), s.cuda_stream))

    call()
    torch.cuda.synchronize()
    want = v.clone(), r.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s, capture_error_mode="thread_local"):
        call()
        call()
    for _ in range(5):
        v.zero_()
        r.fill_(3.0)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(v, want[0]) and torch.equal(r, want[1])

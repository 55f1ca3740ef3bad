"""Kernels that start beside the one before them, with other data in every
call: the element matrices and vectors of a call overwrite those of the one
before, with no wait between the calls, on a stream of the caller's that also
runs the caller's own kernels. A reduction or contraction that read them too
early, or an old copy of them, would give the values of the call before. The
expected values come from the oracle (1e-12 in FP64, 1e-6 in mixed precision,
relative Frobenius)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-12, "factored": 1e-12, "mixed": 1e-6}
SCALES = ((1.0, -3.0, 2.0), (-40.0, 5.0, -1.0), (0.25, 700.0, 30.0), (9.0, 0.0, 0.5))


def rel(a, b):
    nb = np.linalg.norm(b)
    return np.linalg.norm(a - b) / (nb if nb > 0 else 1.0)


def problems(F):
    return {"tri_small": F.config(dim=2, m=5, mesh_order=1, gauss=2, dirichlet=1, dirichlet_value=1.5, source=1),
            "tet_p2": F.config_c2(m=4, order=2), "tet_p3": F.config_c2(m=5, order=3), "tet_p4": F.config_c2(m=2, order=4)}


def terms(F, scale):
    """scale[0] grad u . grad v + scale[1] u v + scale[2] v"""
    arr = (F.TermDesc * 3)()
    for t, kind, c in zip(arr, (F.FG_TERM_GRAD_GRAD, F.FG_TERM_MASS, F.FG_TERM_SOURCE), scale):
        C.memset(C.byref(t), 0, C.sizeof(F.TermDesc))
        t.kind = kind
        t.coef.n_code = 1
        t.coef.code[0].op, t.coef.code[0].re = F.FG_OP_CONST, c
    return arr, 3


def outputs(torch, prob):
    return (torch.zeros(prob.nnz, dtype=torch.complex128, device="cuda"),
            torch.zeros(int(prob.sys.n_rows), dtype=torch.complex128, device="cuda"))


@pytest.mark.parametrize("path", ["fp64", "factored", "mixed"])
@pytest.mark.parametrize("name", ["tri_small", "tet_p2", "tet_p3", "tet_p4"])
def test_other_terms_in_every_call(femg, oracle, cuda, name, path):
    torch = cuda
    prob = femg.Problem(problems(femg)[name])
    sets = [terms(femg, s) for s in SCALES]
    want = [oracle.assemble(prob.arrays(), *t) for t in sets]
    plan = prob.plan()
    if path == "factored":
        plan.set_fp64_method(femg.FG_FP64_FACTORED)
    order = np.random.default_rng(3).integers(0, len(sets), 24)
    out = [outputs(torch, prob) for _ in order]
    seen = torch.zeros(prob.nnz, dtype=torch.complex128, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        for call, (k, (v, r)) in enumerate(zip(order, out)):
            plan.assemble("mixed" if path == "mixed" else "fp64", values=v.data_ptr(), rhs=r.data_ptr(), terms=sets[k],
                          stream=s.cuda_stream)
            if call % 2:
                seen.copy_(v).mul_(2.0)  # the caller's own work on the result
    torch.cuda.synchronize()
    for k, (v, r) in zip(order, out):
        assert rel(v.cpu().numpy(), want[k][0]) <= TOL[path]
        assert rel(r.cpu().numpy(), want[k][1]) <= TOL[path]
    plan.close()


def test_plans_that_share_the_static_scratch(femg, oracle, cuda):
    torch = cuda
    runs = []
    for name, cfg in problems(femg).items():
        prob = femg.Problem(cfg)
        t, nt = terms(femg, SCALES[len(runs)])
        a = prob.arrays()
        plan = prob.plan()
        femg.check(femg.lib().fg_plan_bind_terms(plan.ptr, t, nt, 0.0))
        fixed = torch.from_numpy(a["dirichlet"].view(np.float64).copy()).cuda()
        runs.append((prob, plan, fixed, oracle.assemble(a, t, nt)))
    order = np.random.default_rng(4).integers(0, len(runs), 48)
    out = [outputs(torch, runs[k][0]) for k in order]
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    for k, (v, r) in zip(order, out):
        prob, plan, fixed, _ = runs[k]
        femg.check(femg.lib().fg_assemble_fp64_static(plan.ptr, fixed.data_ptr() if fixed.numel() else None, v.data_ptr(),
                                                      r.data_ptr(), s.cuda_stream))
    torch.cuda.synchronize()
    for k, (v, r) in zip(order, out):
        want_v, want_r = runs[k][3]
        assert rel(v.cpu().numpy(), want_v) <= 1e-12 and rel(r.cpu().numpy(), want_r) <= 1e-12


@pytest.mark.parametrize("path", ["fp64", "mixed"])
def test_calls_that_add_up(femg, oracle, cuda, path):
    """accumulating calls: each adds to what the one before it wrote"""
    torch = cuda
    prob = femg.Problem(problems(femg)["tet_p2"])
    a = prob.arrays()
    plan = prob.plan()
    plan.set_accumulate(True)
    v, r = outputs(torch, prob)
    want_v, want_r, size = 0.0, 0.0, 0.0
    torch.cuda.synchronize()
    for scale in SCALES * 3:
        t = terms(femg, scale)
        plan.assemble(path, values=v.data_ptr(), rhs=r.data_ptr(), terms=t)
        wv, wr = oracle.assemble(a, *t)
        want_v, want_r, size = want_v + wv, want_r + wr, size + np.linalg.norm(wv)
    torch.cuda.synchronize()
    # the terms partly cancel: the error is measured against the summands
    assert np.linalg.norm(v.cpu().numpy() - want_v) <= TOL[path] * size
    assert rel(r.cpu().numpy(), want_r) <= 1e-12
    plan.close()

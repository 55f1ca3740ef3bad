"""Every shape of the CSR reduction (columns per load, loads per lane, component
blocks, one- and two-byte slots) against the oracle, by the FP64 path (1e-12)
and the mixed one (1e-6): element matrices of 3 to 63 columns, rows of one
entry and of hundreds, meshes whose rows do not fill a warp and meshes that
take several rounds; symmetric storage (columns that are not stored); several
groups and frequencies, real and complex; outputs that are added to."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    nb = np.linalg.norm(b)
    return np.linalg.norm(a - b) / (nb if nb > 0 else 1.0)


# name: (config, columns, mixed path applies)
def shapes(F):
    H, X, M, N = F.FG_SPACE_HIERARCHICAL_H1, F.FG_SPACE_HCURL, F.FG_PROBLEM_MAXWELL, F.FG_PROBLEM_NAVIER
    h1 = lambda dim, p, m, **k: F.config(dim=dim, m=m, mesh_order=1, space=H, order=p, gauss=2 * p, k=5.0, **k)  # noqa: E731
    hc = lambda dim, p, m: F.config(kind=M, dim=dim, m=m, mesh_order=1, space=X, order=p, gauss=2 * p + 2, k=5.0, coef_mode=1)  # noqa: E731
    nv = lambda p, m: F.config(kind=N, dim=3, m=m, mesh_order=1, space=H, order=p, gauss=2 * p, omega=3.0)  # noqa: E731
    return {"tri_3": (h1(2, 1, 90), 3, True), "tet_4": (h1(3, 1, 2), 4, True), "tri_6": (h1(2, 2, 31), 6, True),
            "hcurl_tri_8": (hc(2, 1, 9), 8, True), "tet_10": (h1(3, 2, 9), 10, True), "tri_15": (h1(2, 4, 7), 15, True),
            "tet_20": (h1(3, 3, 6), 20, True), "hcurl_tet_20": (hc(3, 1, 3), 20, True), "tri_21": (h1(2, 5, 4), 21, True),
            "tri_28": (h1(2, 6, 5), 28, True), "tet_35": (h1(3, 4, 4), 35, True), "tet_35_coarse": (h1(3, 4, 1), 35, True),
            "hcurl_tri_35": (hc(2, 4, 2), 35, False), "hcurl_tet_45": (hc(3, 2, 2), 45, False),
            "hcurl_tri_63": (hc(2, 6, 1), 63, False), "navier_12": (nv(1, 5), 12, True), "navier_30": (nv(2, 4), 30, True),
            "navier_60": (nv(3, 2), 60, True), "tet_10_upper": (h1(3, 2, 5, upper=1), 10, True),
            "tet_20_upper": (h1(3, 3, 3, upper=1), 20, True)}


NAMES = ["tri_3", "tet_4", "tri_6", "hcurl_tri_8", "tet_10", "tri_15", "tet_20", "hcurl_tet_20", "tri_21", "tri_28", "tet_35",
         "tet_35_coarse", "hcurl_tri_35", "hcurl_tet_45", "hcurl_tri_63", "navier_12", "navier_30", "navier_60", "tet_10_upper",
         "tet_20_upper"]


def tolerance(path):
    return 1e-12 if path == "fp64" else 1e-6


@pytest.mark.parametrize("path", ["fp64", "mixed"])
@pytest.mark.parametrize("name", NAMES)
def test_shapes(femg, oracle, cuda, name, path):
    import torch
    cfg, n, mixed = shapes(femg)[name]
    if path == "mixed" and not mixed:
        pytest.skip("wider than the contraction's tile")
    prob = femg.Problem(cfg)
    assert prob.n == n
    t, nt = prob.terms()
    ref_v, ref_b = oracle.assemble(prob.arrays(), t, nt)
    plan = prob.plan()
    v, b = plan.assemble(path)
    assert rel(v, ref_v) <= tolerance(path) and rel(b, ref_b) <= tolerance(path)
    # added into device outputs
    plan.set_accumulate(True)
    dv = torch.from_numpy(v.copy()).cuda()
    db = torch.ones(len(b), dtype=torch.complex128, device="cuda")
    plan.assemble(path, values=dv.data_ptr(), rhs=db.data_ptr())
    torch.cuda.synchronize()
    assert rel(dv.cpu().numpy(), 2 * ref_v) <= tolerance(path) and rel(db.cpu().numpy(), ref_b + 1.0) <= tolerance(path)
    plan.close()


@pytest.mark.parametrize("how", ["mass_dt2", "damped", "complex"])
@pytest.mark.parametrize("path", ["fp64", "mixed"])
@pytest.mark.parametrize("name", ["tri_3", "tet_4", "tet_10", "tet_20", "tri_21", "tet_35", "navier_12", "navier_30", "navier_60",
                                  "tet_20_upper"])
def test_groups(femg, oracle, cuda, name, path, how):
    """Two real groups, three groups, two complex groups."""
    prob = femg.Problem(shapes(femg)[name][0])
    t, nt = prob.terms()
    extra = (femg.TermDesc * (nt + 1))()
    for i in range(nt):
        C.memmove(C.byref(extra[i]), C.byref(t[i]), C.sizeof(femg.TermDesc))
    C.memset(C.byref(extra[nt]), 0, C.sizeof(femg.TermDesc))
    extra[nt].kind, extra[nt].dt = femg.FG_TERM_MASS, femg.FG_DT_1
    extra[nt].coef.n_code = 1
    extra[nt].coef.code[0].op, extra[nt].coef.code[0].re = femg.FG_OP_CONST, 0.7
    extra[nt - 1].dt = femg.FG_DT_2
    if how == "complex":
        extra[nt].coef.code[0].im = 0.4
        extra[nt].dt = femg.FG_DT_2
    count = nt if how == "mass_dt2" else nt + 1
    omegas = [0.5, 1.5, 4.0]
    a = prob.arrays()
    plan = prob.plan()
    vals, rhs = plan.assemble_multi_freq(omegas, path, terms=(extra, count))
    plan.close()
    for f, w in enumerate(omegas):
        ref_v, ref_b = oracle.assemble(a, extra, count, freq=w)
        assert rel(vals[f], ref_v) <= tolerance(path) and rel(rhs[f], ref_b) <= tolerance(path)

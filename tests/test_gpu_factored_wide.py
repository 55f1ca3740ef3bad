"""The factored FP64 method on the widest elements it takes: it runs where the
caller chose it and a block's shared memory holds the upper triangles of the
reference tensors (HCurl of order 2 on tetrahedra, 45 functions), and the
quadrature loop where it does not (63 functions), against the oracle (1e-12)."""
import pytest

from test_gpu_quadrature_blocks import rel, terms

pytestmark = pytest.mark.gpu


def wide(F):
    hc = lambda dim, p, m: F.config(kind=F.FG_PROBLEM_MAXWELL, dim=dim, m=m, mesh_order=1, space=F.FG_SPACE_HCURL, order=p,  # noqa: E731
                                    gauss=2 * p + 2)
    return {"hcurl_tet_45": (hc(3, 2, 2), 45, True), "hcurl_tri_48": (hc(2, 5, 3), 48, True), "hcurl_tri_63": (hc(2, 6, 2), 63, False)}


@pytest.mark.parametrize("how", ["real", "complex"])
@pytest.mark.parametrize("name", ["hcurl_tet_45", "hcurl_tri_48", "hcurl_tri_63"])
def test_wide(femg, oracle, cuda, name, how):
    cfg, n, fits = wide(femg)[name]
    prob = femg.Problem(cfg)
    assert prob.n == n
    t = terms(femg, prob, how)
    want, _ = oracle.assemble(prob.arrays(), *t)
    plan = prob.plan()
    plan.set_fp64_method(femg.FG_FP64_FACTORED)
    femg.profile_enable(True)
    femg.profile_read()
    try:
        v, _ = plan.assemble("fp64", terms=t)
        kernels = femg.profile_read()
    finally:
        femg.profile_enable(False)
    plan.close()
    assert ("k_element_factored_fp64" in kernels) == fits
    assert rel(v, want) <= 1e-12

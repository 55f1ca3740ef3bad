"""The factored FP64 kernel over its range of element matrices, against the
oracle (1e-12): partial tiles and rounds, odd and even matrix sizes, real and
complex coefficients, a term kind left out, a right-hand side beside it."""
import pytest

from test_gpu_quadrature_blocks import rel, shapes, terms

pytestmark = pytest.mark.gpu


def more(F):
    H = F.FG_SPACE_HIERARCHICAL_H1
    return dict(shapes(F), tri_p4_200=F.config(dim=2, m=10, mesh_order=1, space=H, order=4, gauss=8),
                tri_p9_18=F.config(dim=2, m=3, mesh_order=1, space=H, order=9, gauss=10),
                tri_p2_source=F.config(dim=2, m=8, mesh_order=2, space=F.FG_SPACE_LAGRANGE, gauss=4, source=1, dirichlet=1,
                                       dirichlet_value=1.5))


@pytest.mark.parametrize("how", ["real", "complex", "grad", "mass"])
@pytest.mark.parametrize("shape", ["tri_p1_2", "tri_p1_9522", "tri_p2_lagrange_242", "tri_p4_200", "tri_p6_98", "tri_p9_18",
                                   "tet_p1_6", "tet_p2_4374", "tet_p3_750", "tet_p4_162", "hcurl_tri_0_18", "hcurl_tet_1_750"])
def test_factored_blocks(femg, oracle, cuda, shape, how):
    prob = femg.Problem(more(femg)[shape])
    t = terms(femg, prob, how)
    ref_v, _ = oracle.assemble(prob.arrays(), *t)
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
    assert "k_element_factored_fp64" in kernels
    assert rel(v, ref_v) <= 1e-12


def test_factored_source(femg, oracle, cuda):
    prob = femg.Problem(more(femg)["tri_p2_source"])
    t, nt = prob.terms()
    ref_v, ref_b = oracle.assemble(prob.arrays(), t, nt)
    plan = prob.plan()
    plan.set_fp64_method(femg.FG_FP64_FACTORED)
    v, b = plan.assemble("fp64")
    plan.close()
    assert rel(v, ref_v) <= 1e-12 and rel(b, ref_b) <= 1e-12

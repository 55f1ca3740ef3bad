"""The blocks of the FP64 quadrature kernels at their edges, against the oracle
(1e-12, the FP64 tolerance): element counts around the elements of a block,
from one upper-triangle entry per thread to the largest element matrices, and
each way of summing (real; complex constant coefficients, whose real integrals
are summed apart; complex inside the elements; a term kind left out)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    nb = np.linalg.norm(b)
    return np.linalg.norm(a - b) / (nb if nb > 0 else 1.0)


def shapes(F):
    H, X = F.FG_SPACE_HIERARCHICAL_H1, F.FG_SPACE_HCURL
    M = F.FG_PROBLEM_MAXWELL
    return {"tri_p1_2": F.config(dim=2, m=1, mesh_order=1, space=H, order=1, gauss=2),
            "tri_p1_9522": F.config(dim=2, m=69, mesh_order=1, space=H, order=1, gauss=2),
            "tri_p2_lagrange_242": F.config(dim=2, m=11, mesh_order=2, space=F.FG_SPACE_LAGRANGE, gauss=4),
            "tri_p6_98": F.config(dim=2, m=7, mesh_order=1, space=H, order=6, gauss=6),
            "tet_p1_6": F.config(dim=3, m=1, mesh_order=1, space=H, order=1, gauss=2),
            "tet_p2_4374": F.config(dim=3, m=9, mesh_order=1, space=H, order=2, gauss=4),
            "tet_p3_750": F.config(dim=3, m=5, mesh_order=1, space=H, order=3, gauss=6),
            "tet_p4_162": F.config(dim=3, m=3, mesh_order=1, space=H, order=4, gauss=8),
            "hcurl_tri_0_18": F.config(kind=M, dim=2, m=3, mesh_order=1, space=X, order=0, gauss=2),
            "hcurl_tet_1_750": F.config(kind=M, dim=3, m=5, mesh_order=1, space=X, order=1, gauss=4),
            "hcurl_tri_6_8": F.config(kind=M, dim=2, m=2, mesh_order=1, space=X, order=6, gauss=8),
            "navier_p1_162": F.config(kind=F.FG_PROBLEM_NAVIER, dim=3, m=3, mesh_order=1, space=H, order=1, gauss=2),
            "navier_p2_750": F.config(kind=F.FG_PROBLEM_NAVIER, dim=3, m=5, mesh_order=1, space=H, order=2, gauss=4)}


def terms(F, prob, how):
    """grad (or elastic) and mass terms with the coefficients of `how`"""
    k = lambda re, im=0.0: (F.FG_OP_CONST, 0, re, im)  # noqa: E731
    x, add, mul = (F.FG_OP_X, 0, 0.0, 0.0), (F.FG_OP_ADD, 0, 0.0, 0.0), (F.FG_OP_MUL, 0, 0.0, 0.0)
    first, second = {"real": ([k(1.5)], [k(-3.0)]), "complex": ([k(1.5, 0.5)], [k(-3.0, 0.25)]),
                     "point": ([k(1.5, 0.5), x, k(0.3), mul, add], [k(-3.0), x, k(0.0, 2.0), mul, add]),
                     "grad": ([k(1.5)], None), "mass": (None, [k(-3.0, 1.0)])}[how]
    navier = prob.space.multiplicity == 3
    out = [(F.FG_TERM_ELASTIC if navier else F.FG_TERM_GRAD_GRAD, first), (F.FG_TERM_MASS, second)]
    out = [t for t in out if t[1]]
    arr = (F.TermDesc * len(out))()
    for t, (kind, code) in zip(arr, out):
        C.memset(C.byref(t), 0, C.sizeof(F.TermDesc))
        t.kind = kind
        for ex in (t.coef, t.coef2) if kind == F.FG_TERM_ELASTIC else (t.coef,):
            ex.n_code = len(code)
            for i, (op, arg, re, im) in enumerate(code):
                ex.code[i].op, ex.code[i].arg, ex.code[i].re, ex.code[i].im = op, arg, re, im
    return arr, len(out)


@pytest.mark.parametrize("how", ["real", "complex", "point", "grad", "mass"])
@pytest.mark.parametrize("shape", ["tri_p1_2", "tri_p1_9522", "tri_p2_lagrange_242", "tri_p6_98", "tet_p1_6", "tet_p2_4374",
                                   "tet_p3_750", "tet_p4_162", "hcurl_tri_0_18", "hcurl_tet_1_750", "hcurl_tri_6_8",
                                   "navier_p1_162", "navier_p2_750"])
def test_quadrature_blocks(femg, oracle, cuda, shape, how):
    prob = femg.Problem(shapes(femg)[shape])
    t = terms(femg, prob, how)
    ref_v, ref_b = oracle.assemble(prob.arrays(), *t)
    plan = prob.plan()
    v, b = plan.assemble("fp64", terms=t)
    plan.close()
    assert rel(v, ref_v) <= 1e-12 and rel(b, ref_b) <= 1e-12

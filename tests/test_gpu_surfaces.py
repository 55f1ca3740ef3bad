"""Triangles in a plane of constant z, in a tilted plane and on a curved
surface, and coefficients of real value through every operator that stays
real, on the FP64 path against the oracle (1e-12)."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_quadrature_blocks import rel, terms

pytestmark = pytest.mark.gpu


def lifted(femg, cfg, z):
    """The square's mesh with z(x, y) as its nodes' third coordinate."""
    prob = femg.Problem(cfg)
    xyz = np.ctypeslib.as_array(prob.mesh.node_xyz, shape=(prob.mesh.n_nodes, 3))
    xyz[:, 2] = z(xyz[:, 0], xyz[:, 1])
    return prob


SURFACES = {"flat": lambda x, y: 0.7 + 0.0 * x, "tilted": lambda x, y: 0.3 * x - 0.2 * y, "curved": lambda x, y: 0.4 * x * y + 0.1 * x * x}


def spaces(F):
    return {"p1": F.config(dim=2, m=5, mesh_order=1, space=F.FG_SPACE_LAGRANGE, gauss=2),
            "p2": F.config(dim=2, m=5, mesh_order=2, space=F.FG_SPACE_LAGRANGE, gauss=4),
            "h3": F.config(dim=2, m=4, mesh_order=1, space=F.FG_SPACE_HIERARCHICAL_H1, order=3, gauss=6),
            "hcurl1": F.config(kind=F.FG_PROBLEM_MAXWELL, dim=2, m=4, mesh_order=1, space=F.FG_SPACE_HCURL, order=1, gauss=4)}


@pytest.mark.parametrize("how", ["real", "complex", "point"])
@pytest.mark.parametrize("method", ["quadrature", "factored"])
@pytest.mark.parametrize("surface", list(SURFACES))
@pytest.mark.parametrize("space", ["p1", "p2", "h3", "hcurl1"])
def test_surface(femg, oracle, cuda, space, surface, method, how):
    prob = lifted(femg, spaces(femg)[space], SURFACES[surface])
    t = terms(femg, prob, how)
    ref_v, _ = oracle.assemble(prob.arrays(), *t)
    plan = prob.plan()
    if method == "factored":
        plan.set_fp64_method(femg.FG_FP64_FACTORED)
    v, _ = plan.assemble("fp64", terms=t)
    plan.close()
    assert rel(v, ref_v) <= 1e-12


OPS = ["EXP", "POW2", "POW5", "SIN", "COS", "TAN", "SINH", "COSH", "TANH", "ATAN", "ASINH", "ABS", "CONJ", "REAL", "NEG", "HEAVISIDE",
       "DIV", "ATAN2", "ELEM", "POINT"]


@pytest.mark.parametrize("op", OPS)
def test_real_operator(femg, oracle, cuda, op):
    """m = op(a) and f = op(a) / 2 with the real a = 0.4 + 0.3 x + 0.2 y - 0.5 z."""
    F = femg
    prob = lifted(F, spaces(F)["p2"], SURFACES["flat"])
    a = prob.arrays()
    k = lambda v: (F.FG_OP_CONST, 0, v, 0.0)  # noqa: E731
    o = lambda name, arg=0: (getattr(F, "FG_OP_" + name), arg, 0.0, 0.0)  # noqa: E731
    code = [k(0.4), o("X"), k(0.3), o("MUL"), o("ADD"), o("Y"), k(0.2), o("MUL"), o("ADD"), o("Z"), k(0.5), o("MUL"), o("SUB")]
    table = None
    if op.startswith("POW"):
        code.append(o("POW", int(op[3:])))
    elif op in ("DIV", "ATAN2"):
        code += [k(0.7), o("Y"), o("ADD"), o(op)]
    elif op == "HEAVISIDE":
        code += [k(0.3), o("SUB"), o(op)]
    elif op in ("ELEM", "POINT"):
        count = a["E"] * (a["nq"] if op == "POINT" else 1)
        table = np.zeros((count, 2))
        table[:, 0] = np.random.default_rng(3).uniform(-1.0, 1.0, count)
        code += [o(op), o("MUL")]
    else:
        code.append(o(op))
    t = (F.TermDesc * 3)()
    for i, (kind, c) in enumerate([(F.FG_TERM_GRAD_GRAD, [k(1.0)]), (F.FG_TERM_MASS, code),
                                   (F.FG_TERM_SOURCE, code + [k(0.5), o("MUL")])]):
        C.memset(C.byref(t[i]), 0, C.sizeof(F.TermDesc))
        t[i].kind = kind
        t[i].coef.n_code = len(c)
        for q, (x, arg, re, im) in enumerate(c):
            t[i].coef.code[q].op, t[i].coef.code[q].arg, t[i].coef.code[q].re, t[i].coef.code[q].im = x, arg, re, im
        if i and table is not None:
            t[i].coef.n_arrays = 1
            t[i].coef.elem_values[0] = table.ctypes.data_as(C.POINTER(C.c_double))
    ref_v, ref_b = oracle.assemble(a, t, 3)
    plan = prob.plan()
    v, b = plan.assemble("fp64", terms=(t, 3))
    plan.close()
    assert rel(v, ref_v) <= 1e-12 and rel(b, ref_b) <= 1e-12

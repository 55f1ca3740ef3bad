"""Coefficients that are infinite, NaN or beyond FP32 on one element: what that
element adds to is not finite, and every other entry is bit for bit what it is
with an ordinary coefficient there; through the quadrature loop, the
factorisation and the mixed path (whose finite sums widen from FP32), and the
lean kernels of the reduction."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def terms(F, per_element):
    """c grad u . grad v - 3 u v with c per element"""
    arr = (F.TermDesc * 2)()
    for t, kind in zip(arr, (F.FG_TERM_GRAD_GRAD, F.FG_TERM_MASS)):
        C.memset(C.byref(t), 0, C.sizeof(F.TermDesc))
        t.kind = kind
        t.coef.n_code = 1
    arr[0].coef.code[0].op, arr[0].coef.n_arrays = F.FG_OP_ELEM, 1
    arr[0].coef.elem_values[0] = per_element.ctypes.data_as(C.POINTER(C.c_double))
    arr[1].coef.code[0].op, arr[1].coef.code[0].re = F.FG_OP_CONST, -3.0
    return arr, 2


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 1e300])
@pytest.mark.parametrize("path", ["fp64", "factored", "mixed"])
@pytest.mark.parametrize("dim,order,m", [(2, 2, 6), (3, 1, 3), (3, 3, 2)])
def test_one_element(femg, cuda, dim, order, m, path, value):
    prob = femg.Problem(femg.config(dim=dim, m=m, mesh_order=1, space=femg.FG_SPACE_HIERARCHICAL_H1, order=order, gauss=2 * order))
    a = prob.arrays()
    e = prob.E // 2
    plan = prob.plan()
    if path == "factored":
        plan.set_fp64_method(femg.FG_FP64_FACTORED)
    out = []
    for v in (2.0, value):
        c = np.ones(prob.E, np.complex128)
        c[e] = v
        out.append(plan.assemble("mixed" if path == "mixed" else "fp64", terms=terms(femg, c), rhs=False)[0])
    plan.close()
    ai, aj = a["ai"].astype(np.int64), a["aj"].astype(np.int64)
    mine = np.isin(np.repeat(np.arange(len(ai) - 1), np.diff(ai)), a["edof"][e]) & np.isin(aj, a["edof"][e])
    assert np.array_equal(out[0][~mine].view(np.uint64), out[1][~mine].view(np.uint64)) and np.all(np.isfinite(out[0]))
    if value != 1e300:
        assert not np.any(np.isfinite(out[1][mine]))
    elif path == "mixed":  # beyond FP32
        assert not np.all(np.isfinite(out[1][mine]))
    else:
        assert np.all(np.isfinite(out[1][mine])) and np.abs(out[1][mine]).max() > 1e290

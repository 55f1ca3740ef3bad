"""The FP64 quadrature kernels on flat, sheared elements, entry by entry
against extended precision (numpy longdouble). The reference maps both
functions by J^-T and multiplies physical gradients; an entry's error then
grows as the aspect ratio. A product formed through J^-1 J^-T in reference
coordinates, whose large entries cancel, would lose its square, which a norm of
the whole matrix does not show.

Bound on the error of an entry, with eps = 2^-53 and kappa = |J|_F^3 / |det J|
(for one short direction about the aspect ratio): cofactors and determinant
come with a relative error of a few kappa eps, and a mapped function's sum of
three products, none larger than kappa times the result, with another few, on
both sides; 32 kappa eps of the entry's sum of products of norms covers them.
A bound with kappa^2, which the reference-coordinate product needs, is
thousands of times larger at the aspect ratios here."""
import ctypes as C

import numpy as np
import pytest

from conftest import load_femg

pytestmark = pytest.mark.gpu

L, CL = np.longdouble, np.clongdouble
EPS = 2.0 ** -53


def configs(F):
    H, X, M = F.FG_SPACE_HIERARCHICAL_H1, F.FG_SPACE_HCURL, F.FG_PROBLEM_MAXWELL
    return {"tri_p1": F.config(dim=2, m=3, mesh_order=1, space=H, order=1, gauss=2, jitter=0.0),
            "tri_p3": F.config(dim=2, m=3, mesh_order=1, space=H, order=3, gauss=6, jitter=0.0),
            "tri_lagrange": F.config(dim=2, m=3, mesh_order=2, space=F.FG_SPACE_LAGRANGE, gauss=4, jitter=0.0),
            "tet_p1": F.config(dim=3, m=2, mesh_order=1, space=H, order=1, gauss=2, jitter=0.0),
            "tet_p3": F.config(dim=3, m=2, mesh_order=1, space=H, order=3, gauss=6, jitter=0.0),
            "hcurl_tri": F.config(kind=M, dim=2, m=3, mesh_order=1, space=X, order=1, gauss=4, jitter=0.0),
            "hcurl_tet": F.config(kind=M, dim=3, m=2, mesh_order=1, space=X, order=1, gauss=4, jitter=0.0)}


def stretch(prob, aspect, surface):
    """The problem's nodes, in place: one direction shortened by `aspect`, then
    sheared and turned, in the plane of a 2D mesh (surface: out of it)."""
    m = prob.mesh
    xyz = np.ctypeslib.as_array(m.node_xyz, (3 * m.n_nodes,)).reshape(-1, 3)
    rng = np.random.default_rng(7)
    d = int(m.dim)
    A = np.eye(3)
    A[d - 1, d - 1] = 1.0 / aspect
    S = np.eye(3)
    S[d - 1, 0] = 0.7  # the short direction leans with x
    Q = np.eye(3)
    n = 3 if surface else d
    Q[:n, :n] = np.linalg.qr(rng.standard_normal((n, n)))[0]
    xyz[:] = xyz @ (Q @ S @ A).T


def separate(prob):
    """Gives every element DOFs of its own, so that the CSR values are the
    element matrices: a function that varies along the long directions alone
    does so in some elements and not in their neighbours."""
    y, E, n = prob.sys, prob.E, prob.n
    keep = prob.keep = [np.arange(E * n, dtype=np.uint64), np.full(E * n, load_femg().FG_AT_UNKNOWN, np.int32),
                        np.arange(E * n + 1, dtype=np.uint64) * np.uint64(n),
                        (np.arange(E, dtype=np.uint64)[:, None, None] * np.uint64(n) +
                         np.zeros((1, n, 1), np.uint64) + np.arange(n, dtype=np.uint64)).ravel()]
    y.n_rows, y.n_fixed = E * n, 0
    for name, v in zip(("elem_dof_idx", "elem_dof_type", "ai", "aj"), keep):
        setattr(y, name, v.ctypes.data_as(type(getattr(y, name))))


def expr(F, ex, code):
    ex.n_code, ex.n_arrays = len(code), 0
    for i, (op, re, im) in enumerate(code):
        ex.code[i].op, ex.code[i].arg, ex.code[i].re, ex.code[i].im = op, 0, re, im


SYM = np.array([[2.0, 0.3, 0.2], [0.3, 1.5, -0.4], [0.2, -0.4, 1.2]]) + 1j * np.diag([0.5, -0.25, 0.125])
GEN = np.array([[1.0, 0.5, 0.25], [-0.5, 1.25, 0.125], [0.0, -0.25, 0.75]])
VEC = np.array([0.5, -0.75, 0.25])


def terms(F, form, how):
    """(TermDesc array, count, keep-alive, coefficients): gradient (curl)
    tensor M, mass (tensor) B, value-to-gradient b, gradient-to-value v; M and
    B times 1 + x for "point". Values are exact in binary."""
    one = [(F.FG_OP_CONST, 1.0, 0.0)]
    slope = [(F.FG_OP_CONST, 1.0, 0.0), (F.FG_OP_X, 0.0, 0.0), (F.FG_OP_ADD, 0.0, 0.0)]
    const = lambda z: [(F.FG_OP_CONST, float(np.real(z)), float(np.imag(z)))]  # noqa: E731
    scalar = {"real": (1.5, -3.0), "grad": (1.5, 0.0), "complex": (1.5 + 0.5j, -3.0 + 0.25j), "point": (1.0, 1.0)}
    co = dict(M=np.zeros((3, 3), complex), B=np.zeros((3, 3), complex), b=np.zeros(3), v=np.zeros(3), slope=how == "point")
    out, keep = [], []  # (kind, scalar program, tensor programs)
    if how in scalar:
        cg, cm = scalar[how]
        out.append((F.FG_TERM_GRAD_GRAD, slope if how == "point" else const(cg), None))
        co["M"] = cg * np.eye(3)
        if cm:
            out.append((F.FG_TERM_MASS, slope if how == "point" else const(cm), None))
            co["B"] = cm * np.eye(3)
    elif how == "tensor":
        six = [SYM[0, 0], SYM[1, 1], SYM[2, 2], SYM[0, 1], SYM[0, 2], SYM[1, 2]]
        out.append((F.FG_TERM_GRAD_GRAD_TENSOR, one, [const(z) for z in six]))
        co["M"] = SYM
        if form == F.FG_FORM_1:
            out.append((F.FG_TERM_MASS_TENSOR, one, [const(z) for z in six]))
            co["B"] = SYM
    else:  # "full": every term of the non-symmetric kernel
        out = [(F.FG_TERM_GRAD_GRAD_TENSOR_FULL, one, [const(z) for z in GEN.ravel()]),
               (F.FG_TERM_ADVECTION, one, [const(z) for z in VEC]), (F.FG_TERM_VECTOR_GRAD_TEST, one, [const(z) for z in VEC]),
               (F.FG_TERM_SOURCE_GRAD, one, [const(z) for z in VEC])]
        co.update(M=GEN, b=VEC, v=VEC, f=VEC)
    arr = (F.TermDesc * len(out))()
    for t, (kind, code, ten) in zip(arr, out):
        C.memset(C.byref(t), 0, C.sizeof(F.TermDesc))
        t.kind = kind
        expr(F, t.coef, code)
        if ten:
            ex = (F.Expr * len(ten))()
            for e, c in zip(ex, ten):
                expr(F, e, c)
            keep.append(ex)
            t.tensor = C.cast(ex, C.POINTER(F.Expr))
    return arr, len(out), keep, co


def cross(a, b):
    return np.stack([a[..., 1] * b[..., 2] - a[..., 2] * b[..., 1], a[..., 2] * b[..., 0] - a[..., 0] * b[..., 2],
                     a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]], -1)


def norm(a):
    return np.sqrt((np.abs(a) ** 2).sum(-1))


def exact(a, co):
    """Element matrices and vectors in extended precision, and the bounds of
    their entries in units of 32 eps"""
    X = a["xyz"].astype(L)[a["enodes"]]
    E, n = a["edof"].shape
    ke, bound = np.zeros((E, n, n), CL), np.zeros((E, n, n), L)
    be, bbound = np.zeros((E, n), CL), np.zeros((E, n), L)
    M, B, b, v, f = (np.asarray(co.get(k, np.zeros(3))).astype(CL) for k in ("M", "B", "b", "v", "f"))
    for q in range(a["nq"]):
        dN = a["geo_grad"][q].astype(L)
        col = [np.einsum("ekr,k->er", X, dN[:, c]) for c in range(3)]
        if a["dim"] == 2:
            nrm = cross(col[0], col[1])
            col[2] = nrm / norm(nrm)[:, None]
        cof = [cross(col[1], col[2]), cross(col[2], col[0]), cross(col[0], col[1])]
        det = (col[0] * cof[0]).sum(-1)
        J = np.stack(col, -1)                        # J[e, r, c]
        inv = np.stack(cof, 1) / det[:, None, None]  # J^-1[e, c, r]
        kappa = np.sqrt((J ** 2).sum((1, 2))) ** 3 / np.abs(det)
        gr, va = a["bgrad"][a["orient"], q].astype(L), a["bval"][a["orient"], q].astype(L)
        s = a["w"][q].astype(L) * np.abs(det)
        x = np.einsum("ekr,k->er", X, a["geo_val"][q].astype(L))[:, 0]
        c = 1 + x if co["slope"] else np.ones_like(x)
        if a["form"] == 1:
            G = np.einsum("erc,eic->eir", J, gr) / det[:, None, None]
            P = np.einsum("ecr,eic->eir", inv, va)
        else:
            G, P = np.einsum("ecr,eic->eir", inv, gr), va[..., None] * np.array([1, 0, 0], L)
        MG, BP = np.einsum("rs,ejs->ejr", M, G), np.einsum("rs,ejs->ejr", B, P)
        sc, sb = s * c, s * np.abs(c) * kappa
        U, W = MG + b * P[..., :1], BP + (G @ v)[..., None] * np.array([1, 0, 0], L)
        ke += sc[:, None, None] * (np.einsum("eir,ejr->eij", G, U) + np.einsum("eir,ejr->eij", P, W))
        nU = np.abs(M).sum() * norm(G) + np.abs(b).sum() * norm(P)
        nW = np.abs(B).sum() * norm(P) + np.abs(v).sum() * norm(G)
        bound += sb[:, None, None] * (norm(G)[:, :, None] * nU[:, None, :] + norm(P)[:, :, None] * nW[:, None, :])
        be += s[:, None] * (G @ f)
        bbound += (s * kappa)[:, None] * norm(G) * np.abs(f).sum()
    return ke.ravel(), bound.ravel(), be.ravel(), bbound.ravel()


def worst(got, want, bound):
    """largest error in units of 32 eps times the entry's bound"""
    tiny = L(1e-300)
    return float(np.max(np.abs(got.astype(CL) - want) / (32 * EPS * bound + tiny)))


CASES = [(name, how, surface) for name in ("tri_p1", "tri_p3", "tri_lagrange", "tet_p1", "tet_p3")
         for how in ("real", "grad", "complex", "point", "tensor", "full") for surface in ((False, True) if name == "tri_p3" else (False,))]
CASES += [(name, how, False) for name in ("hcurl_tri", "hcurl_tet") for how in ("real", "complex", "tensor")]


@pytest.mark.parametrize("aspect", [1.0, 1e4])
@pytest.mark.parametrize("name,how,surface", CASES)
def test_entries(femg, cuda, name, how, surface, aspect):
    prob = femg.Problem(configs(femg)[name])
    stretch(prob, aspect, surface)
    separate(prob)
    a = prob.arrays()
    t, nt, keep, co = terms(femg, a["form"], how)
    plan = prob.plan()
    v, r = plan.assemble("fp64", terms=(t, nt))
    plan.close()
    values, vb, rhs, rb = exact(a, co)
    assert worst(v, values, vb) <= 1.0
    assert worst(r, rhs, rb) <= 1.0

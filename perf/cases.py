"""The assembly work that users of the framework have it do, as cases that can be
timed and compared: what each stands for is said at listed().

A case holds plain values. Its problem (mesh, field, terms, pre()) is built by
the host mirror, as a program's own Formulation::pre() would have left it, and a
plan is kept, as a program keeps it; a pass is one call of the library.

A few values follow from a case's order and dimension: the rule is Gauss(2p),
the rule of the repository's own configurations.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _femg():
    if "femg" not in sys.modules:
        spec = importlib.util.spec_from_file_location("femg", os.path.join(ROOT, "fem-g_gb300", "femg.py"))
        mod = importlib.util.module_from_spec(spec)
        sys.modules["femg"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["femg"]


def listed():
    return [
        # the smallest call: a coarse 2D mesh of first-order triangles, its boundary values lifted, a source; launches and host work
        dict(name="tri_p1_m5_fp64", do="assemble", field="h1", dim=2, order=1, m=5, coef="const", dirichlet=True, path="fp64",
             host=False, bound=True),
        # the 2D second-order Lagrange problem of the reference's examples, as the drop-in binding calls it: terms with each call, outputs in host memory
        dict(name="tri_p2_m64_fp64_host", do="assemble", field="lagrange", dim=2, order=2, m=64, coef="const", dirichlet=True,
             path="fp64", host=True, bound=False),
        # the 3D order-3 problem with a coefficient per tetrahedron, in double precision, by the default method
        dict(name="tet_p3_m24_fp64", do="assemble", field="h1", dim=3, order=3, m=24, coef="element", dirichlet=False,
             path="fp64", host=False, bound=True),
        # order 2 with coefficients that vary inside the elements and are complex: an absorbing, graded medium
        dict(name="tet_p2_m21_fp64_point", do="assemble", field="h1", dim=3, order=2, m=21, coef="point", dirichlet=False,
             path="fp64", host=False, bound=True),
        # double precision by the factorisation, chosen by the caller
        dict(name="tet_p3_m30_factored", do="assemble", field="h1", dim=3, order=3, m=30, coef="element", dirichlet=False,
             path="factored", host=False, bound=True),
        # the benchmark's workload: mixed precision, device outputs; the largest listed system
        dict(name="tet_p3_m40_mixed", do="assemble", field="h1", dim=3, order=3, m=40, coef="element", dirichlet=False,
             path="mixed", host=False, bound=True),
        # the widest scalar elements in mixed precision: 35 functions, rows that are not a multiple of a vector
        dict(name="tet_p4_m16_mixed", do="assemble", field="h1", dim=3, order=4, m=16, coef="const", dirichlet=False,
             path="mixed", host=False, bound=True),
        # elasticity, three components, a frequency sweep in one pass
        dict(name="navier_p2_m20_sweep", do="sweep", field="navier", dim=3, order=2, m=20, freqs=8, path="mixed"),
        # elasticity in double precision at one frequency
        dict(name="navier_p2_m15_fp64", do="assemble", field="navier", dim=3, order=2, m=15, coef="element", dirichlet=False,
             path="fp64", host=False, bound=True),
        # Maxwell with edge elements of order 1 (20 functions a tetrahedron), double precision
        dict(name="hcurl_1_m18_fp64", do="assemble", field="hcurl", dim=3, order=1, m=18, coef="element", dirichlet=False,
             path="fp64", host=False, bound=True),
        # many problems of uneven size and order in one graph launch
        dict(name="batch_12_mixed", do="batch", count=12, mix=4, m_lo=4, m_hi=16, path="mixed"),
        # the symbolic phase of the same kind of system: pattern and numbering, host arrays in and out
        dict(name="symbolic_tet_p3_m19", do="symbolic", field="h1", dim=3, order=3, m=19),
    ]


# largest cells per side drawn, by what a case is: none costs more than the largest listed one
_TOP = {("h1", 3, 1): 40, ("h1", 3, 2): 32, ("h1", 3, 3): 26, ("h1", 3, 4): 16, ("h1", 2, 1): 160, ("h1", 2, 2): 128,
        ("h1", 2, 3): 96, ("h1", 2, 4): 64, ("lagrange", 2, 1): 160, ("lagrange", 2, 2): 128, ("lagrange", 3, 2): 20,
        ("navier", 3, 1): 20, ("navier", 3, 2): 15, ("hcurl", 2, 0): 128, ("hcurl", 2, 1): 64, ("hcurl", 3, 0): 28,
        ("hcurl", 3, 1): 18}


def draw(rng):
    do = rng.choice(["assemble"] * 6 + ["sweep", "batch", "symbolic"])
    if do == "batch":
        lo = rng.randint(2, 8)
        return dict(do="batch", count=rng.randint(2, 12), mix=rng.randrange(1 << 20), m_lo=lo, m_hi=lo + rng.randint(2, 10),
                    path="mixed")
    fields = {"sweep": ["navier", "navier", "h1"], "symbolic": ["h1", "h1", "lagrange"]}.get(
        do, ["h1", "h1", "h1", "lagrange", "navier", "hcurl"])
    field = rng.choice(fields)
    if field == "h1":
        dim, order = rng.choice([2, 3, 3, 3]), rng.randint(1, 4)
    elif field == "lagrange":
        dim, order = rng.choice([(2, 1), (2, 2), (3, 2)])
    elif field == "navier":
        dim, order = 3, rng.randint(1, 2)
    else:
        dim, order = rng.choice([2, 3]), rng.randint(0, 1)
    top = _TOP[(field, dim, order)]
    m = int(round(math.exp(rng.uniform(math.log(3), math.log(top)))))
    if do == "symbolic":
        return dict(do=do, field=field, dim=dim, order=order, m=m)
    if do == "sweep":
        return dict(do=do, field=field, dim=dim, order=order, m=m, freqs=rng.randint(2, 8), path=rng.choice(["mixed", "fp64"]))
    coef = rng.choice(["const", "element", "point"])
    if field in ("navier", "hcurl") and coef == "point":
        coef = "element"
    path = "fp64" if coef == "point" else rng.choice(["fp64", "mixed", "mixed", "factored"])
    if path == "factored" and field == "navier":
        path = "fp64"
    fixable = dim == 2 and (field == "lagrange" or (field, order) == ("h1", 1))
    return dict(do=do, field=field, dim=dim, order=order, m=m, coef=coef, dirichlet=fixable and rng.random() < 0.5, path=path,
                host=rng.random() < 0.25, bound=rng.random() < 0.7)


# ------------------------------------------------------------------ problems

K = 20.0  # wavenumber


def _problem(case, seed):
    F = _femg()
    dim, order = case["dim"], case["order"]
    kind = {"navier": F.FG_PROBLEM_NAVIER, "hcurl": F.FG_PROBLEM_MAXWELL}.get(case["field"], F.FG_PROBLEM_HELMHOLTZ)
    space = {"lagrange": F.FG_SPACE_LAGRANGE, "hcurl": F.FG_SPACE_HCURL}.get(case["field"], F.FG_SPACE_HIERARCHICAL_H1)
    lifted = bool(case.get("dirichlet"))
    return F.Problem(F.config(
        kind=kind, dim=dim, m=case["m"], mesh_order=order if case["field"] == "lagrange" else 1, space=space, order=order,
        gauss=2 * (order + 1 if case["field"] == "hcurl" else order), jitter=0.2 if dim == 2 else 0.15, seed=1 + seed, k=K,
        coef_mode=1 if case.get("coef") == "element" or case["field"] == "hcurl" else 0, dirichlet=int(lifted),
        dirichlet_value=1.5 if lifted else 0.0, source=int(lifted), omega=0.0 if case["do"] == "sweep" else 5.0))


def _code(expr, code):
    expr.n_code, expr.n_arrays = len(code), 0
    for k, (op, arg, re, im) in enumerate(code):
        expr.code[k].op, expr.code[k].arg, expr.code[k].re, expr.code[k].im = op, arg, re, im


def _point_terms(dim):
    """c grad u . grad v + m u v + f v with c = 1 + 0.5 x + 0.2 i y^2, m = -k^2 (1 + 0.3 i x y), f = exp(-x) (1 + i y)."""
    F = _femg()
    k = lambda re, im=0.0: (F.FG_OP_CONST, 0, re, im)  # noqa: E731
    x, y = (F.FG_OP_X, 0, 0.0, 0.0), (F.FG_OP_Y, 0, 0.0, 0.0)
    add, mul, neg, exp = ((op, 0, 0.0, 0.0) for op in (F.FG_OP_ADD, F.FG_OP_MUL, F.FG_OP_NEG, F.FG_OP_EXP))
    t = (F.TermDesc * 3)()
    t[0].kind, t[1].kind, t[2].kind = F.FG_TERM_GRAD_GRAD, F.FG_TERM_MASS, F.FG_TERM_SOURCE
    _code(t[0].coef, [k(1.0), k(0.5), x, mul, add, k(0.0, 0.2), y, mul, y, mul, add])
    _code(t[1].coef, [k(1.0), k(0.0, 0.3), x, mul, y, mul, add, k(-K * K), mul])
    _code(t[2].coef, [x, neg, exp, k(1.0), k(0.0, 1.0), y, mul, add, mul])
    return t, 3


def _mix(case):
    """(order, cells per side, wavenumber) of each problem of a batch: the case's own, whatever the seed."""
    rng = np.random.default_rng(case["mix"])
    return [(int(rng.integers(1, 5)), int(rng.integers(case["m_lo"], case["m_hi"] + 1)), float(rng.uniform(5.0, 40.0)))
            for _ in range(case["count"])]


def _omegas(case, seed):
    return np.sort(np.random.default_rng(seed).uniform(1.0, 10.0, case["freqs"]))


def _batch_configs(case, seed):
    F = _femg()
    return [F.config(dim=3, m=m, mesh_order=1, space=F.FG_SPACE_HIERARCHICAL_H1, order=p, gauss=2 * p, jitter=0.15,
                     seed=1 + seed + 1000 * q, k=k) for q, (p, m, k) in enumerate(_mix(case))]


def prepare(case, seed):
    F = _femg()
    s = dict(case=case)
    if case["do"] == "batch":
        s["problems"] = [F.Problem(c) for c in _batch_configs(case, seed)]
        plans = [p.plan() for p in s["problems"]]
        s["batch"] = F.Batch(plans, mixed=case["path"] == "mixed")
        s["values"] = [torch.zeros(p.nnz, dtype=torch.complex128, device="cuda") for p in s["problems"]]
        s["rhs"] = [torch.zeros(int(p.sys.n_rows), dtype=torch.complex128, device="cuda") for p in s["problems"]]
        s["pointers"] = [v.data_ptr() for v in s["values"]], [r.data_ptr() for r in s["rhs"]]
        return s
    p = s["problem"] = _problem(case, seed)
    rows = int(p.sys.n_rows)
    if case["do"] == "symbolic":
        a, d = p.arrays(), p.created_dofs()
        s.update(edof=a["edof"], etype=a["etype"], rows=rows, bbox=p.bbox(), xyz=d["xyz"], types=d["assemble_type"],
                 numbers=p.raw_dofs()["num_dof"])
        return s
    s["plan"] = p.plan()
    if case["path"] == "factored":
        s["plan"].set_fp64_method(F.FG_FP64_FACTORED)
    s["precision"] = "mixed" if case["path"] == "mixed" else "fp64"
    if case["do"] == "sweep":
        s["omegas"] = _omegas(case, seed)
        s["values"] = torch.zeros((case["freqs"], p.nnz), dtype=torch.complex128, device="cuda")
        s["rhs"] = torch.zeros((case["freqs"], rows), dtype=torch.complex128, device="cuda")
        return s
    s["terms"] = _point_terms(case["dim"]) if case["coef"] == "point" else p.terms()
    if case["bound"]:
        F.check(F.lib().fg_plan_bind_terms(s["plan"].ptr, s["terms"][0], s["terms"][1], 0.0))
    if case["host"]:
        s["values"], s["rhs"] = np.zeros(p.nnz, np.complex128), np.zeros(rows, np.complex128)
    else:
        s["values"] = torch.zeros(p.nnz, dtype=torch.complex128, device="cuda")
        s["rhs"] = torch.zeros(rows, dtype=torch.complex128, device="cuda")
    return s


def run(s):
    do = s["case"]["do"]
    if do == "batch":
        s["batch"].run(*s["pointers"])
    elif do == "symbolic":
        F = _femg()
        ai, aj = F.pattern_build(s["edof"], s["etype"], s["rows"])
        numbers = F.hilbert_numbering(s["case"]["dim"], s["bbox"], s["xyz"], s["types"], s["numbers"])
        return ai.view(np.int64), aj.view(np.int64), numbers.view(np.int64)
    elif do == "sweep":
        s["plan"].assemble_multi_freq(s["omegas"], s["precision"], values=s["values"].data_ptr(), rhs=s["rhs"].data_ptr())
    else:
        v, r = s["values"], s["rhs"]
        if not s["case"]["host"]:
            v, r = v.data_ptr(), r.data_ptr()
        s["plan"].assemble(s["precision"], values=v, rhs=r, bound=s["case"]["bound"],
                           terms=None if s["case"]["bound"] else s["terms"])
    return s["values"], s["rhs"]


# ---------------------------------------------------------------------- work

def _cells(dim, m):
    return 6 * m ** 3 if dim == 3 else 2 * m * m


def _functions(field, dim, p):
    if field == "hcurl":
        return (p + 1) * (p + 3) * (p + 4) // 2 if dim == 3 else (p + 1) * (p + 3)
    return (p + 1) * (p + 2) * (p + 3) // 6 if dim == 3 else (p + 1) * (p + 2) // 2


def _size(field, dim, p, m):
    """(elements, functions an element, rows, nonzeros, nodes) of one component on the mesh, nothing fixed."""
    nodes, n = (m + 1) ** dim, _functions(field, dim, p)
    if dim == 2:
        count = [nodes, 3 * m * m + 2 * m, 2 * m * m, 0]
    else:
        count = [nodes, 7 * m ** 3 + 9 * m ** 2 + 3 * m, 12 * m ** 3 + 6 * m ** 2, 6 * m ** 3]
    if field == "hcurl":  # functions on a node, an edge, a face, a cell
        own = [0, p + 1, p * (p + 1), (p - 1) * p * (p + 1) // 2]
    else:
        own = [1, p - 1, (p - 1) * (p - 2) // 2, (p - 1) * (p - 2) * (p - 3) // 6]
    # pairs of functions that meet on a simplex and on none of its sides
    own, below = own[:dim + 1], [[1], [2, 1], [3, 3, 1], [4, 6, 4, 1]]
    pairs = []
    for d in range(dim + 1):
        closed = sum(b * o for b, o in zip(below[d], own))
        pairs.append(closed ** 2 - sum(b * q for b, q in zip(below[d], pairs)))
    return (count[dim], n, sum(c * o for c, o in zip(count, own)), sum(c * q for c, q in zip(count, pairs)), nodes)


def _assembly_work(case, complex_ke, outputs):
    """Coordinates, connectivity, element DOF map and a coefficient an element read once, values and right-hand sides
    written once; the products of an upper triangle by the factorisation over the reference tensors."""
    field, dim = case["field"], case["dim"]
    E, n, rows, nnz, nodes = _size(field, dim, case["order"], case["m"])
    c = 3 if field == "navier" else 1
    nn = n if field == "lagrange" else dim + 1
    read = 24 * nodes + 4 * nn * E + 4 * c * n * E + 16 * E
    factors = {"navier": 10 * 9, "hcurl": 12}.get(field, 7)
    return {"bytes": read + outputs * 16 * (c * c * nnz + c * rows),
            "flops": 2 * factors * (n * (n + 1) // 2) * E * (2 if complex_ke else 1)}


def work(case):
    if case["do"] == "batch":
        each = [_assembly_work(dict(field="h1", dim=3, order=p, m=m), False, 1) for p, m, _ in _mix(case)]
        return {k: sum(e[k] for e in each) for k in ("bytes", "flops")}
    if case["do"] == "symbolic":
        E, n, rows, nnz, _ = _size(case["field"], case["dim"], case["order"], case["m"])
        return {"bytes": E * n * 12 + 8 * (rows + nnz) + rows * (12 + 4 + 8 + 8), "flops": 0}
    return _assembly_work(case, case.get("coef") == "point", case.get("freqs", 1))


# --------------------------------------------------------------------- exact


def _element(a, coef, e0, e1, dev):
    """Element matrices (complex) and vectors of elements e0..e1 by the quadrature sum, in 64 bits.
    coef(e0, e1, x) gives the coefficients at the points x [e, q, 3]: a dict of [e, q] tensors."""
    T = lambda v: torch.as_tensor(np.ascontiguousarray(v), device=dev)  # noqa: E731
    X = T(a["xyz"])[T(a["enodes"][e0:e1])]  # [e, nodes, 3]
    J = torch.einsum("ekr,qkc->eqrc", X, T(a["geo_grad"]))  # dx_r / du_c
    if a["dim"] == 2:
        nrm = torch.linalg.cross(J[..., 0], J[..., 1])
        J[..., 2] = nrm / nrm.norm(dim=-1, keepdim=True)
    det, inv = torch.linalg.det(J), torch.linalg.inv(J)
    x = torch.einsum("ekr,qk->eqr", X, T(a["geo_val"]))
    c = coef(e0, e1, x)
    wd = (T(a["w"]) * det)[..., None]
    o = T(a["orient"][e0:e1].astype(np.int64))
    val, der = T(a["bval"])[o], T(a["bgrad"])[o]  # [e, q, n(, 3)], [e, q, n, 3]
    e, q, n = der.shape[:3]

    def pair(u, v):  # sum over points (and components): [e, q, n, ...] twice
        return torch.bmm(u.movedim(2, 1).reshape(e, n, -1), v.movedim(2, 1).reshape(e, n, -1).transpose(1, 2))

    if a["form"] == 1:
        C = torch.einsum("eqrc,eqnc->eqnr", J, der) / det[..., None, None]
        P = torch.einsum("eqcr,eqnc->eqnr", inv, val)
        return pair(C, C * (wd * c["grad"][..., None])[..., None]) + pair(P, P * (wd * c["mass"][..., None])[..., None]), None
    G = torch.einsum("eqcr,eqnc->eqnr", inv, der)
    if a["mult"] == 3:
        lam, mu, cm = ((wd[..., 0] * c[k])[..., None] for k in ("lam", "mu", "mass"))
        K = torch.zeros((e, n, 3, n, 3), dtype=torch.float64, device=dev)
        dot = pair(G, G * mu[..., None]) + pair(val, val * cm)
        for s in range(3):
            for t in range(3):
                K[:, :, s, :, t] = pair(G[..., s], G[..., t] * lam) + pair(G[..., t], G[..., s] * mu) + (dot if s == t else 0.0)
        return K.reshape(e, 3 * n, 3 * n), None
    parts = []
    for part in ((lambda z: z.real), (lambda z: z.imag)):
        g, m = (part(torch.as_tensor(c[k] + 0j, device=dev)) for k in ("grad", "mass"))
        parts.append(pair(G, G * (wd[..., 0] * g)[..., None, None]) + pair(val, val * (wd * m[..., None])))
        if not any(torch.is_tensor(v) and v.is_complex() for v in c.values()):
            break
    Ke = parts[0] if len(parts) == 1 else torch.complex(*parts)
    be = None if "source" not in c else ((wd[..., 0] * c["source"])[..., None] * val).sum(1)
    return Ke, be


def _assembled(a, coef, dev):
    """CSR values and right-hand side, complex, of the element sums."""
    T = lambda v: torch.as_tensor(np.ascontiguousarray(v), device=dev)  # noqa: E731
    rows, ai = int(a["n_rows"]), T(a["ai"].view(np.int64))
    keys = torch.repeat_interleave(torch.arange(rows, device=dev), ai[1:] - ai[:-1]) * rows + T(a["aj"].view(np.int64))
    values = torch.zeros((2, keys.numel()), dtype=torch.float64, device=dev)
    rhs = torch.zeros((2, rows), dtype=torch.float64, device=dev)
    uD = T(a["dirichlet"]) if a["n_fixed"] else torch.zeros(1, dtype=torch.complex128, device=dev)
    n, step = a["edof"].shape[1], max(1, int(3e7 / (a["edof"].shape[1] * (a["edof"].shape[1] + 4 * a["nq"]))))

    def add(to, at, v):
        to[0].index_add_(0, at, v.real if v.is_complex() else v)
        if v.is_complex():
            to[1].index_add_(0, at, v.imag)

    for e0 in range(0, a["E"], step):
        e1 = min(a["E"], e0 + step)
        Ke, be = _element(a, coef, e0, e1, dev)
        idx, free = T(a["edof"][e0:e1].view(np.int64)), T(a["etype"][e0:e1]) != 1
        both = free[:, :, None] & free[:, None, :]
        at = torch.searchsorted(keys, (idx[:, :, None] * rows + idx[:, None, :])[both])
        add(values, at, Ke[both])
        lift = torch.where(free[:, :, None] & ~free[:, None, :], Ke * uD[torch.where(free, 0, idx)][:, None, :], 0.0).sum(2)
        add(rhs, idx[free], (lift if be is None else lift + be)[free])
    assert n == Ke.shape[1]
    return torch.complex(values[0], values[1]), torch.complex(rhs[0], rhs[1])


def _per_element(p, t, second=False, const=None):
    """The real per-element array of term t's coefficient, or the constant."""
    ex = p.terms()[0][t].coef2 if second else p.terms()[0][t].coef
    return np.ctypeslib.as_array(ex.elem_values[0], shape=(p.E, 2))[:, 0].copy() if ex.n_arrays else np.full(p.E, const)


def exact(case, seed):
    if case["do"] == "symbolic":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["do"] == "batch":
        F, out = _femg(), ([], [])
        for cfg in _batch_configs(case, seed):
            p = F.Problem(cfg)
            for to, v in zip(out, _assembled(p.arrays(), lambda e0, e1, x: {"grad": 1.0, "mass": -cfg.k ** 2}, dev)):
                to.append(v)
        return out
    p = _problem(case, seed)
    a = p.arrays()
    spread = lambda v, e0, e1, x: torch.as_tensor(v[e0:e1], device=dev)[:, None].expand(x.shape[:2])  # noqa: E731
    if case["field"] == "navier":
        lam, mu = _per_element(p, 0), _per_element(p, 0, True)

        def stiff(e0, e1, x, mass):
            return {"lam": spread(lam, e0, e1, x), "mu": spread(mu, e0, e1, x), "mass": torch.full(x.shape[:2], mass, dtype=x.dtype, device=dev)}

        if case["do"] == "assemble":
            return _assembled(a, lambda e0, e1, x: stiff(e0, e1, x, -25.0), dev)
        Kv, Kr = _assembled(a, lambda e0, e1, x: stiff(e0, e1, x, 0.0), dev)
        Mv, Mr = _assembled(a, lambda e0, e1, x: {k: v * 0.0 if k != "mass" else v for k, v in stiff(e0, e1, x, 1.0).items()}, dev)
        w2 = torch.as_tensor(_omegas(case, seed) ** 2, device=dev)[:, None]
        return Kv - w2 * Mv, Kr - w2 * Mr
    if case.get("coef") == "point":
        def coef(e0, e1, x):
            X, Y = x[..., 0], x[..., 1]
            return {"grad": 1.0 + 0.5 * X + 0.2j * Y ** 2, "mass": -K * K * (1.0 + 0.3j * X * Y), "source": torch.exp(-X) * (1.0 + 1j * Y)}
    else:
        mass = _per_element(p, 1, const=-K * K)

        def coef(e0, e1, x):
            c = {"grad": torch.ones(x.shape[:2], dtype=x.dtype, device=dev), "mass": spread(mass, e0, e1, x)}
            if case.get("dirichlet"):  # 1 inside the disk, one half on its edge
                c["source"] = -torch.heaviside(0.01 - (x[..., 0] - 0.5) ** 2 - (x[..., 1] - 0.5) ** 2, torch.full_like(x[..., 0], 0.5))
            return c
    v, r = _assembled(a, coef, dev)
    if case["do"] == "sweep":  # no term with a time derivative: every frequency's system is the same
        return v.expand(case["freqs"], -1).contiguous(), r.expand(case["freqs"], -1).contiguous()
    return v, r

"""The lean kernels of the CSR reduction, real and complex, with every column
stored and with upper storage, into outputs and added to them, over the shapes
of element rows, against the oracle (1e-12 in FP64, 1e-6 in mixed precision);
and batches whose problems need different kernels."""
import numpy as np
import pytest

from test_gpu_quadrature_blocks import terms
from test_gpu_reduction_shapes import rel, shapes, tolerance

pytestmark = pytest.mark.gpu

NAMES = ["tri_3", "tet_4", "tri_6", "hcurl_tri_8", "tet_10", "tri_15", "tet_20", "hcurl_tet_20", "tri_28", "tet_35", "navier_12",
         "navier_30", "navier_60"]


@pytest.mark.parametrize("path", ["fp64", "mixed"])
@pytest.mark.parametrize("how", ["real", "complex"])
@pytest.mark.parametrize("upper", [0, 1])
@pytest.mark.parametrize("name", NAMES)
def test_modes(femg, oracle, cuda, name, upper, how, path):
    torch = cuda
    cfg = shapes(femg)[name][0]
    cfg.upper = upper
    prob = femg.Problem(cfg)
    t = terms(femg, prob, how)
    want, _ = oracle.assemble(prob.arrays(), *t)
    plan = prob.plan()
    v, b = plan.assemble(path, terms=t)
    assert rel(v, want) <= tolerance(path) and np.all(b == 0)
    plan.set_accumulate(True)
    rng = np.random.default_rng(5)
    before = rng.standard_normal(prob.nnz) + 1j * rng.standard_normal(prob.nnz)
    dv = torch.from_numpy(before.copy()).cuda()
    db = torch.full((len(b),), 2.0, dtype=torch.complex128, device="cuda")
    plan.assemble(path, values=dv.data_ptr(), rhs=db.data_ptr(), terms=t)
    torch.cuda.synchronize()
    assert rel(dv.cpu().numpy(), before + want) <= tolerance(path) and torch.all(db == 2.0)
    plan.close()


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("how", ["upper", "upper_and_full", "source"])
def test_batch_of_different_modes(femg, oracle, cuda, how, mixed):
    H = femg.FG_SPACE_HIERARCHICAL_H1
    probs = [femg.Problem(femg.config(dim=2, m=6 + k, mesh_order=1, space=H, order=2, gauss=4, k=5.0, seed=k + 1,
                                      upper=int(how == "upper" or (how == "upper_and_full" and k == 1)),
                                      source=int(how == "source" and k == 1))) for k in range(3)]
    batch = femg.Batch([p.plan() for p in probs], mixed=mixed)
    for _ in range(2):
        values, rhs = batch.run(rhs=[np.zeros(int(p.sys.n_rows), np.complex128) for p in probs])
        for p, v, b in zip(probs, values, rhs):
            want_v, want_b = oracle.assemble(p.arrays(), *p.terms())
            assert rel(v, want_v) <= tolerance("mixed" if mixed else "fp64")
            assert rel(b, want_b) <= 1e-12
    batch.close()

"""The condensed operator of small systems face by face (face_op_kernel in csrc/exa_kernels.cu): w = A v,
and inside GMRES y = P A v in the same launch, at every number of warps per face (blocks of 12 to 150
rows), face blocks of 3 to 25 rows, closed and periodic, in FP64 and with FP32 blocks.

The matvec is compared with the blocks the device holds, summed by numpy: sums of at most 300 terms in
FP64 on either side, 1e-13 of the largest entry.  GMRES is checked by its own claim: the preconditioned
residual of the returned x, formed by numpy, is within the tolerance (1e-6; rounding adds 1e-10)."""
import numpy as np
import pytest

from exasim_b200 import HDGSolver, build as B, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,n,p,mixed", [("cdsin2d", 3, 2, 0), ("cdsin2d", 5, 4, 1), ("ns2d", 4, 3, 0), ("ns2d", 5, 2, 0),
                                             ("convdiff3d", 3, 2, 0), ("convdiff3d", 3, 3, 1), ("convdiff3d", 3, 4, 0),
                                             ("convdiff3d", 5, 4, 1)])
def test_small_operator(tmp_path, model, n, p, mixed):
    import torch
    B.build([model])
    d = str(tmp_path / "datain")
    if model == "cdsin2d":
        cases.cdsin2d_quad(d, n=n, porder=p, kappa=0.1, theta=0.4, gmres_tol=1e-6)
    elif model == "ns2d":
        cases.ns2d_tgv_quad(d, n=n, porder=p, preconditioner=0, gmres_tol=1e-6, newton_tol=1e-12)
    else:
        cases.convdiff3d_hex(d, n=n, porder=p, gmres_tol=1e-6)
    s = HDGSolver(d, model)
    if model != "cdsin2d":
        s.set_time(0.0, 40.0)
        s.set("sdg", 41.0 * s.get("udg")[: s.sizes["n"] * s.sizes["ne"]])
    if mixed:
        s.set_precision(1)
    s.hdgGetQ()
    s.hdgAssembleLinearSystem()
    z = s.sizes
    m, ne, nf, ncf, ncu, N = z["m"], z["ne"], z["nf"], z["npf"] * z["ncu"], z["ncu"], z["ndofuhat"]
    H = s.get("H32" if mixed else "H").reshape(ne, m, m).transpose(0, 2, 1)
    con = (s.connectivity()[1].T[:, :, None] * ncu + np.arange(ncu)).reshape(ne, m)

    def matvec(v):
        w = np.zeros(N)
        np.add.at(w, con, np.einsum("eij,ej->ei", H, v[con]))
        return w

    v = np.random.default_rng(1).standard_normal(N)
    x = torch.tensor(v, dtype=torch.float64, device="cuda")
    w = torch.empty_like(x)
    s.evalMatVec(x.data_ptr(), w.data_ptr())
    ref = matvec(v)
    assert np.abs(w.cpu().numpy() - ref).max() < 1e-13 * np.abs(ref).max()
    s.evalMatVec(x.data_ptr(), x.data_ptr())  # in place
    assert np.abs(x.cpu().numpy() - ref).max() < 1e-13 * np.abs(ref).max()
    s.GMRES()
    b, sol = s.get("b"), s.get("x")

    def pre(r):
        t = torch.tensor(r, dtype=torch.float64, device="cuda")
        y = torch.empty_like(t)
        s.ApplyPreconditioner(t.data_ptr(), y.data_ptr())
        return y.cpu().numpy()

    res = np.linalg.norm(pre(b - matvec(sol))) / np.linalg.norm(pre(b))
    s.close()
    print(model, n, p, mixed, m, ncf, f"{res:.1e}")
    assert res < 1e-6 + 1e-10

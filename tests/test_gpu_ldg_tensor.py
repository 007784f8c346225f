"""The LDG residual of tensor-product hexahedra by sum factorization (csrc/exa_ldg_tp.cuh) against the
oracle's quadrature with the full shape tables, at every order that has an instance and one that has
none (p = 1), on closed and periodic cubes whose element count leaves a partly filled last block,
and the Jacobian product built on it.

Both form the same sums; the oracle's tables differ from the 1D ones by their own rounding (1e-15 to
1e-14 of the derivative entries), which the cancellation in the residual amplifies by |R terms| / |R|,
below 1e3 here: 1e-11.  The product divides the difference of two residuals by eps = 1e-3: 1e-8."""
import numpy as np
import pytest

from exasim_b200 import HDGSolver, build as B, cases
from oracle.ldg import LDGOracle
from oracle.models import MODELS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p,periodic", [(3, 1, True), (3, 2, True), (3, 3, True), (2, 2, False),
                                          (3, 3, False), (1, 3, False)])
def test_residual_and_product_match_oracle(tmp_path, n, p, periodic):
    import torch
    B.build(["euler3d"])
    d = str(tmp_path / "datain")
    cases.euler3d_vortex_hex(d, n=n, porder=p, hybrid=0, periodic=periodic)
    s, o = HDGSolver(d, "euler3d"), LDGOracle(d, MODELS["euler3d"]())
    rng = np.random.default_rng(n + 10 * p)
    u = o.udg[:, :o.ncu] * (1.0 + 1e-2 * rng.standard_normal(o.udg[:, :o.ncu].shape))
    sdg = 60.0 * u * (1.0 + 1e-2 * rng.standard_normal(u.shape))
    o.time, o.dtfactor, o.sdg = 0.01, 68.28427124746192, sdg
    o.sdgg = np.einsum("gj,jce->gec", o.shapegt[:, :, 0], sdg)
    ref = o.residual_ldg(u)
    s.set_time(o.time, o.dtfactor)
    s.set("sdg", sdg)
    s.set("udg", u)
    nrm = s.evalResidual()
    got = s.get("Ru")
    rel = np.linalg.norm(got - ref.ravel(order="F")) / np.linalg.norm(ref)
    v = rng.standard_normal(u.shape)
    x = torch.tensor(v.ravel(order="F"), dtype=torch.float64, device="cuda")
    w = torch.empty_like(x)
    s.evalMatVec(x.data_ptr(), w.data_ptr())
    wref = o.matvec_fd(u, ref, v).ravel(order="F")
    wrel = np.linalg.norm(w.cpu().numpy() - wref) / np.linalg.norm(wref)
    s.close()
    print(n, p, periodic, f"{rel:.1e} {wrel:.1e}")
    assert abs(nrm - np.linalg.norm(ref)) < 1e-11 * nrm
    assert rel < 1e-11
    assert wrel < 1e-8

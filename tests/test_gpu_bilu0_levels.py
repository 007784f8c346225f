"""The block ILU(0) application's level schedule (csrc/exa_bilu0.cpp, exa_bilu0_dev.cu) on sub-domains
larger than the other tests use: levels of many rows, levels cut at the buffers' limits (64 rows, 96
blocks: 4 x 4 x 4 hexahedra have levels of 56 rows and of more than 96 blocks), and blocks of 2 to 16
rows.  Against the oracle's sweeps row by row; the tolerance is that of the blocks' comparison in
test_gpu_bilu0.py, 1e-11 of the largest entry."""
import numpy as np
import pytest

from exasim_b200 import HDGSolver, build as B, cases
from oracle.hdg import HDGOracle
from oracle.models import MODELS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,n,p,cgp", [("poisson2d", 16, 1, (2, 16, 16, 8, 8, 0)),
                                           ("poisson2d", 12, 3, (2, 12, 12, 12, 12, 0)),
                                           ("ns2d", 4, 3, (2, 4, 4, 4, 4, 0)),
                                           ("convdiff3d", 4, 1, (3, 4, 4, 4, 4, 4, 4, 0)),
                                           ("convdiff3d", 4, 2, (3, 4, 4, 4, 4, 4, 2, 1))])
def test_apply_matches_oracle(tmp_path, model, n, p, cgp):
    import torch
    B.build([model])
    d = str(tmp_path / "datain")
    if model == "poisson2d":
        cases.poisson2d_quad(d, n=n, porder=p, preconditioner=2, cartgridpart=cgp)
    elif model == "ns2d":
        cases.ns2d_tgv_quad(d, n=n, porder=p, preconditioner=2, block=4, periodic=False)
    else:
        cases.convdiff3d_hex(d, n=n, porder=p, nsteps=1, preconditioner=2, cartgridpart=cgp)
    s, o = HDGSolver(d, model), HDGOracle(d, MODELS[model]())
    if o.tdep:
        o.sdg = 41.0 * o.udg[:, :o.ncu]
        o.sdgg = np.einsum("gj,jce->gec", o.shapegt[:, :, 0], o.sdg)
        o.time, o.dtfactor = 0.01, 40.0
        s.set("sdg", o.sdg)
        s.set_time(o.time, o.dtfactor)
    s.hdgGetQ()
    o.get_q(o.udg, o.uh)
    s.hdgAssembleLinearSystem()
    o.assemble()
    o.build_precond()
    v = np.random.default_rng(5).standard_normal(s.sizes["ndofuhat"])
    x = torch.tensor(v, dtype=torch.float64, device="cuda")
    y = torch.empty_like(x)
    s.ApplyPreconditioner(x.data_ptr(), y.data_ptr())
    ref = o.apply_precond(v.reshape(o.ncu, o.npf, o.nf, order="F")).ravel(order="F")
    err = np.abs(y.cpu().numpy() - ref).max() / np.abs(ref).max()
    s.close()
    print(model, n, p, f"{err:.1e}")
    assert err < 1e-11

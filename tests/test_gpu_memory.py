"""Device memory of a context against the estimate that the server admits it by: at least what it holds,
and not so much more that contexts which fit are kept waiting.  The estimate bounds the number of faces
by those of all elements (up to twice the true one) and adds 16 MB, so: above the bytes held by at most
the Krylov basis and the preconditioner's face blocks once more, and 24 MB."""
import pytest

from exasim_b200 import build as B, cases, read_datain
from exasim_b200.serve import Server

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,n,p,precision", [("convdiff3d", 6, 4, 0), ("convdiff3d", 6, 4, 1), ("convdiff3d", 8, 2, 0),
                                                 ("convdiff3d", 3, 1, 0), ("euler3d", 4, 3, 0), ("euler3d", 4, 3, 1),
                                                 ("euler3d", 6, 2, 0), ("ns2d", 16, 3, 0), ("cdsin2d", 40, 4, 0),
                                                 ("poisson2d", 24, 3, 0), ("poisson2d", 24, 3, 1),
                                                 ("ns2d_ilu", 16, 3, 0), ("euler3d_ldg", 6, 3, 0)])
def test_estimate_covers_what_is_held(tmp_path, model, n, p, precision):
    ilu, ldg, model = model.endswith("_ilu"), model.endswith("_ldg"), model.split("_")[0]
    B.build([model])
    d = str(tmp_path / "datain")
    if model == "poisson2d":
        cases.poisson2d_tri(d, n=n, porder=p)
    elif model == "cdsin2d":
        cases.cdsin2d_quad(d, n=n, porder=p, kappa=0.1)
    elif model == "convdiff3d":
        cases.convdiff3d_hex(d, n=n, porder=p, nsteps=1)
    elif model == "ns2d":
        cases.ns2d_tgv_quad(d, n=n, porder=p, nsteps=1, preconditioner=2 if ilu else 0)
    else:
        cases.euler3d_vortex_hex(d, n=n, porder=p, nsteps=1, hybrid=0 if ldg else 1)
    blobs = read_datain(d)
    with Server(model, slots=1) as srv:
        srv.wait(srv.submit(blobs, precision=precision))
        st = srv.stats()
    held, est = st["bytes_held"], st["peak_bytes_held"]
    nd = {"convdiff3d": 3, "euler3d": 3}.get(model, 2)
    ncu, restart = {"euler3d": 5, "ns2d": 4}.get(model, 1), {"ns2d": 100}.get(model, 50)
    quad = model != "poisson2d"
    ne = n**nd if quad else 2 * n * n
    ncf, nf = ncu * (p + 1) ** (nd - 1), ne * (2 * nd if quad else 3) / 2
    slack = 8 * nf * ncf * (restart + 7 + ncf) + (24 << 20)
    # the mixed form has freed its FP64 blocks by now, which are part of what it needs at most
    m = ncf * (2 * nd if quad else 3)
    npe = (p + 1) ** nd if quad else (p + 1) * (p + 2) // 2
    if ilu:  # face blocks: each face's own and those of the other faces of its elements, at most
        slack += 8 * 2 * nf * ncf * ncf * (1 + 2 * (2 * nd - 1))
    if precision:
        slack += 8 * ne * m * (m + npe * ncu)
    print(model, n, p, precision, held >> 20, est >> 20, int(slack) >> 20)
    assert held <= est <= held + slack

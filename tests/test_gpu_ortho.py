"""The Gram-Schmidt of GMRES (csrc/exa_ortho.cu) against modified Gram-Schmidt in numpy: restarted
GMRES on the assembled condensed system, at trace lengths on both sides of the limits of its forms
(one to eight CTAs of a cluster, the whole-GPU kernels with one and several rows per thread) and
restarts within and beyond a panel of 64 basis vectors.

Both runs do the same steps, so the iteration counts agree up to one step that lands on the
tolerance by rounding.  With equal counts the solutions differ by the rounding of the two runs
only: 1e-16 per operation, some 1e4 operations per entry and the condition of the preconditioned
system (below 1e4 here) leave 1e-8; one step more or less moves them within the solve's tolerance
times that condition."""
import numpy as np
import pytest
import scipy.sparse as sp

from exasim_b200 import HDGSolver, build as B, cases

pytestmark = pytest.mark.gpu


def mgs_gmres(op, b, restart, tol):
    x, its, nrm = np.zeros_like(b), 0, np.linalg.norm(b)
    while its < 4000:
        r = b - op(x) if its else b.copy()
        beta = np.linalg.norm(r)
        if beta / nrm < tol:
            break
        V, H = np.zeros((restart + 1, b.size)), np.zeros((restart + 1, restart))
        V[0] = r / beta
        for j in range(restart):
            w = op(V[j])
            for k in range(j + 1):
                H[k, j] = V[k] @ w
                w = w - H[k, j] * V[k]
            H[j + 1, j] = np.linalg.norm(w)
            V[j + 1] = w / H[j + 1, j]
            its += 1
            e = np.zeros(j + 2)
            e[0] = beta
            y, res = np.linalg.lstsq(H[:j + 2, :j + 1], e, rcond=None)[:2]
            if np.linalg.norm(H[:j + 2, :j + 1] @ y - e) / nrm < tol:
                return x + y @ V[:j + 1], its
        x = x + y @ V[:restart]
    return x, its


# trace lengths 120 (one CTA), 720 (two), 1680 (four), 10080 (eight), 16560 (past the cluster's
# limit of 16384), 82500 (two rows per thread; a stage system of the 3D model)
@pytest.mark.parametrize("model,n,p,restart,tol", [("cdsin2d", 4, 2, 50, 1e-10), ("cdsin2d", 8, 4, 50, 1e-10),
                                                   ("cdsin2d", 14, 3, 70, 1e-10), ("cdsin2d", 35, 3, 130, 1e-8),
                                                   ("cdsin2d", 45, 3, 70, 1e-8), ("convdiff3d", 10, 4, 50, 1e-10)])
def test_gmres_matches_numpy_mgs(tmp_path, model, n, p, restart, tol):
    B.build([model])
    d = str(tmp_path / "datain")
    if model == "cdsin2d":
        cases.cdsin2d_quad(d, n=n, porder=p, kappa=0.1, theta=0.7, gmres_tol=tol, restart=restart)
    else:
        cases.convdiff3d_hex(d, n=n, porder=p, gmres_tol=tol, restart=restart)
    s = HDGSolver(d, model)
    if model == "convdiff3d":
        s.set_time(0.0, 229.0)
    s.hdgGetQ()
    s.hdgAssembleLinearSystem()
    its, _ = s.GMRES()
    x, b, z = s.get("x"), s.get("b"), s.sizes
    m, ne, ncf, nf, N = z["m"], z["ne"], z["npf"], z["nf"], z["ndofuhat"]
    H = s.get("H").reshape(ne, m, m).transpose(0, 2, 1)
    con = s.connectivity()[1].T
    P = s.get("P").reshape(nf, ncf, ncf).transpose(0, 2, 1)
    s.close()
    A = sp.csr_matrix((H.ravel(), (np.repeat(con, m, axis=1).ravel(), np.tile(con, (1, m)).ravel())), shape=(N, N))
    pre = lambda v: np.einsum("fij,fj->fi", P, v.reshape(nf, ncf)).ravel()
    ref, rits = mgs_gmres(lambda v: pre(A @ v), pre(b), restart, tol)
    rel = np.linalg.norm(x - ref) / np.linalg.norm(ref)
    print(n, p, N, restart, its, rits, f"{rel:.1e}")
    assert abs(its - rits) <= 1, (its, rits)
    assert rel < (1e-8 if its == rits else 1e4 * tol), rel

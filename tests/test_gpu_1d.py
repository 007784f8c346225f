"""A scalar model without q on a 1D mesh, whose faces have one node and one unknown: the condensed blocks,
the element solves and the Newton solution against the oracle.  Sums of at most 10 terms and inverses of
blocks of condition 1e2: 1e-12; the solution to the solve's 1e-10."""
import importlib.util
import os

import numpy as np
import pytest

from exasim_b200 import HDGSolver, build as B, inputs as I
from oracle.hdg import HDGOracle
from oracle.models import _PointModel

MODEL = "burgers1d"


def flux(uq, mu):
    return mu[0] * uq[0] + uq[0] * uq[0] / 2


class Burgers1D(_PointModel):
    """u_t + (c u + u^2 / 2)_x = 0, boundary flux f(u) . n + tau (u - uhat)."""

    def __init__(self):
        self.nd, self.ncu, self.nc = 1, 1, 1

    @staticmethod
    def _flux(uq, param):
        return flux(uq.T, param)[:, None, None]

    def initu(self, x, param):
        return 1.0 + 0.3 * np.sin(2 * np.pi * x)


def datain(d, ne, p):
    grid = I.Grid(p=np.sort(np.linspace(0, 1, ne + 1) ** 1.1)[None], t=np.array([np.arange(ne), np.arange(1, ne + 1)]),
                  elemtype=1)
    master = I.make_master(1, 1, p, 2 * p)
    master.perm = master.perm.reshape(1, 2)  # one node on each of the two faces
    app = I.PDEApp(nd=1, ncu=1, model="ModelC", NewtonIter=20, NewtonTol=1e-9, GMRESiter=200, GMRESrestart=50,
                   GMREStol=1e-10, RBdim=0, ppdegree=1, tau=[2.0], torder=1, nstage=1, dt=[0.05],
                   physicsparam=[0.5], externalparam=[0.0, 0.0])
    os.makedirs(d, exist_ok=True)
    I.write_app_bin(os.path.join(d, "app.bin"), app)
    I.write_master_bin(os.path.join(d, "master.bin"), master)
    I.write_mesh_bin(os.path.join(d, "mesh.bin"), grid, master, I.assign_bf(grid, [lambda x: True], [1]), [1])
    I.write_sol_bin(os.path.join(d, "sol.bin"), I.dgnodes(grid, master), nc=1, ncu=1)


def oracle(d):
    o = HDGOracle(d, Burgers1D())
    o.time, o.dtfactor = 0.0, 20.0
    o.sdg = 20.0 * o.udg * 1.01
    o.sdgg = np.einsum("gj,jce->gec", o.shapegt[:, :, 0], o.sdg)
    return o


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    spec = importlib.util.spec_from_file_location("make_models", os.path.join(B.MODELS, "make_models.py"))
    mm = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mm)
    mm.HERE = src = str(tmp_path_factory.mktemp("models"))
    import sympy as sp
    mm.write_symbolic_case(MODEL, 1, 1, False, 1, lambda uq, x, mu: [[flux(uq, mu)]], lambda uq, x, mu: [sp.Integer(0)],
                           lambda uq, x, mu, uh, nl, t0: mm._tau_fbou([[flux(uq, mu)]], uq, uh, nl, t0, 1, 1),
                           lambda x, mu: [1 + sp.Rational(3, 10) * sp.sin(2 * sp.pi * x[0])])
    B.build(sources={MODEL: os.path.join(src, MODEL)})
    return MODEL


def test_oracle_runs_in_1d(tmp_path):
    d = str(tmp_path / "datain")
    datain(d, 5, 3)
    o = oracle(d)
    H, Rh, F, Ru = o.assemble()
    assert H.shape == (2, 2, 5) and F.shape == (4, 2, 5) and np.isfinite(H).all()


@pytest.mark.gpu
@pytest.mark.parametrize("ne,p", [(1, 1), (7, 3), (64, 4)])
def test_blocks_and_solution_match_oracle(tmp_path, library, ne, p):
    d = str(tmp_path / "datain")
    datain(d, ne, p)
    o, s = oracle(d), HDGSolver(d, library)
    s.set_time(o.time, o.dtfactor)
    s.set("sdg", o.sdg)
    err = lambda a, b: np.abs(a - np.asarray(b).ravel(order="F")).max() / np.abs(b).max()
    assert err(s.get("udg"), o.udg) < 1e-14
    H, Rh, F, Ru = o.assemble()
    s.hdgAssembleLinearSystem()
    for name, ref in (("H", H), ("F", F), ("Ru", Ru), ("Rh", Rh)):
        assert err(s.get(name), ref) < 1e-12, name
    s.NewtonSolver()
    o.newton()
    assert err(s.get("uh"), o.uh) < 1e-9 and err(s.get("udg"), o.udg) < 1e-9
    s.close()

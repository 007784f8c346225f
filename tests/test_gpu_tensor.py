"""Tensor-product elements (quadrilaterals, hexahedra) at every order with an instance and one beside
them (p = 1), scalar and systems, with and without q, closed and periodic: q recovery, the residual and
the assembled blocks against the oracle's dense quadrature.

Tolerances: q and the residual vectors differ by the rounding of sums of up to 1e3 terms and of the
element tables (1e-14 of the derivative entries), against terms that cancel to 1e-2 of their size:
1e-11 of the largest entry; the condensed blocks and D^-1 F pass through the explicit inverse of
blocks of condition 1e3: 5e-12 as in the reference comparison, 2e-11 for p = 4."""
import numpy as np
import pytest

from exasim_b200 import HDGSolver, build as B, cases
from oracle.hdg import HDGOracle
from oracle.models import MODELS

pytestmark = pytest.mark.gpu
CASES = [("cdsin2d", 3, p) for p in (1, 2, 3, 4)] + [("convdiff3d", 2, p) for p in (1, 2, 3, 4)] + \
        [("ns2d", 3, p) for p in (2, 3, 4)] + [("ns2d_closed", 3, 3), ("euler3d", 3, 2), ("euler3d", 2, 3)]


@pytest.mark.parametrize("model,n,p", CASES)
def test_residual_and_blocks_match_oracle(tmp_path, model, n, p):
    d = str(tmp_path / "datain")
    lib = "ns2d" if model == "ns2d_closed" else model
    B.build([lib])
    if lib == "cdsin2d":
        cases.cdsin2d_quad(d, n=n, porder=p, kappa=0.05, theta=0.6)
    elif lib == "convdiff3d":
        cases.convdiff3d_hex(d, n=n, porder=p, nsteps=1)
    elif lib == "ns2d":
        cases.ns2d_tgv_quad(d, n=n, porder=p, preconditioner=0, periodic=model == "ns2d")
    else:
        cases.euler3d_vortex_hex(d, n=n, porder=p, periodic=n > 2)
    s, o = HDGSolver(d, lib), HDGOracle(d, MODELS[lib]())
    rng = np.random.default_rng(p)
    udg, uh = o.udg.copy(), o.uh.copy()
    udg[:, :o.ncu] = udg[:, :o.ncu] * (1 + 1e-2 * rng.standard_normal(udg[:, :o.ncu].shape)) + 1e-3
    uh = uh * (1 + 1e-2 * rng.standard_normal(uh.shape)) + 1e-3
    s.set("udg", udg)
    s.set("uh", uh)
    o.udg, o.uh = udg.copy(), uh.copy()
    if o.tdep:
        o.sdg = 40.0 * udg[:, :o.ncu]
        o.sdgg = np.einsum("gj,jce->gec", o.shapegt[:, :, 0], o.sdg)
        o.time, o.dtfactor = 0.01, 45.0
        s.set("sdg", o.sdg)
        s.set_time(o.time, o.dtfactor)
    s.hdgGetQ()
    if o.ncq:
        o.get_q(o.udg, o.uh)
    err = lambda a, b: np.abs(a - np.asarray(b).ravel(order="F")).max() / np.abs(b).max()
    e = {"udg": err(s.get("udg"), o.udg)}
    s.set("udg", o.udg)
    s.hdgAssembleResidual()
    r = o.residual()
    Ru, Rh = np.asarray(r[0]), np.asarray(r[1])
    e["Ru"], e["Rh"] = err(s.get("Ru"), Ru), err(s.get("Rh"), Rh)
    s.hdgAssembleLinearSystem()
    H, Rhc, F, Ruc = o.assemble()
    e["H"], e["F"] = err(s.get("H"), H), err(s.get("F"), F)
    s.close()
    print(model, n, p, {k: f"{v:.1e}" for k, v in e.items()})
    assert e["udg"] < 1e-11 and e["Ru"] < 1e-11 and e["Rh"] < 1e-11
    assert max(e["H"], e["F"]) < (2e-11 if p == 4 else 5e-12)


@pytest.mark.parametrize("off", [3e-14, 1e-9])
def test_tables_that_are_no_products_are_used_as_they_are(tmp_path, off):
    """A master file whose element tables differ from the Kronecker products of its 1D ones by more than
    rounding: q and the residual are those of the file's tables (sums of 1e3 terms in another order: 2e-12 of
    the largest entry), not of the products, which 3e-14 would put ten times as far off."""
    from exasim_b200 import inputs as I
    B.build(["convdiff3d"])
    d = str(tmp_path / "datain")
    cases.convdiff3d_hex(d, n=2, porder=4, nsteps=1)
    m = I.make_master(3, 1, 4, 8)
    rng = np.random.default_rng(5)
    shap = m.shapegt + off * np.abs(m.shapegt).max() * rng.uniform(-1, 1, m.shapegt.shape)
    m.shapegt, m.shapegw = I._shapes_t_w(np.transpose(shap, (1, 0, 2)), m.gwe, 4)
    I.write_master_bin(d + "/master.bin", m)
    s, o = HDGSolver(d, "convdiff3d"), HDGOracle(d, MODELS["convdiff3d"]())
    udg, uh = rng.standard_normal(o.udg.shape), rng.standard_normal(o.uh.shape)
    o.udg, o.uh = udg.copy(), uh.copy()
    o.time, o.dtfactor = 0.01, 45.0
    o.sdg = 40.0 * udg[:, :1]
    o.sdgg = np.einsum("gj,jce->gec", o.shapegt[:, :, 0], o.sdg)
    s.set("udg", udg)
    s.set("uh", uh)
    s.set("sdg", o.sdg)
    s.set_time(o.time, o.dtfactor)
    s.hdgGetQ()
    o.get_q(o.udg, o.uh)
    err = lambda a, b: np.abs(a - np.asarray(b).ravel(order="F")).max() / np.abs(b).max()
    e = {"udg": err(s.get("udg"), o.udg)}
    s.set("udg", o.udg)
    s.hdgAssembleResidual()
    Ru, Rh = o.residual()[:2]
    e["Ru"], e["Rh"] = err(s.get("Ru"), Ru), err(s.get("Rh"), Rh)
    s.close()
    print(off, {k: f"{v:.1e}" for k, v in e.items()})
    assert max(e.values()) < 2e-12

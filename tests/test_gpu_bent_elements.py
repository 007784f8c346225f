"""The sum-factorized kernels on elements that are no boxes and whose neighbours meet them rotated
(tests/bent.py): q recovery, residual, condensed blocks, condensed operator, both forms, and the LDG residual
and product, against the oracle's dense quadrature.

Tolerances as on boxes (tests/test_gpu_tensor.py, test_gpu_qelim.py, test_gpu_ldg_tensor.py): 1e-11 for
sums, 2e-11 behind D^-1; FP32 5e-6 and 2e-4 behind D^-1; products by differences with a step of 1e-3 1e-8."""
import numpy as np
import pytest

from bent import bend, rotations
from exasim_b200 import HDGSolver, build as B, cases
from oracle.hdg import HDGOracle
from oracle.ldg import LDGOracle
from oracle.models import MODELS


def err(a, b):
    return np.abs(a - np.asarray(b).ravel(order="F")).max() / np.abs(b).max()


def write(d, model, n, p, **kw):
    if model == "cdsin2d":
        cases.cdsin2d_quad(d, n=n, porder=p, kappa=0.05, theta=0.6)
    elif model == "convdiff3d":
        cases.convdiff3d_hex(d, n=n, porder=p, nsteps=1)
    elif model == "ns2d":
        cases.ns2d_tgv_quad(d, n=n, porder=p, preconditioner=0, **kw)
    else:
        cases.euler3d_vortex_hex(d, n=n, porder=p, **kw)


def state(s, o, p):
    """The same perturbed state, stage source and time in both."""
    rng = np.random.default_rng(p)
    o.udg[:, :o.ncu] = o.udg[:, :o.ncu] * (1 + 1e-2 * rng.standard_normal(o.udg[:, :o.ncu].shape)) + 1e-3
    o.uh = o.uh * (1 + 1e-2 * rng.standard_normal(o.uh.shape)) + 1e-3
    s.set("udg", o.udg)
    s.set("uh", o.uh)
    if o.tdep:
        o.sdg = 40.0 * o.udg[:, :o.ncu]
        o.sdgg = np.einsum("gj,jce->gec", o.shapegt[:, :, 0], o.sdg)
        o.time, o.dtfactor = 0.01, 45.0
        s.set("sdg", o.sdg)
        s.set_time(o.time, o.dtfactor)


def test_meshes_are_bent_and_rotated(tmp_path, monkeypatch):
    assert len(rotations(2)) == 4 and len(rotations(3)) == 24
    bend(monkeypatch)
    d = str(tmp_path / "datain")
    write(d, "convdiff3d", 3, 2)
    o = HDGOracle(d, MODELS["convdiff3d"]())
    X = np.abs(o.Xx)                                                    # [nge, nd nd, ne]
    assert o.jac.min() > 0 and np.ptp(o.jac, axis=0).min() > 1e-2 * o.jac.mean()
    assert X[:, [1, 2, 3, 5, 6, 7]].mean() > 0.05 * X[:, [0, 4, 8]].mean()
    e2, l2 = o.f2e[2], o.f2e[3]
    met = {tuple(o.elemcon.reshape(o.npf, o.nfe, -1, order="F")[:, l, e] - o.npf * f)
           for f, (e, l) in enumerate(zip(e2, l2)) if e >= 0}
    assert len(met) == 4                                                # all ways two faces can meet


@pytest.mark.gpu
@pytest.mark.parametrize("model,n,p", [("cdsin2d", 4, 2), ("cdsin2d", 3, 3), ("cdsin2d", 3, 4), ("convdiff3d", 3, 2),
                                       ("convdiff3d", 2, 3), ("convdiff3d", 2, 4), ("ns2d", 4, 2), ("ns2d", 3, 3),
                                       ("ns2d", 3, 4), ("euler3d", 3, 2), ("euler3d", 3, 3)])
def test_residual_and_blocks_match_oracle(tmp_path, monkeypatch, model, n, p):
    import torch
    bend(monkeypatch, seed=n + p)
    B.build([model])
    d = str(tmp_path / "datain")
    write(d, model, n, p)
    s, o = HDGSolver(d, model), HDGOracle(d, MODELS[model]())
    state(s, o, p)
    s.hdgGetQ()
    if o.ncq:
        o.get_q(o.udg, o.uh)
    e = {"udg": err(s.get("udg"), o.udg)}
    s.set("udg", o.udg)
    s.hdgAssembleResidual()
    Ru, Rh = o.residual()[:2]
    e["Ru"], e["Rh"] = err(s.get("Ru"), Ru), err(s.get("Rh"), Rh)
    s.hdgAssembleLinearSystem()
    H, Rhc, F, Ruc = o.assemble()
    b = {k: err(s.get(k), v) for k, v in (("H", H), ("F", F), ("K", o.K), ("Ru", Ruc), ("Rh", Rhc))}
    if model == "convdiff3d":
        ref = o._volume(o.udg)[2] + o._faces(o.udg, o.uh)["Dface"][:, :, :, :, 1:]
        e["B"] = err(s.get("B"), ref[:, :, :, 0].transpose(0, 1, 3, 2))
    v = np.random.default_rng(1).standard_normal(o.uh.size)
    x = torch.tensor(v, dtype=torch.float64, device="cuda")
    w = torch.empty_like(x)
    s.evalMatVec(x.data_ptr(), w.data_ptr())
    b["Av"] = err(w.cpu().numpy(), o.matvec(v.reshape(o.uh.shape, order="F")))
    s.close()
    print(model, n, p, {k: f"{v:.1e}" for k, v in {**e, **b}.items()})
    assert max(e.values()) < 1e-11 and max(b.values()) < 2e-11


@pytest.mark.gpu
@pytest.mark.parametrize("model,n,p", [("convdiff3d", 3, 2), ("convdiff3d", 5, 3), ("convdiff3d", 3, 4), ("cdsin2d", 3, 3),
                                       ("euler3d", 3, 2)])
def test_mixed_blocks_match_oracle(tmp_path, monkeypatch, model, n, p):
    bend(monkeypatch, seed=n + p)
    B.build([model])
    d = str(tmp_path / "datain")
    write(d, model, n, p)
    s, o = HDGSolver(d, model), HDGOracle(d, MODELS[model]())
    s.set_precision(1)
    state(s, o, p)
    if o.ncq:
        o.get_q(o.udg, o.uh)
        s.set("udg", o.udg)
    s.hdgAssembleLinearSystem()
    H, Rh, F, Ru = o.assemble()
    e = {k: err(s.get(k), v) for k, v in (("K32", o.K), ("H32", H), ("F32", F), ("Rh", Rh), ("Ru", Ru))}
    s.close()
    print(model, n, p, {k: f"{v:.1e}" for k, v in e.items()})
    assert e.pop("K32") < 5e-6 and max(e.values()) < 2e-4


@pytest.mark.gpu
@pytest.mark.parametrize("n,p,periodic", [(3, 2, True), (3, 3, True), (3, 2, False), (2, 3, False), (1, 3, False)])
def test_ldg_residual_and_product_match_oracle(tmp_path, monkeypatch, n, p, periodic):
    import torch
    bend(monkeypatch, seed=n + p)
    B.build(["euler3d"])
    d = str(tmp_path / "datain")
    write(d, "euler3d", n, p, hybrid=0, periodic=periodic)
    s, o = HDGSolver(d, "euler3d"), LDGOracle(d, MODELS["euler3d"]())
    rng = np.random.default_rng(n + 10 * p)
    u = o.udg[:, :o.ncu] * (1.0 + 1e-2 * rng.standard_normal(o.udg[:, :o.ncu].shape))
    o.sdg = 60.0 * u * (1.0 + 1e-2 * rng.standard_normal(u.shape))
    o.sdgg = np.einsum("gj,jce->gec", o.shapegt[:, :, 0], o.sdg)
    o.time, o.dtfactor = 0.01, 68.28427124746192
    ref = o.residual_ldg(u)
    s.set_time(o.time, o.dtfactor)
    s.set("sdg", o.sdg)
    s.set("udg", u)
    s.evalResidual()
    rel = np.linalg.norm(s.get("Ru") - ref.ravel(order="F")) / np.linalg.norm(ref)
    v = rng.standard_normal(u.shape)
    x = torch.tensor(v.ravel(order="F"), dtype=torch.float64, device="cuda")
    w = torch.empty_like(x)
    s.evalMatVec(x.data_ptr(), w.data_ptr())
    wref = o.matvec_fd(u, ref, v).ravel(order="F")
    wrel = np.linalg.norm(w.cpu().numpy() - wref) / np.linalg.norm(wref)
    s.close()
    print(n, p, periodic, f"{rel:.1e} {wrel:.1e}")
    assert rel < 1e-11 and wrel < 1e-8

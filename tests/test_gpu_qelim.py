"""q elimination of scalar models on tensor-product hexahedra (csrc/exa_qelim_tp.cuh), from meshes with
several blocks per element to one, every order with an instance: the eliminated blocks K and H and the
block B, which is formed when it is read, against the oracle's dense products.

Tolerances: K and B are sums of at most 1e3 terms over tables of rounding 1e-14 of their largest entries:
1e-11 of the largest entry; H passes through D^-1 of condition 1e3: 2e-11."""
import numpy as np
import pytest
import torch

from exasim_b200 import ExaError, HDGSolver, build as B, cases
from oracle.hdg import HDGOracle
from oracle.models import MODELS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p", [(2, 2), (3, 3), (2, 4), (9, 2)])
def test_eliminated_blocks_match_oracle(tmp_path, n, p):
    d = str(tmp_path / "datain")
    B.build(["convdiff3d"])
    cases.convdiff3d_hex(d, n=n, porder=p, nsteps=1)
    s, o = HDGSolver(d, "convdiff3d"), HDGOracle(d, MODELS["convdiff3d"]())
    o.sdg = 40.0 * o.udg[:, :o.ncu]
    o.sdgg = np.einsum("gj,jce->gec", o.shapegt[:, :, 0], o.sdg)
    o.time, o.dtfactor = 0.01, 45.0
    s.set("sdg", o.sdg.ravel(order="F"))
    s.set_time(o.time, o.dtfactor)
    rng = np.random.default_rng(p)
    err = lambda a, b: np.abs(a - np.asarray(b).ravel(order="F")).max() / np.abs(b).max()

    def step():
        udg = rng.standard_normal(o.udg.shape)
        uh = rng.standard_normal(o.uh.shape)
        s.set("udg", udg)
        s.set("uh", uh)
        o.udg, o.uh = udg.copy(), uh.copy()
        s.hdgAssembleLinearSystem()
        H = o.assemble()[0]
        b = o._volume(udg)[2] + o._faces(udg, uh)["Dface"][:, :, :, :, 1:]
        return H, b[:, :, :, 0].transpose(0, 1, 3, 2)

    H, b = step()
    assert err(s.get("K"), o.K) < 1e-11 and err(s.get("H"), H) < 2e-11
    assert err(s.get("B"), b) < 1e-11
    ptr, size = s.field_ptr("B")  # the pointer shows B of each later assembly
    view = type("View", (), {"__cuda_array_interface__": {"data": (ptr, False), "shape": (size,), "typestr": "<f8",
                                                          "version": 3}})()
    H, b = step()
    torch.cuda.synchronize()
    assert err(torch.as_tensor(view, device="cuda").cpu().numpy(), b) < 1e-11
    H, b = step()
    s.set("B", 2.0 * s.get("B"))
    assert err(s.get("B"), 2.0 * b) < 1e-11  # what was written is read back
    assert err(s.get("H"), H) < 2e-11
    s.close()


@pytest.mark.parametrize("n,p", [(3, 2), (2, 3)])
def test_blocks_without_q_are_assembled_again(tmp_path, n, p):
    """Without q only the entries that couple a face with its own nodes are written again by an assembly:
    H, F and K of a second state, and after a caller wrote into K, against the oracle."""
    d = str(tmp_path / "datain")
    B.build(["euler3d"])
    cases.euler3d_vortex_hex(d, n=n, porder=p, periodic=n > 2)
    s, o = HDGSolver(d, "euler3d"), HDGOracle(d, MODELS["euler3d"]())
    o.sdg = 40.0 * o.udg[:, :o.ncu]
    o.sdgg = np.einsum("gj,jce->gec", o.shapegt[:, :, 0], o.sdg)
    o.time, o.dtfactor = 0.01, 45.0
    s.set("sdg", o.sdg.ravel(order="F"))
    s.set_time(o.time, o.dtfactor)
    rng = np.random.default_rng(n)
    u0, h0 = o.udg.copy(), o.uh.copy()
    err = lambda a, b: np.abs(a - np.asarray(b).ravel(order="F")).max() / np.abs(b).max()
    for written in (False, False, True):
        o.udg = u0 * (1 + 1e-2 * rng.standard_normal(u0.shape)) + 1e-3
        o.uh = h0 * (1 + 1e-2 * rng.standard_normal(h0.shape)) + 1e-3
        s.set("udg", o.udg)
        s.set("uh", o.uh)
        if written:
            s.set("K", rng.standard_normal(o.K.size))
        s.hdgAssembleLinearSystem()
        H, Rh, F, Ru = o.assemble()
        for name, ref in (("H", H), ("F", F), ("Ru", Ru), ("Rh", Rh)):
            assert err(s.get(name), ref) < 5e-12, name
    assert err(s.get("K"), o.K) < 1e-11
    s.close()


def test_reading_a_block_does_not_form_it_for_good(tmp_path):
    """get() of B forms B once (two launches) and leaves the later assemblies as they were; a pointer to it
    makes each of them form it."""
    B.build(["convdiff3d"])
    d = str(tmp_path / "datain")
    cases.convdiff3d_hex(d, n=2, porder=3)
    s = HDGSolver(d, "convdiff3d")
    s.set_time(0.01, 45.0)

    def launches(call):
        before = s.lib.exa_launch_count()
        call()
        return s.lib.exa_launch_count() - before

    s.hdgAssembleLinearSystem()
    first = launches(s.hdgAssembleLinearSystem)
    assert s.field_size("B") == s.sizes["n"] * 3 * s.sizes["n"] * s.sizes["ne"]
    b = []
    assert launches(lambda: b.append(s.get("B"))) == 2 and np.abs(b[0]).max() > 0
    assert launches(s.hdgAssembleLinearSystem) == first
    s.field_ptr("B")
    assert launches(s.hdgAssembleLinearSystem) == first + 2
    s.close()


@pytest.mark.parametrize("model,p", [("euler3d", 2), ("convdiff3d", 2)])
def test_schur_products_are_counted_as_they_run(tmp_path, model, p):
    """The products of the Schur phase: D^-1 F and K D^-1 F with all n rows, or (without q) those of a face."""
    B.build([model])
    d = str(tmp_path / "datain")
    if model == "euler3d":
        cases.euler3d_vortex_hex(d, n=2, porder=p, periodic=False)
    else:
        cases.convdiff3d_hex(d, n=2, porder=p)
    s = HDGSolver(d, model)
    s.set_time(0.01, 45.0)
    s.set("sdg", 45.0 * s.get("udg")[:s.sizes["n"] * s.sizes["ne"]])
    s.hdgAssembleLinearSystem()
    s.profile(True)
    s.hdgAssembleLinearSystem()
    z, flops = s.sizes, s.profile_read()["schur"][2]
    s.profile(False)
    n, m, ne = z["n"], z["m"], z["ne"]
    k = z["npf"] * z["ncu"] if model == "euler3d" else n
    assert flops == 2.0 * ne * (n * m * k + n * n + m * m * k + m * n)
    s.close()


def test_trace_rows_are_timed_within_the_q_elimination(tmp_path):
    """Phase qelim_trace of the profile: one region per mixed assembly, within those of qelim; none in FP64."""
    B.build(["convdiff3d"])
    d = str(tmp_path / "datain")
    cases.convdiff3d_hex(d, n=3, porder=4)
    s = HDGSolver(d, "convdiff3d")
    s.set_time(0.01, 45.0)
    for mixed in (0, 1):
        s.set_precision(mixed)
        s.profile(True)
        s.hdgAssembleLinearSystem()
        p = s.profile_read()
        s.profile(False)
        assert p["qelim"][1] == 1 and p["qelim_trace"][1] == mixed
        assert 0.0 <= p["qelim_trace"][0] < p["qelim"][0]
    s.close()


def test_refused_calls_for_k_change_nothing(tmp_path):
    """Once a caller holds or has written K, each assembly sets its zeros again (two more memory sets per
    chunk); a call for it that is refused does not count."""
    from torch.profiler import ProfilerActivity, profile
    B.build(["euler3d"])
    d = str(tmp_path / "datain")
    cases.euler3d_vortex_hex(d, n=2, porder=2, periodic=False)
    s = HDGSolver(d, "euler3d")
    s.set_time(0.01, 45.0)
    s.set("sdg", 45.0 * s.get("udg"))

    def sets():
        s.hdgAssembleLinearSystem()
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            s.hdgAssembleLinearSystem()
            torch.cuda.synchronize()
        names = [e.name for e in prof.events()]
        if not any("face_kernel" in n for n in names):
            pytest.skip("no device activities recorded")
        return sum(n.startswith("Memset (") for n in names)

    before = sets()
    for call in (lambda: s.set("K", np.zeros(3)), lambda: s.lib.exa_field_ptr(s.h, b"K", None, None)):
        try:
            assert call() not in (None, 0)
        except ExaError:
            pass
        assert sets() == before
    s.set("K", s.get("K"))
    assert sets() == before + 2
    s.close()


@pytest.mark.parametrize("n,p", [(2, 2), (3, 3), (2, 4), (3, 4), (5, 2)])
def test_mixed_blocks_match_oracle(tmp_path, n, p):
    """K and H of the mixed form, whose trace rows are eliminated face by face in FP32 (rounding 6e-8 of
    sums that cancel to a tenth: 5e-6), H behind a D^-1 of condition 1e3 (2e-4)."""
    d = str(tmp_path / "datain")
    B.build(["convdiff3d"])
    cases.convdiff3d_hex(d, n=n, porder=p, nsteps=1)
    s, o = HDGSolver(d, "convdiff3d"), HDGOracle(d, MODELS["convdiff3d"]())
    s.set_precision(1)
    o.sdg = 40.0 * o.udg[:, :o.ncu]
    o.sdgg = np.einsum("gj,jce->gec", o.shapegt[:, :, 0], o.sdg)
    o.time, o.dtfactor = 0.01, 45.0
    s.set("sdg", o.sdg.ravel(order="F"))
    s.set_time(o.time, o.dtfactor)
    rng = np.random.default_rng(p)
    o.udg, o.uh = rng.standard_normal(o.udg.shape), rng.standard_normal(o.uh.shape)
    err = lambda a, b: np.abs(a - np.asarray(b).ravel(order="F")).max() / np.abs(b).max()
    for _ in range(2):
        s.set("udg", o.udg)
        s.set("uh", o.uh)
        s.hdgAssembleLinearSystem()
        H, Rh, F, Ru = o.assemble()
        e = {k: err(s.get(k), v) for k, v in (("K32", o.K), ("H32", H), ("F32", F), ("Rh", Rh))}
        print(n, p, e)
        assert e["K32"] < 5e-6 and max(e["H32"], e["F32"], e["Rh"]) < 2e-4
        o.udg = rng.standard_normal(o.udg.shape)
    s.close()

"""Assemblies of meshes that take several element chunks (at most 65535 elements, or 8 GB of blocks, each):
the blocks of elements on both sides of a chunk's end and at the mesh's, against a context for these
elements alone, which the oracle tests cover.  The same kernels see the same element data: 1e-12 in FP64
(products may be split otherwise), 1e-5 for the FP32 blocks behind D^-1 of condition 1e3."""
import os

import numpy as np
import pytest

from exasim_b200 import HDGSolver, build as B, cases, inputs as I

pytestmark = pytest.mark.gpu


class View:
    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def blocks(s, name, elems):
    """The blocks of some elements of a device array [.., ne]."""
    import torch
    ptr, n = s.field_ptr(name)
    ne = s.sizes["ne"]
    t = torch.as_tensor(View(ptr, (ne, n // ne), "<f4" if name.endswith("32") else "<f8"), device="cuda")
    return t[torch.as_tensor(elems, device="cuda")].double().cpu().numpy()


@pytest.mark.parametrize("model,n,mixed", [("convdiff3d", 41, 0), ("convdiff3d", 41, 1), ("euler3d", 23, 0)])
def test_elements_of_every_chunk(tmp_path, monkeypatch, model, n, mixed):
    B.build([model])
    kept = {}
    write = cases.write_case

    def keep(datain, grid, master, app, exprs, bcs, *args):
        kept.update(grid=grid, master=master, app=app, bf=I.assign_bf(grid, exprs, bcs), bcs=bcs)
        return write(datain, grid, master, app, exprs, bcs, *args)

    monkeypatch.setattr(cases, "write_case", keep)
    big, small = str(tmp_path / "big"), str(tmp_path / "small")
    if model == "convdiff3d":
        cases.convdiff3d_hex(big, n=n, porder=2, nsteps=1)
    else:
        cases.euler3d_vortex_hex(big, n=n, porder=2, nsteps=1)
    s = HDGSolver(big, model)
    z = s.sizes
    ne, nb = z["ne"], z["neb"]
    assert nb < ne, "one chunk holds the mesh"
    grid, master = kept["grid"], kept["master"]
    elems = np.unique(np.concatenate([np.arange(3), np.arange(nb - 20, nb + 20), np.arange(ne - 20, ne)]))
    sub = I.Grid(p=grid.p, t=grid.t[:, elems], elemtype=1, tp=None if grid.tp is None else grid.tp[:, elems])
    os.makedirs(small)
    I.write_app_bin(os.path.join(small, "app.bin"), kept["app"])
    I.write_master_bin(os.path.join(small, "master.bin"), master)
    I.write_mesh_bin(os.path.join(small, "mesh.bin"), sub, master, kept["bf"][:, elems], kept["bcs"])
    I.write_sol_bin(os.path.join(small, "sol.bin"), I.dgnodes(sub, master), nc=kept["app"].nc, ncu=kept["app"].ncu)
    q = HDGSolver(small, model)
    ncu, npe = z["ncu"], z["npe"]
    rng = np.random.default_rng(0)
    u = s.get("udg").reshape(ne, -1, npe)
    u[:, :ncu] = u[:, :ncu] * (1 + 1e-2 * rng.standard_normal((ne, ncu, npe))) + 1e-3
    u[:, ncu:] = 0.1 * rng.standard_normal(u[:, ncu:].shape)
    uh = s.get("uh").reshape(-1, ncu)
    uh = uh * (1 + 1e-2 * rng.standard_normal(uh.shape)) + 1e-3
    sdg = 40.0 * u[:, :ncu]
    con, qcon = s.connectivity()[1], q.connectivity()[1]
    quh = np.zeros((q.sizes["ndofuhat"] // ncu, ncu))
    quh[qcon.T.ravel()] = uh[con[:, elems].T.ravel()]
    for c, e, h in ((s, slice(None), uh), (q, elems, quh)):
        if mixed:
            c.set_precision(1)
        c.set_time(0.01, 45.0)
        c.set("udg", u[e].ravel())
        c.set("uh", h.ravel())
        c.set("sdg", sdg[e].ravel())
        c.hdgAssembleLinearSystem()
    mine = np.arange(elems.size)
    for name in ("H32", "F32", "K32", "Dinv32", "Ru", "Rh") if mixed else ("H", "F", "Ru", "Rh"):
        a, b = blocks(s, name, elems), blocks(q, name, mine)
        e = np.abs(a - b).max() / np.abs(b).max()
        print(model, name, f"{e:.1e}")
        assert np.isfinite(a).all() and e < (1e-5 if mixed else 1e-12)
    s.close()
    q.close()

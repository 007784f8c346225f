"""Meshes for the tests whose quadrilaterals and hexahedra are no boxes: every element is numbered from a
vertex of its own (neighbours meet rotated) and the element nodes are moved by a smooth map, periodic on the
domain, so that the geometry factors are full matrices that vary over each element."""
import itertools
import os

import numpy as np

from exasim_b200 import cases, inputs as I


def rotations(nd):
    """The proper rotations of the reference element as lists of its vertices."""
    quad = [(0, 0), (1, 0), (1, 1), (0, 1)]
    x = np.array(quad if nd == 2 else [q + (0,) for q in quad] + [q + (1,) for q in quad]) * 2 - 1
    out = []
    for perm in itertools.permutations(range(nd)):
        for sign in itertools.product((1, -1), repeat=nd):
            R = np.zeros((nd, nd), dtype=int)
            R[range(nd), perm] = sign
            if round(np.linalg.det(R)) == 1:
                y = x @ R.T
                out.append([int(np.flatnonzero((x == v).all(1))[0]) for v in y])
    return out


def bend(monkeypatch, seed=0, amp=0.03, rotate=True):
    """Make the case writers of exasim_b200.cases write such meshes."""
    write = cases.write_case

    def bent(datain, grid, master, app, exprs, bcs, *args):
        rng = np.random.default_rng(seed)
        if rotate:
            rots = rotations(grid.nd)
            for e in range(grid.ne):
                r = rots[rng.integers(len(rots))]
                grid.t[:, e] = grid.t[r, e]
                if grid.tp is not None:
                    grid.tp[:, e] = grid.tp[r, e]
        write(datain, grid, master, app, exprs, bcs, *args)
        x = I.dgnodes(grid, master)                                     # [npe, nd, ne]
        lo, L = grid.p.min(1), np.ptp(grid.p, axis=1)
        s = (x - lo[:, None]) / L[:, None]
        for d in range(grid.nd):
            k = rng.integers(1, 3, grid.nd)
            x[:, d] += amp * L[d] * np.sin(2 * np.pi * np.einsum("ide,d->ie", s, k) + rng.uniform(0, 6))
        I.write_sol_bin(os.path.join(datain, "sol.bin"), x, nc=app.nc, ncu=app.ncu)

    monkeypatch.setattr(cases, "write_case", bent)

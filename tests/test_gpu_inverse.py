"""The batched explicit inverse (exa_dinverse_batched, the reference's Inverse,
backend/Common/pblas.h:163) against LAPACK through numpy, for every kernel shape: one warp
per matrix (n <= 32), the register-tiled kernel (n <= 160) and the 2 x 2 blocked form
(n <= 320).  Matrices are diagonally weighted random blocks with cond ~ 1e2; tolerance
1e-12 of max |inverse| (Gauss-Jordan with partial pivoting against getrf + getri).  A
singular block sets the flag."""
import ctypes

import numpy as np
import pytest

from exasim_b200 import build as B, load_library

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    B.build(["poisson2d"])
    return load_library("poisson2d")


@pytest.mark.parametrize("n", [1, 5, 25, 32, 33, 64, 96, 125, 128, 150, 160, 200, 320])
def test_inverse_matches_lapack(lib, n):
    import torch
    rng = np.random.default_rng(n)
    batch = 37
    A = rng.standard_normal((batch, n, n)) + np.eye(n) * (2.0 * np.sqrt(n))
    # column-major blocks spaced n^2 apart
    dev = torch.tensor(np.ascontiguousarray(np.transpose(A, (0, 2, 1))).ravel(), dtype=torch.float64, device="cuda")
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    st = lib.exa_dinverse_batched(ctypes.c_void_p(dev.data_ptr()), n, n * n, batch, ctypes.c_void_p(flag.data_ptr()),
                                  None)
    assert st == 0, lib.exa_last_error().decode()
    torch.cuda.synchronize()
    got = np.transpose(dev.cpu().numpy().reshape(batch, n, n), (0, 2, 1))
    ref = np.linalg.inv(A)
    assert int(flag.item()) == 0
    err = np.abs(got - ref).max() / np.abs(ref).max()
    assert err < 1e-12, err


@pytest.mark.parametrize("n", [25, 125, 160, 170, 201, 250, 320])
def test_fp32_inverse_matches_lapack(lib, n):
    """exa_sinverse_batched, the mixed form's FP32 inverse: register kernels up to 160, the
    recursive blocked form with 3xTF32 tensor-core products above (one level at 170, two at
    201, 250 and 320; 170, 201 and 250 have halves that are not multiples of 16, so the
    packed operands carry padding).  FP32 rounding of the input and of the elimination:
    within 2e-5 of max |inverse| at cond ~ 1e2."""
    import torch
    rng = np.random.default_rng(1000 + n)
    batch = 37
    A = (rng.standard_normal((batch, n, n)) + np.eye(n) * (2.0 * np.sqrt(n))).astype(np.float32)
    dev = torch.tensor(np.ascontiguousarray(np.transpose(A, (0, 2, 1))).ravel(), dtype=torch.float32, device="cuda")
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    for _ in range(2):  # the second call reuses the stream-ordered workspace memory
        d = dev.clone()
        st = lib.exa_sinverse_batched(ctypes.c_void_p(d.data_ptr()), n, n * n, batch,
                                      ctypes.c_void_p(flag.data_ptr()), None)
        assert st == 0, lib.exa_last_error().decode()
        torch.cuda.synchronize()
        assert int(flag.item()) == 0
        got = np.transpose(d.cpu().numpy().reshape(batch, n, n), (0, 2, 1)).astype(np.float64)
        ref = np.linalg.inv(A.astype(np.float64))
        err = np.abs(got - ref).max() / np.abs(ref).max()
        assert err < 2e-5, err


@pytest.mark.parametrize("n", [125, 250])
def test_fp32_singular_block_sets_flag(lib, n):
    """A zero pivot column in the block (the leading diagonal block of the blocked form at
    250) sets the flag in the FP32 inverse as in the FP64 one."""
    import torch
    A = np.eye(n, dtype=np.float32)
    A[3, 3] = 0.0
    dev = torch.tensor(A.T.ravel(), dtype=torch.float32, device="cuda")
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert lib.exa_sinverse_batched(ctypes.c_void_p(dev.data_ptr()), n, n * n, 1, ctypes.c_void_p(flag.data_ptr()),
                                    None) == 0
    torch.cuda.synchronize()
    assert int(flag.item()) == 1


@pytest.mark.parametrize("n", [8, 125])
def test_singular_block_sets_flag(lib, n):
    import torch
    A = np.eye(n)
    A[3, 3] = 0.0
    dev = torch.tensor(A.T.ravel(), dtype=torch.float64, device="cuda")
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert lib.exa_dinverse_batched(ctypes.c_void_p(dev.data_ptr()), n, n * n, 1, ctypes.c_void_p(flag.data_ptr()),
                                    None) == 0
    torch.cuda.synchronize()
    assert int(flag.item()) == 1


@pytest.mark.parametrize("n", [8, 25, 32, 64, 96, 128, 129, 135, 150, 160])
@pytest.mark.parametrize("fp32", [False, True])
def test_negative_zeros_are_no_pivots(lib, n, fp32):
    """Rows of a diagonal matrix in any order with -0 beside the entries (a product of a zero and a negative
    number): the pivot of each column is its one entry, not a -0, and the inverse is exact."""
    import torch
    rng = np.random.default_rng(n)
    A = np.full((5, n, n), -0.0)
    for M in A:
        M[rng.permutation(n), np.arange(n)] = 2.0 ** rng.integers(-3, 4, n) * rng.choice([-1.0, 1.0], n)
    ref = np.linalg.inv(A)
    dt, inv = (torch.float32, lib.exa_sinverse_batched) if fp32 else (torch.float64, lib.exa_dinverse_batched)
    dev = torch.tensor(np.ascontiguousarray(np.transpose(A, (0, 2, 1))).ravel(), dtype=dt, device="cuda")
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    st = inv(ctypes.c_void_p(dev.data_ptr()), n, n * n, 5, ctypes.c_void_p(flag.data_ptr()), None)
    assert st == 0, lib.exa_last_error().decode()
    torch.cuda.synchronize()
    got = np.transpose(dev.cpu().numpy().reshape(5, n, n), (0, 2, 1))
    assert int(flag.item()) == 0 and np.array_equal(got, ref)


@pytest.mark.parametrize("fp64", [0, 1])
def test_every_tuned_shape_gives_the_same_bits(lib, fp64):
    """exa_inverse_autotune picks one of the column-by-warp shapes per order; whatever it
    picks, the inverse is the same to the bit, because every shape performs the same
    operations with the same pivots.  The same blocks of orders 96 and 125 are inverted with
    the untuned default shape and again after tuning: the results must be identical.  (In a
    session where an earlier test already tuned the order, both runs use the tuned shape and
    the check holds trivially.)"""
    import torch
    dt, inv = (torch.float64, lib.exa_dinverse_batched) if fp64 else (torch.float32, lib.exa_sinverse_batched)
    for n in (96, 125):
        rng = np.random.default_rng(100 + n)
        batch = 300
        # diagonally weighted (cond ~ 1e2), then the rows shuffled, so partial pivoting has to
        # find the permutation
        A = rng.standard_normal((batch, n, n)) + np.eye(n) * (2.0 * np.sqrt(n))
        A = np.stack([a[rng.permutation(n)] for a in A])
        host = np.ascontiguousarray(np.transpose(A, (0, 2, 1))).ravel()
        outs = []
        for tune in (False, True):
            if tune:
                v = ctypes.c_int(-2)
                assert lib.exa_inverse_autotune(n, fp64, batch, None, ctypes.byref(v)) == 0, lib.exa_last_error().decode()
                assert 0 <= v.value <= 3
                w = ctypes.c_int(-2)
                assert lib.exa_inverse_autotune(n, fp64, batch, None, ctypes.byref(w)) == 0
                assert w.value == v.value                       # kept after the first call
            dev = torch.tensor(host, dtype=dt, device="cuda")
            flag = torch.zeros(1, dtype=torch.int32, device="cuda")
            st = inv(ctypes.c_void_p(dev.data_ptr()), n, n * n, batch, ctypes.c_void_p(flag.data_ptr()), None)
            assert st == 0, lib.exa_last_error().decode()
            torch.cuda.synchronize()
            outs.append(dev.cpu().numpy())
        assert np.array_equal(outs[0], outs[1])
        ref = np.linalg.inv(A)
        got = np.transpose(outs[1].reshape(batch, n, n), (0, 2, 1))
        tol = 1e-12 if fp64 else 1e-4
        assert np.abs(got - ref).max() / np.abs(ref).max() < tol
    v = ctypes.c_int(-2)
    assert lib.exa_inverse_autotune(200, fp64, 8, None, ctypes.byref(v)) == 0 and v.value == -1


@pytest.mark.parametrize("n", [193, 200, 250, 319, 320])
@pytest.mark.parametrize("lead", ["zero", "tiny", "regular"])
def test_pivots_are_found_beyond_the_leaves(lib, n, lead):
    """Blocks whose leading quarter is singular (or scaled by 1e-9) while their leading half is regular and
    well conditioned: the halves are [[e R, Q], [Q', R']] with orthogonal Q, in both diagonal places.  Without
    pivots from outside the quarter the scaled one loses nine digits and the singular one everything; every
    other matrix of the batch is an ordinary one, and must not be affected.  The blocks have cond 5: pivoting
    over the halves leaves 2e-14 in a 64-bit restatement of the steps (leaves of 96 rows: 1e-6 and NaN);
    1e-12 as above."""
    import torch
    rng = np.random.default_rng(n)
    batch = 12
    h, q = (n + 1) // 2, ((n + 1) // 2 + 1) // 2
    eps = {"zero": 0.0, "tiny": 1e-9, "regular": 1.0}[lead]
    orth = lambda k: np.linalg.qr(rng.standard_normal((k, k)))[0]

    def half(k, lead_rows):
        M = 0.1 * rng.standard_normal((k, k)) / np.sqrt(k)
        r = k - lead_rows
        M[:lead_rows, :lead_rows] = eps * orth(lead_rows)
        M[:r, lead_rows:] += orth(r)
        M[lead_rows:, :r] += orth(r)
        if lead_rows > r:  # one more leading row than there are others: it needs an entry of its own
            M[r, r] = 1.0
        return M

    A = 0.02 * rng.standard_normal((batch, n, n)) / np.sqrt(n)
    for b in range(batch):
        if b % 2 == 0:
            A[b, :h, :h] = half(h, q)
            A[b, h:, h:] = half(n - h, (n - h + 1) // 2)
        else:
            A[b] += rng.standard_normal((n, n)) + np.eye(n) * (2.0 * np.sqrt(n))
    assert np.linalg.cond(A).max() < 10
    ref = np.linalg.inv(A)
    dev = torch.tensor(np.ascontiguousarray(np.transpose(A, (0, 2, 1))).ravel(), dtype=torch.float64, device="cuda")
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    st = lib.exa_dinverse_batched(ctypes.c_void_p(dev.data_ptr()), n, n * n, batch, ctypes.c_void_p(flag.data_ptr()),
                                  None)
    assert st == 0, lib.exa_last_error().decode()
    torch.cuda.synchronize()
    got = np.transpose(dev.cpu().numpy().reshape(batch, n, n), (0, 2, 1))
    err = np.abs(got - ref).max((1, 2)) / np.abs(ref).max((1, 2))
    print(n, lead, f"{err.max():.1e}")
    assert int(flag.item()) == 0
    assert err.max() < 1e-12
    # a singular block sets the flag at these orders too
    A[0] = 0.0
    dev = torch.tensor(np.ascontiguousarray(np.transpose(A, (0, 2, 1))).ravel(), dtype=torch.float64, device="cuda")
    assert lib.exa_dinverse_batched(ctypes.c_void_p(dev.data_ptr()), n, n * n, batch, ctypes.c_void_p(flag.data_ptr()),
                                    None) == 0
    torch.cuda.synchronize()
    assert int(flag.item()) == 1


@pytest.mark.parametrize("dtfactor", [45.0, 0.1, 1e-6, 0.0])
def test_euler_blocks_with_a_weak_time_term(tmp_path, dtfactor):
    """The p = 3 blocks of 3D Euler, whose leading 80 rows (density and one layer of x momentum) become
    singular as the time term goes: D^-1, D^-1 F and H against the oracle's LAPACK.  cond(D) is 2.8e3; pivoting
    within 160 rows, as the kernel promises, leaves 1e-12 of D^-1 in 64-bit numpy (leaves of 80 rows: 1e-2 at
    1e-6), times 1e2 for the products: 1e-10."""
    from exasim_b200 import HDGSolver, cases
    from oracle.hdg import HDGOracle
    from oracle.models import MODELS
    B.build(["euler3d"])
    d = str(tmp_path / "datain")
    cases.euler3d_vortex_hex(d, n=3, porder=3)
    s, o = HDGSolver(d, "euler3d"), HDGOracle(d, MODELS["euler3d"]())
    rng = np.random.default_rng(0)
    o.udg = o.udg * (1 + 1e-2 * rng.standard_normal(o.udg.shape))
    o.time, o.dtfactor = 0.01, dtfactor
    o.sdg = dtfactor * o.udg[:, :o.ncu]
    o.sdgg = np.einsum("gj,jce->gec", o.shapegt[:, :, 0], o.sdg)
    s.set("udg", o.udg)
    s.set("sdg", o.sdg)
    s.set_time(o.time, o.dtfactor)
    s.hdgAssembleLinearSystem()
    H, Rh, F, Ru = o.assemble()
    err = lambda a, b: np.abs(a - np.asarray(b).ravel(order="F")).max() / np.abs(b).max()
    e = {k: err(s.get(k), v) for k, v in (("Dinv", o.Dinv), ("F", F), ("H", H), ("Ru", Ru), ("Rh", Rh))}
    s.close()
    print(dtfactor, {k: f"{v:.1e}" for k, v in e.items()})
    assert max(e.values()) < 1e-10

"""The Gram-Schmidt step of the Krylov loops (exa_mgs in csrc/exa_ortho.cu) and the update of the iterate
(exa_gemv_add) on vectors of their own, against the same recurrence vector by vector in torch: every number
of rows per thread of the whole-GPU kernels (a step of 75776 entries), one tile per block and more (from
606208 entries), the cluster's sizes, lengths that are no multiples of 32, and bases within a panel of 64
vectors and across two and three.

The triangular form and the recurrence differ by rounding: sums of n terms of size |w|, on a basis that is
orthonormal to 1e-14: 1e-13 of |w| = sqrt(n) per coefficient and of 1 per vector of unit norm."""
import ctypes

import pytest
import torch

from exasim_b200 import build as B, load_library

pytestmark = pytest.mark.gpu
P = ctypes.c_void_p


@pytest.fixture(scope="module")
def lib():
    B.build(["poisson2d"])
    L = load_library("poisson2d")
    # C++ functions of the library, by their mangled names
    mgs, add, size = (L[k] for k in ("_Z7exa_mgsPdPKdxiS_S_iPK9ExaGivensP11CUstream_st",
                                     "_Z12exa_gemv_addPdPKdS1_xiP11CUstream_st", "_Z14exa_ortho_worki"))
    mgs.argtypes = [P, P, ctypes.c_longlong, ctypes.c_int, P, P, ctypes.c_int, P, P]
    add.argtypes = [P, P, P, ctypes.c_longlong, ctypes.c_int, P]
    size.argtypes, size.restype = [ctypes.c_int], ctypes.c_size_t
    return mgs, add, size


CASES = [(n, 6) for n in (1, 31, 512, 513, 1025, 2049, 4097, 8193, 16383, 16384, 16385, 40001, 75776, 75777, 151553,
                          227329, 303105, 378881, 454657, 530433, 606207, 606208, 606209, 650003, 1212417)]


@pytest.mark.parametrize("n,K", CASES + [(700, 130), (16384, 130), (20011, 130), (300000, 70), (650003, 66)])
def test_step_and_update_match_the_recurrence(lib, n, K):
    mgs, add, size = lib
    K = min(K, n)
    g = torch.Generator(device="cuda").manual_seed(n)
    V = torch.empty(K + 1, n, dtype=torch.float64, device="cuda")
    V[0] = torch.randn(n, generator=g, dtype=torch.float64, device="cuda")
    V[0] /= V[0].norm()
    work = torch.zeros(size(K), dtype=torch.float64, device="cuda")
    h = torch.zeros(K + 1, dtype=torch.float64, device="cuda")
    worst = 0.0
    for k in range(1, K + 1):
        w = torch.randn(n, generator=g, dtype=torch.float64, device="cuda")
        scale = w.norm()
        V[k] = w
        torch.cuda.synchronize()
        assert mgs(V[k].data_ptr(), V.data_ptr(), n, k, h.data_ptr(), work.data_ptr(), K, None, None) == 0
        torch.cuda.synchronize()
        ref = torch.zeros_like(h)
        for j in range(k):
            ref[j] = V[j] @ w
            w = w - ref[j] * V[j]
        ref[k] = w.norm()
        e = ((h[:k + 1] - ref[:k + 1]).abs().max() / scale).item()
        if k < n:  # the last vector of a full basis is rounding alone
            e = max(e, (V[k] - w / ref[k]).abs().max().item())
        else:
            V[k] = 0.0
        worst = max(worst, e)
    y = torch.randn(K, generator=g, dtype=torch.float64, device="cuda")
    x = torch.randn(n, generator=g, dtype=torch.float64, device="cuda")
    ref = x + y @ V[:K]
    torch.cuda.synchronize()
    assert add(x.data_ptr(), V.data_ptr(), y.data_ptr(), n, K, None) == 0
    torch.cuda.synchronize()
    worst = max(worst, (x - ref).abs().max().item() / ref.abs().max().item())
    print(n, K, f"{worst:.1e}")
    assert worst < 1e-13

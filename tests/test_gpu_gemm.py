"""The complex GEMMs of the path (q3b_gemm FP64, q3b_gemm_single on the tensor
cores) against numpy, over tile edges, split-K and odd leading dimensions.

Bars: FP64 within 1e-13 of sum |a||b| per entry; FP32 (TF32 split into hi+lo,
three products, FP32 accumulation) within 2e-6 of sum |a||b| per entry --
the accuracy of an FP32 GEMM.
"""
import ctypes as C

import numpy as np
import pytest

from q3_b200._lib import Cplx64, Cplx128, check

pytestmark = pytest.mark.gpu

SHAPES = [
    # (trans_a, m, n, k)
    ("C", 512, 256, 23847),   # <beta|psi> of the 64-atom cell
    ("C", 130, 70, 1000),     # tile edges on M and N
    ("C", 17, 9, 33),         # below one tile
    ("C", 256, 256, 6000),    # subspace block V^H HV
    ("N", 23847, 256, 512),   # beta (D <beta|psi>)
    ("N", 1000, 65, 129),     # edges on every axis
    ("N", 3000, 48, 96),      # corrections of config 2
    ("N", 64, 8, 7),
]


@pytest.fixture(scope="module")
def ctx(cuda_device):
    from q3_b200.applicator import Context
    return Context()


def _mats(rng, ta, m, n, k, lda_pad=1):
    ar = (k, m) if ta == "C" else (m, k)
    a = rng.standard_normal(ar) + 1j * rng.standard_normal(ar)
    b = rng.standard_normal((k, n)) + 1j * rng.standard_normal((k, n))
    c = rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))
    return a, b, c


def _dev(x, dtype, pad=0):
    """Column-major device copy with leading dimension rows + pad."""
    import torch
    rows, cols = x.shape
    buf = np.zeros((cols, rows + pad), dtype=dtype)
    buf[:, :rows] = x.T
    return torch.from_numpy(buf).cuda(), rows + pad


@pytest.mark.parametrize("ta,m,n,k", SHAPES)
@pytest.mark.parametrize("single", [False, True], ids=["fp64", "fp32"])
def test_gemm(ctx, ta, m, n, k, single):
    import torch
    rng = np.random.default_rng(m * 7 + n * 3 + k)
    a, b, c = _mats(rng, ta, m, n, k)
    alpha, beta = 0.75 - 0.5j, (0.25 + 0.125j if k % 2 else 0.0)
    ref = alpha * ((a.conj().T if ta == "C" else a) @ b) + beta * c
    scale = np.abs(alpha) * ((np.abs(a).T if ta == "C" else np.abs(a)) @ np.abs(b)) + np.abs(beta) * np.abs(c)
    dt = np.complex64 if single else np.complex128
    A, lda = _dev(a, dt, pad=1)
    B, ldb = _dev(b, dt, pad=3)
    Cd, ldc = _dev(c, dt, pad=0)
    lib, h = ctx.lib, ctx.handle
    if single:
        rc = lib.q3b_gemm_single(h, ta.encode(), b"N", m, n, k, Cplx64(alpha.real, alpha.imag), A.data_ptr(),
                                 lda, B.data_ptr(), ldb, Cplx64(beta.real, beta.imag), Cd.data_ptr(), ldc)
    else:
        rc = lib.q3b_gemm(h, ta.encode(), b"N", m, n, k, Cplx128(alpha.real, alpha.imag), A.data_ptr(), lda,
                          B.data_ptr(), ldb, Cplx128(beta.real, beta.imag), Cd.data_ptr(), ldc)
    check(h, rc)
    ctx.synchronize()
    got = Cd.cpu().numpy()[:, :m].T.astype(np.complex128)
    err = np.max(np.abs(got - ref) / scale)
    assert err < (2e-6 if single else 1e-13), err


def test_gemm_rejects_unsupported(ctx):
    from q3_b200._lib import Q3BError
    lib, h = ctx.lib, ctx.handle
    rc = lib.q3b_gemm(h, b"T", b"N", 4, 4, 4, Cplx128(1, 0), None, 4, None, 4, Cplx128(0, 0), None, 4)
    with pytest.raises(Q3BError):
        check(h, rc)


def test_gemm_long_operands(ctx):
    """What the FP64 units took stays accepted: more rows than a grid of 32-row tiles has."""
    import torch
    m, n, k = 2_097_153, 8, 8
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    a, b = (torch.randn(k, r, dtype=torch.complex128, device="cuda", generator=g) for r in (m, n))
    b = b.T.contiguous()  # column-major k x n
    c = torch.empty(n, m, dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    check(ctx.handle, ctx.lib.q3b_gemm(ctx.handle, b"N", b"N", m, n, k, Cplx128(1, 0), a.data_ptr(), m,
                                       b.data_ptr(), k, Cplx128(0, 0), c.data_ptr(), m))
    ctx.synchronize()
    # 8 k rounded FMAs a part
    err = float(((c - b @ a).abs() / (b.abs() @ a.abs())).max())
    assert err < 32 * k * 2.0 ** -53, err


@pytest.mark.parametrize("ta,m,n,k", [("C", 512, 256, 24000), ("N", 24000, 256, 512)])
def test_gemm_keeps_small_entries(ctx, ta, m, n, k):
    """q3b_gemm's bar is per entry, also where a row's large entries meet a column's tiny ones."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(m)

    def rand(*shape):
        return torch.randn(*shape, dtype=torch.complex128, device="cuda", generator=g)

    front = (torch.arange(k, device="cuda") < k // 2).double()
    a = rand(m, k) * (front + 1e-25 * (1 - front))   # op(A)
    b = rand(k, n) * (1e-25 * front + 1 - front)[:, None]
    A = (a.conj() if ta == "C" else a.T).resolve_conj().contiguous()  # column-major K x M, or M x K
    B, c = b.T.contiguous(), torch.empty(n, m, dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    check(ctx.handle, ctx.lib.q3b_gemm(ctx.handle, ta.encode(), b"N", m, n, k, Cplx128(1, 0), A.data_ptr(),
                                       k if ta == "C" else m, B.data_ptr(), k, Cplx128(0, 0), c.data_ptr(), m))
    ctx.synchronize()
    err = (c.T - a @ b).abs() / (a.abs() @ b.abs())
    assert float(err.max()) < 1e-13


def test_residue_products_end_where_their_byte_sums_do(ctx):
    """257 K ranges of 16384 are the most whose bytes add up in 16 bits."""
    worth = ctx.lib["_ZN3q3b4zmod5worthEbiiib"]  # bool q3b::zmod::worth(bool, int, int, int, bool)
    worth.restype, worth.argtypes = C.c_bool, [C.c_bool, C.c_int, C.c_int, C.c_int, C.c_bool]
    for packed in (False, True):
        assert worth(True, 2048, 1024, 257 * 16384, packed)
        assert not worth(True, 2048, 1024, 257 * 16384 + 1, packed)
        assert not worth(False, 2048, 1024, 257 * 16384 + 1, packed)

"""The FP64 complex products on the integer tensor cores (q3b_gemm_residue, and the library's own
large products), entry by entry against exactly rounded sums.

Bound: both operands are rounded to integers of row norm at least 2^(c-1), c = 58.39, with an
error of at most 1/2 in each real number, so an entry is off by at most
2 sqrt(2 K) 2^-58.39 |a| |b| (|a|, |b| the norms of its row and column), and by a few roundings
of its value, of alpha times it and of beta C.
"""
import math

import numpy as np
import pytest

from q3_b200._lib import Cplx128, check

pytestmark = pytest.mark.gpu

# tile edges (128 rows, 64 columns, 128 of K), one partial sum's longest K (16384) and beyond
SHAPES = [
    ("C", 257, 257, 16384), ("C", 300, 193, 16385), ("C", 260, 130, 40007), ("C", 513, 257, 1023),
    ("N", 6200, 256, 384), ("N", 4097, 321, 257), ("N", 130, 65, 16500), ("N", 512, 512, 512),
    ("C", 1, 1, 1), ("N", 3, 2, 5),
]


@pytest.fixture(scope="module")
def ctx(cuda_device):
    from q3_b200.applicator import Context
    return Context()


def _gemm(ctx, ta, a, b, c, alpha, beta, pad=1):
    import torch

    def dev(x, extra):
        buf = np.full((x.shape[1], x.shape[0] + extra), np.nan + 0j)
        buf[:, :x.shape[0]] = x.T
        return torch.from_numpy(buf).cuda(), x.shape[0] + extra

    (A, lda), (B, ldb), (C, ldc) = dev(a, pad), dev(b, 2 * pad), dev(c, pad)
    m, n, k = c.shape[0], c.shape[1], b.shape[0]
    before = ctx.lib.q3b_kernel_launches()
    check(ctx.handle, ctx.lib.q3b_gemm_residue(ctx.handle, ta.encode(), b"N", m, n, k,
                                               Cplx128(alpha.real, alpha.imag), A.data_ptr(), lda, B.data_ptr(), ldb,
                                               Cplx128(beta.real, beta.imag), C.data_ptr(), ldc))
    ctx.synchronize()
    # two kernels pack each operand, two make the product (the FP64 units' path has two at most)
    assert ctx.lib.q3b_kernel_launches() - before >= 6
    out = C.cpu().numpy()
    assert np.isnan(out[:, m:]).all()  # rows beyond M stay untouched
    return out[:, :m].T


def _exact(x, y):
    """sum x_k y_k with one rounding per part."""
    re, im = [], []
    for p, q, sign in ((x.real, y.real, 1), (x.imag, y.imag, -1)):
        h, l = _product(p, q)
        re += list(sign * h) + list(sign * l)
    for p, q in ((x.real, y.imag), (x.imag, y.real)):
        h, l = _product(p, q)
        im += list(h) + list(l)
    return complex(math.fsum(re), math.fsum(im))


def _product(p, q):
    """p q as an unevaluated sum of two doubles (Dekker)."""
    def split(v):
        t = 134217729.0 * v
        h = t - (t - v)
        return h, v - h
    (ph, pl), (qh, ql) = split(p), split(q)
    h = p * q
    return h, ((ph * qh - h) + ph * ql + pl * qh) + pl * ql


def _operand(rng, kind, rows, cols):
    x = rng.standard_normal((rows, cols)) + 1j * rng.standard_normal((rows, cols))
    if kind == "graded":  # falls off along both axes, as projectors and bands do
        x *= np.exp(-18.0 * np.linspace(0, 1, rows))[:, None] * 10.0 ** rng.uniform(-12, 3, cols)[None, :]
    return x


@pytest.mark.parametrize("kind", ["normal", "graded"])
@pytest.mark.parametrize("ta,m,n,k", SHAPES)
def test_entries_against_exact_sums(ctx, ta, m, n, k, kind):
    rng = np.random.default_rng(m + 3 * n + 7 * k)
    a = _operand(rng, kind, *((k, m) if ta == "C" else (m, k)))
    b = _operand(rng, kind, k, n)
    c = _operand(rng, "normal", m, n)
    alpha, beta = 0.75 - 0.5j, (0.25 + 0.125j if k % 2 else 0.0j)
    got = _gemm(ctx, ta, a, b, c, alpha, beta)
    rows = sorted({0, m - 1, min(m - 1, 127), *rng.integers(0, m, 6).tolist()})
    cols = sorted({0, n - 1, min(n - 1, 63), *rng.integers(0, n, 4).tolist()})
    for i in rows:
        x = a[:, i].conj() if ta == "C" else a[i, :]
        for j in cols:
            s = _exact(x, b[:, j])
            bound = 2.0 * math.sqrt(2 * k) * 2.0 ** -58.39 * np.linalg.norm(x) * np.linalg.norm(b[:, j])
            want = alpha * s + beta * c[i, j]
            slack = abs(alpha) * bound + 8 * 2.0 ** -53 * (abs(alpha) * abs(s) + abs(beta) * abs(c[i, j]))
            assert abs(got[i, j] - want) <= slack, (i, j, abs(got[i, j] - want), slack)


def test_scales_along_k_do_not_count(ctx):
    """N,N: the scales of A's columns and B's rows against each other, as in a basis of unequal
    norms times the inverse of its Cholesky factor, leave every bit as it is without them."""
    rng = np.random.default_rng(11)
    m, n, k = 1000, 130, 257
    a, b = _operand(rng, "normal", m, k), _operand(rng, "normal", k, n)
    scale = 2.0 ** rng.integers(-40, 41, k)
    zero = np.zeros((m, n), complex)
    want = _gemm(ctx, "N", a, b, zero, 1 + 0j, 0j)
    got = _gemm(ctx, "N", a * scale[None, :], b / scale[:, None], zero, 1 + 0j, 0j)
    assert np.array_equal(got, want)
    far = 2.0 ** rng.integers(-400, 401, k)  # beyond what is balanced: the bits are those of the largest
    got = _gemm(ctx, "N", a * far[None, :], b / far[:, None], zero, 1 + 0j, 0j)
    assert np.isfinite(got).all()


@pytest.mark.parametrize("ta", ["C", "N"])
def test_scales_zeros_and_non_finite(ctx, ta):
    """Rows far out of the usual range (their squares leave it), zero rows, and rows with an
    infinity or a NaN, which spoil their own outputs only."""
    rng = np.random.default_rng(5)
    m, n, k = (256, 256, 8200) if ta == "C" else (8200, 256, 256)
    a = _operand(rng, "normal", *((k, m) if ta == "C" else (m, k)))
    b = _operand(rng, "normal", k, n)
    rows = a.T if ta == "C" else a  # a view: row i of op(A)
    scale = {1: 1e200, 2: 1e-200, 3: 5e-324 * 2 ** 40, 4: 1e150, 5: 0.0}
    for i, s in scale.items():
        rows[i] *= s
    b[:, 7] *= 1e-100
    b[:, 8] = 0.0
    rows[130, 17] = np.inf
    rows[140, 3] = complex(0.0, np.nan)
    b[9, 70] = -np.inf
    got = _gemm(ctx, ta, a, b, np.zeros((m, n), complex), 1 + 0j, 0j)
    bad = np.zeros((m, n), bool)
    bad[[130, 140]] = True
    bad[:, 70] = True
    assert not np.isfinite(got[bad]).any()
    assert np.isfinite(got[~bad]).all()
    assert np.all(got[5][~bad[5]] == 0) and np.all(got[:, 8][~bad[:, 8]] == 0)
    for i in (0, 1, 2, 3, 4, 200):
        x = rows[i].conj() if ta == "C" else rows[i]
        for j in (0, 7, 255):
            s = _exact(x * 2.0 ** 600 if i == 3 else x, b[:, j])
            w = got[i, j] * 2.0 ** 600 if i == 3 else got[i, j]
            bound = 2.0 * math.sqrt(2 * k) * 2.0 ** -58.39 * (np.linalg.norm(np.abs(x) / np.abs(x).max())
                                                             * np.abs(x).max() * (2.0 ** 600 if i == 3 else 1.0)
                                                             * np.linalg.norm(b[:, j]))
            # the bound |row| <= max sqrt(2 K) of rows whose squares leave the range costs sqrt(K) more;
            # an output among the denormals is rounded to 2^-1074
            bound *= math.sqrt(2 * k) if i in (1, 2, 3) else 1.0
            bound += 2.0 ** -1073 * (2.0 ** 600 if i == 3 else 1.0)
            assert abs(w - s) <= bound + 4 * 2.0 ** -53 * abs(s), (i, j)

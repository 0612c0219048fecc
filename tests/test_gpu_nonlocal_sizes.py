"""The projector products of H|psi> (FP32 on split FP16 tiles, FP64 on residue tiles or the FP64
units, by size) on their own: no potential, no kinetic energy, no plane wave on the grid, so
that H psi = beta D beta^H psi.

Bounds per entry, S = sum |beta| |D| sum |beta| |psi| over projectors and plane waves: FP32
4e-6 S (each product within 2e-6 of its sum of magnitudes, test_gpu_gemm.py's bar); FP64 1e-15 S (the
rounding of the operands leaves 1.6e-18 |a| |b| of the balanced rows and columns, at most 4 times
their sum of magnitudes here; six times that, and a few roundings of the coefficients and the result).
The inputs are uniform, graded along the plane waves with projectors of unequal norms, or such that
the large entries of beta meet the small ones of its partner: bands of the highest plane waves only,
and projectors whose norms the D blocks make up for.
"""
import numpy as np
import pytest

from q3_b200._lib import FP64, MIXED

pytestmark = pytest.mark.gpu

# edges of 256-row, 128-column and 64-column tiles and of 64 and 128 of K, on the FP16 tiles (from
# 2e9 multiply-adds of half as many bands as projectors) and, first and last, the TF32 ones
SIZES = [(5000, 136, 130), (12289, 640, 130), (4097, 1032, 65), (2100, 1400, 257), (23847, 512, 33), (769, 640, 257)]


def _inputs(npw, nproj, nvec, kind):
    rng = np.random.default_rng(npw + nproj + nvec)
    beta = rng.standard_normal((npw, nproj)) + 1j * rng.standard_normal((npw, nproj))
    psi = rng.standard_normal((npw, nvec)) + 1j * rng.standard_normal((npw, nvec))
    if kind == "graded":  # projectors and bands fall off along the plane waves, and differ in size
        fall = np.exp(-16.0 * np.linspace(0.0, 1.0, npw))[:, None]
        beta *= fall * 10.0 ** rng.uniform(-3, 3, nproj)[None, :]
        psi *= fall ** 0.25 * 10.0 ** rng.uniform(-6, 3, nvec)[None, :]
    d = rng.uniform(-1.0, 1.0, (nproj // 8, 8, 8))
    d = d + d.transpose(0, 2, 1)
    if kind == "opposed":
        beta *= np.exp(-16.0 * np.linspace(0.0, 1.0, npw))[:, None]
        psi[:4 * npw // 5] = 0.0
        norms = 10.0 ** rng.uniform(-3, 3, nproj)
        beta *= norms[None, :]
        d /= norms.reshape(-1, 8, 1) * norms.reshape(-1, 1, 8)
    return beta, psi, d


@pytest.mark.parametrize("kind", ["normal", "graded", "opposed"])
@pytest.mark.parametrize("npw,nproj,nvec", SIZES)
def test_projector_products(cuda_device, npw, nproj, nvec, kind):
    import torch
    from q3_b200.applicator import PlanewaveHamiltonianApplicator
    beta, psi, d = _inputs(npw, nproj, nvec, kind)
    ap = PlanewaveHamiltonianApplicator()
    ap.update_potential(np.zeros(16 ** 3), (16, 16, 16))
    ap.prepare_kpoint(0, npw, np.full(npw, -1, np.int32), np.zeros(npw), beta,
                      np.arange(0, nproj + 1, 8, dtype=np.int32), d.transpose(0, 2, 1).reshape(-1))
    x = torch.from_numpy(np.ascontiguousarray(psi.T)).cuda()
    inner = beta.conj().T @ psi
    want = beta @ np.einsum("aij,ajv->aiv", d, inner.reshape(nproj // 8, 8, nvec)).reshape(nproj, nvec)
    mag = np.abs(beta) @ np.einsum("aij,ajv->aiv", np.abs(d), (np.abs(beta).T @ np.abs(psi)).reshape(
        nproj // 8, 8, nvec)).reshape(nproj, nvec)
    for precision, tol in ((MIXED, 4e-6), (FP64, 1e-15)):
        y = torch.full_like(x, np.nan)
        ap.apply_batch(x, y, nvec, precision)
        torch.cuda.synchronize()
        got = y.cpu().numpy().T
        assert np.max(np.abs(got - want) / mag) < tol, precision


@pytest.mark.parametrize("precision,scale,tol", [(MIXED, 3e-38, 4e-6), (FP64, 1e-290, 1e-15)], ids=["mixed", "fp64"])
def test_tiny_projectors_with_zeros_among_them(cuda_device, precision, scale, tol):
    """Projectors near the end of the range, a projector of zeros and plane waves that no projector
    reaches: scales and balance together stay in range, and the zeros contribute nothing."""
    import torch
    from q3_b200.applicator import PlanewaveHamiltonianApplicator
    npw, nproj, nvec = 12289, 640, 130
    beta, psi, _ = _inputs(npw, nproj, nvec, "normal")
    beta[:, 17] = 0.0
    beta[1000:1200] = 0.0
    ap = PlanewaveHamiltonianApplicator()
    ap.update_potential(np.zeros(16 ** 3), (16, 16, 16))
    # D takes the scale out of the coefficients again, so that the result is beta's size
    ap.prepare_kpoint(0, npw, np.full(npw, -1, np.int32), np.zeros(npw), scale * beta,
                      np.arange(0, nproj + 1, 8, dtype=np.int32), np.tile(np.eye(8).reshape(-1) / scale, nproj // 8))
    x = torch.from_numpy(np.ascontiguousarray(psi.T)).cuda()
    y = torch.full_like(x, np.nan)
    ap.apply_batch(x, y, nvec, precision)
    torch.cuda.synchronize()
    want = beta @ (beta.conj().T @ psi)
    mag = np.abs(beta) @ (np.abs(beta).T @ np.abs(psi))
    got = y.cpu().numpy().T / scale
    assert np.all(got[1000:1200] == 0.0)
    keep = mag > 0.0
    assert np.max(np.abs(got - want)[keep] / mag[keep]) < tol

"""H|psi> under an HBM budget that has no room for the optional buffers (packed projector copies,
workspace of the tensor-core products): they are left out or given back, and the result stays."""
import numpy as np
import pytest

from q3_b200._lib import FP64, MIXED

pytestmark = pytest.mark.gpu

NPW, NPROJ, NVEC = 12000, 256, 128


def _held_and_result(budget, precision):
    import torch
    from q3_b200.applicator import PlanewaveHamiltonianApplicator
    rng = np.random.default_rng(3)
    beta = rng.standard_normal((NPW, NPROJ)) + 1j * rng.standard_normal((NPW, NPROJ))
    d = rng.uniform(-1.0, 1.0, (NPROJ // 8, 8, 8))
    psi = rng.standard_normal((NVEC, NPW)) + 1j * rng.standard_normal((NVEC, NPW))
    ap = PlanewaveHamiltonianApplicator(hbm_budget=budget)
    ap.update_potential(np.zeros(16 ** 3), (16, 16, 16))
    ap.prepare_kpoint(0, NPW, np.full(NPW, -1, np.int32), np.zeros(NPW), beta,
                      np.arange(0, NPROJ + 1, 8, dtype=np.int32), (d + d.transpose(0, 2, 1)).reshape(-1))
    x = torch.from_numpy(psi).cuda()
    y = torch.empty_like(x)
    ap.apply_batch(x, y, NVEC, precision)
    torch.cuda.synchronize()
    return ap.ctx.device_bytes(), y.cpu().numpy()


@pytest.mark.parametrize("precision,tol", [(FP64, 1e-13), (MIXED, 1e-5)])
def test_tight_budgets(cuda_device, precision, tol):
    held, want = _held_and_result(0, precision)
    # what the calls cannot do without: projectors in FP64 and FP32 and their TF32 tiles (npw and
    # the projectors padded to 128), the bands' FP32 copies and coefficients, and 16 MB for the rest
    padded = -(-NPW // 128) * 128
    least = NPW * NPROJ * 24 + 2 * padded * NPROJ * 16 + 2 * NPW * NVEC * 8 + 4 * NPROJ * NVEC * 16 + (80 << 20)
    for budget in (held, (held + least) // 2, least):
        got_held, got = _held_and_result(budget, precision)
        assert got_held <= budget
        assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)

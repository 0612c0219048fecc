"""q3b_prepare_kpoint has finished its device work when it returns: the caller may apply H on
another stream at once."""
import numpy as np
import pytest

from q3_b200._lib import FP64, MIXED

pytestmark = pytest.mark.gpu


# TF32 and residue tiles (5000 x 256), FP16 and residue tiles (24000 x 512)
@pytest.mark.parametrize("npw,nproj", [(5000, 256), (24000, 512)])
def test_apply_on_another_stream_right_after_preparing(cuda_device, npw, nproj):
    import torch
    from q3_b200.applicator import PlanewaveHamiltonianApplicator
    rng = np.random.default_rng(npw)
    nvec = nproj // 2
    beta = np.asfortranarray(rng.standard_normal((npw, nproj)) + 1j * rng.standard_normal((npw, nproj)))
    d = rng.uniform(-1.0, 1.0, (nproj // 8, 8, 8))
    psi = torch.from_numpy(rng.standard_normal((nvec, npw)) + 1j * rng.standard_normal((nvec, npw))).cuda()
    ap = PlanewaveHamiltonianApplicator()
    ap.update_potential(np.zeros(16 ** 3), (16, 16, 16))
    other = torch.cuda.Stream()
    own = torch.cuda.ExternalStream(ap.ctx.stream)

    def prepare(b):
        ap.prepare_kpoint(0, npw, np.full(npw, -1, np.int32), np.zeros(npw), b,
                          np.arange(0, nproj + 1, 8, dtype=np.int32), (d + d.transpose(0, 2, 1)).reshape(-1))

    def apply(precision):
        y = torch.full_like(psi, np.nan)
        ap.apply_batch(psi, y, nvec, precision)
        torch.cuda.synchronize()
        return y

    prepare(beta)
    want = [apply(p) for p in (FP64, MIXED)]
    for precision, ref in zip((FP64, MIXED), want):
        ap.ctx.set_stream(None)
        prepare(-2.0 * beta)  # the buffers hold other projectors, as between two k-points
        torch.cuda.synchronize()
        prepare(beta)
        assert own.query()  # nothing of it is still running
        ap.ctx.set_stream(other.cuda_stream)
        assert torch.equal(apply(precision), ref)
    ap.ctx.set_stream(None)

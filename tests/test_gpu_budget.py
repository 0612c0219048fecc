"""H|psi> under an HBM budget that has no room for the optional buffers (residue tiles of the
projectors, workspace of the tensor-core products): they are left out or given back, and the result
stays."""
import numpy as np
import pytest

from q3_b200._lib import FP64, MIXED

pytestmark = pytest.mark.gpu

NPW, NPROJ, NVEC = 12000, 256, 128


def _held_and_result(budget, precision, npw=NPW, nproj=NPROJ, nvec=NVEC):
    """Bytes held, the result and the kernels launched for one application (after a first one)."""
    import torch
    from q3_b200.applicator import PlanewaveHamiltonianApplicator
    rng = np.random.default_rng(3)
    beta = rng.standard_normal((npw, nproj)) + 1j * rng.standard_normal((npw, nproj))
    d = rng.uniform(-1.0, 1.0, (nproj // 8, 8, 8))
    psi = rng.standard_normal((nvec, npw)) + 1j * rng.standard_normal((nvec, npw))
    ap = PlanewaveHamiltonianApplicator(hbm_budget=budget)
    ap.update_potential(np.zeros(16 ** 3), (16, 16, 16))
    ap.prepare_kpoint(0, npw, np.full(npw, -1, np.int32), np.zeros(npw), beta,
                      np.arange(0, nproj + 1, 8, dtype=np.int32), (d + d.transpose(0, 2, 1)).reshape(-1))
    x = torch.from_numpy(psi).cuda()
    y = torch.empty_like(x)
    ap.apply_batch(x, y, nvec, precision)
    before = ap.lib.q3b_kernel_launches()
    ap.apply_batch(x, y, nvec, precision)
    launches = ap.lib.q3b_kernel_launches() - before
    torch.cuda.synchronize()
    return ap.ctx.device_bytes(), y.cpu().numpy(), launches


@pytest.mark.parametrize("precision,tol", [(FP64, 1e-13), (MIXED, 1e-5)])
def test_tight_budgets(cuda_device, precision, tol):
    held, want, _ = _held_and_result(0, precision)
    # what the calls cannot do without: projectors in FP64 and FP32 and their TF32 tiles (npw and
    # the projectors padded to 128), the bands' FP32 copies and coefficients, and 16 MB for the rest
    padded = -(-NPW // 128) * 128
    least = NPW * NPROJ * 24 + 2 * padded * NPROJ * 16 + 2 * NPW * NVEC * 8 + 4 * NPROJ * NVEC * 16 + (80 << 20)
    for budget in (held, (held + least) // 2, least):
        got_held, got, _ = _held_and_result(budget, precision)
        assert got_held <= budget
        assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)


def test_large_fp32_sets_keep_their_tiles(cuda_device):
    """FP32 projectors of large sets stay packed (16 B an entry, half of what the TF32 tiles of smaller
    sets take) where a budget has no room for the FP64 residues: the same kernels, the same bits."""
    npw, nproj, nvec = 16000, 512, 96
    held, want, launches = _held_and_result(0, MIXED, npw, nproj, nvec)
    residues = 60 * npw * nproj  # 15 bytes a part, in two forms
    got_held, got, got_launches = _held_and_result(held - residues // 2, MIXED, npw, nproj, nvec)
    assert got_held <= held - residues // 2
    assert got_launches == launches and np.array_equal(got, want)


def test_optional_buffers_leave_room_on_the_device_and_come_back(cuda_device):
    """Without a budget, an eighth of the device is left to others; once there is room again, the next
    k-point has its fast products, residues and workspace, as if there had always been."""
    import torch
    from q3_b200.applicator import PlanewaveHamiltonianApplicator
    rng = np.random.default_rng(5)
    beta = rng.standard_normal((NPW, NPROJ)) + 1j * rng.standard_normal((NPW, NPROJ))
    x = torch.from_numpy(rng.standard_normal((NVEC, NPW)) + 1j * rng.standard_normal((NVEC, NPW))).cuda()

    def apply(ap):
        ap.prepare_kpoint(0, NPW, np.full(NPW, -1, np.int32), np.zeros(NPW), beta,
                          np.arange(0, NPROJ + 1, 8, dtype=np.int32), np.ones(8 * NPROJ))
        y = torch.empty_like(x)
        ap.apply_batch(x, y, NVEC, FP64)
        torch.cuda.synchronize()
        return ap.ctx.device_bytes(), y

    def fresh():
        ap = PlanewaveHamiltonianApplicator()
        ap.update_potential(np.zeros(16 ** 3), (16, 16, 16))
        return ap

    roomy, want = apply(fresh())
    free, total = torch.cuda.mem_get_info()
    assert free > total // 4
    ap = fresh()
    other = torch.empty(free - total // 10, dtype=torch.uint8, device="cuda")  # leaves a tenth
    tight, got = apply(ap)
    assert tight < roomy - 60 * NPW * NPROJ  # no residues
    assert float((got - want).norm() / want.norm()) < 1e-13
    del other
    torch.cuda.empty_cache()
    again, got = apply(ap)
    assert again == roomy and torch.equal(got, want)


def test_a_basis_packed_for_two_products_stays_within_bounds(cuda_device):
    """The workspace in which the Davidson's basis is packed whole, once for both subspace rows, ends
    at 4 GB of packed basis (30 bytes an entry, rows padded to 256): above, each product packs it a
    panel at a time, and its workspace is that of one product."""
    import ctypes as C
    from q3_b200 import _lib
    lib = _lib.load()
    two = lib["_ZN3q3b22cgemm_two_wanted_bytesIdEEmiii"]  # size_t q3b::cgemm_two_wanted_bytes<double>(int, int, int)
    two.restype, two.argtypes = C.c_size_t, [C.c_int] * 3
    below, above = 128 * (4 * 2 ** 30 // (128 * 30 * 1024)), 160000
    assert two(1024, 512, below) >= 30 * 1024 * below
    assert two(1024, 512, above) == 0

"""The plane, stick and density kernels for compile-time lengths at every length they exist for,
and the general kernels where an axis has none, against the CPU oracle.

Bars as in test_gpu_hpsi.py and test_gpu_density.py: FP64 1e-12, FP32 2e-5 relative to the
largest entry.  The sphere is off-centre (k != 0) and its stick count is no multiple of the 32
sticks a block takes.
"""
import math

import numpy as np
import pytest

from oracle import density as odens
from oracle import hpsi as ohpsi
from q3_b200 import synthetic
from q3_b200._lib import FP64, MIXED

pytestmark = pytest.mark.gpu

LENGTHS = (16, 18, 20, 24, 25, 27, 30, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 75, 80, 81, 90, 96, 100, 108)
# no square plane, or a stick length without a kernel (12, 15), or a plane length without one
MIXED_GRIDS = ((24, 25, 27), (32, 32, 12), (15, 15, 36), (40, 40, 100), (64, 30, 30))


def _system(grid, nbands):
    shortest = min(grid)
    a = 0.4 * shortest
    gmax = 2.0 * math.pi / a * shortest / 4.4  # products of two bands stay on the grid
    return synthetic.small_system(grid=grid, a=a, ecut=gmax * gmax, natoms=1, nbands=nbands, seed=sum(grid),
                                  k_frac=(0.25, -0.125, 0.375))


@pytest.mark.parametrize("grid", [(n, n, n) for n in LENGTHS] + list(MIXED_GRIDS), ids=str)
def test_kernels_match_the_oracle(cuda_device, grid):
    import torch
    from q3_b200.applicator import PlanewaveHamiltonianApplicator
    sy = _system(grid, 3)
    kp, psi = sy.kpoints[0], sy.psi0[0]
    ap = PlanewaveHamiltonianApplicator()
    ap.update_potential(sy.v_r, sy.cell.grid)
    ap.prepare_system_kpoint(sy)
    ref = ohpsi.apply_h(psi, kp, sy.v_r, sy.cell.grid, threads=8)
    x = torch.from_numpy(np.ascontiguousarray(psi.T)).cuda()
    for precision, tol in ((FP64, 1e-12), (MIXED, 2e-5)):
        for choice in (128, 256, 512):
            ap.set_local_kernel(choice, precision)
            y = torch.full_like(x, np.nan)
            ap.apply_batch(x, y, 3, precision)
            torch.cuda.synchronize()
            assert np.max(np.abs(y.cpu().numpy().T - ref)) / np.max(np.abs(ref)) < tol, (choice, precision)
    w = np.array([0.7, 0.0, 0.3])
    rho = torch.zeros(int(np.prod(grid)), dtype=torch.float64, device="cuda")
    ap.accumulate_density(x, w, rho)
    torch.cuda.synchronize()
    want = odens.accumulate(psi, kp.g_to_grid, sy.cell.grid, w)
    assert np.max(np.abs(rho.cpu().numpy() - want)) / np.max(np.abs(want)) < 1e-12


def test_contexts_that_meet_a_grid_at_once_choose_one_kernel(cuda_device):
    """The tuner's choice is one for all contexts of a process, also when several tune at the same time
    (a server's workers on the first requests): another kernel rounds otherwise."""
    import threading
    from q3_b200.applicator import PlanewaveHamiltonianApplicator
    for n in (30, 36, 45, 48, 54):
        sy = _system((n, n, n), 3)
        aps = [PlanewaveHamiltonianApplicator() for _ in range(8)]
        for ap in aps:
            ap.update_potential(sy.v_r, sy.cell.grid)
            ap.prepare_system_kpoint(sy)
        start, chosen = threading.Barrier(len(aps)), [None] * len(aps)

        def tune(i):
            start.wait()
            chosen[i] = [aps[i].local_kernel(precision) for precision in (FP64, MIXED)]

        threads = [threading.Thread(target=tune, args=(i,)) for i in range(len(aps))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert all(c == chosen[0] for c in chosen), (n, chosen)

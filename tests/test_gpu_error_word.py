"""The device word that a bounded wait sets when it runs out: calls that return host data report it,
and a call that fails on what such a wait left behind reports and clears it.

No wait runs out here.  The word of the context is found by its record {context, address, 16 bytes}
at the front of the context and set from the host, as a kernel would have set it.
"""
import ctypes as C

import numpy as np
import pytest

from q3_b200._lib import ERR_CUDA, ERR_LINALG, Q3BError, check

pytestmark = pytest.mark.gpu


def _set_word(handle):
    words = (C.c_uint64 * 64).from_address(handle)
    at = [words[i + 1] for i in range(62) if words[i] == handle and words[i + 2] == 16]
    assert len(at) == 1
    cudart = C.CDLL("libcudart.so.12")
    cudart.cudaMemset.argtypes = [C.c_void_p, C.c_int, C.c_size_t]
    assert cudart.cudaMemset(at[0], 1, 4) == 0 and cudart.cudaDeviceSynchronize() == 0


@pytest.fixture()
def ap(cuda_device):
    from q3_b200.applicator import PlanewaveHamiltonianApplicator
    ap = PlanewaveHamiltonianApplicator()
    ap.update_potential(np.zeros(512), (8, 8, 8))
    ap.prepare_kpoint(0, 37, (np.arange(37) * 7) % 512, 1.0 + 0.5 * np.arange(37))
    return ap


def _code(call):
    with pytest.raises(Q3BError) as e:
        call()
    return e.value.code


def test_projections_and_rotation_report_it(ap):
    from q3_b200.starting import StartingSubspaceSolver
    sol = StartingSubspaceSolver(ap)
    rng = np.random.default_rng(3)
    chi = rng.standard_normal((37, 4)) + 1j * rng.standard_normal((37, 4))
    sol.apply_hamiltonian(chi, 4)
    for call in (sol.project, lambda: sol.rotate_into_bands(np.eye(4, 2, dtype=complex), 2)):
        _set_word(ap.h)
        assert _code(call) == ERR_CUDA
        call()  # reported once


def test_a_failed_solve_reports_and_clears_it(ap):
    from q3_b200.davidson import hegv
    eye, bad = np.eye(70, dtype=complex), -np.eye(70, dtype=complex)
    assert _code(lambda: hegv(ap, eye, bad)) == ERR_LINALG
    _set_word(ap.h)
    assert _code(lambda: hegv(ap, eye, bad)) == ERR_CUDA
    ap.ctx.synchronize()
    # an error of the arguments leaves it to the call that waits for the work
    _set_word(ap.h)
    assert ap.lib.q3b_apply_h(ap.h, None, None, -1, 0) != 0
    assert _code(ap.ctx.synchronize) == ERR_CUDA
    ap.ctx.synchronize()

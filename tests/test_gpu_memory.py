"""Device memory that the faster moment loops take: none at the upload beyond a byte per site,
none for sets that do not run in strips, and none where it is short (the set then runs step by
step, with the same moments)."""
from __future__ import annotations

import numpy as np
import pytest

import gpuqt_b200 as g
from test_gpu_strip import SQUARE, lattice

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _free():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _phases(n):
    a = np.random.default_rng(n).uniform(0, 2 * np.pi, n)
    return np.cos(a), np.sin(a)


@pytest.mark.parametrize("n0,n1", [(2000, 2001), (400000, 10)])  # in strips; too thin for them
def test_upload_takes_the_operator_alone(n0, n1):
    ell = lattice(SQUARE, n0, n1)
    g.Hamiltonian(**lattice(SQUARE, 8, 8)).close()  # the library's own first allocations
    before = _free()
    H = g.Hamiltonian(**ell)
    # rows of four: neighbour, hopping, xx and code of each entry, the potential; a byte of
    # row pattern; allocations are rounded up to 2 MiB
    assert before - _free() <= ell["n"] * (4 * (4 + 16 + 8 + 1) + 8 + 1) + 16 * MIB
    H.close()


def test_only_sets_in_strips_take_their_memory():
    ell = lattice(SQUARE, 2000, 2001)
    n = ell["n"]
    H = g.Hamiltonian(**ell)
    phi = g.Vector.from_host(*_phases(n))
    used = []
    for window, M in ((0, 2), (4, 30), (0, 30)):
        H.set_loop(window)
        before = _free()
        g.moments(H, phi, phi, M)
        g.moments_doubled(H, phi, min(M, 3))
        used.append(before - _free())
    vectors = 2 * 16 * n
    assert used[0] <= vectors + 80 * MIB  # the recurrence's two vectors, the partial sums
    assert used[1] <= 16 * MIB + 80 * MIB  # the wavefront loop has its own counters
    assert vectors + 15 * n <= used[2] <= vectors + 16 * n + 16 * MIB
    H.close()


def test_short_memory_runs_step_by_step():
    import torch

    ell = lattice(SQUARE, 2400, 2501)
    H = g.Hamiltonian(**ell)
    phi = g.Vector.from_host(*_phases(ell["n"]))

    def run(M):
        g.reset_launch_count()
        mu = g.moments(H, phi, phi, M)
        return mu[0] + 1j * mu[1], g.launch_count()

    # the strip loop would take three times 96 MB; an eighth of what is left is less
    filler = torch.empty(_free() - 1300 * MIB, dtype=torch.uint8, device="cuda")
    tight, steps = run(24)
    assert steps >= 24
    del filler
    torch.cuda.empty_cache()
    again, same = run(24)  # the captured loop
    assert same == steps and np.array_equal(tight, again)
    wide, launches = run(23)
    assert launches < 23
    np.testing.assert_allclose(wide, tight[:23], rtol=0, atol=1e-15 * ell["n"])
    H.close()

"""The benchmark's byte models follow the loop that runs: step by step, or several Chebyshev
steps per launch as the launch counts tell."""
from __future__ import annotations

import pytest

import bench


def test_bytes_per_site_by_the_loop():
    # operator entries and potential, then four (three) streams of 16 bytes
    assert bench.fp64_bytes_per_site(z=6) == 6 + 8 + 64
    assert bench.fp64_bytes_per_site(z=3, coded=False) == 60 + 8 + 64
    assert bench.fp64_pair_bytes_per_site_step(z=6) == 6 + 8 + 48
    # in strips: five (four) vectors and a record per launch
    assert bench.fp64_bytes_per_site(steps=3) == pytest.approx(96 / 3)
    assert bench.fp64_pair_bytes_per_site_step(steps=4) == pytest.approx(80 / 4)


@pytest.mark.parametrize("steps", [1, 3, 4, 6])
@pytest.mark.parametrize("symmetric", [False, True])
def test_steps_per_launch_from_launch_counts(steps, symmetric):
    class Library:
        """Counts launches as the moment loops do: mu_0, T_1, the steps, their sums."""
        count = 0

        def reset_launch_count(self):
            self.count = 0

        def launch_count(self):
            return self.count

        def _set(self, chebyshev_steps):
            self.count += 2 + -(-chebyshev_steps // steps) + (chebyshev_steps > 0)

        def moments(self, H, left, right, n):
            self._set(n - 2)

        def moments_doubled(self, H, x, n):
            self._set(n // 2 - 1)
            self.count += 1

    assert bench.steps_per_launch(Library(), None, None, symmetric) == steps

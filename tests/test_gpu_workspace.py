"""Device memory of a plan: a run of a batch adds its fields and the two stacks of
mean-flow matrices that the step reads (Linv R and Linv, three stages each)."""
import numpy as np
import pytest

from jax_spectral_dns._plan import StepPlan
from jax_spectral_dns.seeds import cheb_points, mode_counts

pytestmark = pytest.mark.gpu


def test_a_run_holds_two_matrix_stacks(cuda):
    ny = 195
    modes, phys = mode_counts((4, ny, 4))
    size = [StepPlan(modes, phys, 2 * np.pi, np.pi, 1, [3000.0] * runs, 0.01, linearise=True,
                     base_u=1 - cheb_points(ny) ** 2).workspace_bytes() for runs in (2, 3)]
    stack = 3 * (2 * ny) ** 2 * 8
    fields = 24 * 16 * ny * modes[0] * modes[2]  # a linearised plan holds 20 fields and some rows per run
    assert 2 * stack < size[1] - size[0] < 2 * stack + fields < 3 * stack

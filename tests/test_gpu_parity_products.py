"""FP64 products on even and odd parts (k_parity) inside the step, against the
oracle: Ny at the edges of the kernel's row tiles (16 j + 1 points: one row
beyond; even Ny: no mid-plane; the smallest that has the form and one below it;
the largest, and one beyond it on the whole operators), column counts that
leave a ragged last tile. Tolerance: the FP64 parity bar of the package."""
import numpy as np
import pytest
import torch

import jsd_oracle as O
from conftest import rel
from jax_spectral_dns._plan import StepPlan, to_device_layout, to_reference_layout
from jax_spectral_dns.seeds import cheb_points, mode_counts, seeded_velocity_hat

pytestmark = pytest.mark.gpu
LX, LZ, RE, DT = 2 * np.pi, np.pi, 4000.0, 0.005


@pytest.mark.parametrize("ny", [9, 10, 17, 18, 19, 34, 49, 50, 66, 82, 98, 130, 131, 145, 161, 193, 195])
@pytest.mark.parametrize("linearise", [False, True])
def test_step_on_even_and_odd_parts(cuda, ny, linearise):
    shape = (4, ny, 8)
    u0 = seeded_velocity_hat(shape, (LX, LZ), (2, 4), 1e-3, seed=ny)
    modes, phys = mode_counts(shape)
    plan = StepPlan(modes, phys, LX, LZ, 1, RE, DT, linearise=linearise, base_u=1 - cheb_points(ny) ** 2)
    st = to_device_layout(u0)
    plan.step(st, torch.zeros(1, dtype=torch.float64, device="cuda"), 0, 2)
    want, _, _ = O.run(O.make_stepper("perturbation", shape, LX, LZ, RE, DT, linearise=linearise), u0, 2)
    assert rel(to_reference_layout(st).cpu().numpy(), want) < 1e-10

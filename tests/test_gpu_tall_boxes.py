"""FP64 steps on both sides of the eigen update's split by Ny (eight parts of the
rows up to 202 points, four beyond), to heights where eight parts would exceed
the shared memory of a block, against the oracle. Tolerance: the FP64 parity bar
of the package, 1e-10 at the bar's tallest box (195), growing like Ny^4 with the
round-off of the second derivative."""
import numpy as np
import pytest
import torch

import jsd_oracle as O
from conftest import rel
from jax_spectral_dns._plan import StepPlan, pack_runs, to_device_layout, to_reference_layout, unpack_runs
from jax_spectral_dns.seeds import cheb_points, mode_counts, seeded_velocity_hat

pytestmark = pytest.mark.gpu
LX, LZ, RE, DT = 2 * np.pi, np.pi, 4000.0, 0.005


@pytest.mark.parametrize("ny", [202, 203, 402, 403, 451])
def test_step(cuda, ny):
    shape = (4, ny, 4)
    u0 = seeded_velocity_hat(shape, (LX, LZ), (2, 2), 1e-3, seed=ny)
    modes, phys = mode_counts(shape)
    plan = StepPlan(modes, phys, LX, LZ, 1, RE, DT, base_u=1 - cheb_points(ny) ** 2)
    st = to_device_layout(u0)
    plan.step(st, torch.zeros(1, dtype=torch.float64, device="cuda"), 0, 1)
    want, _, _ = O.run(O.make_stepper("perturbation", shape, LX, LZ, RE, DT, linearise=False), u0, 1)
    assert rel(to_reference_layout(st).cpu().numpy(), want) < 1e-10 * max(1.0, (ny / 195) ** 4)


@pytest.mark.parametrize("ny", [202, 203])
def test_batch_step(cuda, ny):
    shape = (4, ny, 8)
    modes, phys = mode_counts(shape)
    runs = [(RE, 1e-3), (0.5 * RE, 1e-2)]
    u0 = [seeded_velocity_hat(shape, (LX, LZ), (2, 4), e0, seed=i) for i, (_, e0) in enumerate(runs)]
    plan = StepPlan(modes, phys, LX, LZ, 1, [re for re, _ in runs], DT, base_u=1 - cheb_points(ny) ** 2)
    st = pack_runs(u0)
    plan.step(st, torch.zeros(1, dtype=torch.float64, device="cuda"), 0, 1)
    for got, u, (re, _) in zip(unpack_runs(st), u0, runs):
        want, _, _ = O.run(O.make_stepper("perturbation", shape, LX, LZ, re, DT, linearise=False), u, 1)
        assert rel(got.cpu().numpy(), want) < 1e-10 * max(1.0, (ny / 195) ** 4)

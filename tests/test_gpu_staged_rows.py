"""Inverse z pass with staged input rows: batches large enough to take it, run by
run against plans of one run, which do not (and which the oracle tests cover);
the dual's two field sets at the side that always takes it, against the oracle.
Run counts leave a ragged last block. Tolerances: FP64 1e-12, the bar of a batch
against single runs; mixed 1e-6, the FP32 rounding of its terms; dual 1e-10, the
FP64 parity bar."""
import numpy as np
import pytest
import torch

import jsd_oracle as O
from conftest import rel
from jax_spectral_dns._plan import StepPlan, pack_runs, to_device_layout, to_reference_layout, unpack_runs
from jax_spectral_dns.adjoint import GainProblem, dual_gradient
from jax_spectral_dns.seeds import cheb_points, mode_counts, seeded_velocity_hat

pytestmark = pytest.mark.gpu
LX, LZ, RE, DT = 2 * np.pi, np.pi, 4000.0, 0.005
STAGED = 1 << 19  # entries per field from which the rows are staged


@pytest.mark.parametrize("nz,precision", [(40, "fp64"), (48, "fp64"), (64, "fp64"), (88, "fp64"), (120, "fp64"),
                                          (32, "mixed"), (64, "mixed"), (120, "mixed")])
def test_batch_against_single_runs(cuda, nz, precision):
    shape = (4, 18, nz)
    modes, phys = mode_counts(shape)
    runs = -(-STAGED // int(np.prod(modes)))
    u0 = [seeded_velocity_hat(shape, (LX, LZ), (2, nz // 2), 1e-3, seed=i) for i in range(3)]
    base = 1 - cheb_points(shape[1]) ** 2
    plan = StepPlan(modes, phys, LX, LZ, 1, [RE] * runs, DT, base_u=base, precision=precision)
    st = pack_runs([u0[i % 3] for i in range(runs)])
    plan.step(st, torch.zeros(1, dtype=torch.float64, device="cuda"), 0, 1)
    got = unpack_runs(st)
    one = StepPlan(modes, phys, LX, LZ, 1, RE, DT, base_u=base, precision=precision)
    want = []
    for u in u0:
        s = to_device_layout(u)
        one.step(s, torch.zeros(1, dtype=torch.float64, device="cuda"), 0, 1)
        want.append(to_reference_layout(s))
    for i, g in enumerate(got):
        w = want[i % 3]
        assert float((g - w).norm() / w.norm()) < (1e-12 if precision == "fp64" else 1e-6), i


def test_dual_sets(cuda):
    shape, n = (4, 17, 144), 2
    modes, phys = mode_counts(shape)
    u0 = seeded_velocity_hat(shape, (LX, LZ), (2, 8), 1e-4, seed=5)
    p = GainProblem(modes, phys, LX, LZ, RE, DT, n * DT, False, checkpoint_every=1, gradient="dual")
    g, grad = dual_gradient(torch.as_tensor(u0), p)
    want, gain, _, _ = O.dual_gradient(shape, LX, LZ, RE, DT, n, u0, False)
    assert rel(grad.cpu().numpy(), want) < 1e-10
    assert abs(g / gain - 1) < 1e-10


@pytest.mark.parametrize("runs", [48, 49, 98, 99])
def test_parts_of_the_field_list(cuda, runs):
    """Block counts on both sides of the lines between six, three and one part
    of the field list (24 lines per block: 102, 105, 209 and 211 blocks)."""
    shape = (4, 17, 16)
    modes, phys = mode_counts(shape)
    base = 1 - cheb_points(shape[1]) ** 2
    u = seeded_velocity_hat(shape, (LX, LZ), (2, 8), 1e-3, seed=runs)
    plan = StepPlan(modes, phys, LX, LZ, 1, [RE] * runs, DT, base_u=base)
    st = pack_runs([u] * runs)
    plan.step(st, torch.zeros(1, dtype=torch.float64, device="cuda"), 0, 1)
    want, _, _ = O.run(O.make_stepper("perturbation", shape, LX, LZ, RE, DT, linearise=False), u, 1)
    for got in unpack_runs(st):
        assert rel(got.cpu().numpy(), want) < 1e-10

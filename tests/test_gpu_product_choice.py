"""Which kernel an FP64 plan's y-products run: on even and odd parts for 10 to 194
Chebyshev points, whole operators beyond, and the tile the caller sets for a call
site in place of either. Tolerance: the FP64 parity bar of the package, 1e-10
(1e-12 of |S x| |y| for the transpose)."""
import numpy as np
import pytest
import torch

from conftest import rel
from jax_spectral_dns import _native
from jax_spectral_dns._plan import StepPlan, to_device_layout
from jax_spectral_dns.seeds import cheb_points, mode_counts, seeded_velocity_hat

pytestmark = pytest.mark.gpu
LX, LZ, RE, DT = 2 * np.pi, np.pi, 4000.0, 0.005


def _plan(ny, linearise=False, **kw):
    modes, phys = mode_counts((4, ny, 8))
    return StepPlan(modes, phys, LX, LZ, 1, RE, DT, linearise=linearise, base_u=1 - cheb_points(ny) ** 2, **kw)


def _forms(plan):
    return [plan.even_odd_products(site) for site in _native.GEMM_SITES]


def _step(plan, ny, n=2):
    st = to_device_layout(seeded_velocity_hat((4, ny, 8), (LX, LZ), (2, 4), 1e-3, seed=ny))
    plan.step(st, torch.zeros(1, dtype=torch.float64, device="cuda"), 0, n)
    return st


@pytest.mark.parametrize("ny", [8, 9, 10, 17, 18, 19, 34, 49, 50, 65, 66, 82, 98, 129, 130, 131, 145, 161, 193, 194,
                                195, 196])
def test_form_by_points(cuda, ny):
    even_odd = 10 <= ny <= 194
    plan = _plan(ny)
    assert _forms(plan) == [even_odd] * 3
    assert _forms(_plan(ny, linearise=True)) == [even_odd] * 3
    assert _forms(_plan(ny, precision="mixed")) == [False] * 3
    default = _step(plan, ny)
    for site in _native.GEMM_SITES:
        plan.set_gemm_config(site, 1)
    assert _forms(plan) == [False] * 3
    whole = _step(plan, ny)
    # another order of summation: other bits, the same numbers
    assert torch.equal(whole, default) == (not even_odd)
    assert rel(whole.cpu().numpy(), default.cpu().numpy()) < 1e-10


def test_set_tiles_take_effect_site_by_site_and_agree(cuda):
    ny, out = 33, []
    for config in range(_native.DGEMM_CONFIGS):
        plan = _plan(ny)
        for i, site in enumerate(_native.GEMM_SITES):
            plan.set_gemm_config(site, config)
            assert _forms(plan) == [j > i for j in range(3)]
        out.append(_step(plan, ny))
    assert all(torch.equal(o, out[0]) for o in out)  # every tile sums over K in the same order


def test_int8_products_take_the_place_of_either(cuda):
    plan = _plan(33)
    plan.set_eig_kernel(1, 1)
    assert _forms(plan) == [True, False, True]
    plan.set_eig_kernel(1, 0)
    assert _forms(plan) == [True] * 3


def test_autotune_returns_to_the_plans_own_choice(cuda):
    plan, fresh = _plan(33), _plan(33)
    for site in _native.GEMM_SITES:
        plan.set_gemm_config(site, 0)
    plan.autotune()
    assert _forms(plan) == [True] * 3
    plan.set_xmid_variant(fresh.xmid_variant()[0])
    assert torch.equal(_step(plan, 33), _step(fresh, 33))


@pytest.mark.parametrize("ny", [10, 17, 18, 33, 130, 145, 193, 195])
@pytest.mark.parametrize("tiles", [False, True])
def test_adjoint_is_the_transpose_in_either_form(cuda, ny, tiles):
    plan = _plan(ny, linearise=True)
    if tiles:
        for site in _native.GEMM_SITES:
            plan.set_gemm_config(site, 0)
    mx, _, mz = plan.modes
    gen = torch.Generator(device="cpu").manual_seed(ny)
    x, y = (torch.randn((3, ny, mx, mz), dtype=torch.complex128, generator=gen).cuda() for _ in range(2))
    sx, sty = x.clone(), y.clone()
    plan.step(sx, torch.zeros(1, dtype=torch.float64, device="cuda"), 0, 1)
    plan.step_adjoint(sty, 1)
    dot = lambda a, b: torch.sum(a.real * b.real + a.imag * b.imag).item()  # noqa: E731
    assert abs(dot(sx, y) - dot(x, sty)) < 1e-12 * (sx.abs().norm() * y.abs().norm()).item()


@pytest.mark.parametrize("ny", [10, 33, 34, 195])
@pytest.mark.parametrize("tiles", [False, True])
def test_profile_counts_the_operations_that_run(cuda, ny, tiles):
    """FLOPs of the product class over one step: D on three (first stage) or two
    fields, three products into the eigenbasis and one more in the first stage
    (V^-1 omega_y) with V^-1 v, three out of it; on even and odd parts each whole
    product M x K counts M / 2 x K / 2 twice (halves rounded up and down)."""
    plan = _plan(ny)
    if tiles:
        for site in _native.GEMM_SITES:
            plan.set_gemm_config(site, 0)
    plan.profile(True)
    _step(plan, ny, 1)
    _, _, work = plan.profile_read("gemm")
    plan.profile(False)
    mx, _, mz = plan.modes
    halves = 10 <= ny <= 194 and not tiles

    def product(m, k, crossed):
        if not halves:
            return m * k
        (me, mo), (ke, ko) = ((m + 1) // 2, m // 2), ((k + 1) // 2, k // 2)
        return me * ko + mo * ke if crossed else me * ke + mo * ko

    n = ny - 2
    d, vd, vi, v, dv = (product(ny, ny, True), product(n, ny, True), product(n, n, False), product(ny, n, False),
                        product(ny, n, True))
    fields = (3 + 2 + 2) * d + 3 * (vd + 2 * vi + 2 * v + dv) + 2 * vi
    assert work == 2.0 * fields * 2 * mx * mz

"""GPU tests of the FP64 transforms in block fixed point: the sizes and radix
orders at which their passes change, the spectra that ask for the fewest and
the most shifted bits, and the range of exponents.

Tolerances: one right-hand side against the FP64 oracle has the repository's
bar of 1e-13 (relative L2); what must not depend on the launch shape or the
exponent is compared bit for bit."""

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mods(built_lib):
    from spectral2d_gb300 import Ensemble, Spectral2D
    return Ensemble, Spectral2D


def _rhs_error(S2D, n, w, plan=0, form="basdevant", nu=0.01):
    g = O.get_grid_size(n, n)
    w = O.truncate(w, g)
    psi = O.truncate(O.compute_psi(w, g), g)
    with S2D(n, nu=nu, nonlinear_form=form) as s:
        s.fft_plan = plan
        s.set_state(w)
        dW = s.compute_rhs()
    ref, _ = O.compute_rhs(w, psi, g, nu, round_trip=False)
    return O.rel_l2(dW, O.truncate(ref, g))


# radices 3,4 / 3,2,4 / 3,3,4 / ... / 3^4,4; 512 | 576: the last size with 4
# elements per thread and the first with 12
@pytest.mark.parametrize("plan", [0, 1, 2])
@pytest.mark.parametrize("n", [8, 16, 24, 48, 72, 144, 216, 432, 512, 576, 768])
def test_rhs_at_every_kind_of_plan(mods, n, plan):
    _, S2D = mods
    w = O.random_state(O.get_grid_size(n, n), 7 + n, decay=0.02)
    assert _rhs_error(S2D, n, w, plan) < 1e-13


def _transform_bound(w, g, form):
    """2-norm of the right-hand side's error if every transform is exact to
    2e-16 of its result's 2-norm (what an FP64 FFT of these lengths has): four
    transforms and two roundings stand between w and F[product], whose modes
    the form weights by up to K^2 or K; the oracle has the same error."""
    K, M = g.nx // 2, g.nxG
    kx = np.arange(g.cISize)[None, :]
    ky = np.fft.fftfreq(M, 1.0 / M)[:, None]
    psi = O.truncate(O.compute_psi(w, g), g)
    phys = lambda f: np.fft.irfft(np.fft.ifft(f, axis=0) * M, n=M, axis=1) * M   # noqa: E731
    spec = lambda p: np.linalg.norm(np.fft.rfft2(p)) / M ** 2                   # noqa: E731
    u, v, wp = phys(1j * ky * psi), phys(-1j * kx * psi), phys(w)
    if form == "basdevant":
        weight, size = K * K, spec(u * v) + spec(v * v - u * u)
    else:
        weight, size = K, spec(u * wp) + spec(v * wp)
    return 2 * 6 * 2e-16 * weight * size


@pytest.mark.parametrize("form", ["basdevant", "conservative"])
@pytest.mark.parametrize("kind", ["white", "steep", "one_mode", "one_mode_and_noise", "zero"])
@pytest.mark.parametrize("n", [64, 648])
def test_rhs_of_white_steep_and_single_mode_spectra(mods, n, kind, form):
    """Steep spectra have right-hand sides far smaller than their transforms'
    terms, so the error is held to the transforms' accuracy, not to a fraction
    of the result."""
    _, S2D = mods
    g = O.get_grid_size(n, n)
    rnd = O.random_state(g, 3, decay=0.0)
    if kind == "white":
        w = rnd
    elif kind == "steep":
        w = O.random_state(g, 3, decay=0.6)
    else:
        w = np.zeros_like(rnd)
        if kind != "zero":
            w[3, 2] = 1.0 + 0.5j
            w[1, 5] = 0.25j
        if kind == "one_mode_and_noise":
            w = w + 1e-9 * rnd
    w = O.truncate(w, g)
    with S2D(n, nu=0.01, nonlinear_form=form) as s:
        s.set_state(w)
        dW = s.compute_rhs()
    if kind == "zero":
        assert np.all(dW == 0.0)
        return
    ref, _ = O.compute_rhs(w, O.truncate(O.compute_psi(w, g), g), g, 0.01, round_trip=False)
    visc = 4 * 2.0 ** -53 * 0.01 * (n // 2) ** 2 * np.linalg.norm(w)
    assert np.linalg.norm(dW - O.truncate(ref, g)) <= _transform_bound(w, g, form) + visc


@pytest.mark.parametrize("n", [48, 576])
@pytest.mark.parametrize("k", [-300, -1, 200])
def test_rhs_scales_exactly_with_powers_of_two(mods, n, k):
    """Without viscosity the right-hand side is quadratic: w 2^k gives 2^(2k)
    times the same bits, for exponents far from 0 too."""
    _, S2D = mods
    w = O.truncate(O.random_state(O.get_grid_size(n, n), 5, decay=0.05), O.get_grid_size(n, n))
    out = []
    with S2D(n, nu=0.0) as s:
        for e in (0, k):
            s.set_state(w * 2.0 ** e)
            out.append(s.compute_rhs())
    assert np.array_equal(out[1], out[0] * 2.0 ** (2 * k))


@pytest.mark.parametrize("n", [64, 576])
def test_an_infinity_reaches_every_mode(mods, n):
    _, S2D = mods
    g = O.get_grid_size(n, n)
    w = O.truncate(O.random_state(g, 5, decay=0.05), g)
    w[2, 3] = complex(np.inf, 0.0)
    with S2D(n, nu=0.01) as s:
        s.set_state(w)
        dW = s.compute_rhs()
    keep = O.truncate(np.ones_like(w), g) != 0
    assert not np.any(np.isfinite(dW[keep]))


@pytest.mark.parametrize("n", [256, 512])
def test_four_and_twelve_elements_per_thread_give_the_same_bits(mods, n):
    """A batch runs 12 elements per thread at every size, a run alone 4."""
    Ensemble, S2D = mods
    w = O.truncate(O.random_state(O.get_grid_size(n, n), 9, decay=0.05), O.get_grid_size(n, n))
    with Ensemble([n], [1e-3]) as ens, S2D(n, nu=1e-3) as s:
        ens.runs[0].set_state(w)
        ens.set_dt([1e-3])
        ens.integrate_steps(2)
        s.set_state(w)
        s.integrate_steps(2, 1e-3)
        assert np.array_equal(ens.runs[0].get_state()[0], s.get_state()[0])


# the conservative x-pass: three groups of 4 elements per thread up to n = 256
# (FP64) or 384 (FP32), three of 12 up to 576, one group above; the orders of
# the radices at each
@pytest.mark.parametrize("plan", [0, 1, 2])
@pytest.mark.parametrize("precision, tol", [("fp64", 1e-13), ("fp32", 5e-6)])
@pytest.mark.parametrize("n", [8, 24, 256, 288, 384, 432, 576, 648])
def test_conservative_rhs_at_the_sizes_where_its_kernel_changes(mods, n, precision, tol, plan):
    _, S2D = mods
    g = O.get_grid_size(n, n)
    w = O.truncate(O.random_state(g, 7 + n, decay=0.02), g)
    with S2D(n, nu=0.01, nonlinear_form="conservative", precision=precision) as s:
        s.fft_plan = plan
        s.set_state(w)
        dW = s.compute_rhs()
    ref, _ = O.compute_rhs(w, O.truncate(O.compute_psi(w, g), g), g, 0.01, round_trip=False)
    assert O.rel_l2(dW, O.truncate(ref, g)) < tol

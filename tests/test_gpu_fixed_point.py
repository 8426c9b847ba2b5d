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


def _flow_of_y_and_perturbation(n, amp):
    """A vorticity that depends on y alone, and a perturbation (kx > 0) of largest mode amp times its own."""
    g = O.get_grid_size(n, n)
    ky = np.fft.fftfreq(g.nyG, 1.0 / g.nyG)
    base = np.zeros((g.nyG, g.cISize), complex)
    base[np.abs(ky) == 4, 0] = 2.0
    pert = O.truncate(O.random_state(g, 3, decay=0.2), g)
    pert[:, 0] = 0
    return g, base, pert * (2.0 * amp / np.abs(pert).max())


def _perturbed_tendency(g, base, pert, form):
    """The inviscid tendency of base + pert from the products of base and perturbation, formed apart (so that its errors
    are relative to the perturbation), and the bounds on the 2-norm of a right-hand side's error in kx > 0 and in kx = 0:
    _transform_bound with the products that are linear in the perturbation, and with the quadratic ones."""
    M, K = g.nxG, g.nx // 2
    kx = np.arange(g.cISize)[None, :]
    ky = np.fft.fftfreq(M, 1.0 / M)[:, None]
    phys = lambda f: np.fft.irfft(np.fft.ifft(f, axis=0) * M, n=M, axis=1) * M   # noqa: E731
    spec = lambda p: np.fft.rfft2(p) / M ** 2                                   # noqa: E731
    norm = lambda *ps: sum(np.linalg.norm(spec(p)) for p in ps)                 # noqa: E731
    psi0, psi1 = (O.truncate(O.compute_psi(w, g), g) for w in (base, pert))
    u0, w0 = phys(1j * ky * psi0), phys(base)
    u1, v1, w1 = phys(1j * ky * psi1), phys(-1j * kx * psi1), phys(pert)
    lin = -1j * kx * spec(u0 * w1 + w0 * u1) - 1j * ky * spec(v1 * w0)
    lin[:, 0] = 0   # its x-means vanish
    dW = O.truncate(lin - 1j * kx * spec(u1 * w1) - 1j * ky * spec(v1 * w1), g)
    if form == "basdevant":
        weight, linear, quad = K * K, norm(u0 * v1, 2 * u0 * u1), norm(u1 * v1, v1 * v1 - u1 * u1)
    else:
        weight, linear, quad = K, norm(u0 * w1, w0 * u1, v1 * w0), norm(u1 * w1, v1 * w1)
    per = 2 * 6 * 2e-16 * weight
    return dW, per * (linear + quad), per * quad


# plan 2 (FP64): the general transform; 64 | 768: 4 and 12 elements per thread,
# three groups and one; amp 0.1: the means stay in the transforms, or not, row by row
@pytest.mark.parametrize("form", ["basdevant", "conservative"])
@pytest.mark.parametrize("plan", [0, 2])
@pytest.mark.parametrize("amp", [0.1, 1e-3, 1e-6, 1e-10])
@pytest.mark.parametrize("n", [64, 96, 768])
def test_weak_perturbations_keep_their_bits_beside_a_large_mean(mods, n, amp, plan, form):
    """An FP64 transform of u + i v adds a row's mean u in butterflies without
    twiddles, so a weak v keeps its own 53 bits; ky = 0 and kx = 0 (in which
    the base flow has no linear term of u u) show it."""
    _, S2D = mods
    g, base, pert = _flow_of_y_and_perturbation(n, amp)
    ref, bound, bound0 = _perturbed_tendency(g, base, pert, form)
    with S2D(n, nu=0.0, nonlinear_form=form) as s:
        s.fft_plan = plan
        s.set_state(base)
        alone = s.compute_rhs()
        s.set_state(base + pert)
        dW = s.compute_rhs()
    assert np.all(alone == 0.0)
    err = dW - ref
    assert np.linalg.norm(err[:, 1:]) <= bound
    if amp <= 1e-3:   # (else not all rows' means stand apart)
        assert np.linalg.norm(err[:, 0]) <= bound0
        assert np.all(np.abs(err[0, 1:5]) <= 5e-14 * np.abs(ref[0, 1:5]))


def test_a_batch_and_a_run_alone_agree_beside_a_large_mean(mods):
    Ensemble, S2D = mods
    for n, amp in ((64, 1e-6), (128, 0.1)):
        _, base, pert = _flow_of_y_and_perturbation(n, amp)
        with Ensemble([n], [1e-3]) as ens, S2D(n, nu=1e-3) as s:
            ens.runs[0].set_state(base + pert)
            ens.set_dt([1e-3])
            ens.integrate_steps(2)
            s.set_state(base + pert)
            s.integrate_steps(2, 1e-3)
            assert np.array_equal(ens.runs[0].get_state()[0], s.get_state()[0])


@pytest.mark.parametrize("form", ["basdevant", "conservative"])
@pytest.mark.parametrize("plan", [0, 2])
@pytest.mark.parametrize("n", [64, 576, 768])
def test_results_below_the_normal_range_are_gradual(mods, n, plan, form):
    """w 2^k, k chosen so that the products' spectra are subnormal numbers: 2^(2k) times the right-hand side to the
    rounding of the x-pass's results and of K3's, half of 2^-1074 each: M rows are summed, and a mode's two products
    weighed by up to K^2 (four parts, real and imaginary)."""
    _, S2D = mods
    g = O.get_grid_size(n, n)
    w = O.truncate(O.random_state(g, 5, decay=0.1), g)
    with S2D(n, nu=0.0, nonlinear_form=form) as s:
        s.fft_plan = plan
        s.set_state(w)
        dW = s.compute_rhs()
        k = -int((1040 + np.log2(np.abs(dW).max())) / 2)
        s.set_state(w * 2.0 ** k)
        low = s.compute_rhs()
    K = n // 2
    weight = K * K if form == "basdevant" else K
    ulp = 2.0 ** -1074
    want = dW * 2.0 ** k * 2.0 ** k
    assert np.abs(want).max() > 1000 * weight * ulp
    assert np.abs(low - want).max() <= 4 * weight * (g.nxG / 2 + 1) * ulp


@pytest.mark.parametrize("n", [8, 64, 96])
def test_the_allocation_free_rhs_keeps_weak_perturbations_too(built_lib, n):
    """Its x-pass scales the products itself (u and v come unscaled); 8^2: one
    thread per transform, 32 of them in a CTA."""
    torch = pytest.importorskip("torch")
    import ctypes as C

    from spectral2d_gb300 import _lib as L
    g, base, pert = _flow_of_y_and_perturbation(n, 1e-6)
    ref, bound, bound0 = _perturbed_tendency(g, base, pert, "basdevant")
    w = torch.from_numpy((base + pert).view(np.float64).copy()).cuda()
    dW = torch.full_like(w, float("nan"))
    torch.cuda.synchronize()
    assert L.lib().s2d_compute_rhs_noalloc(n, 0.0, C.c_void_p(w.data_ptr()), C.c_void_p(dW.data_ptr()), None) == 0
    torch.cuda.synchronize()
    err = dW.cpu().numpy().view(np.complex128).reshape(ref.shape) - ref
    assert np.linalg.norm(err[:, 1:]) <= bound and np.linalg.norm(err[:, 0]) <= bound0

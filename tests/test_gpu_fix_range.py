"""Exponents of the FP64 form's fixed-point passes: components of very different
sizes beside each other, and states near the ends of the double range."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def field(n, seed):
    """Random solenoidal velocity coefficients of order n^3, Nyquist-free."""
    rng = np.random.default_rng(seed)
    k = np.fft.fftfreq(n, 1.0 / n)
    kx, ky, kz = k[:, None, None], k[None, :, None], np.arange(n // 2 + 1)[None, None, :].astype(float)
    k2 = kx * kx + ky * ky + kz * kz
    amp = np.exp(-k2 / 18.0) * (np.sqrt(k2) < n // 2)
    u = [np.fft.rfftn(rng.standard_normal((n, n, n))) * amp for _ in range(3)]
    d = (kx * u[0] + ky * u[1] + kz * u[2]) / np.where(k2 > 0, k2, 1.0)
    return [u[0] - kx * d, u[1] - ky * d, u[2] - kz * d]


def nonlinear(n, u):
    import vonkarman_gb300 as vk
    from vonkarman_gb300.solver import compute_nonlinear

    with vk.Periodic3D(vk.GridSpec(n), 1e-3, field(n, 1), vk.SolverOptions()) as s:
        return [np.array(c) for c in compute_nonlinear(s, u)]


# padded lines of 24 and 96 points (two stages) and 192 (three)
@pytest.mark.parametrize("n", [16, 64, 128])
@pytest.mark.parametrize("p", [-450, -300, 300, 450])
def test_nonlinear_scales_with_the_square(n, p):
    # a power of two commutes with every rounding inside the double range
    u = field(n, 5)
    one = nonlinear(n, u)
    got = nonlinear(n, [np.ldexp(c.real, p) + 1j * np.ldexp(c.imag, p) for c in u])
    for a, b in zip(got, one):
        assert np.array_equal(np.ldexp(a.real, -2 * p), b.real)
        assert np.array_equal(np.ldexp(a.imag, -2 * p), b.imag)


def test_nonlinear_past_the_range():
    u = field(16, 6)
    for c in nonlinear(16, [np.ldexp(c.real, -600) + 1j * np.ldexp(c.imag, -600) for c in u]):
        assert not c.any()
    big = nonlinear(16, [np.ldexp(c.real, 560) + 1j * np.ldexp(c.imag, 560) for c in u])
    assert not all(np.isfinite(c).all() for c in big)
    for c in nonlinear(16, [np.zeros_like(c) for c in u]):
        assert not c.any()


@pytest.mark.parametrize("n", [16, 64, 128])
@pytest.mark.parametrize("p", [40, 120])
def test_small_component_beside_large_ones(n, p):
    # u_x, u_y and u_z depend on x and y alone: the nonlinear term's z component is
    # linear in u_z.  Its error is relative to itself: a few roundings of the
    # passes, which differ with the exponents (2^-53 each, eight passes)
    rng = np.random.default_rng(7)
    k = np.fft.fftfreq(n, 1.0 / n)
    k2 = k[:, None] ** 2 + k[None, :] ** 2
    amp = np.exp(-k2 / 18.0) * (np.sqrt(k2) < n // 2)
    psi, w = (np.fft.fft2(rng.standard_normal((n, n))) * amp * n for _ in range(2))
    u = [np.zeros((n, n, n // 2 + 1), dtype=complex) for _ in range(3)]
    u[0][:, :, 0], u[1][:, :, 0] = 1j * k[None, :] * psi, -1j * k[:, None] * psi
    u[2][:, :, 0] = w
    one = nonlinear(n, u)[2]
    u[2] = u[2] * 2.0 ** -p
    got = nonlinear(n, u)[2] * 2.0 ** p
    assert np.linalg.norm(one) > 0.0
    assert np.linalg.norm(got - one) < 2.0 ** -50 * np.linalg.norm(one)


@pytest.mark.parametrize("shape", [(8, 12, 16), (16, 16, 192)])
def test_denormals(shape):
    # whole multiples of 2^-1074 below 2^-1042: every pass rounds to that unit, of
    # values around 2^29 of them
    import vonkarman_gb300 as vk

    m = np.random.default_rng(9).integers(-2 ** 31, 2 ** 31, shape).astype(float)
    f = vk.GpuFftBackend(*shape)
    got = f.r2c_3d(np.ldexp(m, -1074))
    f.close()
    got = np.ldexp(got.real, 1074) + 1j * np.ldexp(got.imag, 1074)
    want = np.fft.rfftn(m)
    assert np.linalg.norm(got - want) < 2.0 ** -26 * np.linalg.norm(want)


@pytest.mark.parametrize("n", [16, 64])
def test_columns_of_very_different_sizes(n):
    # a narrow vortex: the columns fall from 1 to round-off within the box
    from oracle import vk_oracle as vo

    g = vo.Grid(n)
    x = 2.0 * np.pi * np.arange(n) / n - np.pi
    r2 = x[:, None, None] ** 2 + x[None, :, None] ** 2 + 0.3 * x[None, None, :] ** 2
    psi = np.fft.rfftn(np.exp(-r2 / 0.3))
    k = np.fft.fftfreq(n, 1.0 / n)
    k[n // 2] = 0.0
    u = [1j * k[None, :, None] * psi, -1j * k[:, None, None] * psi, np.zeros_like(psi)]
    u = [c * (np.arange(n // 2 + 1) < n // 2) for c in u]
    want = vo.compute_nonlinear(vo.SpectralOps(g), [c.copy() for c in u])
    got = nonlinear(n, u)
    err = np.sqrt(sum(np.linalg.norm(a - b) ** 2 for a, b in zip(got, want)))
    assert err < 1e-13 * np.sqrt(sum(np.linalg.norm(b) ** 2 for b in want))

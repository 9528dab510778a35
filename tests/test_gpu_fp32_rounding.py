"""Rounding of the state in a step of the FP32-bulk form."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def field(n, seed):
    rng = np.random.default_rng(seed)
    k = np.fft.fftfreq(n, 1.0 / n)
    kx, ky, kz = k[:, None, None], k[None, :, None], np.arange(n // 2 + 1)[None, None, :].astype(float)
    k2 = kx * kx + ky * ky + kz * kz
    amp = np.exp(-k2 / 18.0) * (np.sqrt(k2) < n // 2)
    u = [np.fft.rfftn(rng.standard_normal((n, n, n))) * amp for _ in range(3)]
    d = (kx * u[0] + ky * u[1] + kz * u[2]) / np.where(k2 > 0, k2, 1.0)
    return k2, [(c - q * d).astype(np.complex64).astype(complex) for c, q in zip(u, (kx, ky, kz))]


@pytest.mark.parametrize("variant", ["reference", "cox-matthews"])
@pytest.mark.parametrize("n", [16, 64])
def test_one_rounding_at_the_size_of_the_state(n, variant):
    # u' = E u + increment with E rounded to single precision: half a unit of u' for
    # the sum, and for the increment, below 2^-6 of u', its own few 2^-24 (0.1 of a unit)
    import vonkarman_gb300 as vk

    nu, dt = 1e-3, 2e-4
    k2, u = field(n, 3)
    out = []
    for precision in ("fp64", "fp32bulk"):
        opts = vk.SolverOptions(precision=precision, etd_variant=variant, dt_mode="fixed", dt_fixed=dt)
        with vk.Periodic3D(vk.GridSpec(n), nu, u, opts) as s:
            s.step(1)
            out.append([np.array(c) for c in s.u_hat()])
    e = np.exp(-nu * k2 * dt)
    e32 = e.astype(np.float32).astype(float)
    worst, count = 0.0, 0
    for c in range(3):
        want = out[0][c] + (e32 - e) * u[c]
        inc = out[0][c] - e * u[c]
        for w, g, d in ((want.real, out[1][c].real, inc.real), (want.imag, out[1][c].imag, inc.imag)):
            big = (np.abs(w) > 64.0 * np.abs(d)) & (np.abs(w) > np.abs(w).max() / 64.0)
            ulp = np.spacing(np.abs(w[big]).astype(np.float32)).astype(float)
            worst, count = max(worst, float((np.abs(g - w)[big] / ulp).max())), count + int(big.sum())
    assert count > 1000
    assert worst < 0.6

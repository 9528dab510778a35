"""Exact zeros on the FP64 form's main path: a flow that does not depend on one
direction stays two-dimensional."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def planar_state(n, axis, seed):
    """Random solenoidal field that does not depend on `axis`, without a
    component along it."""
    rng = np.random.default_rng(seed)
    k = np.fft.fftfreq(n, 1.0 / n)
    p, q = [a for a in range(3) if a != axis]
    kp, kq = k[:, None], k[None, :]
    amp = np.exp(-np.hypot(kp, kq) / 3.0) * (np.hypot(kp, kq) < n // 2)
    psi = np.fft.ifft2(np.fft.fft2(rng.standard_normal((n, n))) * amp)
    hat = np.fft.fft2(psi.real)
    plane = {p: 1j * kq * hat, q: -1j * kp * hat}
    u = []
    for c in range(3):
        full = np.zeros((n, n, n), dtype=complex)
        if c != axis:
            index = [slice(None)] * 3
            index[axis] = 0
            full[tuple(index)] = plane[c] * n
        u.append(full[:, :, :n // 2 + 1].copy())
    return u


# two-stage lines of 24 and 96 points and three-stage ones of 192
@pytest.mark.parametrize("n", [16, 64, 128])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("integrator", ["etd-rk4", "rk4"])
def test_planar_flow_stays_planar(n, axis, integrator):
    import vonkarman_gb300 as vk

    u = planar_state(n, axis, 3)
    opts = vk.SolverOptions(integrator=integrator, dt_mode="fixed", dt_fixed=1e-3)
    with vk.Periodic3D(vk.GridSpec(n), 1e-3, u, opts) as s:
        s.step(3)
        out = s.u_hat()
    moved = 0.0
    for c in range(3):
        index = [slice(None)] * 3
        index[axis] = slice(1, None)
        assert not out[c][tuple(index)].any(), c   # no other wave number along the axis
        if c == axis == 2:   # (the others share a packed z line with a component that is not zero)
            assert not out[c].any()
        moved = max(moved, float(np.abs(out[c] - u[c]).max()))
    assert moved > 0.0

"""The FP64 form's fixed-point transforms on the GPU at the edges of their
ranges: line classes (zero, tiny, huge, non-finite) and mixed axis lengths."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# each axis pass is within 2^-52 of the norm (vk_fix.cuh), numpy's own error is
# of the same order: four ulps for the three passes and the comparison
TOL = 4.0 * 2.0 ** -52


def backend(shape):
    import vonkarman_gb300 as vk

    return vk.GpuFftBackend(*shape)


def rel(a, b, scale):
    return np.linalg.norm((a - b) / scale) / np.linalg.norm(b / scale)


@pytest.mark.parametrize("shape", [(8, 12, 16), (24, 32, 48), (64, 96, 8), (12, 8, 128), (192, 24, 24), (16, 48, 256),
                                   (8, 384, 12), (512, 8, 64), (8, 16, 768), (768, 12, 8)])
@pytest.mark.parametrize("scale", [1e-290, 1.0, 1e290])
def test_lengths_and_ranges(shape, scale):
    x = np.random.default_rng(3).standard_normal(shape)
    f = backend(shape)
    want = np.fft.rfftn(x)
    got = f.r2c_3d(x * scale)
    assert rel(got, want * scale, scale) < TOL
    assert rel(f.c2r_3d(want * scale), x * scale, scale) < 2 * TOL   # the error of `want` itself included
    f.close()


@pytest.mark.parametrize("shape", [(16, 16, 16), (48, 32, 64), (96, 192, 24)])
def test_zero_lines_stay_zero(shape):
    f = backend(shape)
    x = np.zeros(shape)
    assert not f.r2c_3d(x).any()
    x[1, 2, 3] = 1.0      # most z and y lines are zero
    assert rel(f.r2c_3d(x), np.fft.rfftn(x), 1.0) < TOL
    x[...] = 0.0
    x[:, :, 0] = 1e-200   # tiny lines beside zero lines
    assert rel(f.r2c_3d(x), np.fft.rfftn(x), 1e-200) < TOL
    f.close()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_lines(bad):
    shape = (32, 24, 64)
    f = backend(shape)
    x = np.random.default_rng(4).standard_normal(shape)
    x[5, 6, 7] = bad
    assert not np.isfinite(f.r2c_3d(x)).any()   # every output sums the bad input
    f.close()

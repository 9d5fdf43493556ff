"""Spectra, correlations and quadrants of fields whose sizes change the
kernels' shapes: lengths 1 and 2, odd, even, prime and multiples of eight
around eight lags per thread, lines long enough that a block takes fewer
values or reads its twiddles from global memory, and fewer planes than a
group of values.  The sums are FP64 over at most n terms of one size: errors
of order n * 2^-53 of the sum of the terms' magnitudes (n < 2e4: 1e-11 of the
largest value with a margin of five)."""
import numpy as np
import pytest

import dnslbm
import inputs

pytestmark = pytest.mark.gpu
SHAPES = [(1, 1, 1), (2, 3, 1), (7, 8, 2), (16, 17, 5), (31, 64, 6), (67, 40, 9), (2048, 3, 1), (5, 1500, 2)]


def _field(nx, ny, nz, seed):
    rng = np.random.default_rng(seed)
    vel = np.zeros((nx, ny, nz + 2, 3))
    vel[:, :, 1:-1] = 0.05 * rng.standard_normal((nx, ny, nz, 3)) + [0.08, 0.0, 0.0]
    return vel


def _close(got, want):
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-11 * max(np.abs(want).max(), 1e-300))


@pytest.mark.parametrize("shape", SHAPES + [(7200, 2, 1), (2, 2900, 1)])
def test_spectra(shape):
    nx, ny, nz = shape
    vel = _field(nx, ny, nz, 3)
    c = np.fft.fft(np.fft.rfft(vel[:, :, 1:-1], axis=1), axis=0) / (nx * ny)
    c[0, 0] = 0
    p = 0.5 * np.abs(c) ** 2
    p[:, 1:] *= 2
    ex, ey = dnslbm.spectra_vel(vel)
    _close(ex[:, :, 1:-1], p.sum(1).transpose(2, 0, 1))
    _close(ey[:, :, 1:-1], p.sum(0).transpose(2, 0, 1))
    assert not ex[:, :, [0, -1]].any() and not ey[:, :, [0, -1]].any()


@pytest.mark.parametrize("shape", SHAPES)
def test_correlations(shape):
    nx, ny, nz = shape
    vel = _field(nx, ny, nz, 4)
    m = vel[:, :, 1:-1].mean((0, 1))
    m = 0.5 * (m + m[::-1] * [1, 1, -1])
    q = vel.copy()
    q[:, :, 1:-1] -= m
    xc, yc, ua = dnslbm.correlations_vel(vel)
    for axis, got, n in ((0, xc, nx), (1, yc, ny)):
        want = np.stack([(q * np.roll(q, -d, axis)).sum((0, 1)) for d in range(n)], 1)
        _close(got, want)
    _close(ua[1:-1], m[:, 0])


@pytest.mark.parametrize("shape", SHAPES[3:])
def test_quadrants(shape):
    nx, ny, nz = shape
    vel = _field(nx, ny, nz, 5)
    inner = vel[:, :, 1:-1]
    d = inner - inner.mean((0, 1))
    u, w = d[..., 0], d[..., 2]
    _, dq, uw = dnslbm.quadrant_vel(vel)
    for i, s in enumerate(((u > 0) & (w > 0), (u < 0) & (w > 0), (u < 0) & (w < 0), (u > 0) & (w < 0))):
        _close(dq[i, 1:-1], (u * w * s).sum((0, 1)) / (nx * ny))
    _close(uw[1:-1], (u * w).sum((0, 1)) / (nx * ny))


@pytest.mark.parametrize("prec", [64, 32, 16])
@pytest.mark.parametrize("shape", [(33, 5, 6), (32, 3, 14), (2, 2, 3), (70, 4, 9)])
def test_moments_of_a_state(shape, prec):
    """Tiles of 32 x 8 planes (walls included) of one y: edges of both.  The
    fields against the stored populations: 19 FP64 additions in the same order
    and one division, up to the stored values' own rounding (none here: they
    are read back from the same state); wall planes are zero."""
    nx, ny, nz = shape
    with dnslbm.Channel(nx, ny, nz, 1.7, gx=2e-5, precision=prec) as ch:
        ch.load_state(inputs.laminar_state(nx, ny, nz, 0.06, 0.1, 3))
        for steps in (0, 1, 1):
            ch.step(steps)
            f = ch.store_state()
            vel, den = ch.moments()
            e = np.asarray(inputs.E, float)
            rho = f.sum(-1)
            np.testing.assert_allclose(den, rho, rtol=0, atol=1e-14)
            j = f @ e
            j[:, :, 1:-1] /= rho[:, :, 1:-1, None]
            np.testing.assert_allclose(vel, j, rtol=0, atol=1e-14)
            assert not vel[:, :, [0, -1]].any() and not den[:, :, [0, -1]].any()

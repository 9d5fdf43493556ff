"""The persistent time-loop kernel against the per-thread kernels, at the
sizes where its order, its row groups or its copies change: the smallest grid,
a last group of fewer rows, rows that tensor copies cannot take, calls that
end in the middle of a launch's steps, two steps at once (states beyond L2),
and planes with link masks whose rows are alike, mixed or both.  With a fixed
force both run the same operations per cell: populations equal bit for bit.
Logs come from sums in another order: FP64 sums of at most 2e6 values of one
size differ by less than 2e6 * 2^-53 relative; FP32 partial sums of about 30
cells by 30 * 2^-24 of the largest term."""
import os

import numpy as np
import pytest

import dnslbm
import inputs

pytestmark = pytest.mark.gpu


def _run(path, shape, flags, prec, calls, general=False, monkeypatch=None):
    monkeypatch.setenv("DNSLBM_PATH", path) if path else monkeypatch.delenv("DNSLBM_PATH", raising=False)
    nx, ny, nz = shape
    with dnslbm.Channel(nx, ny, nz, 1.7, gx=2e-5, precision=prec,
                        bc_mode=dnslbm.BC_GENERAL if general else dnslbm.BC_REFERENCE) as ch:
        ch.set_flags(flags)
        ch.load_state(inputs.laminar_state(nx, ny, nz, 0.06, 0.1, 7))
        for n in calls:
            ch.step(n)
        return ch.kernel, ch.store_state(), ch.logs()


def _compare(shape, flags, prec, calls, monkeypatch, general=False):
    kernel, state, logs = _run(None, shape, flags, prec, calls, general, monkeypatch)
    assert "persist_batch_kernel" in kernel
    other, want, wlogs = _run("scalar", shape, flags, prec, calls, general, monkeypatch)
    assert "per-thread" in other
    np.testing.assert_array_equal(state, want)
    rtol = 1e-9 if prec == 64 else 1e-5
    np.testing.assert_allclose(logs, wlogs, rtol=rtol, atol=1e-12)
    return kernel


@pytest.mark.parametrize("prec", [64, 32, 16])
@pytest.mark.parametrize("shape", [(2, 2, 3), (3, 9, 4), (45, 17, 5), (70, 33, 6)])
def test_small_grids(shape, prec, monkeypatch):
    nx, ny, nz = shape
    _compare(shape, inputs.flags_longitudinal(nx, ny, nz, 1, 1), prec, (1, 66, 5), monkeypatch)


@pytest.mark.parametrize("prec,shape", [(64, (301, 57, 44)), (32, (402, 75, 52)), (16, (640, 83, 60))])
def test_two_steps_at_once(prec, shape, monkeypatch):
    kernel = _compare(shape, inputs.flags_smooth(*shape), prec, (3, 70), monkeypatch)
    assert "2 steps per sweep" in kernel, kernel


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("walls", ["riblets", "blocks", "both"])
def test_planes_with_link_masks(prec, walls, monkeypatch):
    shape = nx, ny, nz = 44, 26, 14
    flags = inputs.flags_riblets(nx, ny, nz, 3, 6) if walls != "blocks" else inputs.flags_smooth(nx, ny, nz)
    if walls != "riblets":  # a block in the flow: rows of solid and fluid cells
        flags[5:11, 8:15, 5:9] = -1
    _compare(shape, flags, prec, (1, 9), monkeypatch, general=True)


def _beyond_l2(texture, prec):
    """A grid whose state does not stay in L2; FP32 rows of 402 cells are 1616
    bytes, three to a group, which tensor copies cannot take."""
    shape = {64: (301, 57, 44), 32: (402, 75, 52), 16: (640, 83, 60)}[prec]
    if texture == "grooves":
        return shape, inputs.flags_longitudinal(*shape, 3, 5), False
    flags = inputs.flags_riblets(*shape, 3, 6)  # rows alike, and a block in the flow: mixed rows
    flags[5:11, 8:15, 20:24] = -1
    return shape, flags, True


@pytest.mark.parametrize("prec", [64, 32, 16])
@pytest.mark.parametrize("texture", ["grooves", "riblets and a block"])
def test_two_steps_at_once_with_wall_links(texture, prec, monkeypatch):
    """Results written by the threads themselves (links of a textured wall, of
    mixed rows) and read by another step's copies two steps deep, over calls of
    odd and even lengths."""
    shape, flags, general = _beyond_l2(texture, prec)
    kernel = _compare(shape, flags, prec, (3, 70, 1), monkeypatch, general)
    assert "2 steps per sweep" in kernel, kernel


def test_two_steps_at_once_in_a_batch(monkeypatch):
    """A channel two steps deep between channels of one step at a time."""
    monkeypatch.delenv("DNSLBM_BATCH", raising=False)
    shape, flags, general = _beyond_l2("riblets and a block", 32)
    small = 45, 17, 5
    specs = [(small, inputs.flags_longitudinal(*small, 1, 1), False), (shape, flags, general), (small, inputs.flags_smooth(*small), False)]
    decks = [dnslbm.deck(*s, 1.7, gx=2e-5, precision=32, bc_mode=dnslbm.BC_GENERAL if g else dnslbm.BC_REFERENCE)
             for s, _, g in specs]
    with dnslbm.Batch(decks) as b:
        for ch, (s, fl, _) in zip(b.channels, specs):
            ch.set_flags(fl)
            ch.load_state(inputs.laminar_state(*s, 0.06, 0.1, 7))
        for n in (3, 70, 1):
            b.step(n)
        got = [ch.store_state() for ch in b.channels]
    for (s, fl, g), state in zip(specs, got):
        _, want, _ = _run("scalar", s, fl, 32, (3, 70, 1), g, monkeypatch)
        np.testing.assert_array_equal(state, want)

"""A channel of a batch stepped by itself: the single-channel calls take the
batch's stages and their own kernel's threads and shared memory, whichever
kernel steps the batch."""
import numpy as np
import pytest

import dnslbm
import inputs

pytestmark = pytest.mark.gpu
SPECS = [(40, 24, 10, "g", "smooth"), (63, 31, 16, "g", "grooves"), (300, 12, 9, "g", "smooth"), (26, 12, 7, "q", "smooth"),
         (48, 20, 12, "g", "riblets")]


def _make(spec, prec):
    nx, ny, nz, force, tex = spec
    fl = {"smooth": inputs.flags_smooth, "grooves": lambda *s: inputs.flags_longitudinal(*s, 3, 5),
          "riblets": lambda *s: inputs.flags_riblets(*s, 3, 6)}[tex](nx, ny, nz)
    kw = dict(ubulk=0.06, gx=2e-5, force_mode=dnslbm.CONST_G if force == "g" else dnslbm.CONST_Q, precision=prec,
              bc_mode=dnslbm.BC_GENERAL if tex == "riblets" else dnslbm.BC_REFERENCE)
    return (nx, ny, nz), fl, inputs.rest_solids(inputs.laminar_state(nx, ny, nz, 0.08, 0.1, 11), fl), kw


@pytest.mark.parametrize("mode", ["persistent", "launch"])
@pytest.mark.parametrize("prec", [64, 32, 16])
def test_channel_of_a_batch_stepped_by_itself(prec, mode, monkeypatch):
    monkeypatch.setenv("DNSLBM_BATCH", mode)
    chans = [_make(s, prec) for s in SPECS]
    with dnslbm.Batch([dnslbm.deck(*shape, 1.7, **kw) for shape, _, _, kw in chans]) as b:
        for ch, (_, fl, st, _) in zip(b.channels, chans):
            ch.set_flags(fl)
            ch.load_state(st)
        b.step(5)
        for ch in b.channels:
            ch.step(37)
            ch.step_timed(4)
        b.step(33)
        got = [ch.store_state() for ch in b.channels]
    for (shape, fl, st, kw), state, spec in zip(chans, got, SPECS):
        with dnslbm.Channel(*shape, 1.7, **kw) as ch:
            ch.set_flags(fl)
            ch.load_state(st)
            ch.step(79)
            want = ch.store_state()
        if spec[3] == "g":
            np.testing.assert_array_equal(state, want, err_msg=str(spec))
        else:  # sums in another order: the force's rounding, and in FP32 and FP16 the state's
            np.testing.assert_allclose(state, want, rtol=0, atol={64: 1e-11, 32: 1e-5, 16: 1e-3}[prec], err_msg=str(spec))

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


@pytest.mark.parametrize("count,shape,prec", [(10, (720, 3, 4), 64), (3, (740, 3, 4), 64), (60, (628, 3, 4), 64),
                                              (58, (1256, 3, 4), 32), (450, (8, 4, 3), 64), (2, (2960, 3, 4), 16)])
def test_number_of_channels_costs_no_shared_memory(count, shape, prec, monkeypatch):
    """Rows that fill two stages, and many channels: every batch whose widest
    row fits twice is taken, whatever the number of channels."""
    monkeypatch.delenv("DNSLBM_BATCH", raising=False)
    states = [inputs.laminar_state(*shape, 0.05, 0.1, i) for i in range(4)]
    with dnslbm.Batch([dnslbm.deck(*shape, 1.6, gx=1e-5 * (1 + i % 3), precision=prec) for i in range(count)]) as b:
        for i, ch in enumerate(b.channels):
            ch.load_state(states[i % 4])
        b.step(3)
        b.step(40)
        got = [ch.store_state() for ch in b.channels]
    want = {}
    for i, state in enumerate(got):
        key = i % 4, i % 3
        if key not in want:
            with dnslbm.Channel(*shape, 1.6, gx=1e-5 * (1 + i % 3), precision=prec) as ch:
                ch.load_state(states[i % 4])
                ch.step(43)
                want[key] = ch.store_state()
        np.testing.assert_array_equal(state, want[key], err_msg=f"channel {i}")


@pytest.mark.parametrize("mode", ["persistent", "launch"])
@pytest.mark.parametrize("prec", [64, 16])
def test_autotune_of_a_batch_channel_leaves_the_batch_its_shape(prec, mode, monkeypatch):
    """The channel's own search ends with the batch's launch shape: the batch
    kernel's stages are as large as the batch made them."""
    monkeypatch.setenv("DNSLBM_BATCH", mode)
    chans = [_make(s, prec) for s in (SPECS[0], SPECS[2], SPECS[4])]
    with dnslbm.Batch([dnslbm.deck(*shape, 1.7, **kw) for shape, _, _, kw in chans]) as b:
        kernel = b.kernel
        for ch in b.channels:
            assert "best of" in ch.autotune(2)
        assert b.kernel == kernel
        for ch, (_, fl, st, _) in zip(b.channels, chans):
            ch.set_flags(fl)
            ch.load_state(st)
        b.step(38)
        got = [ch.store_state() for ch in b.channels]
    for (shape, fl, st, kw), state in zip(chans, got):
        with dnslbm.Channel(*shape, 1.7, **kw) as ch:
            ch.set_flags(fl)
            ch.load_state(st)
            ch.step(38)
            np.testing.assert_array_equal(state, ch.store_state())


@pytest.mark.parametrize("prec", [64, 32])
def test_wait_limit_set_after_a_chunk_of_steps(prec, monkeypatch):
    """The limit of channel 0 holds for the chunks replayed from a graph too: a
    limit shorter than any load ends the next chunk, and the states can be
    loaded again."""
    monkeypatch.delenv("DNSLBM_BATCH", raising=False)
    chans = [_make(s, prec) for s in SPECS[:2]]
    with dnslbm.Batch([dnslbm.deck(*shape, 1.7, **kw) for shape, _, _, kw in chans]) as b:
        def load():
            for ch, (_, fl, st, _) in zip(b.channels, chans):
                ch.set_flags(fl)
                ch.load_state(st)
        load()
        b.step(64)
        want = [ch.store_state() for ch in b.channels]
        b.channels[0].set_wait_limit(1e-5)
        with pytest.raises(dnslbm.DnsLbmError) as e:
            b.step(64)
        assert e.value.code == dnslbm.ERR_TIMEOUT
        b.channels[0].set_wait_limit(1000)
        load()
        b.step(64)
        for ch, w in zip(b.channels, want):
            np.testing.assert_array_equal(ch.store_state(), w)

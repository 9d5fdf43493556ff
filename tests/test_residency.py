"""The persistent time loop makes progress whatever number of its blocks is on
the GPU at once: with one block, with a few, and with many times more than the
GPU holds (3000 planes, so that under a plane-per-block split most planes
would belong to blocks that never start while others wait), and with several
contexts stepped at once from threads of their own.  The results are those of
the kernel's own number of blocks: the sums do not depend on who takes what."""
import threading

import numpy as np
import pytest

import dnslbm
import inputs

pytestmark = pytest.mark.gpu


def _channel(shape, force, prec=64, wait_ms=1000.0):
    ch = dnslbm.Channel(*shape, 1.7, ubulk=0.06, gx=2e-5, force_mode=dnslbm.CONST_Q if force == "q" else dnslbm.CONST_G,
                        precision=prec)
    ch.set_wait_limit(wait_ms)
    ch.load_state(inputs.laminar_state(*shape, 0.06, 0.1, 3))
    return ch


@pytest.mark.parametrize("force", ["g", "q"])
@pytest.mark.parametrize("shape,blocks", [((4, 3, 3000), 6000), ((20, 9, 40), 4000), ((20, 9, 40), 1), ((70, 33, 12), 3)])
def test_any_number_of_blocks(shape, blocks, force):
    out = []
    for n in (0, blocks):
        with _channel(shape, force, wait_ms=200.0) as ch:
            ch.test_blocks(n)
            ch.step(1)
            ch.step(70)
            out.append((ch.store_state(), ch.logs()))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("force", ["g", "q"])
def test_contexts_stepped_at_once(force):
    shapes = [(64, 32, 40), (300, 61, 40), (48, 17, 90), (201, 50, 30)]
    want = []
    for s in shapes:
        with _channel(s, force) as ch:
            ch.step(400)
            want.append(ch.store_state())
    chans = [_channel(s, force) for s in shapes]
    errors = []

    def work(ch):
        try:
            for _ in range(8):
                ch.step(50)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(ch,)) for ch in chans]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for ch, w in zip(chans, want):
        np.testing.assert_array_equal(ch.store_state(), w)
        ch.close()

"""What a channel takes of the device's memory, and when: all at its creation,
none at a step; and rows that were made longer for tensor copies do not refuse
a grid whose rows as they are fit."""
import pytest
import torch

import dnslbm

pytestmark = pytest.mark.gpu


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("batch", [False, True])
def test_steps_take_no_memory(batch):
    shape = 8, 240, 400  # 12000 row groups: 6 MB of sums
    deck = dnslbm.deck(*shape, 1.6, gx=1e-5)
    with dnslbm.Channel(16, 8, 8, 1.6, gx=1e-5) as ch:  # the kernels are loaded
        ch.init_rest()
        ch.step(66)
    with dnslbm.Batch([dnslbm.deck(16, 8, 8, 1.6, gx=1e-5)]) as b:
        b.channels[0].init_rest()
        b.step(66)
    owner = dnslbm.Batch([deck]) if batch else dnslbm.Channel(*shape, 1.6, gx=1e-5)
    with owner as o:
        (o.channels[0] if batch else o).init_rest()
        before = _free()
        o.step(1)
        o.step(66)
        assert _free() == before


def test_longer_rows_give_way_to_memory():
    shape = 628, 157, 128  # FP64 rows of 640 cells, 29 MB longer in all
    kw = dict(gx=1e-5, log_capacity=64)
    longer = 19 * 8 * 12 * 157 * 128
    with dnslbm.Channel(*shape, 1.6, **kw):  # the kernels are loaded
        pass
    before = _free()
    with dnslbm.Channel(*shape, 1.6, **kw):
        need = before - _free()
    keep = need - longer // 2  # too little for longer rows by 14 MB
    chunks, left = [], _free() - keep
    try:
        while left >= 2 << 20:
            n = min(left, 16 << 30) >> 21 << 21
            chunks.append(torch.empty(n, dtype=torch.uint8, device="cuda"))
            left -= n
        assert need - longer < _free() < need
        with dnslbm.Channel(*shape, 1.6, **kw) as ch:
            ch.init_rest()
            ch.step(2)
    finally:
        chunks.clear()
        torch.cuda.empty_cache()


@pytest.mark.parametrize("shape,kept", [((400, 400, 140), False), ((200, 60, 40), True)])
def test_large_workspaces_are_given_back(shape, kept):
    """Spectra's workspace is about nx * ny / 2 * nz * 48 bytes; above 512 MB
    it lives for the call."""
    with dnslbm.Channel(*shape, 1.6, gx=1e-5, precision=16) as ch:
        ch.init_rest()
        ch.quadrant()  # takes the velocity field's memory
        before = _free()
        ch.spectra()
        after = _free()
        assert before - after <= (512 << 20 if kept else 0)
        ch.spectra()
        assert _free() == after

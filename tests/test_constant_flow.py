"""Constant flow rate: the force of a step is a small difference (1e-6 of 0.07)
of sums over the state before it.

FP32 and FP16 take it rounded to FP32, so the last bits of the FP64 sums decide
now and then which way, and a state is reproducible only if the sums keep their
order -- each block's rows thread by thread, then blocks, then planes.  The
values below are those of that order (default launch shapes of a B200): the
forces of the 41st and the last step, and the SHA-256 of the state.  FP64 takes
the force unrounded: the persistent time loop, over launches and calls of even
and odd lengths, agrees with the per-thread kernels to the rounding of the sums
(a force of magnitude 0.07 * 2^-52 * sqrt(cells) apart at worst, 5e-14 of a
population after the 273 steps here; bound 1e-11)."""
import hashlib

import numpy as np
import pytest

import dnslbm
import inputs

pytestmark = pytest.mark.gpu
CALLS = (3, 70, 200)

ALONE = {  # 70 x 24 x 31: force[40], force[272], state
    (32, "smooth"): ("0x1.c607e9bf66052p-16", "0x1.848859d5750a4p-16", "038bfebc1acfedbf"),
    (32, "grooves"): ("0x1.5e3ea2ceb2148p-16", "0x1.5515d2d85f666p-16", "9e3184867b599911"),
    (32, "riblets"): ("0x1.ae1f1b98dfe3dp-15", "0x1.2212d96842a14p-15", "a3a822ca610a42e9"),
    (16, "smooth"): ("0x1.c63e959a5819ap-16", "0x1.84bd3576a0e14p-16", "aa5a01f704e375f8"),
    (16, "grooves"): ("0x1.5ea2debeb775cp-16", "0x1.550e67dccf8f6p-16", "bfea8ff0749075fe"),
    (16, "riblets"): ("0x1.ae2f9cd0a2ca4p-15", "0x1.220b4f591fb5cp-15", "c1103f020f8020bd"),
}
BATCH = {  # states of the channels below
    32: ["51e1762ea7a986d5", "1c873a942bb63520", "ea141d4d9514e4f9", "48e9c3cd5a531f86", "ce1abe4e9735cbfc"],
    16: ["5fa8098401e1c39a", "43c77c0d871ce33a", "8f841f8b846f657e", "266d64c0b2b4fbdf", "350ed7b0ff267693"],
}
CHANNELS = [(40, 24, 10, 1.8, "smooth", True), (63, 31, 16, 1.9, "grooves", False), (26, 12, 7, 1.6, "smooth", False),
            (48, 20, 12, 1.75, "riblets", False), (642, 16, 20, 1.7, "smooth", False)]


def _flags(texture, nx, ny, nz):
    if texture == "smooth":
        return inputs.flags_smooth(nx, ny, nz)
    return inputs.flags_longitudinal(nx, ny, nz, 3, 5) if texture == "grooves" else inputs.flags_riblets(nx, ny, nz, 3, 6)


def _load(ch, texture, shape, seed):
    fl = _flags(texture, *shape)
    ch.set_flags(fl)
    ch.load_state(inputs.rest_solids(inputs.laminar_state(*shape, 0.08, 0.1, seed), fl))


def _mode(texture):
    return dnslbm.BC_GENERAL if texture == "riblets" else dnslbm.BC_REFERENCE


def _digest(a):
    return hashlib.sha256(np.ascontiguousarray(a).tobytes()).hexdigest()[:16]


@pytest.mark.parametrize("prec,texture", list(ALONE))
def test_low_precision_sums_keep_their_order(prec, texture, monkeypatch):
    """With riblets either of a step's two kernels may run its tail: the force
    is the same from both."""
    for e in ("PATH", "GROUP_ROWS", "STAGES", "THREADS", "BLOCKS_PER_SM", "ROW_ALIGN"):
        monkeypatch.delenv("DNSLBM_" + e, raising=False)
    shape = 70, 24, 31
    with dnslbm.Channel(*shape, 1.7, ubulk=0.06, force_mode=dnslbm.CONST_Q, precision=prec, bc_mode=_mode(texture)) as ch:
        _load(ch, texture, shape, 7)
        for n in CALLS:
            ch.step(n)
        force = ch.logs()[:, 0]
        got = (float(force[40]).hex(), float(force[272]).hex(), _digest(ch.store_state()))
    assert got == ALONE[prec, texture]


@pytest.mark.parametrize("mode", ["persistent", "launch"])
@pytest.mark.parametrize("prec", [32, 16])
def test_low_precision_batch_keeps_its_order(prec, mode, monkeypatch):
    monkeypatch.setenv("DNSLBM_BATCH", mode)
    decks = [dnslbm.deck(nx, ny, nz, om, ubulk=0.06, gx=2e-5, force_mode=dnslbm.CONST_G if g else dnslbm.CONST_Q,
                         precision=prec, bc_mode=_mode(tex)) for nx, ny, nz, om, tex, g in CHANNELS]
    with dnslbm.Batch(decks) as b:
        for i, (ch, (nx, ny, nz, _, tex, _)) in enumerate(zip(b.channels, CHANNELS)):
            _load(ch, tex, (nx, ny, nz), 30 + i)
        for n in CALLS:
            b.step(n)
        assert [_digest(ch.store_state()) for ch in b.channels] == BATCH[prec]


@pytest.mark.parametrize("texture", ["smooth", "grooves", "riblets"])
def test_fp64_over_launches_matches_the_per_thread_kernels(texture, monkeypatch):
    shape, out = (70, 24, 31), []
    for path in (None, "scalar"):
        monkeypatch.setenv("DNSLBM_PATH", path) if path else monkeypatch.delenv("DNSLBM_PATH", raising=False)
        with dnslbm.Channel(*shape, 1.7, ubulk=0.06, force_mode=dnslbm.CONST_Q, bc_mode=_mode(texture)) as ch:
            _load(ch, texture, shape, 7)
            for n in CALLS:
                ch.step(n)
            assert ("persist_batch_kernel" in ch.kernel) == (path is None), ch.kernel
            out.append((ch.store_state(), ch.logs()))
    np.testing.assert_allclose(out[0][0], out[1][0], rtol=0, atol=1e-11)
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=1e-9, atol=1e-11)

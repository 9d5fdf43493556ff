"""Timed cases of the channel-flow library, through its public entry points.

What a user of the library has it do: advance one channel between two output
events (``Channel.step`` and the state that comes back), advance a batch of
channels (a parameter study), advance caller-owned device memory
(``dnslbm_step_f64_noalloc``), compute the output event's fields and plane
statistics, and post-process a velocity field (two-point correlations, energy
spectra, quadrants), on the live state or from a ``vel`` file.  Channels are
created with the library's default launch shapes, as ``run-dns`` does.

Grids are those of ``inputs.py`` -- the laminar 64 x 32 x 64 channel, the
(2 pi h) x (pi h) x (2 h) channels of half-height h = 20 .. 100, rows of up to
1256 cells -- and odd sizes in between; x is streamwise, y spanwise, z
wall-normal (fluid planes).
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dns-solvers_b200"))
import dnslbm  # noqa: E402
import inputs  # noqa: E402

U_TAU = 0.005
SIZE = {64: 8, 32: 4, 16: 2}


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the laminar validation channel: 1000 steps on a state that stays in
        # cache, so launches and step ends count
        dict(name="steps_laminar64_f64", kind="steps", nx=64, ny=32, nz=64, precision=64, force="g", texture="smooth",
             re=24.0, steps=1000),
        # a host code that owns its device memory, a few steps per call
        dict(name="noalloc_64x32x64", kind="noalloc", nx=64, ny=32, nz=64, precision=64, force="g", texture="smooth",
             re=24.0, steps=10),
        # the reference's own mode (constant flow rate, FP64) on a coarse channel
        dict(name="steps_h32_f64_q", kind="steps", nx=201, ny=101, nz=64, precision=64, force="q", texture="smooth",
             re=100.0, steps=300),
        # a grooved channel with constant flow rate in FP32 storage
        dict(name="steps_h48_f32_q_grooves", kind="steps", nx=302, ny=151, nz=96, precision=32, force="q",
             texture="grooves", re=150.0, steps=400),
        # solids inside the flow: riblets on both walls
        dict(name="steps_h64_f32_riblets", kind="steps", nx=402, ny=201, nz=128, precision=32, force="g",
             texture="riblets", re=180.0, steps=300),
        # the headline Re_tau 180 channel, 39.4 M cells, in each storage type
        dict(name="steps_h100_f64", kind="steps", nx=628, ny=314, nz=200, precision=64, force="g", texture="smooth",
             re=180.0, steps=150),
        dict(name="steps_h100_f32_grooves", kind="steps", nx=628, ny=314, nz=200, precision=32, force="g",
             texture="grooves", re=180.0, steps=250),
        dict(name="steps_h100_f16", kind="steps", nx=628, ny=314, nz=200, precision=16, force="g", texture="smooth",
             re=180.0, steps=300),
        # a parameter study: eight channels of four sizes and mixed walls
        dict(name="batch8_f32", kind="batch", channels=8, first=0, precision=32, steps=160),
        # an output event after an odd number of steps: fields and statistics
        dict(name="output_h64_f64", kind="output", nx=402, ny=201, nz=128, precision=64, force="g", texture="grooves",
             re=180.0, steps=1),
        # post-processing of the running state
        dict(name="analysis_h64_f32", kind="analysis", nx=402, ny=201, nz=128, precision=32, force="g",
             texture="smooth", re=180.0, steps=0),
        # post-processing of a vel file of odd sizes
        dict(name="field_251x127x95", kind="field", nx=251, ny=127, nz=95, re=180.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: sizes over their logarithm, odd ones among
    them, up to about 20 M cells.  The Reynolds number goes down with the
    height, so that narrow or short channels stay stable over many passes."""
    kind = rng.choice(["steps"] * 6 + ["batch", "noalloc", "output", "analysis", "field"])
    if kind == "batch":
        return dict(kind=kind, channels=rng.randint(2, 7), first=rng.randint(1, 500), precision=rng.choice([64, 32]),
                    steps=rng.randint(40, 130))
    most = {"steps": 20e6, "noalloc": 5e6, "output": 10e6, "analysis": 8e6, "field": 3e6}[kind]
    while True:
        nx, ny, nz = _log_int(rng, 48, 1256), _log_int(rng, 24, 314), _log_int(rng, 24, 200)
        cells = nx * ny * nz
        if cells <= most and nx >= ny // 2:
            break
    re = round(min(rng.uniform(60, 150), 1.25 * nz), 1)
    if kind == "field":
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, re=re)
    precision = 64 if kind == "noalloc" else rng.choice([64, 32, 16])
    force = rng.choice("gq") if kind == "steps" and precision != 16 else "g"
    texture = rng.choice(["smooth", "grooves", "riblets"] if kind == "steps" else ["smooth", "grooves"])
    steps = {"steps": max(60, min(1000, int(4e9 / cells))), "noalloc": rng.randint(1, 20), "output": rng.randint(0, 3),
             "analysis": 0}[kind]
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, precision=precision, force=force, texture=texture,
                re=re, steps=steps)


# ---------------------------------------------------------------- channels
class _Spec:
    """Parameters of one channel of a case."""

    def __init__(self, nx, ny, nz, re, precision, force, texture, tex):
        self.nx, self.ny, self.nz, self.precision, self.force = nx, ny, nz, precision, force
        h = nz / 2.0
        self.omega = 1.0 / (0.5 + 3.0 * U_TAU * h / re)
        self.gx = U_TAU ** 2 / h
        self.ubulk = 15.7 * U_TAU * (re / 180.0) ** (1 / 7)
        make = {"smooth": inputs.flags_smooth, "longitudinal": inputs.flags_longitudinal,
                "transverse": inputs.flags_transverse, "riblets": inputs.flags_riblets}[texture]
        self.flags = make(nx, ny, nz, **tex)
        self.general = texture == "riblets"
        self.smooth = texture == "smooth"

    @property
    def cells(self):
        return self.nx * self.ny * self.nz

    def deck(self):
        return dict(ubulk=self.ubulk, gx=self.gx, force_mode=dnslbm.CONST_Q if self.force == "q" else dnslbm.CONST_G,
                    precision=self.precision, bc_mode=dnslbm.BC_GENERAL if self.general else dnslbm.BC_REFERENCE)


def _specs(case):
    if case["kind"] == "batch":
        out = []
        for w in inputs.batch_channels(case["first"] + case["channels"], 0)[case["first"]:]:
            s = _Spec(w.nx, w.ny, w.nz, 180.0, case["precision"], "g", w.texture, w.tex)
            s.omega, s.gx, s.ubulk = w.omega, w.gx, w.ubulk
            out.append(s)
        return out
    texture, tex = case.get("texture", "smooth"), {}
    if texture == "grooves":
        texture, tex = "longitudinal", {"gap": 16, "width": 16}
    elif texture == "riblets":
        tex = {"height": 6, "spacing": 12}
    return [_Spec(case["nx"], case["ny"], case["nz"], case["re"], case.get("precision", 64), case.get("force", "g"),
                  texture, tex)]


class _Host:
    """The program's page-locked buffer for states and fields: one, grown to
    what the largest case needs and kept, as a program writes one checkpoint
    after another from the same memory."""

    buf = None

    @classmethod
    def take(cls, *shapes):
        sizes = [int(np.prod(s)) for s in shapes]
        if cls.buf is None or cls.buf.array.size < sum(sizes):
            cls.buf = dnslbm.PinnedArray((sum(sizes),))
        out, o = [], 0
        for s, n in zip(shapes, sizes):
            out.append(cls.buf.array[o:o + n].reshape(s))
            o += n
        return out


# ---------------------------------------------------------------- inputs
def _velocity(spec, seed):
    """(nx, ny, nz, 3) FP64 on the GPU: a laminar profile of the bulk velocity
    and a divergence-free perturbation of 10 % (the curl of a low-pass vector
    potential that vanishes at both walls), every number from the seed."""
    nx, ny, nz = spec.nx, spec.ny, spec.nz
    rng = np.random.default_rng(seed)
    modes, kmax = 3, 6
    kx = np.fft.fftfreq(nx, 1.0 / nx)[:, None]
    ky = np.fft.rfftfreq(ny, 1.0 / ny)[None, :]
    mask = (np.abs(kx) <= kmax) & (np.abs(ky) <= kmax) & ((kx != 0) | (ky != 0))
    shape = (3, modes, nx, ny // 2 + 1)
    spec_c = torch.zeros(shape, dtype=torch.complex128)
    at = np.argwhere(mask)
    g = rng.standard_normal((3, modes, len(at), 2))
    spec_c[:, :, at[:, 0], at[:, 1]] = torch.view_as_complex(torch.from_numpy(g))
    spec_c = spec_c.cuda()
    back = lambda s: torch.fft.irfft2(s, s=(nx, ny)) * (nx * ny / 100.0)  # noqa: E731
    b = back(spec_c)
    bx = back(spec_c * torch.from_numpy(2j * np.pi * kx / nx).cuda())
    by = back(spec_c * torch.from_numpy(2j * np.pi * ky / ny).cuda())
    z = (torch.arange(1, nz + 1, dtype=torch.float64, device="cuda") - 0.5) / nz
    m = torch.arange(1, modes + 1, dtype=torch.float64, device="cuda")[:, None]
    pz = torch.sin(math.pi * z) * torch.sin(m * math.pi * z)
    dpz = (math.pi / nz) * (torch.cos(math.pi * z) * torch.sin(m * math.pi * z)
                            + m * torch.sin(math.pi * z) * torch.cos(m * math.pi * z))
    mul = lambda f, p: torch.einsum("mxy,mz->xyz", f, p)  # noqa: E731
    u = torch.empty((nx, ny, nz, 3), dtype=torch.float64, device="cuda")
    u[..., 0] = mul(by[2], pz) - mul(b[1], dpz)
    u[..., 1] = mul(b[0], dpz) - mul(bx[2], pz)
    u[..., 2] = mul(bx[1], pz) - mul(by[0], pz)
    u *= 0.1 * spec.ubulk / u.square().sum(-1).mean().sqrt()
    # small-scale noise, so that no wave number is empty
    gen = torch.Generator(device="cuda").manual_seed(seed)
    for x0 in range(0, nx, 64):
        n = min(64, nx - x0)
        u[x0:x0 + n] += 0.01 * spec.ubulk * (torch.rand((n, ny, nz, 3), generator=gen, dtype=torch.float64,
                                                        device="cuda") - 0.5)
    u[..., 0] += 1.5 * spec.ubulk * 4 * z * (1 - z)
    return u


E = torch.tensor(inputs.E)
W = torch.tensor(inputs.W)


def _equilibrium(u):
    """(..., 19) populations of density 1 at velocity u (..., 3)."""
    e, w = E.to(u.device), W.to(u.device)
    eu = u @ e.T
    return w * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * u.square().sum(-1, keepdim=True))


def _fill_state(spec, u, out):
    """The lbf state (nx, ny, nz + 2, 19) of velocity u into a host array."""
    t = torch.from_numpy(out)
    step = max(1, (1 << 24) // (spec.ny * (spec.nz + 2)))
    for x0 in range(0, spec.nx, step):
        part = u[x0:x0 + step]
        chunk = torch.zeros((part.shape[0], spec.ny, spec.nz + 2, 19), dtype=torch.float64, device="cuda")
        chunk[:, :, 1:-1] = _equilibrium(part)
        t[x0:x0 + step].copy_(chunk)
    torch.cuda.synchronize()


# ---------------------------------------------------------------- prepare, run
def _load(ch, spec, seed, buf):
    ch.set_flags(spec.flags)
    u = _velocity(spec, seed)
    _fill_state(spec, u, buf)
    ch.load_state(buf)


def _wall_bits(flags):
    """Wall-link bits [2][ny][nx] of dnslbm_step_f64_noalloc."""
    nx, ny, _ = flags.shape
    out = np.zeros((2, ny, nx), np.uint8)
    for w, k in enumerate((0, -1)):
        s = flags[:, :, k].T
        for b, (dx, dy) in enumerate(((0, 0), (1, 0), (-1, 0), (0, 1), (0, -1))):
            t = np.roll(np.roll(s, -dx, axis=1), -dy, axis=0)
            out[w] |= (((t == -1) & (s == -1)).astype(np.uint8) << b)
    return out


def prepare(case, seed):
    kind, specs = case["kind"], _specs(case)
    st = dict(case=case)
    if kind == "batch":
        st["out"] = _Host.take(*[(s.nx, s.ny, s.nz + 2, 19) for s in specs])
        b = st["batch"] = dnslbm.Batch([dnslbm.deck(s.nx, s.ny, s.nz, s.omega, **s.deck()) for s in specs])
        for i, (c, s) in enumerate(zip(b.channels, specs)):
            _load(c, s, seed * 64 + i, st["out"][i])
        return st
    s = specs[0]
    if kind == "field":
        vel = np.zeros((s.nx, s.ny, s.nz + 2, 3))
        vel[:, :, 1:-1] = _velocity(s, seed).cpu().numpy()
        st["vel"] = vel
        return st
    if kind == "noalloc":
        soa = torch.empty((19, s.nz, s.ny, s.nx), dtype=torch.float64, device="cuda")
        soa.copy_(_equilibrium(_velocity(s, seed)).permute(3, 2, 1, 0))
        st.update(pop=soa, parity=0, spec=s,
                  bits=None if s.smooth else torch.from_numpy(_wall_bits(s.flags)).cuda())
        return st
    ch = st["channel"] = dnslbm.Channel(s.nx, s.ny, s.nz, s.omega, **s.deck())
    state = (s.nx, s.ny, s.nz + 2, 19)
    st["out"], = _Host.take(state)
    _load(ch, s, seed, st["out"])
    if kind == "output":
        ch.step(case["steps"])
        st["vel"], st["den"] = _Host.take(state[:3] + (3,), state[:3])
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "steps":
        ch = st["channel"]
        ch.step(case["steps"])
        out = {"state": torch.from_numpy(ch.store_state(st["out"]))}
        if case["precision"] == 64:
            out["logs"] = ch.logs(ch.steps_done - case["steps"])
        return out
    if kind == "batch":
        st["batch"].step(case["steps"])
        return [torch.from_numpy(c.store_state(o)) for c, o in zip(st["batch"].channels, st["out"])]
    if kind == "noalloc":
        s, L = st["spec"], dnslbm.lib()
        f = L.dnslbm_step_f64_noalloc
        err = ctypes.create_string_buffer(256)
        bits = st["bits"]
        rc = f(ctypes.c_void_p(st["pop"].data_ptr()), ctypes.c_size_t(s.cells), s.nx, s.ny, s.nz,
               ctypes.c_double(s.omega), ctypes.c_double(s.gx),
               ctypes.c_void_p(None if bits is None else bits.data_ptr()), st["parity"], ctypes.c_long(case["steps"]),
               ctypes.c_void_p(None), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), err,
               ctypes.c_size_t(256))
        if rc:
            raise RuntimeError(err.value.decode())
        st["parity"] = (st["parity"] + case["steps"]) % 2
        return st["pop"]
    if kind == "output":
        ch = st["channel"]
        ch.moments(st["vel"], st["den"])
        return {"statistics": ch.statistics(), "vel": torch.from_numpy(st["vel"]), "den": torch.from_numpy(st["den"])}
    if kind == "analysis":
        ch = st["channel"]
        return {"correlations": ch.correlations(), "spectra": ch.spectra(), "quadrant": ch.quadrant()}
    vel = st["vel"]
    return {"correlations": dnslbm.correlations_vel(vel), "spectra": dnslbm.spectra_vel(vel),
            "quadrant": dnslbm.quadrant_vel(vel)}


# ---------------------------------------------------------------- work
def work(case):
    """A pass of K steps cannot do without reading the populations once,
    writing them once and K collisions per cell (about 300 operations); the
    per-step traffic of the stepping schemes is what the code may choose."""
    specs = _specs(case)
    cells = float(sum(s.cells for s in specs))
    column = float(sum(s.nx * s.ny * (s.nz + 2) for s in specs))
    kind = case["kind"]
    if kind in ("steps", "batch"):
        return {"bytes": 2 * 19 * SIZE[case["precision"]] * cells + 19 * 8 * column,
                "flops": 300.0 * cells * case["steps"]}
    if kind == "noalloc":
        return {"bytes": 2 * 19 * 8 * cells, "flops": 300.0 * cells * case["steps"]}
    if kind == "output":
        return {"bytes": 19 * SIZE[case["precision"]] * cells + 4 * 8 * column, "flops": 60.0 * cells}
    nx, ny = case["nx"], case["ny"]
    fft = 3 * 2.5 * math.log2(nx * ny) * cells  # the 2-D real transforms of each plane
    lags = 2 * 3 * 5 * math.log2(nx * ny) * cells  # correlations by way of them
    read = 19 * SIZE[case["precision"]] * cells if kind == "analysis" else 24 * column
    return {"bytes": read + 48.0 * (case["nz"] + 2) * (nx + ny), "flops": fft + lags + 20 * cells}


# ---------------------------------------------------------------- 64-bit values
EX, EY, EZ = (inputs.E[:, i].astype(int) for i in range(3))
OPP = [0, 2, 1, 4, 3, 6, 5, 9, 10, 7, 8, 13, 14, 11, 12, 17, 18, 15, 16]
MIR = [next(b for b in range(19) if (EX[b], EY[b], EZ[b]) == (EX[a], EY[a], -EZ[a])) for a in range(19)]


def _collide(f, omega, g):
    """BGK with the body force g, in place, f a list of 19 arrays."""
    rho = f[0].clone()
    j = [torch.zeros_like(rho) for _ in range(3)]
    for a in range(1, 19):
        rho += f[a]
        for d, ed in enumerate((EX[a], EY[a], EZ[a])):
            if ed:
                j[d].add_(f[a], alpha=int(ed))
    u = [x.div_(rho) for x in j]
    usq = 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])
    for a in range(19):
        w, ex = float(inputs.W[a]), int(EX[a])
        if a == 0:
            t = 1 - usq
            force = u[0] * (-3 * w * g)
        else:
            eu = sum(int(e) * x for e, x in zip((EX[a], EY[a], EZ[a]), u) if e)
            t = eu * eu
            t.mul_(4.5).add_(eu, alpha=3).sub_(usq).add_(1)
            force = u[0] * (-3 * w * g)
            force.add_(3 * w * g * ex)
            if ex:
                force.add_(eu, alpha=9 * w * g * ex)
        t.mul_(rho).mul_(w * omega)
        f[a].mul_(1 - omega).add_(t).add_(force)


class _Exact:
    """The channel in FP64 with plain torch: arrays (nz, ny, nx)."""

    def __init__(self, spec, u):
        self.s = spec
        f = _equilibrium(u)
        self.f = [f[..., a].permute(2, 1, 0).contiguous() for a in range(19)]
        del f
        fl = torch.from_numpy(spec.flags).cuda().permute(2, 1, 0)
        self.solid = fl[1:-1] == -1
        self.band = None
        if bool(self.solid.any()):
            for a in range(19):
                self.f[a][self.solid] = float(inputs.W[a])
            planes = self.solid.flatten(1).any(1)
            near = planes.clone()
            near[1:] |= planes[:-1]
            near[:-1] |= planes[1:]
            self.band = near.nonzero().flatten()
        # the link of cell P toward wall cell T bounces back iff both P's own
        # wall cell and T are no-slip
        self.bounce = {}
        for w, k in ((-1, 0), (1, -1)):
            s = fl[k] == -1
            for a in range(19):
                if EZ[a] == w:
                    self.bounce[a] = s & torch.roll(s, (-int(EY[a]), -int(EX[a])), (0, 1))

    def step(self):
        s, f = self.s, self.f
        g = s.gx
        if s.force == "q":
            n = float(s.cells)
            rho = sum(float(x.sum()) for x in f) / n
            jx = sum(int(EX[a]) * float(f[a].sum()) for a in range(19) if EX[a]) / n
            g = rho * s.ubulk - jx
        _collide(f, s.omega, g)
        if self.band is not None:
            for a in range(19):
                f[a][self.solid] = float(inputs.W[a])
            near = {a: f[a][self.band] for a in range(19)}
        walls = {a: f[a][0 if EZ[a] < 0 else -1].clone() for a in range(19) if EZ[a]}
        for a in range(1, 19):
            r = torch.roll(f[a], (int(EY[a]), int(EX[a])), (1, 2)) if EX[a] or EY[a] else f[a]
            if EZ[a]:
                n = torch.empty_like(r)
                if EZ[a] > 0:
                    n[1:] = r[:-1]
                else:
                    n[:-1] = r[1:]
                r = n
            f[a] = r
        for a, v in walls.items():
            k, m = (0 if EZ[a] < 0 else -1), self.bounce[a]
            f[OPP[a]][k][m] = v[m]
            q = torch.roll(~m, (int(EY[a]), int(EX[a])), (0, 1))
            f[MIR[a]][k][q] = torch.roll(v, (int(EY[a]), int(EX[a])), (0, 1))[q]
        if self.band is not None:
            for a in range(1, 19):
                tgt = torch.roll(self.solid, (-int(EY[a]), -int(EX[a])), (1, 2))
                if EZ[a] > 0:
                    tgt = torch.cat([tgt[1:], torch.zeros_like(tgt[:1])])
                elif EZ[a] < 0:
                    tgt = torch.cat([torch.zeros_like(tgt[:1]), tgt[:-1]])
                hit = (tgt & ~self.solid)[self.band]
                plane = f[OPP[a]][self.band]
                plane[hit] = near[a][hit]
                f[OPP[a]][self.band] = plane
            for a in range(19):
                f[a][self.solid] = float(inputs.W[a])

    def soa(self):
        return torch.stack(self.f)

    def state(self):
        s = self.s
        out = torch.zeros((s.nx, s.ny, s.nz + 2, 19), dtype=torch.float64)
        for a in range(19):
            out[:, :, 1:-1, a] = self.f[a].permute(2, 1, 0).cpu()
        return out

    def moments(self):
        """(vel (nx, ny, nz + 2, 3), den (nx, ny, nz + 2)) on the GPU."""
        s = self.s
        vel = torch.zeros((s.nx, s.ny, s.nz + 2, 3), dtype=torch.float64, device="cuda")
        den = torch.zeros((s.nx, s.ny, s.nz + 2), dtype=torch.float64, device="cuda")
        rho = sum(self.f)
        for d, e in enumerate((EX, EY, EZ)):
            j = sum(int(e[a]) * self.f[a] for a in range(19) if e[a])
            vel[:, :, 1:-1, d] = (j / rho).permute(2, 1, 0)
        den[:, :, 1:-1] = rho.permute(2, 1, 0)
        return vel, den


def _field_values(vel):
    """correlations, spectra and quadrants of vel (nx, ny, zd, 3)."""
    nx, ny, zd, _ = vel.shape
    n = nx * ny
    inner = vel[:, :, 1:-1]
    mean = inner.mean((0, 1))  # (nz, 3)
    sym = 0.5 * (mean + mean.flip(0) * torch.tensor([1.0, 1.0, -1.0], dtype=vel.dtype, device=vel.device))
    q = vel.clone()
    q[:, :, 1:-1] -= sym

    def line(dim, length):  # sum over the plane of u'(p) u'(p + d), all periodic lags d
        p = torch.fft.rfft(q, dim=dim).abs().square().sum(1 - dim, keepdim=True)
        return torch.fft.irfft(p, n=length, dim=dim).squeeze(1 - dim)  # (length, zd, 3)

    xc, yc = line(0, nx).permute(1, 0, 2), line(1, ny).permute(1, 0, 2)
    ua = torch.zeros(zd, dtype=vel.dtype, device=vel.device)
    ua[1:-1] = sym[:, 0]
    c = torch.fft.fft(torch.fft.rfft(inner, dim=1), dim=0)
    c = c / n
    c[0, 0] = 0
    p = 0.5 * c.abs().square()
    p[:, 1:] *= 2
    ex = torch.zeros((3, nx, zd), dtype=vel.dtype, device=vel.device)
    ey = torch.zeros((3, ny // 2 + 1, zd), dtype=vel.dtype, device=vel.device)
    ex[:, :, 1:-1] = p.sum(1).permute(2, 0, 1)
    ey[:, :, 1:-1] = p.sum(0).permute(2, 0, 1)
    d = inner - mean
    u, w = d[..., 0], d[..., 2]
    uw = u * w
    quad, dquad = (torch.zeros((4, zd), dtype=vel.dtype, device=vel.device) for _ in range(2))
    for i, m in enumerate(((u > 0) & (w > 0), (u < 0) & (w > 0), (u < 0) & (w < 0), (u > 0) & (w < 0))):
        s, cnt = (uw * m).sum((0, 1)), m.sum((0, 1))
        quad[i, 1:-1] = s / cnt
        dquad[i, 1:-1] = s / n
    um = torch.zeros(zd, dtype=vel.dtype, device=vel.device)
    um[1:-1] = uw.sum((0, 1)) / n
    return {"correlations": (xc, yc, ua), "spectra": (ex, ey), "quadrant": (quad, dquad, um)}


def _statistics(vel, den):
    zd = den.shape[2]
    out = torch.zeros((9, zd), dtype=vel.dtype, device=vel.device)
    v, r = vel[:, :, 1:-1], den[:, :, 1:-1]
    m, rm = v.mean((0, 1)), r.mean((0, 1))
    d, dr = v - m, r - rm
    out[0:3, 1:-1] = m.T
    out[3:6, 1:-1] = d.square().mean((0, 1)).sqrt().T
    out[6, 1:-1] = (d[..., 0] * d[..., 2]).mean((0, 1))
    out[7, 1:-1] = rm
    out[8, 1:-1] = dr.square().mean((0, 1)).sqrt()
    return out


def exact(case, seed):
    kind, specs = case["kind"], _specs(case)
    if sum(s.cells for s in specs) * case.get("steps", 0) > 12e9:
        return None  # tens of seconds in plain torch
    if kind == "field":
        s = specs[0]
        vel = torch.zeros((s.nx, s.ny, s.nz + 2, 3), dtype=torch.float64, device="cuda")
        vel[:, :, 1:-1] = _velocity(s, seed)
        return _field_values(vel)
    done = []
    for i, s in enumerate(specs):
        x = _Exact(s, _velocity(s, seed * 64 + i if kind == "batch" else seed))
        for _ in range(case["steps"]):
            x.step()
        if kind == "steps":
            out = {"state": x.state()}
            return {**out, "logs": None} if s.precision == 64 else out
        if kind == "noalloc":
            if case["steps"] % 2:
                return None  # left in the odd layout
            return x.soa()
        if kind == "output":
            vel, den = x.moments()
            return {"statistics": _statistics(vel, den), "vel": vel, "den": den}
        if kind == "analysis":
            return _field_values(x.moments()[0])
        done.append(x.state())
        del x
        torch.cuda.empty_cache()
    return done

"""The work that a program using this library has it do, as measurable cases.

Five kinds of work, each through the public entry points (dropfluid.DropFluid
and the C ABI that it binds):

  box      windows of the closed-box drop simulation from a saved state
           (seek and replay: load_state, step, the fields read back): the
           48^3-class box stepped interactively with every step's statistics,
           a box whose dims are odd multiples of 8 (no exact coarsest grid,
           rows that are not multiples of 8 on the coarse grids), the
           192x256x192 box in FP32 and mixed precision, and a larger box
  ref      a seek of the reference setup (BloodDropEngine's seekToSimTime):
           drop lifecycle, wave solver, free-surface top, parcels, 2x dye,
           light volume, one uniform block per substep
  adjoint  forward and backward of a recorded trajectory (gradients of the
           initial state, as a fitting loop takes them)
  render   one frame: lighting passes and the plume march into a host image
  psolve   the pressure solve alone on a host program's own device buffers

Sizes are the repository's own scenes, tests and benchmark sizes, or generic.
A pass starts from the same saved state every time, so passes are alike.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "drop-of-blood_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from dropfluid import DropFluid, abi, load  # noqa: E402
from dropfluid import uniforms as U  # noqa: E402
from dropfluid._lib import check  # noqa: E402
from dropfluid.adjoint import DropTrajectory  # noqa: E402
from dropfluid.sequencer import SubstepSequencer  # noqa: E402

DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _box(name, nx, ny, nz, steps, parcels, prec="fp32", pipelined=False):
    c = {"kind": "box", "nx": nx, "ny": ny, "nz": nz, "steps": steps, "parcels": parcels, "prec": prec,
         "pipelined": pipelined}
    return dict(c, name=name) if name else c


def _ref(name, nx, ny, nz, levels, prec, substeps, parcels):
    c = {"kind": "ref", "nx": nx, "ny": ny, "nz": nz, "levels": levels, "prec": prec, "substeps": substeps,
         "parcels": parcels}
    return dict(c, name=name) if name else c


def _adjoint(name, nx, ny, nz, steps, every, prec):
    c = {"kind": "adjoint", "nx": nx, "ny": ny, "nz": nz, "steps": steps, "every": every, "prec": prec}
    return dict(c, name=name) if name else c


def _render(name, width, height, prec):
    c = {"kind": "render", "width": width, "height": height, "prec": prec}
    return dict(c, name=name) if name else c


def _psolve(name, nx, ny, nz, bc, levels):
    c = {"kind": "psolve", "nx": nx, "ny": ny, "nz": nz, "bc": bc, "levels": levels}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the small interactive box: one step in flight, every step's statistics read on the host
        _box("box48_interactive", 48, 64, 48, 16, 8192, pipelined=True),
        # a box that a user sized for the scene: 72 = 8*9, 104 = 8*13, 56 = 8*7 (three grids, swept coarsest)
        _box("box_ragged", 72, 104, 56, 16, 5001),
        # the benchmark scene's box, both storage modes
        _box("box192_fp32", 192, 256, 192, 24, 393216),
        _box("box192_mixed", 192, 256, 192, 24, 393216, prec="mixed"),
        # a production-size box (25 million cells)
        _box("box256_fp32", 256, 384, 256, 24, 393216),
        # one simulated second of the reference engine's own setup
        _ref("ref96_seek", 96, 128, 96, 4, "fp32", 60, 393216),
        # the same engine with its binary16 textures on a reduced grid
        _ref("ref48_fp16", 48, 64, 48, 3, "fp16", 24, 49152),
        # gradients over a trajectory with one recomputed segment, and a small mixed one
        _adjoint("adjoint96", 96, 128, 96, 16, 8, "fp32"),
        _adjoint("adjoint64_mixed", 64, 96, 64, 8, 8, "mixed"),
        # a half-resolution 1080p frame of the plume
        _render("render_960x540", 960, 540, "fp32"),
        # the pressure solve of a host that owns its memory: the reference's grid, and a small closed box
        _psolve("psolve96_ref", 96, 128, 96, "ref", 4),
        _psolve("psolve_small", 40, 56, 24, "box", 3),
    ]


def draw(rng):
    def dim(lo, hi, m):
        return max(m, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / m)) * m)

    kind = rng.choice(["box", "box", "box", "ref", "adjoint", "render", "psolve", "psolve"])
    if kind == "box":
        prec = rng.choice(["fp32", "fp32", "mixed"])
        nx, ny, nz = dim(32, 256, 8), dim(48, 384, 8), dim(32, 256, 8)
        return _box(None, nx, ny, nz, rng.randint(6, 24), rng.randint(1000, 393216), prec, rng.random() < 0.3)
    if kind == "ref":
        return _ref(None, dim(32, 96, 8), dim(48, 128, 8), dim(32, 96, 8), 3, rng.choice(["fp32", "fp16"]),
                    rng.randint(4, 40), rng.randint(16384, 393216))
    if kind == "adjoint":
        every = rng.choice([4, 8])
        return _adjoint(None, dim(32, 96, 8), dim(48, 128, 8), dim(32, 96, 8), rng.randint(4, 12), every,
                        rng.choice(["fp32", "mixed"]))
    if kind == "render":
        return _render(None, rng.randint(160, 960), rng.randint(90, 540), rng.choice(["fp32", "fp16"]))
    return _psolve(None, dim(24, 96, 8), dim(24, 128, 8), dim(24, 96, 8), rng.choice(["box", "ref"]), 3)


PREC = {"fp32": abi.DOB_PREC_FP32, "mixed": abi.DOB_PREC_MIXED, "fp16": abi.DOB_PREC_REFERENCE_FP16}
BOX_FIELDS = {"u": abi.FIELD_VEL_U, "v": abi.FIELD_VEL_V, "w": abi.FIELD_VEL_W, "p": abi.FIELD_PRESSURE,
              "dye": abi.FIELD_CONC}


# ---- inputs -------------------------------------------------------------------------------------

def _box_config(case):
    c = abi.config_closed_box(case["nx"], case["ny"], case["nz"])
    c.precision_mode = PREC[case.get("prec", "fp32")]
    if case.get("prec") == "mixed":
        c.mg_cycles = 3
    c.parcel_capacity = case.get("parcels", 1024)
    return c


def _box_state(case, seed):
    """Drops on their way down: for each, a divergence-free Gaussian vortex
    of 1.5 cells per step with face noise, a soft ball of dye and parcels in
    it, over a weak large-scale circulation; float32 numpy arrays."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    r = max(3.0, min(nx, ny, nz) / 16.0)
    n_drops = 3 if min(nx, ny, nz) >= 64 else 1
    cell = 1.0 / 0.02  # one cell per step in world units
    drops = [np.array([rng.uniform(2 * r, n - 2 * r) for n in (nx, ny, nz)]) for _ in range(n_drops)]
    back = [(rng.uniform(0.05, 0.1) * cell, rng.uniform(0, 2 * np.pi)) for _ in range(3)]
    gen = torch.Generator(device=DEV).manual_seed(int(seed) * 7 + 1)
    ax = [torch.arange(n, dtype=torch.float64, device=DEV) for n in (nz, ny, nx)]

    def at(ox, oy, oz):
        return (ax[2] + ox)[None, None, :], (ax[1] + oy)[None, :, None], (ax[0] + oz)[:, None, None]

    out = {}
    for k, (name, off) in enumerate((("u", (1.0, 0.5, 0.5)), ("v", (0.5, 1.0, 0.5)), ("w", (0.5, 0.5, 1.0)))):
        x, y, z = at(*off)
        amp, ph = back[k]
        a, b = [(y / ny, z / nz), (z / nz, x / nx), (x / nx, y / ny)][k]
        f = amp * torch.sin(2 * np.pi * a + ph) * torch.cos(2 * np.pi * b) + torch.zeros((nz, ny, nx), device=DEV)
        for c in drops:
            d = (x - c[0], y - c[1], z - c[2])
            r2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
            g = torch.exp(-r2 / (2 * r * r))
            f = f - 1.5 * cell * g * ((1.0 - r2 / (2 * r * r) if k == 1 else 0.0) + d[k] * d[1] / (2 * r * r))
            noise = torch.randn((nz, ny, nx), generator=gen, dtype=torch.float32, device=DEV)
            f = f + (0.05 * cell) * noise * (g > 0.5)
        f[(slice(None),) * (2 - k) + (-1,)] = 0.0
        out[name] = f.to(torch.float32).cpu().numpy()
    x, y, z = at(0.5, 0.5, 0.5)
    dye = torch.zeros((nz, ny, nx), dtype=torch.float64, device=DEV)
    for c in drops:
        d = torch.sqrt((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2)
        t = ((r + 1.0 - d) / 2.0).clamp(0.0, 1.0)
        dye = dye + t * t * (3.0 - 2.0 * t)
    out["dye"] = dye.to(torch.float32).cpu().numpy()
    if PREC[case.get("prec", "fp32")] == abi.DOB_PREC_MIXED:
        out["dye"] = out["dye"].astype(np.float16).astype(np.float32)
    out["p"] = np.zeros((nz, ny, nx), np.float32)
    n = case.get("parcels", 1024)
    q = rng.normal(size=(n, 3))
    q *= (r * rng.random(n) ** (1 / 3) / np.linalg.norm(q, axis=1))[:, None]
    par = np.zeros((n, 8), np.float32)
    par[:, :3] = q + np.stack(drops)[np.arange(n) % n_drops]
    par[:, 3] = 0.134
    out["parcels"] = par
    return out


def _load_box(sim, st):
    for k, f in BOX_FIELDS.items():
        sim.set_field(f, st[k])
    sim.run_stage(abi.STAGE_MAC_TO_CENTER)


def _ref_sim(case, seed, warm, flags):
    """A reference-mode context `warm` substeps into the drop lifecycle."""
    c = abi.config_reference()
    c.nx, c.ny, c.nz = case.get("nx", 96), case.get("ny", 128), case.get("nz", 96)
    c.mg_levels = case.get("levels", 4)
    c.precision_mode = PREC[case["prec"]]
    c.physics_flags = abi.DOB_PHYS_REFERENCE_ALL | flags
    c.parcel_capacity = case.get("parcels", 393216)
    sim = DropFluid(c)
    rng = np.random.default_rng(seed)
    seq = SubstepSequencer(parcel_capacity=c.parcel_capacity, seed=1.0 + seed % 89)
    sim.set_uniforms(seq.reset_simulation(1.0 + seed % 89, tuple(rng.uniform(-0.1, 0.1, 2))))
    sim.reset()
    sim.step_uniforms(np.stack([seq.advance_substep()[0] for _ in range(warm)]))
    return sim, seq


def _psolve_inputs(case, seed):
    """A drop step's right-hand side (divergence of a noisy vortex field) and
    a smooth initial pressure, on the device."""
    g = torch.Generator().manual_seed(int(seed))
    shape = (case["nz"], case["ny"], case["nx"])
    b = torch.randn(shape, generator=g, dtype=torch.float32)
    z, y, x = (torch.linspace(0, 2 * math.pi, n) for n in shape)
    ph = torch.rand(3, generator=g) * 6.0
    smooth = torch.sin(z + ph[0])[:, None, None] * torch.sin(y + ph[1])[None, :, None] * torch.sin(x + ph[2])[None, None, :]
    b = 0.2 * b + smooth
    if case["bc"] == "box":
        b = b - b.double().mean().float()
    p0 = 20.0 * smooth + torch.randn(shape, generator=g, dtype=torch.float32)
    return b.to(DEV).contiguous(), p0.to(DEV).contiguous()


def _psolve_config(case):
    if case["bc"] == "box":
        c = abi.config_closed_box(case["nx"], case["ny"], case["nz"])
        k = c.mg_levels - 1
        if (c.nx >> k) * (c.ny >> k) * (c.nz >> k) > 2304:  # more than this entry point solves exactly
            c.mg_coarse_sweeps = 6
        return c
    c = abi.config_reference()
    c.nx, c.ny, c.nz, c.mg_levels = case["nx"], case["ny"], case["nz"], case["levels"]
    return c


def prepare(case, seed):
    kind = case["kind"]
    if kind == "box":
        sim = DropFluid(_box_config(case))
        st = _box_state(case, seed)
        _load_box(sim, st)
        sim.set_parcels(st["parcels"])
        sim.save_state(0)
        return {"case": case, "sim": sim}
    if kind == "ref":
        sim, seq = _ref_sim(case, seed, 52, abi.DOB_PHYS_WAVE | abi.DOB_PHYS_LIGHTING)
        sim.save_state(0)
        blocks = np.stack([seq.advance_substep()[0] for _ in range(case["substeps"])])
        return {"case": case, "sim": sim, "blocks": blocks}
    if kind == "adjoint":
        sim = DropFluid(_box_config(case))
        st = _box_state(case, seed)
        _load_box(sim, st)
        sim.save_state(0)
        g = _dye_gradient(case, seed)
        return {"case": case, "sim": sim, "grad": g, "traj": DropTrajectory(sim, case["every"])}
    if kind == "render":
        sim, seq = _ref_sim(case, seed, 90, abi.DOB_PHYS_WAVE)
        eye, target = (0.0, 0.16, 0.6), (0.0, 0.2, 0.0)
        vp, ivp = U.camera_matrices(eye, target, 40.0, case["width"] / case["height"])
        block = U.SimUniformPacker().pack(
            drops=seq.drops.snapshot().snapshot, dt=U.FIXED_SIM_DT, frame_index=seq.frame_index,
            global_seed=seq.drop_seed, inv_view_proj=ivp, view_proj=vp, camera_pos=eye, camera_target=target,
            viewport_width=case["width"], viewport_height=case["height"]).copy()
        sim.set_uniforms(block)
        sim.set_spectral_lut(U.synthetic_spectral_lut(seed % 1000))
        return {"case": case, "sim": sim}
    b, p0 = _psolve_inputs(case, seed)
    return {"case": case, "cfg": _psolve_config(case), "b": b, "p0": p0, "lib": load()}


def _dye_gradient(case, seed):
    """d loss / d final dye of a least-squares fit: a smooth random mismatch."""
    rng = np.random.default_rng(seed + 5)
    z, y, x = (np.linspace(0, 2 * np.pi, n) for n in (case["nz"], case["ny"], case["nx"]))
    ph = rng.uniform(0, 6, 3)
    g = np.sin(2 * z + ph[0])[:, None, None] * np.cos(y + ph[1])[None, :, None] * np.sin(x + ph[2])[None, None, :]
    return g.astype(np.float32)


# ---- one pass -----------------------------------------------------------------------------------

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "psolve":
        p = state["p0"].clone()
        stream = torch.cuda.current_stream()
        check(state["lib"].dob_pressure_solve_noalloc(C.byref(state["cfg"]), C.c_void_p(state["b"].data_ptr()),
                                                      C.c_void_p(p.data_ptr()), C.c_void_p(stream.cuda_stream)),
              "dob_pressure_solve_noalloc")
        return {"p": p}
    sim = state["sim"]
    if kind == "box":
        sim.load_state(0)
        if case["pipelined"]:
            stats = sim.run_pipelined(case["steps"])
            out = {"alive": stats[-1]["parcels_alive"]}
        else:
            sim.step(case["steps"])
            out = {}
        out.update({k: sim.get_field(f) for k, f in BOX_FIELDS.items()})
        out["parcels"] = sim.get_parcels()
        return out
    if kind == "ref":
        sim.load_state(0)
        sim.step_uniforms(state["blocks"])
        out = {k: sim.get_field(f) for k, f in BOX_FIELDS.items()}
        out.update(wave=sim.get_field(abi.FIELD_WAVE), light=sim.get_field(abi.FIELD_LIGHT),
                   bricks=sim.get_field(abi.FIELD_BRICKS), parcels=sim.get_parcels())
        return out
    if kind == "adjoint":
        sim.load_state(0)
        dye = state["traj"].forward(case["steps"])
        return {"dye": dye, "grad": state["traj"].backward(state["grad"])}
    return {"image": sim.render_plume(case["width"], case["height"]).view(np.float16)}


def work(case):
    """Minimum traffic and arithmetic of one pass.  Per closed-box step and
    cell: velocity, pressure and dye read and written once (40 B; the dye at
    2 B in mixed mode), and about 1000 operations (three RK2 traces with their
    samples 400, Casson 60, 16 smoothing sweeps and transfers 250, projection
    20, dye 250); a parcel is 64 B and 300 operations a step."""
    kind = case["kind"]
    if kind == "render":
        px = case["width"] * case["height"]
        # the image, the light volume and the 4-channel dye once; some 50 march samples a pixel
        return {"bytes": 16.0 * px + 96 * 128 * 96 * (8 + 8 * 16), "flops": 50 * 200.0 * px}
    n = float(case["nx"] * case["ny"] * case["nz"])
    if kind == "box":
        s = case["steps"]
        b = 36 if case["prec"] == "mixed" else 40
        return {"bytes": s * (b * n + 64 * case["parcels"]), "flops": s * (1000 * n + 300 * case["parcels"])}
    if kind == "ref":
        s, e = case["substeps"], 2 if case["prec"] == "fp16" else 4
        # faces and pressure of the velocity grid, 4-channel dye on 8 times the cells, the wave field
        return {"bytes": s * (n * (6 * e + 8 + 64 * e) + 32 * 512 * 512), "flops": s * (900 * n + 8 * n * 100 + 400 * 512 * 512)}
    if kind == "adjoint":
        s = case["steps"]
        return {"bytes": 3 * s * 40 * n, "flops": 3 * s * 1000 * n}
    cycles = 4 if case["bc"] == "box" else 1
    return {"bytes": 12 * n, "flops": cycles * 60 * n}


# ---- the same results in 64 bits --------------------------------------------------------------------

def _centre(u, v, w):
    def mean(a, dim):
        lo = torch.zeros_like(a.narrow(dim, 0, 1))
        return 0.5 * (a + torch.cat([lo, a.narrow(dim, 0, a.shape[dim] - 1)], dim))

    return torch.stack([mean(u, 2), mean(v, 1), mean(w, 0)])


def _shift(a, dim, step):
    """a at index + step along dim, the edge value beyond the ends."""
    n = a.shape[dim]
    if step > 0:
        return torch.cat([a.narrow(dim, 1, n - 1), a.narrow(dim, n - 1, 1)], dim)
    return torch.cat([a.narrow(dim, 0, 1), a.narrow(dim, 0, n - 1)], dim)


def _taps(n, t):
    f = torch.floor(t)
    i = f.long()
    return i.clamp(0, n - 1), (i + 1).clamp(0, n - 1), t - f


def _corners(shape, uvw):
    (x0, x1, fx), (y0, y1, fy), (z0, z1, fz) = (_taps(n, t * n - 0.5) for n, t in zip(shape[::-1], uvw))
    nz, ny, nx = shape
    idx = [(z * ny + y) * nx + x for z in (z0, z1) for y in (y0, y1) for x in (x0, x1)]
    return idx, (fx, fy, fz)


def _mix8(c, f):
    fx, fy, fz = f
    a = [p + (q - p) * fx for p, q in zip(c[0::2], c[1::2])]
    b = [p + (q - p) * fy for p, q in zip(a[0::2], a[1::2])]
    return b[0] + (b[1] - b[0]) * fz


def _sample(fields, uvw):
    """Trilinear samples of the (nz, ny, nx) fields at uvw, clamped at the edges."""
    idx, f = _corners(fields[0].shape, uvw)
    return [_mix8([a.reshape(-1)[i] for i in idx], f) for a in fields]


class _Poisson:
    """The V-cycles of the pressure solve (and the exact solve) in float64."""

    def __init__(self, cfg, dev):
        self.ref = cfg.bc_mode == abi.DOB_BC_REFERENCE
        self.cfg, self.lv = cfg, []
        for l in range(cfg.mg_levels):
            shape = (cfg.nz >> l, cfg.ny >> l, cfg.nx >> l)
            one = torch.ones(shape, dtype=torch.float64, device=dev)
            diag = self._sum(one) + (self._top(one) if self.ref else 0.0)
            z, y, x = (torch.arange(n, device=dev) for n in shape)
            red = (z[:, None, None] + y[None, :, None] + x[None, None, :]) % 2 == 0
            self.lv.append((shape, float(4 ** l), diag, red))
        self.dev = dev
        self.basis = {}

    @staticmethod
    def _sum(a):
        s = torch.zeros_like(a)
        for dim in range(3):
            n = a.shape[dim]
            z = torch.zeros_like(a.narrow(dim, 0, 1))
            s = s + torch.cat([z, a.narrow(dim, 0, n - 1)], dim) + torch.cat([a.narrow(dim, 1, n - 1), z], dim)
        return s

    @staticmethod
    def _top(a):
        t = torch.zeros_like(a)
        t[:, -1, :] = 1.0
        return t

    def _sweep(self, l, e, b, n):
        _, h2, diag, red = self.lv[l]
        for _ in range(n):
            for mask in (red, ~red):
                e = torch.where(mask, (self._sum(e) - h2 * b) / diag, e)
        return e

    def _axis(self, n, dirichlet):
        if (n, dirichlet) not in self.basis:
            k = torch.arange(n, dtype=torch.float64, device=self.dev)
            t = math.pi * (k + 0.5) / (n + 0.5) if dirichlet else math.pi * k / n
            v = torch.cos(t[:, None] * (k[None, :] + 0.5))
            v = v / v.norm(dim=1, keepdim=True)
            mu = 2.0 - 2.0 * torch.cos(t)
            if not dirichlet:
                mu[0] = 0.0
            self.basis[n, dirichlet] = v, mu
        return self.basis[n, dirichlet]

    def direct(self, l, b):
        (nz, ny, nx), h2, _, _ = self.lv[l]
        (vx, mx), (vy, my), (vz, mz) = self._axis(nx, False), self._axis(ny, self.ref), self._axis(nz, False)
        c = torch.einsum("kz,zyx->kyx", vz, torch.einsum("ky,zyx->zkx", vy, torch.einsum("kx,zyx->zyk", vx, b)))
        mu = mz[:, None, None] + my[None, :, None] + mx[None, None, :]
        c = torch.where(mu > 0, c / mu.clamp(min=1e-300), torch.zeros_like(c))
        return -h2 * torch.einsum("kz,kyx->zyx", vz, torch.einsum("ky,zkx->zyx", vy, torch.einsum("kx,zyk->zyx", vx, c)))

    def _prolong(self, e):
        for dim in (2, 1, 0):
            lo, hi = _shift(e, dim, -1), _shift(e, dim, 1)
            if self.ref and dim == 1:
                hi = torch.cat([hi.narrow(1, 0, hi.shape[1] - 1), torch.zeros_like(hi.narrow(1, 0, 1))], 1)
            e = torch.stack([0.75 * e + 0.25 * lo, 0.75 * e + 0.25 * hi], dim + 1).flatten(dim, dim + 1)
        return e

    def cycle(self, l, e, b):
        c = self.cfg
        top = l == 0 and c.reference_schedule
        if l == c.mg_levels - 1:
            if c.mg_levels == 1:
                return self._sweep(l, e, b, c.mg_pre + c.mg_post)
            return self.direct(l, b) if c.mg_coarse_sweeps < 0 else self._sweep(l, e, b, c.mg_coarse_sweeps)
        e = self._sweep(l, e, b, 1 if top else c.mg_pre)
        (nz, ny, nx), h2, diag, _ = self.lv[l]
        r = b - (self._sum(e) - diag * e) / h2
        r = r.reshape(nz // 2, 2, ny // 2, 2, nx // 2, 2).mean(dim=(1, 3, 5))
        e = e + self._prolong(self.cycle(l + 1, torch.zeros_like(r), r))
        return self._sweep(l, e, b, 1 if top else c.mg_post)

    def solve(self, p, b):
        if self.cfg.precision_mode == abi.DOB_PREC_MIXED:
            return self.direct(0, b)
        for _ in range(self.cfg.mg_cycles):
            p = self.cycle(0, p, b)
        return p if self.ref else p - p.mean()


def _trace(cen, uvw, dt, size, lo, hi, at=None, sign=1.0):
    """(departure point, start velocity) of the midpoint trace from uvw."""
    v0 = at if at is not None else _sample(cen, [t.clamp(lo, hi) for t in uvw])
    mid = [(t - sign * 0.5 * v * dt / s).clamp(lo, hi) for t, v, s in zip(uvw, v0, size)]
    vm = _sample(cen, mid)
    return [(t - sign * v * dt / s).clamp(lo, hi) for t, v, s in zip(uvw, vm, size)], v0


def _wall(a, dim):
    """a with its last layer along dim zeroed."""
    return torch.cat([a.narrow(dim, 0, a.shape[dim] - 1), torch.zeros_like(a.narrow(dim, 0, 1))], dim)


def _div(u, v, w):
    d = torch.zeros_like(u)
    for a, dim in ((u, 2), (v, 1), (w, 0)):
        a = _wall(a, dim)
        d = d + a - torch.cat([torch.zeros_like(a.narrow(dim, 0, 1)), a.narrow(dim, 0, a.shape[dim] - 1)], dim)
    return d


def _exact_step(cfg, mg, u, v, w, p, dye, cen, parcels=None):
    nx, ny, nz = cfg.nx, cfg.ny, cfg.nz
    size, dt, dx = (float(nx), float(ny), float(nz)), float(cfg.dt), float(cfg.dx)
    dev = u.device
    x = ((torch.arange(nx, dtype=torch.float64, device=dev) + 0.5) / nx)[None, None, :].expand(nz, ny, nx)
    y = ((torch.arange(ny, dtype=torch.float64, device=dev) + 0.5) / ny)[None, :, None].expand(nz, ny, nx)
    z = ((torch.arange(nz, dtype=torch.float64, device=dev) + 0.5) / nz)[:, None, None].expand(nz, ny, nx)
    half = (0.5 / nx, 0.5 / ny, 0.5 / nz)
    c3, new = [cen[0], cen[1], cen[2]], []
    for k, a in enumerate((u, v, w)):
        face = [t + half[j] if j == k else t for j, t in enumerate((x, y, z))]
        end, _ = _trace(c3, face, dt, size, 0.002, 0.998)
        end[k] = end[k] - half[k]
        new.append(_wall(_sample([a], [t.clamp(0.001, 0.999) for t in end])[0] * float(cfg.vel_damping), 2 - k))
    u, v, w = new
    d2, lap = 0.0, [-6.0 * a for a in (u, v, w)]
    for dim in range(3):
        for k, a in enumerate((u, v, w)):
            hi, lo = _shift(a, dim, 1), _shift(a, dim, -1)
            d2 = d2 + (hi - lo) ** 2
            lap[k] = lap[k] + hi + lo
    c = dye.clamp(0.0, 1.5)
    # the root of the shear rate has no slope at rest: its limit there is 0
    gdot = torch.where(d2 > 0, d2, torch.ones_like(d2)).sqrt() * (d2 > 0) / (2 * dx)
    yield_ = c * torch.sqrt(float(cfg.casson_tau_y) / (gdot + 0.4))
    nu = (math.sqrt(cfg.casson_mu_p) + yield_) ** 2
    alpha = (nu * dt / (dx * dx)).clamp(max=0.125)
    u, v, w = (_wall(a + alpha * l, 2 - k) for k, (a, l) in enumerate(zip((u, v, w), lap)))
    b = _div(u, v, w)
    p = mg.solve(p, b - b.mean())
    u, v, w = (_wall(a - (_shift(p, 2 - k, 1) - p), 2 - k) for k, a in enumerate((u, v, w)))
    cen = _centre(u, v, w)
    c3 = [cen[0], cen[1], cen[2]]
    if parcels is not None:
        def vel(q):
            return torch.stack(_sample(c3, [(q[:, k] / size[k]).clamp(0.002, 0.998) for k in range(3)]), 1)

        k1 = vel(parcels)
        k2 = vel(parcels + 0.5 * dt * k1)
        k3 = vel(parcels + 0.75 * dt * k2)
        s = torch.tensor(size, dtype=torch.float64, device=dev)
        parcels = torch.minimum(torch.maximum(parcels + dt * (2 * k1 + 3 * k2 + 4 * k3) / 9, 0.002 * s), 0.998 * s)
    back, v0 = _trace(c3, [x, y, z], dt, size, 0.001, 0.999, at=c3)
    idx, f = _corners(dye.shape, back)
    taps = [dye.reshape(-1)[i] for i in idx]
    pred = _mix8(taps, f)
    lo, hi = taps[0], taps[0]
    for t in taps[1:]:
        lo, hi = torch.minimum(lo, t), torch.maximum(hi, t)
    fwd = [(t + q * dt / s).clamp(0.001, 0.999) for t, q, s in zip((x, y, z), v0, size)]
    est = _sample([pred], fwd)[0]
    dye = torch.minimum(torch.maximum(pred + 0.45 * float(cfg.dye_sharpness) * (dye - est), lo), hi)
    return u, v, w, p, dye, cen, parcels


def exact(case, seed):
    kind = case["kind"]
    if kind in ("ref", "render"):
        # binary16 textures, drops, parcels with thresholds: no plain 64-bit value to hold them to
        return None
    if kind == "psolve":
        b, p0 = _psolve_inputs(case, seed)
        cfg = _psolve_config(case)
        return {"p": _Poisson(cfg, b.device).solve(p0.double(), b.double())}
    cfg = _box_config(case)
    st = {k: torch.from_numpy(a).to(DEV).double() for k, a in _box_state(case, seed).items()}
    mg = _Poisson(cfg, torch.device(DEV))
    if kind == "box":
        with torch.no_grad():
            s = tuple(st[k] for k in ("u", "v", "w", "p", "dye"))
            s += (_centre(*s[:3]), st["parcels"][:, :3])
            for _ in range(case["steps"]):
                s = _exact_step(cfg, mg, *s)
        out = dict(zip(("u", "v", "w", "p", "dye"), s[:5]))
        out["parcels"] = torch.cat([s[6], st["parcels"][:, 3:]], 1)
        if case["pipelined"]:
            out["alive"] = None
        return out
    # the gradient by automatic differentiation, one step's graph at a time
    names = ("u", "v", "w", "p", "dye")
    states = [tuple(st[k] for k in names)]
    with torch.no_grad():
        for _ in range(case["steps"]):
            s = states[-1]
            states.append(_exact_step(cfg, mg, *s, _centre(*s[:3]))[:5])
    g = [torch.zeros_like(st["u"]) for _ in range(4)] + [torch.from_numpy(_dye_gradient(case, seed)).to(DEV).double()]
    for s in reversed(states[:-1]):
        s = [a.detach().requires_grad_(True) for a in s]
        out = _exact_step(cfg, mg, *s, _centre(*s[:3]))[:5]
        g = torch.autograd.grad(out, s, grad_outputs=g, allow_unused=True)
        g = [torch.zeros_like(a) if h is None else h for a, h in zip(s, g)]
    # in clear water every tap of the limiter is equal: there the loss has no
    # derivative in the dye, and each convention gives another value
    return {"dye": states[-1][4], "grad": dict(zip(names, g), dye=None)}

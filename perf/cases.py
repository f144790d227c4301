"""The performance cases: what users of this framework have it do, through its
public entry points, over the sizes, precisions and options they use.

  transform  `Mesh.transform2d_dev`: a batch of half-integer transforms of
             device planes (the plug-in call of the reference).
  march      `Mesh.move_all_split_layers` with the driver held, as a scan over
             plasma parameters runs it, then the on-axis wake, the potential
             and the tail layer's longitudinal field.
  step       `Mesh.step_host`: the beam in from pinned host memory, the beam
             push, the march, beam and on-axis wake back (a simulation's loop).
  adjoint    `autograd.wake_loss` forward and backward: the gradient of a loss
             on the wake with respect to the driver's charge profile.

Everything is made from the seed: the driver is a sampled bi-Gaussian bunch
whose radius and density vary by a few per cent with it.  Results of a march
in 32 bits are given as float32 and those of one in 64 bits as float64 (the
calls return both in float64 arrays).

`exact` holds a plain torch restatement in 64 bits: dense transform matrices,
the per-mode maps of the Guess and the Iterate, the particle push, the NGP and
CIC deposits and the beam deposit, differentiable for the adjoint.
"""
from __future__ import annotations

import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from tertia_b200.abi import (PRECISIONS, QS_F_EX, QS_REDFT11, QS_RODFT11, QS_SHAPE_CIC,
                             QS_SHAPE_NGP, default_config)
from tertia_b200.autograd import wake_loss, xi_bins
from tertia_b200.mesh import Mesh

F64 = ("fp64", "fp64fft")
BINS = 64


def listed():
    march = dict(kind="march", ppc=4, n_iter=1, shape="cic", beam=100_000)
    return [
        # three small planes: one call is all launches and latency
        dict(name="transform_128_fp32", kind="transform", precision="fp32", ny=128, nz=128,
             batch=3, kz="C", ky="S"),
        # the six field planes of a layer at the benchmark's transverse size
        dict(name="transform_512_fp32", kind="transform", precision="fp32", ny=512, nz=512,
             batch=6, kz="C", ky="C"),
        # the largest 64-bit transforms, on a rectangular grid
        dict(name="transform_1024_fp64fft", kind="transform", precision="fp64fft", ny=1024, nz=512,
             batch=4, kz="S", ky="C"),
        # the smallest march: a quick look with the reference's live particle shape
        dict(march, name="march_64_ngp_fp32", precision="fp32", ny=64, nz=64, nx=32, shape="ngp",
             beam=20_000),
        # the benchmark's plain 64-bit configuration (128 x 128 x 256)
        dict(march, name="march_128_fp64", precision="fp64", ny=128, nz=128, nx=256),
        # sizes that are no power of two, nine particles per cell, two iterations
        dict(march, name="march_ragged_fp32", precision="fp32", ny=96, nz=160, nx=48, ppc=9,
             n_iter=2),
        # the default precision at the benchmark's transverse size, the head of its box
        dict(march, name="march_512_fp32", precision="fp32", ny=512, nz=512, nx=128),
        # the 64-bit path for production accuracy at that size
        dict(march, name="march_512_fp64fft", precision="fp64fft", ny=512, nz=512, nx=64),
        # the transverse size of the two largest configurations
        dict(march, name="march_1024_fp32", precision="fp32", ny=1024, nz=1024, nx=48),
        # split-precision transforms on the tensor cores (the precision study)
        dict(march, name="march_512_bf16x3", precision="bf16x3", ny=512, nz=512, nx=48),
        # the gradient configuration's grid, 64 bins, checkpoints every 32 layers
        dict(name="adjoint_256_fp32", kind="adjoint", precision="fp32", ny=256, nz=256, nx=256,
             ppc=4, n_iter=1, shape="cic", beam=200_000, every=32),
        # the benchmark itself: one whole beam step of 512 x 512 x 1024, warm plasma
        dict(name="step_512_fp32", kind="step", precision="fp32", ny=512, nz=512, nx=1024, ppc=4,
             n_iter=1, shape="cic", beam=1_000_000, thermal=0.01),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _plane(rng, precision, lo, hi, most):
    """ny, nz of a transverse grid: powers of two, and other multiples of 8
    where the precision takes them; at most `most` cells."""
    while True:
        if precision == "bf16x3":
            ny, nz = 128 * rng.randint(1, 5), 128 * rng.randint(1, 5)
        elif precision != "fp64fft" and rng.random() < (0.2 if precision == "fp32" else 0.5):
            ny, nz = 8 * _log(rng, lo / 8, 32), 8 * _log(rng, lo / 8, 32)
        else:
            e = (int(math.log2(lo)), int(math.log2(hi)))
            ny = 1 << rng.randint(*e)
            nz = ny if rng.random() < 0.6 else 1 << rng.randint(*e)
        if ny * nz <= most:
            return ny, nz


def draw(rng):
    kind = rng.choice(["transform", "transform", "march", "march", "march", "march", "adjoint",
                       "step"])
    if kind == "transform":
        precision = rng.choice(["fp32", "fp32", "fp64fft", "fp64", "bf16x3"])
        ny, nz = _plane(rng, precision, 32, 256 if precision == "fp64" else 1024, 1 << 20)
        return dict(kind=kind, precision=precision, ny=ny, nz=nz, batch=_log(rng, 1, 8),
                    kz=rng.choice("CS"), ky=rng.choice("CS"))
    if kind == "march":
        precision = rng.choice(["fp32", "fp32", "fp32", "fp64fft", "fp64", "bf16x3"])
        ny, nz = _plane(rng, precision, 64, 256 if precision == "fp64" else 1024, 1 << 20)
        shape = rng.choice(["cic", "cic", "cic", "ngp"])
        # an NGP deposit jumps where a particle crosses a cell boundary, and a
        # wake carries the jump on: those boxes stay short
        nx = _log(rng, 16, min(48 if shape == "ngp" else 192, (1 << 26) // (ny * nz)))
        return dict(kind=kind, precision=precision, ny=ny, nz=nz, nx=nx, shape=shape,
                    ppc=rng.choice([1, 2, 4, 4, 4, 5, 9]), n_iter=rng.choice([1, 1, 1, 2]),
                    beam=_log(rng, 10_000, 300_000))
    precision = rng.choice(["fp32", "fp32", "fp64fft"])
    ny, nz = _plane(rng, "fp64fft", 128, 512, 1 << 18)
    n = ny * nz
    if kind == "adjoint":
        nx = _log(rng, 40, min(256, (1 << 24) // n))
        return dict(kind=kind, precision=precision, ny=ny, nz=nz, nx=nx,
                    ppc=4, n_iter=1, shape="cic", beam=_log(rng, 20_000, 300_000),
                    every=_log(rng, 8, 64))
    nx = _log(rng, 40, min(512, (1 << 26) // n))
    return dict(kind=kind, precision=precision, ny=ny, nz=nz, nx=nx,
                ppc=4, n_iter=1, shape="cic", beam=_log(rng, 50_000, 1_000_000),
                thermal=rng.choice([0.0, 0.01]))


# ---------------------------------------------------------------- the inputs

def _cell(n):
    """Cell size of n cells across the box: 0.05 / k_p, coarser on small grids
    so that the driver and its blowout fit."""
    return max(0.05, 6.4 / n)


def _config(case):
    c = default_config(ny=case["ny"], nz=case["nz"], nx=case.get("nx", 1),
                       hy=_cell(case["ny"]), hz=_cell(case["nz"]),
                       precision=PRECISIONS[case["precision"]])
    if case["kind"] != "transform":
        c.shape = QS_SHAPE_CIC if case["shape"] == "cic" else QS_SHAPE_NGP
        c.ppc, c.n_iter = case["ppc"], case["n_iter"]
        c.pspread_x = c.pspread_y = c.pspread_z = case.get("thermal", 0.0)
    if case["kind"] in ("march", "adjoint"):   # the driver stands where it was sampled
        c.ts, c.synchrotron = 0.0, 0
    return c


def _driver(case, seed):
    """A bi-Gaussian electron bunch near the front of the box, in (cell,
    fraction) form: numpy arrays."""
    rng = np.random.default_rng(seed)
    n, h = case["beam"], (0.05, _cell(case["ny"]), _cell(case["nz"]))
    size = (case["nx"], case["ny"], case["nz"])
    length = size[0] * h[0]
    s_xi = min(1.0, length / 8.0)
    s_r = 0.5 * rng.uniform(0.97, 1.03)
    density = 0.5 * rng.uniform(0.95, 1.05)
    mid = (length - 4.0 * s_xi, size[1] * h[1] / 2, size[2] * h[2] / 2)
    b = {}
    for a, (cell, frac) in enumerate((("i", "x"), ("j", "y"), ("k", "z"))):
        g = mid[a] + (s_xi if a == 0 else s_r) * rng.standard_normal(n)
        g = np.clip(g / h[a], 0.0, size[a] - 1e-9)
        b[cell] = np.floor(g).astype(np.int32)
        b[frac] = g - b[cell]
    b["px"] = np.full(n, math.sqrt(1000.0 ** 2 - 1.0))
    b["py"], b["pz"] = np.zeros(n), np.zeros(n)
    w = density * (2 * math.pi) ** 1.5 * s_xi * s_r ** 2 / (n * h[0] * h[1] * h[2])
    b["w"] = np.full(n, w)
    return b


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.from_numpy(a).dtype, pin_memory=True)
    t.numpy()[:] = a
    return t.numpy()


def _window(case):
    """The witness window: layers whose on-axis field the loss adds up."""
    nx = case["nx"]
    lo = max(1, nx - 200)
    return lo, min(nx - 1, lo + 20)


def _bin_weights(seed):
    g = torch.Generator().manual_seed(seed)
    return 1.0 + 0.1 * torch.rand(BINS, generator=g)


def _bins(case, beam, cfg):
    return xi_bins(beam, cfg, BINS, 0.0, cfg.nx * cfg.hx)


def _planes(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = torch.float64 if case["precision"] in F64 else torch.float32
    return torch.randn(case["batch"], case["nz"], case["ny"], generator=g, device="cuda",
                       dtype=dt)


class State:
    """One mesh and what its caller keeps beside it."""


def prepare(case, seed):
    s = State()
    s.case = case
    cfg = _config(case)
    s.mesh = Mesh(cfg)
    if case["kind"] == "transform":
        s.x = _planes(case, seed)
        s.y = torch.empty_like(s.x)
        kinds = {"C": QS_REDFT11, "S": QS_RODFT11}
        s.args = (kinds[case["kz"]], kinds[case["ky"]], case["batch"], s.x.data_ptr(),
                  s.y.data_ptr())
        return s
    s.beam = {k: _pinned(v) for k, v in _driver(case, seed).items()}
    if case["kind"] == "march":
        s.mesh.load_beam(s.beam)
        s.mesh.move_beam_particles()
    elif case["kind"] == "step":
        s.seed = seed & 0xffff
        s.out = {k: _pinned(np.empty_like(s.beam[k])) for k in "ijk"}
        s.out.update({k: _pinned(np.empty_like(s.beam[k])) for k in ("x", "y", "z", "px", "py",
                                                                     "pz")})
    else:
        s.mesh.seed_front_plasma(0)
        s.mesh.adjoint_checkpoints(case["every"])
        s.bins = _bins(case, s.beam, cfg)
        s.coeff = np.zeros(cfg.nx)
        lo, hi = _window(case)
        s.coeff[lo:hi] = cfg.hx
        s.weights = _bin_weights(seed).requires_grad_(True)
    return s


def _typed(case, a):
    return np.asarray(a, dtype=np.float64 if case["precision"] in F64 else np.float32)


def run(s):
    case, m = s.case, s.mesh
    if case["kind"] == "transform":
        m.transform2d_dev(*s.args)
        return s.y
    if case["kind"] == "march":
        m.move_all_split_layers()
        return {"ex_onaxis": _typed(case, m.onaxis_ex()), "psi": _typed(case, m.psi()),
                "ex_tail": _typed(case, m.get_field3d(QS_F_EX, 0))}
    if case["kind"] == "step":
        m.seed_front_plasma(s.seed)
        b, ex = m.step_host(s.beam, out=s.out)
        got = {"ex_onaxis": _typed(case, ex)}
        for cell, frac in ("ix", "jy", "kz"):
            got[frac] = _typed(case, b[cell] + b[frac])
            got["p" + frac] = _typed(case, b["p" + frac])
        return got
    loss = wake_loss(s.weights, m, s.beam, s.bins, s.coeff)
    grad, = torch.autograd.grad(loss, s.weights)
    return {"loss": loss.detach(), "grad": grad}


def work(case):
    """One pass's reads and writes that no arrangement saves, and operations:
    a layer's particles do not fit on the chip beside its planes, so that each
    of its n_iter + 1 pushes reads them (and the last writes them back); the
    spectra of the beam's two planes are read and the six field planes
    written.  A transform of n points of a row counts 2.5 n log2 n."""
    size = 8 if case["precision"] in F64 else 4
    n = case["ny"] * case["nz"]
    per_plane = 2.5 * n * math.log2(n)
    if case["kind"] == "transform":
        return {"bytes": 2.0 * size * n * case["batch"], "flops": per_plane * case["batch"]}
    pushes = case["n_iter"] + 1
    parts = n * case["ppc"]
    # y, z, px, py, pz, w and a 4-byte cell in; y, z, px, py, pz (and the cell) out
    bytes_ = parts * (pushes * (6 * size + 4) + 5 * size + 4) + 8.0 * size * n
    flops = parts * pushes * 200.0 + (6 + 9 * pushes) * per_plane + 150.0 * n * pushes
    layers = case["nx"]
    total = {"bytes": bytes_ * layers, "flops": flops * layers}
    if case["kind"] == "adjoint":
        # each swept layer: its state read by both push adjoints, five
        # particle adjoints read and written by each, the gathered fields read
        swept = layers - _window(case)[0]
        back = parts * pushes * (6 * size + 4 + 10 * size) + 6.0 * pushes * size * n
        total["bytes"] += back * swept
        total["flops"] += 2.5 * flops * swept
    if case["kind"] in ("step", "adjoint"):
        total["bytes"] += case["beam"] * 2 * (3 * 4 + 7 * 8)
        total["flops"] += case["beam"] * 400.0
    return total


# ------------------------------------------------- the same in 64 bits, plain

def _dtt(n, kind):
    i = torch.arange(n, device="cuda", dtype=torch.int64)
    # (2j+1)(2k+1) in units of pi/(4n), reduced exactly
    q = ((2 * i[:, None] + 1) * (2 * i[None, :] + 1)) % (8 * n)
    a = q.double() * (math.pi / (4.0 * n))
    return 2.0 * (torch.cos(a) if kind == "C" else torch.sin(a))


class _March:
    """The march in float64 on dense matrices (planes are nz x ny)."""

    # z and y kinds of the planes
    EB = ("CC", "CS", "SC", "SS", "SC", "CS")     # Ex Ey Ez Bx By Bz
    J = ("CC", "CS", "SC")

    def __init__(self, case):
        self.case = case
        self.ny, self.nz, self.nx = case["ny"], case["nz"], case["nx"]
        self.hx, self.hy, self.hz = 0.05, _cell(self.ny), _cell(self.nz)
        self.my = {k: _dtt(self.ny, k) for k in "CS"}
        self.mz = {k: _dtt(self.nz, k) for k in "CS"}
        ar = lambda n: torch.arange(n, device="cuda", dtype=torch.float64) + 0.5  # noqa: E731
        self.ky = (math.pi / (self.ny * self.hy)) * ar(self.ny)[None, :]
        self.kz = (math.pi / (self.nz * self.hz)) * ar(self.nz)[:, None]
        self.k2 = self.ky ** 2 + self.kz ** 2

    def transform(self, x, kinds):
        return self.mz[kinds[0]] @ x @ self.my[kinds[1]]

    def fields(self, spec):
        s = 1.0 / (4.0 * self.ny * self.nz)
        return torch.stack([s * self.transform(x, k) for x, k in zip(spec, self.EB)])

    def beam_spectra(self, b, w, drift):
        """Spectra of RhoBeam and JxBeam of layers 0..nx, of the bunch after
        `drift` of its own motion in empty space."""
        t = {k: torch.as_tensor(v, device="cuda") for k, v in b.items()}
        gamma = torch.sqrt(1.0 + t["px"] ** 2 + t["py"] ** 2 + t["pz"] ** 2)
        vx = t["px"] / gamma
        x = t["i"].double() + t["x"] + (vx - 1.0) * drift / self.hx
        i = torch.floor(x).long()
        out = torch.zeros(2, self.nx + 1, self.nz, self.ny, device="cuda", dtype=torch.float64)
        out = out.reshape(2, -1)
        j, k = t["j"].long(), t["k"].long()
        q = -w
        for di in (0, 1):
            for dj in (0, 1):
                for dk in (0, 1):
                    a = ((x - i) if di else 1.0 - (x - i)) * (t["y"] if dj else 1.0 - t["y"]) * \
                        (t["z"] if dk else 1.0 - t["z"])
                    ii, jj, kk = i + di, j + dj, k + dk
                    ok = (ii >= 0) & (ii <= self.nx) & (jj < self.ny) & (kk < self.nz)
                    at = ((ii * self.nz + kk) * self.ny + jj)[ok]
                    add = torch.stack([q * a, q * vx * a])[:, ok]
                    out = out.index_add(1, at, add)
        out = out.reshape(2, self.nx + 1, self.nz, self.ny)
        return self.mz["C"] @ out @ self.my["C"], x

    def front(self):
        ppc, n = self.case["ppc"], self.ny * self.nz
        side = int(math.sqrt(ppc - 1) + 1.0)
        at = []
        for s in range(ppc):
            if ppc <= 3:
                at.append((0.5, 0.5))
            elif ppc == 4:
                at.append(((1.0 + s % 2) / 3.0, (1.0 + s // 2) / 3.0))
            else:
                at.append(((s % side + 0.5) / side, (s // side + 0.5) / side))
        at = torch.tensor(at, device="cuda", dtype=torch.float64).repeat(n, 1)
        cell = torch.arange(n, device="cuda").repeat_interleave(ppc)
        zero = torch.zeros(n * ppc, device="cuda", dtype=torch.float64)
        return cell, at[:, 0], at[:, 1], zero, zero, zero

    def corners(self, cell, y, z):
        j, k = cell % self.ny, cell // self.ny
        j1, k1 = (j + 1) % self.ny, (k + 1) % self.nz
        return ((j + self.ny * k, (1 - y) * (1 - z)), (j1 + self.ny * k, y * (1 - z)),
                (j + self.ny * k1, (1 - y) * z), (j1 + self.ny * k1, y * z))

    def push(self, state, avg):
        """The deposit of Jx, Jy, Jz and the state after the move."""
        cic = self.case["shape"] == "cic"
        cell, y, z, px, py, pz = state
        flat = avg.reshape(6, -1)
        if cic:
            f = sum(w * flat[:, c] for c, w in self.corners(cell, y, z))
        else:
            f = flat[:, cell]
        half = -0.5 * self.hx                        # q/m hx/2
        g = torch.sqrt(1 + px ** 2 + py ** 2 + pz ** 2)
        vx0, vy0, vz0 = px / g, py / g, pz / g
        kick = half / (1 - vx0)
        ex, ey, ez = f[0] * kick, f[1] * kick, f[2] * kick
        px, py, pz = px + ex, py + ey, pz + ez
        kick = kick / torch.sqrt(1 + px ** 2 + py ** 2 + pz ** 2)
        bx, by, bz = f[3] * kick, f[4] * kick, f[5] * kick
        co = 2 / (1 + bx ** 2 + by ** 2 + bz ** 2)
        qx, qy, qz = ((py * bz - pz * by + px) * co, (pz * bx - px * bz + py) * co,
                      (px * by - py * bx + pz) * co)
        px, py, pz = (px + ex + qy * bz - qz * by, py + ey + qz * bx - qx * bz,
                      pz + ez + qx * by - qy * bx)
        g = torch.sqrt(1 + px ** 2 + py ** 2 + pz ** 2)
        vx, vy, vz = px / g, py / g, pz / g
        inv = 1 / (1 - 0.5 * (vx + vx0))
        dj = torch.stack([-vx, -vy, -vz]) * (inv / self.case["ppc"])
        dy = 0.5 * (vy + vy0) * self.hx / self.hy * inv
        dz = 0.5 * (vz + vz0) * self.hx / self.hz * inv
        step = torch.clamp(torch.maximum(dy.abs(), dz.abs()), min=1.0)
        done = 0                                     # sub-steps of at most one cell
        dep = torch.zeros(3, self.ny * self.nz, device="cuda", dtype=torch.float64)
        j0, k0 = cell % self.ny, cell // self.ny
        j, k = j0, k0
        while True:
            left = step - done
            live = left > 0
            ps = torch.where(live, torch.where(left > 1, 1 / step, left / step), 0.0)
            uy, uz = y + dy * ps, z + dz * ps
            sy, sz = torch.floor(uy.detach()), torch.floor(uz.detach())
            bj, bk = (j, k) if cic else (j0, k0)
            nj = (bj + sy.long()) % self.ny
            nk = (bk + sz.long()) % self.nz
            j, k = torch.where(live, nj, j), torch.where(live, nk, k)
            y, z = torch.where(live, uy - sy, y), torch.where(live, uz - sz, z)
            now = j + self.ny * k
            if cic:
                for c, w in self.corners(now, y, z):
                    dep = dep.index_add(1, c, dj * (ps * w))
            else:
                dep = dep.index_add(1, now, dj * ps)
            done += 1
            if not bool((step > done).any()):
                break
        new = (j + self.ny * k) if cic else cell
        return dep.reshape(3, self.nz, self.ny), (new, y, z, px, py, pz)

    def layer(self, bank, pf, state, rb, jxb, rbp):
        """One layer: the P bank (rho, E, J spectra), the P fields and the
        particles; returns those of the layer."""
        hx, ky, kz, k2 = self.hx, self.ky, self.kz, self.k2
        rho_p, ex_p, ey_p, ez_p, jx_p, jy_p, jz_p = bank
        dh2 = hx * hx
        den = 4.0 + dh2
        rbs = rb + rbp
        rho = ((4 - dh2) * rho_p - rbs * dh2 + 4 * hx * ex_p * (k2 + 1)) / den
        ex = ((4 - dh2) * ex_p - 2 * hx * (2 * rho_p + rbs) / (k2 + 1)) / den
        src = (rbs + rho_p + rho) / (k2 + 1)
        ey, ez = -ey_p + ky * src, -ez_p + kz * src
        jx = jx_p + 0.5 * hx * (ex + ex_p)
        jy = jy_p + 0.5 * hx * (ey + ey_p)
        jz = jz_p + 0.5 * hx * (ez + ez_p)

        def magnetic(jx, jy, jz, ey, ez):
            return ((kz * jy - ky * jz) / k2, (-kz * (jx + jxb) + ez) / k2,
                    (ky * (jx + jxb) - ey) / k2)

        cf = self.fields((ex, ey, ez) + magnetic(jx, jy, jz, ey, ez))
        for it in range(self.case["n_iter"] + 1):
            dep, moved = self.push(state, 0.5 * (pf + cf))
            jx, jy, jz = (self.transform(d, k) for d, k in zip(dep, self.J))
            src = (rbs + rho_p + rho) / (k2 + 1)
            rho = rho_p + jx - jx_p - 0.5 * hx * (ky * (jy + jy_p) + kz * (jz + jz_p))
            ex = -(ky * jy + kz * jz) / k2
            ey, ez = -ey_p + ky * src, -ez_p + kz * src
            cf = self.fields((ex, ey, ez) + magnetic(jx, jy, jz, ey, ez))
        return (rho, ex, ey, ez, jx, jy, jz), cf, moved

    def run(self, beam, w, drift=0.0, grad=False):
        """On-axis Ex of every layer, the tail's Ex plane, the beam's x."""
        (rb, jxb), x = self.beam_spectra(beam, w, drift)
        zero = torch.zeros(self.nz, self.ny, device="cuda", dtype=torch.float64)
        bank, pf, state = (zero,) * 7, torch.stack([zero] * 6), self.front()
        axis = [None] * self.nx
        for i in range(self.nx - 1, -1, -1):
            args = (bank, pf, state, rb[i], jxb[i], rb[i + 1] if i < self.nx - 1 else zero)
            bank, pf, state = (checkpoint(self.layer, *args, use_reentrant=False) if grad
                               else self.layer(*args))
            axis[i] = pf[0, self.nz // 2, self.ny // 2]
        return torch.stack(axis), pf[0], x


def exact(case, seed):
    if case["kind"] == "transform":
        x = _planes(case, seed).double()
        return _dtt(case["nz"], case["kz"]) @ x @ _dtt(case["ny"], case["ky"])
    if case.get("thermal"):
        return None   # the front plasma's momenta are the device generator's own
    m = _March(case)
    b = _driver(case, seed)
    w = torch.as_tensor(b["w"], device="cuda")
    if case["kind"] == "adjoint":
        cfg = _config(case)
        bins = torch.as_tensor(_bins(case, b, cfg), device="cuda")
        beta = _bin_weights(seed).double().cuda().requires_grad_(True)
        axis, _, _ = m.run(b, w * beta[bins], grad=True)
        lo, hi = _window(case)
        loss = m.hx * axis[lo:hi].sum()
        grad, = torch.autograd.grad(loss, beta)
        return {"loss": loss.detach(), "grad": grad}
    with torch.no_grad():
        axis, tail, x = m.run(b, w, drift=1.0 if case["kind"] == "step" else 0.0)
    if case["kind"] == "step":
        got = {"ex_onaxis": axis, "x": x}
        for cell, frac in ("jy", "kz"):
            got[frac] = b[cell] + b[frac]
        got.update({p: b[p] for p in ("px", "py", "pz")})
        return got
    ahead = torch.cat([axis[1:], torch.zeros_like(axis[:1])])
    psi = torch.flip(torch.cumsum(torch.flip(0.5 * m.hx * (axis + ahead), [0]), 0), [0])
    return {"ex_onaxis": axis, "psi": psi, "ex_tail": tail}

"""The work a SWAP user has this library do, as cases with a size, timed through its public entries.

A case is a dict of plain values with a ``kind``:

* ``subcycle``: one field subcycle through the per-subroutine entries (maind.f:430-462), as SWAP's own
  driver calls them on resident arrays.
* ``particles``: the particle entries of one ion step up to improve_up (maind.f:385-402), one by one.
* ``steps``: whole FP64 ion steps (``swap_run``) between two outputs.
* ``f32``: whole ion steps of the FP32 form between two outputs, in a context of 4-byte reals (SWAP's
  makefile builds with -real-size 32).
* ``moments``: the update_up deposit on the caller's own device arrays (``swap_update_up_noalloc``).
* ``grads``: the field surrogate's loss and weight gradients on one training pair (forward and backward).

The oracle in ``exact`` is the ion step on a periodic box of unit spacing in 64 bits, written with torch.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from swap_gb300.hybrid import Hybrid, Surrogate, config

# Floating point operations, counted from the formulas: one ion through one ion step, one node through one
# field subcycle (predictor and corrector).
ION_FLOPS, NODE_FLOPS = 600, 260


def listed():
    return [
        # the smallest calls: a ragged test box, where launches and waits count
        dict(name="subcycle 18x11x14", kind="subcycle", cx=18, cy=11, cz=14),
        # an ordinary field subcycle of a driver that keeps its own loop
        dict(name="subcycle 128x64x64", kind="subcycle", cx=128, cy=64, cz=64),
        # the particle entries one by one on a ragged box with two species
        dict(name="particles 45x22x31", kind="particles", cx=45, cy=22, cz=31, ppc=7, heavy=2),
        # the uniform periodic box at its stated size, from a fresh load, ten steps between outputs
        dict(name="steps 64x32x32", kind="steps", cx=64, cy=32, cz=32, ppc=16, heavy=0, n=10, x_open=False,
             mature=False),
        # solar wind through the box: inflow, outflow and the compaction that goes with them
        dict(name="steps open 128x64x64", kind="steps", cx=128, cy=64, cz=64, ppc=16, heavy=0, n=2, x_open=True,
             mature=False),
        # a run after thousands of steps: the array order of the ions no longer follows their cells
        dict(name="steps mature 64x64x64", kind="steps", cx=64, cy=64, cz=64, ppc=32, heavy=0, n=2, x_open=False,
             mature=True),
        # the FP32 form on its smallest boxes: launch latency
        dict(name="f32 16x8x12", kind="f32", cx=16, cy=8, cz=12, ppc=8, heavy=0, n=20, x_open=False),
        # the FP32 form on the uniform periodic box at its stated size
        dict(name="f32 64x32x32", kind="f32", cx=64, cy=32, cz=32, ppc=16, heavy=0, n=20, x_open=False),
        # two species on an ordinary box
        dict(name="f32 128x64x64", kind="f32", cx=128, cy=64, cz=64, ppc=28, heavy=4, n=20, x_open=False),
        # the benchmark's workload: 134M ions, x inflow and outflow, 20 steps between outputs
        dict(name="f32 open 256x128x128", kind="f32", cx=256, cy=128, cz=128, ppc=32, heavy=0, n=20, x_open=True),
        # a caller with its own device arrays
        dict(name="moments 96x80x64", kind="moments", cx=96, cy=80, cz=64, ppc=8),
        # one training pair of the surrogate at the size of its training boxes
        dict(name="grads 64x64x64", kind="grads", cx=64, cy=64, cz=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["subcycle", "particles", "steps", "steps", "f32", "f32", "moments", "grads"])
    if kind == "grads":  # the network wants a multiple of 128 voxels
        return dict(kind=kind, cx=rng.choice([8, 16, 32, 64, 128]), cy=4 * _log(rng, 2, 16), cz=4 * _log(rng, 2, 16))
    if kind == "f32":  # 8..1024 cells per axis, multiples of 4
        cells = [4 * _log(rng, 2, 32), 4 * _log(rng, 2, 16), 4 * _log(rng, 2, 16)]
        return dict(kind=kind, cx=cells[0], cy=cells[1], cz=cells[2], ppc=rng.randint(8, 28),
                    heavy=rng.choice([0, 0, 2, 4]), n=rng.randint(5, 20), x_open=rng.random() < 0.3)
    cells = [_log(rng, 8, 100), _log(rng, 8, 80), _log(rng, 8, 80)]
    c = dict(kind=kind, cx=cells[0], cy=cells[1], cz=cells[2])
    if kind == "subcycle":
        return c
    c["ppc"] = rng.randint(5, 16)
    if kind == "moments":
        return c
    c["heavy"] = rng.choice([0, 0, 1, 3])
    if kind == "steps":
        c.update(n=rng.randint(1, 4), x_open=rng.random() < 0.3, mature=rng.random() < 0.5)
        c["ppc"] = rng.randint(8, 16)
    return c


# ---- inputs ------------------------------------------------------------------------------------------------


def _cells(case):
    return case["cx"], case["cy"], case["cz"]


def _gen(seed, device="cuda"):
    return torch.Generator(device=device).manual_seed(seed)


def _ion_columns(cells, ppc, u, vth, g):
    """Columns x, y, z, vx, vy, vz (FP64, on the GPU): ppc ions per cell, uniform in it, drifting Maxwellian,
    in the loader's order (by 4x4x4 bricks where the cells allow it, else x fastest)."""
    ncx, ncy, ncz = cells
    n = ncx * ncy * ncz
    c = torch.arange(n, device="cuda")
    if ncx % 4 == 0 and ncy % 4 == 0 and ncz % 4 == 0:
        b, l = c // 64, c % 64
        nbx, nby = ncx // 4, ncy // 4
        ijk = (4 * (b % nbx) + l % 4, 4 * (b // nbx % nby) + l // 4 % 4, 4 * (b // (nbx * nby)) + l // 16)
    else:
        ijk = (c % ncx, c // ncx % ncy, c // (ncx * ncy))
    for i in ijk:  # cell i spans q(i+1)..q(i+2) of the unit grid; kept off the faces, in 4-byte reals too
        yield (i + 1).repeat_interleave(ppc).double() + 1e-4 + (1 - 2e-4) * torch.rand(
            n * ppc, generator=g, device="cuda", dtype=torch.float64)
    for m in range(3):
        yield u[m] + vth * torch.randn(n * ppc, generator=g, device="cuda", dtype=torch.float64) / math.sqrt(2)


def _perturbed_b(cells, b0, g, amp=0.05):
    """b0 along z plus a few long waves and noise on the nodes, with periodic ghost planes."""
    ncx, ncy, ncz = cells
    x, y, z = torch.meshgrid(*(2 * math.pi * torch.arange(n, device="cuda", dtype=torch.float64) / n
                               for n in cells), indexing="ij")
    b = torch.empty(ncx, ncy, ncz, 3, device="cuda", dtype=torch.float64)
    ph = 2 * math.pi * torch.rand(9, generator=g, device="cuda", dtype=torch.float64)
    for m, (p, q, r) in enumerate(((y, z, x), (z, x, y), (x, y, z))):
        b[..., m] = amp * (torch.sin(p + ph[3 * m]) + torch.cos(q + ph[3 * m + 1]) + 0.5 * torch.sin(
            2 * r + ph[3 * m + 2]))
    b += 0.4 * amp * torch.randn(b.shape, generator=g, device="cuda", dtype=torch.float64)
    b[..., 2] += b0
    return _ghosts(b)


def _ghosts(a):
    """Interior (ncx,ncy,ncz,...) to nodes with the periodic ghost planes (node 1 = node n-1, node n = node 2)."""
    for ax in range(3):
        n = a.shape[ax]
        a = torch.cat([a.narrow(ax, n - 1, 1), a, a.narrow(ax, 0, 1)], ax)
    return a


def _config(case, seed):
    cells, ppc = _cells(case), case.get("ppc", 1)
    cfg = config(1 if case.get("x_open") else 0, cells=cells, ppc=ppc, seed=seed)
    return cfg


def _put(dst, src):
    torch.from_numpy(dst).copy_(src)


def _load(h, case, seed):
    """A user's arrays before the first call: ions and a perturbed field, already on the device."""
    cfg, cells, g = h.cfg, _cells(case), _gen(seed)
    if "ppc" in case:
        n1 = int(np.prod(cells)) * case["ppc"]
        n = n1 + int(np.prod(cells)) * case.get("heavy", 0)
        perm = torch.randperm(n, generator=g, device="cuda") if case.get("mature") else None
        light = _ion_columns(cells, case["ppc"], cfg.u, cfg.vth, g)
        heavy = _ion_columns(cells, case["heavy"], (0.2, 0.0, 0.0), 0.2, g) if case.get("heavy") else None
        for q, col in enumerate(light):
            if heavy is not None:
                col = torch.cat([col, next(heavy)])
            if perm is not None:
                col = col[perm]
            _put((h.xp if q < 3 else h.vp)[:n, q % 3], col)
            if q >= 3:  # v one step back: not quite v
                _put(h.vp1[:n, q % 3], col + 0.02 * torch.randn(n, generator=g, device="cuda", dtype=torch.float64))
        if heavy is not None:  # pickup ions: mass 4, two per light ion's weight
            col = torch.ones(n, device="cuda", dtype=torch.float64)
            for dst, v in ((h.mrat, 0.25), (h.beta_p, 2.0)):
                col[n1:] = v
                _put(dst[:n], col if perm is None else col[perm])
        h.ni_tot[0] = n
    b = _perturbed_b(cells, cfg.b0, g)
    for a in (h.b1, h.b12, h.b1p2, h.bt):
        _put(a, b)
    if case["kind"] == "subcycle":  # np, up and the level one subcycle back come from the particle half
        d = lambda *s: torch.randn(*s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
        _put(h.np, _ghosts(1 + 0.2 * torch.tanh(d(*cells))))
        _put(h.up, _ghosts(0.1 * d(*cells, 3) + torch.tensor(cfg.u, device="cuda", dtype=torch.float64)))
        _put(h.b12, b + 0.004 * _ghosts(d(*cells, 3)))
    h.mark_host_dirty()
    h.sync_to_device()


def _room(case, cfg):
    n = int(np.prod(_cells(case))) * (case.get("ppc", 0) + case.get("heavy", 0))
    return int(1.1 * n) + 4096 if case.get("x_open") else max(n, 1)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "grads":
        dims, g = _cells(case), _gen(seed)
        V = dims[0] * dims[1] * dims[2]
        net = Surrogate(seed=seed % 1000 + 1)
        net.set_curl_weight(1.0, 2.5)  # the bench trains with the curl term
        net.norm(*_norm())
        return dict(kind=kind, net=net, dims=dims, vin=torch.randn(V, Surrogate.NIN, generator=g, device="cuda"),
                    tgt=torch.randn(V, 3, generator=g, device="cuda"))
    cfg = _config(case, seed)
    if kind == "moments":
        nodes, n = cfg.nodes, cfg.n_particles
        h = Hybrid(config(0, cells=(4, 3, 3), ppc=1))  # its library handle; the entry itself takes no context
        from swap_gb300 import abi
        from swap_gb300.grid import Coords, grd7

        co = grd7(*nodes)
        g = _gen(seed)
        cols = list(_ion_columns(_cells(case), case["ppc"], cfg.u, cfg.vth, g))
        dens = _ghosts(1 + 0.2 * torch.tanh(torch.randn(*_cells(case), generator=g, device="cuda",
                                                        dtype=torch.float64)))
        return dict(kind=kind, lib=h.lib, n=n, co=co, nodes=nodes, dims=abi.Dims(*nodes, 8, n),
                    prm=abi.Params(cfg.dt, cfg.alpha, cfg.beta, co.dx, co.dy, 0.0, cfg.ntsub, 0),
                    coords=abi.Coords(*[abi.dptr(getattr(co, a)) for a in Coords.ARRAYS]),
                    x=torch.cat(cols[:3]), v=torch.cat(cols[3:]),
                    bp=torch.ones(n, device="cuda", dtype=torch.float64),
                    np=dens.permute(2, 1, 0).contiguous(),
                    up=torch.zeros(3, nodes[2], nodes[1], nodes[0], device="cuda", dtype=torch.float64))
    h = Hybrid(cfg, ni_max=_room(case, cfg), work_arrays=kind == "particles", real_bytes=4 if kind == "f32" else 8)
    if cfg.sources:
        h.set_sources(cfg.make_sources())
    _load(h, case, seed)
    if kind == "f32" and not case["x_open"]:
        h.f32_begin()
    return dict(kind=kind, h=h, n=case.get("n", 1), x_open=case.get("x_open", False))


def _norm():
    return (np.full(Surrogate.NIN, 0.1), np.full(Surrogate.NIN, 1.5), np.array([0.5, -0.25, 0.0]),
            np.array([0.75, 0.5, 2.0]))


# ---- one pass ----------------------------------------------------------------------------------------------


def _fetch(h, *names):
    """The named arrays as the caller reads them: brought to the host (the ions' up to Ni_tot)."""
    for k in names:
        h.sync_to_host(getattr(h, k))
    return {k: getattr(h, k) for k in names}


def run(s):
    kind = s["kind"]
    if kind == "grads":
        loss, g = s["net"].grads(s["dims"], s["vin"].data_ptr(), s["tgt"].data_ptr())
        return dict(loss=loss, grads=g)
    if kind == "moments":
        p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
        rc = s["lib"].swap_update_up_noalloc(C.byref(s["dims"]), C.byref(s["prm"]), C.byref(s["coords"]), p(s["x"]),
                                             p(s["v"]), p(s["bp"]), s["n"], p(s["np"]), p(s["up"]),
                                             C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0, rc
        return s["up"]
    h = s["h"]
    if kind == "subcycle":  # maind.f:430-462; f_update_tlev is left to the caller, so that a pass can be repeated
        dtsub = h.cfg.dt / h.cfg.ntsub
        h.curlB(h.bt, h.np, h.aj)
        h.predict_B(h.b0, h.b1, h.b12, h.b1p2, h.bt, h.E, h.aj, h.up, h.np, h.nu, dtsub)
        h.correct_B(h.b0, h.b1, h.b1p2, h.E, h.aj, h.up, h.np, h.nu, dtsub)
        return _fetch(h, "b1p2", "E", "aj")
    if kind == "particles":
        h.get_interp_weights(h.xp)
        h.update_np(h.np)
        h.update_up(h.vp, h.np, h.up)
        h.curlB(h.bt, h.np, h.aj)
        h.edge_to_center(h.bt, h.btc)
        h.extrapol_up(h.up, h.vp, h.vp1, h.np)
        h.get_Ep(h.Ep, h.aj, h.np, h.up, h.btc, h.nu)
        h.get_vplus_vminus(h.Ep, h.btc, h.vp, h.vplus, h.vminus)
        h.improve_up(h.vp1, h.vplus, h.vminus, h.up, h.np)
        return _fetch(h, "np", "up", "btc", "Ep", "vplus", "vminus", "vp1")
    if kind == "steps":
        h.run(s["n"])
        return dict(_fetch(h, "xp", "vp", "vp1", "b1", "b12", "b1p2", "bt", "np", "up", "aj", "E"), ni_tot=h.ni_tot)
    # The FP32 form hands its ions back in the order of its sort, where one last-bit difference in a position
    # moves every later ion of the array by a place: the outputs are the fields and moments.
    if s["x_open"]:  # sources: the FP32 state is begun again after each write-back
        h.f32_begin()
    h.f32_run(s["n"])
    h.f32_end()
    return _fetch(h, "b1", "b12", "np", "up", "aj", "E")


# ---- what a pass cannot do without ---------------------------------------------------------------------------


def work(case):
    ncell = int(np.prod(_cells(case)))
    kind = case["kind"]
    if kind == "grads":
        # 27 taps x the four layers' true channels, forward, data gradient and weight gradient
        macs = 27 * (14 * 16 + 2 * 16 * 16 + 16 * 3)
        return {"bytes": ncell * (14 + 3) * 4, "flops": 3 * 2 * macs * ncell}
    nodes = int(np.prod([c + 2 for c in _cells(case)]))
    if kind == "subcycle":  # bt, b1, b12, up (3 each), np, nu in; b1p2, E, aj out
        return {"bytes": 8 * nodes * (12 + 2 + 9), "flops": NODE_FLOPS * ncell}
    ions = ncell * (case["ppc"] + case.get("heavy", 0))
    if kind == "moments":  # x, v, beta_p and np in, up out
        return {"bytes": 56 * ions + 32 * nodes, "flops": 80 * ions}
    if kind == "particles":  # x, v, vp1, mrat, beta_p in; Ep, v+, v-, vp1 out; bt in, np, up, btc out
        return {"bytes": (88 + 96) * ions + 8 * nodes * 10, "flops": 400 * ions}
    n, r = case["n"], 4 if kind == "f32" else 8
    # each step: the ions' x, v, vp1 read and written, mrat and beta_p (the FP32 form: a species byte) read; and
    # per subcycle b1, b12, up, np, nu read and the new B written
    ion = 2 * 9 * r + (16 if r == 8 else 1)
    return {"bytes": n * (ion * ions + 10 * r * 14 * nodes), "flops": n * (ION_FLOPS * ions + 10 * NODE_FLOPS * ncell)}


# ---- the oracle: the ion step on the periodic box of unit spacing, in 64 bits ---------------------------------


def _m(a, ax):  # the value at node - e_ax
    return torch.roll(a, 1, ax)


def _p(a, ax):  # the value at node + e_ax
    return torch.roll(a, -1, ax)


class _Box:
    """Fields as interior tensors (ncx,ncy,ncz[,3]); node p holds the reference's node p+2."""

    def __init__(self, cfg, cells):
        self.cfg, self.cells = cfg, cells
        self.dt, self.nu, self.alpha = cfg.dt, cfg.nu, cfg.alpha

    # grid_interp.f, gutsf.f
    def to_center(self, v):
        return torch.stack([0.5 * (v[..., m] + _m(v[..., m], m)) for m in range(3)], -1)

    def to_face(self, v):
        return torch.stack([0.5 * (v[..., m] + _p(v[..., m], m)) for m in range(3)], -1)

    def edge_to_center(self, b):
        out = []
        for m in range(3):
            c = b[..., m]
            for ax in (q for q in range(3) if q != m):
                c = 0.5 * (c + _m(c, ax))
            out.append(c)
        return torch.stack(out, -1)

    def curl_b(self, b, dens):
        B1, B2, B3 = b.unbind(-1)
        c = ((B3 - _m(B3, 1)) + (_m(B2, 2) - B2), (B1 - _m(B1, 2)) + (_m(B3, 0) - B3),
             (B2 - _m(B2, 0)) + (_m(B1, 1) - B1))
        return torch.stack([c[m] / (0.5 * (dens + _p(dens, m)) * self.alpha) for m in range(3)], -1)

    def curl_e(self, e):
        E1, E2, E3 = e.unbind(-1)
        return torch.stack([(_p(E3, 1) - E3) + (E2 - _p(E2, 2)), (E3 - _p(E3, 0)) + (_p(E1, 2) - E1),
                            (E1 - _p(E1, 1)) + (_p(E2, 0) - E2)], -1)

    def e_field(self, aj, up, btc):
        ct = torch.linalg.cross(self.to_center(aj - up), btc)
        return self.to_face(ct) + self.nu * aj

    def predict(self, s, dtsub):
        s["aj"] = self.curl_b(s["bt"], s["np"])
        s["E"] = self.e_field(s["aj"], s["up"], self.edge_to_center(s["bt"]))
        s["b1p2"] = s["b12"] - 2 * dtsub * self.curl_e(s["E"])

    def correct(self, s, dtsub):
        bh = 0.5 * (s["b1p2"] + s["b1"])
        s["aj"] = self.curl_b(bh, s["np"])
        btc = self.to_center(self.to_face(self.edge_to_center(bh)))
        s["E"] = self.e_field(s["aj"], s["up"], btc)
        s["b1p2"] = s["b1"] - dtsub * self.curl_e(s["E"])

    # gutsp.f
    def locate(self, x):
        """Per corner the flat node and weight of every ion."""
        ncx, ncy, ncz = self.cells
        lo = [torch.ceil(x[0]) - 1, torch.floor(x[1]), torch.ceil(x[2]) - 1]
        f = [x[m] - lo[m] for m in range(3)]
        lo = [c.long() for c in lo]
        out = []
        for c in range(8):
            d = (c & 1, c >> 1 & 1, c >> 2)
            i, j, k = ((lo[m] + d[m] - 2) % self.cells[m] for m in range(3))
            w = 1.0
            for m in range(3):
                w = w * (f[m] if d[m] else 1 - f[m])
            out.append(((i * ncy + j) * ncz + k, w))
        return out

    def deposit(self, at, q):
        acc = torch.zeros(int(np.prod(self.cells)), device=q.device, dtype=torch.float64)
        for node, w in at:
            acc.index_add_(0, node, w * q)
        return acc.view(self.cells)

    def density(self, at, qw):
        return self.deposit(at, qw)

    def flow(self, at, qw, v, dens):
        return self.to_face(torch.stack([self.deposit(at, qw * v[m]) / dens for m in range(3)], -1))

    def gather(self, at, f):
        f = f.reshape(-1, 3)
        out = [torch.zeros_like(at[0][1]) for _ in range(3)]
        for node, w in at:
            g = f[node]
            for m in range(3):
                out[m] += w * g[:, m]
        return out

    def ep(self, s, at, btc, mrat):
        a = self.gather(at, self.to_center(s["aj"]) - self.to_center(s["up"]))
        b = self.gather(at, btc)
        return [(a[1] * b[2] - a[2] * b[1]) * mrat, (a[2] * b[0] - a[0] * b[2]) * mrat,
                (a[0] * b[1] - a[1] * b[0]) * mrat], b

    def rotate(self, v, ep, b, mrat):
        dt = self.dt
        vm = [v[m] + 0.5 * dt * ep[m] for m in range(3)]
        B = [b[m] * mrat for m in range(3)]
        b2 = B[0] ** 2 + B[1] ** 2 + B[2] ** 2
        ad = 1 / (1 + 0.25 * b2 * dt * dt)
        a1, a2, a3 = (1 - 0.25 * b2 * dt * dt) * ad, dt * ad, 0.5 * dt * dt * ad
        vdb = vm[0] * B[0] + vm[1] * B[1] + vm[2] * B[2]
        vxb = [vm[1] * B[2] - vm[2] * B[1], vm[2] * B[0] - vm[0] * B[2], vm[0] * B[1] - vm[1] * B[0]]
        return [a1 * vm[m] + a2 * vxb[m] + a3 * vdb * B[m] for m in range(3)], vm

    def move(self, x, v):
        for m in range(3):
            n = float(self.cells[m])
            y = x[m] + 0.5 * self.dt * v[m]
            y = torch.where(y > n + 1, y - n, torch.where(y <= 1, y + n, y))
            x[m] = y

    def moments(self, s, x, v, qw):
        at = self.locate(x)
        s["np"] = self.density(at, qw)
        s["up"] = self.flow(at, qw, v, s["np"])
        return at

    def push(self, s, x, v, v1, qw, mrat):
        """maind.f:385-402: the moments, Ep, v+, v- and improve_up; (at, Ep, v+, v-, btc)."""
        at = self.moments(s, x, v, qw)
        s["aj"] = self.curl_b(s["bt"], s["np"])
        btc = self.edge_to_center(s["bt"])
        s["up"] = self.flow(at, qw, [1.5 * v[m] - 0.5 * v1[m] for m in range(3)], s["np"])
        ep, b = self.ep(s, at, btc, mrat)
        vpl, vmi = self.rotate(v, ep, b, mrat)
        s["up"] = self.flow(at, qw, [0.5 * (vpl[m] + vmi[m]) for m in range(3)], s["np"])
        return at, ep, vpl, vmi, btc

    def step(self, s, x, v, v1, qw, mrat):
        at, _, _, _, btc = self.push(s, x, v, v1, qw, mrat)
        ep, b = self.ep(s, at, btc, mrat)
        vpl, _ = self.rotate(v, ep, b, mrat)
        for m in range(3):
            v1[m] = v[m]
            v[m] = vpl[m] + 0.5 * self.dt * ep[m]
        del at, ep, b, vpl
        self.move(x, v)
        self.moments(s, x, v, qw)
        dtsub = self.dt / self.cfg.ntsub
        for _ in range(self.cfg.ntsub):
            self.predict(s, dtsub)
            self.correct(s, dtsub)
            s["bt"], s["b12"], s["b1"] = s["b1p2"], s["b1"], s["b1p2"]
        self.move(x, v)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda().double()


def _host(a):
    return a.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if case.get("x_open"):
        return None  # inflow draws its ions from this repository's generator
    if kind == "grads":
        return _exact_grads(case, seed)
    ions = int(np.prod(_cells(case))) * (case.get("ppc", 0) + case.get("heavy", 0))
    if ions * case.get("n", 1) > 4e8:
        return None
    box = _Box(_config(case, seed), _cells(case))
    if kind == "moments":
        s = prepare(case, seed)
        x, v = s["x"].view(3, -1).unbind(0), s["v"].view(3, -1).unbind(0)
        dens = s["np"].permute(2, 1, 0)[1:-1, 1:-1, 1:-1].contiguous()
        qw = torch.full_like(x[0], 1 / box.cfg.beta)
        up = _ghosts(box.flow(box.locate(x), qw, v, dens))
        return up.permute(3, 2, 1, 0).contiguous()
    # the inputs as prepare() makes them, without running anything
    cfg = box.cfg
    h = _Arrays(case, cfg, np.float32 if kind == "f32" else np.float64)
    _load(h, case, seed)
    s = {k: _dev(getattr(h, k)[1:-1, 1:-1, 1:-1]) for k in ("b1", "b12", "b1p2", "bt", "np", "up")}
    full = lambda *names: {k: _host(_ghosts(s[k])) for k in names}  # noqa: E731
    dtsub = cfg.dt / cfg.ntsub
    if kind == "subcycle":
        box.predict(s, dtsub)
        box.correct(s, dtsub)
        out = full("b1p2", "E")
        aj = np.zeros_like(out["E"])  # curlB leaves the ghost nodes of aj as they are
        aj[1:-1, 1:-1, 1:-1] = _host(s["aj"])
        return dict(out, aj=aj)
    x, v, v1 = ([_dev(a[:, m]) for m in range(3)] for a in (h.xp, h.vp, h.vp1))
    mrat = _dev(h.mrat)
    qw = 1 / (cfg.beta * _dev(h.beta_p))
    if kind == "particles":
        _, ep, vpl, vmi, s["btc"] = box.push(s, x, v, v1, qw, mrat)
        st = lambda c: _host(torch.stack(c, -1))  # noqa: E731
        return dict(full("np", "up", "btc"), Ep=st(ep), vplus=st(vpl), vminus=st(vmi),
                    vp1=st([0.5 * (vpl[m] + vmi[m]) for m in range(3)]))
    for _ in range(case["n"]):
        box.step(s, x, v, v1, qw, mrat)
    if kind == "f32":
        return full("b1", "b12", "np", "up", "aj", "E")
    out = full("b1", "b12", "b1p2", "bt", "np", "up", "E")
    out.update({k: _host(torch.stack(a, -1)) for k, a in (("xp", x), ("vp", v), ("vp1", v1))})
    return dict(out, aj=None, ni_tot=None)  # the ghosts of aj are those of an earlier call


class _Arrays:
    """The arrays of maind.f that _load() fills, on the host alone."""

    def __init__(self, case, cfg, dtype):
        n = _room(case, cfg)
        self.cfg = cfg
        self.xp, self.vp, self.vp1 = (np.zeros((n, 3), dtype, order="F") for _ in range(3))
        self.mrat, self.beta_p = np.ones(n, dtype), np.ones(n, dtype)
        self.ni_tot = np.zeros(1, np.int32)
        for k in ("b1", "b12", "b1p2", "bt", "up"):
            setattr(self, k, np.zeros(cfg.nodes + (3,), dtype, order="F"))
        self.np = np.zeros(cfg.nodes, dtype, order="F")

    def mark_host_dirty(self):
        pass

    sync_to_device = mark_host_dirty


def _exact_grads(case, seed):
    """The surrogate's loss and gradients by autograd in 64 bits, without its 16-bit activations."""
    s = prepare(case, seed)
    nx, ny, nz = s["dims"]
    mean, std, omean, ostd = (torch.as_tensor(a, device="cuda", dtype=torch.float64) for a in _norm())
    tgt = s["tgt"].double()
    h = torch.nn.functional.pad((s["vin"].double() - mean) / std, (0, 2))
    params = []
    taps = [(dz, dy, dx) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]
    for l in range(len(s["net"].layers)):
        w, b = (torch.tensor(a, device="cuda", dtype=torch.float64, requires_grad=True) for a in s["net"].weights(l))
        params.append((w, b))
        f = h.view(nz, ny, nx, -1)
        z = b.expand(nx * ny * nz, -1)
        for t, (dz, dy, dx) in enumerate(taps):
            z = z + torch.roll(f, (-dz, -dy, -dx), (0, 1, 2)).reshape(nx * ny * nz, -1) @ w[t].T
        h = torch.nn.functional.gelu(z, approximate="tanh") if l < len(s["net"].layers) - 1 else z
    out = h[:, :3]
    loss = 0.5 * ((out - (tgt - omean) / ostd) ** 2).mean()
    e = (out * ostd + omean - tgt).view(nz, ny, nx, 3)
    D = lambda q, d: torch.roll(e[..., q], -1, d) - e[..., q]  # noqa: E731
    k2 = (D(2, 1) - D(1, 0)) ** 2 + (D(0, 0) - D(2, 2)) ** 2 + (D(1, 2) - D(0, 1)) ** 2
    (loss + 0.5 * k2.mean() / 2.5).backward()
    return dict(loss=None, grads=[(w.grad.cpu().numpy(), b.grad.cpu().numpy()) for w, b in params])

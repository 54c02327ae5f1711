"""Performance cases: the work users of this framework have it do.

Four kinds of work through the public entry points, over the sizes of the
repository's tests, smoke run and benchmark:

  rhs    the per-block drop-in operator, CCZ4Evolution::computeRHS, on device
         buffers (granite_ccz4_compute_rhs_device) or on host blocks
         (CCZ4Evolution.computeRHSVacuum);
  step   one resident block advanced by SSP-RK3 steps: initial data in, `steps`
         steps, final state out (Evolver.upload, rk3_step, download), as a
         program does between two outputs;
  hier   the same over a Berger-Oliger hierarchy of uneven blocks
         (Evolver.hierarchy_step), in both AMR modes;
  norms  the constraint monitor of a resident state (Evolver.constraint_norms).

The state restarts from its initial data in every pass, so a pass always
advances the same finite state. Inputs are Brill-Lindquist punctures with
seeded masses, positions and noise, the gauge wave, and, for the operator
alone, puncture data with smooth perturbations of every field.

`exact` restates the evolution system, the RK3 step, the ghost fills and the
inter-level transfers in plain torch FP64 over flat per-level storage.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import granite_b200 as gb

NV, NG = 22, 4
CHI, GXX, AXX, KTR, GHX, THETA, ALPHA, BETAX = 0, 1, 7, 13, 14, 17, 18, 19
F_INF_ONE = (0, 1, 4, 6, 18)  # chi, the diagonal of the metric and the lapse tend to 1
CFL = 0.25
NOISE = 1e-10


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def _rhs(n, precision="fp64", matter=False, host=False):
    return dict(kind="rhs", nx=n[0], ny=n[1], nz=n[2], precision=precision, matter=matter, host=host)


def _step(n, steps, precision="fp64", data="puncture", chi_fp64=0.0, matter=False):
    return dict(kind="step", nx=n[0], ny=n[1], nz=n[2], steps=steps, precision=precision, data=data,
                chi_fp64=chi_fp64, matter=matter)


def _hier(levels, coarse_n, extent, sizes, blocks, steps, precision="mixed", chi_fp64=0.5, amr="ghosts", layout=2024):
    return dict(kind="hier", levels=levels, coarse_n=coarse_n, extent=extent, sizes=sizes, min_blocks=blocks[0],
                max_blocks=blocks[1], steps=steps, precision=precision, chi_fp64=chi_fp64, amr=amr, layout=layout)


def listed():
    return [
        # the reference's call pattern: its evolve function calls computeRHS for
        # every block of a level, here on a small block whose data is on the device
        dict(name="rhs_32_fp64", **_rhs((32, 32, 32))),
        # a ragged block with an odd row length and matter sources, mixed precision
        dict(name="rhs_45x37x29_mixed_matter", **_rhs((45, 37, 29), "mixed", matter=True)),
        # an ordinary large block
        dict(name="rhs_128x96x80_fp64", **_rhs((128, 96, 80))),
        # the operator on host GridBlocks, the call that needs no change in a CPU code
        dict(name="rhs_host_48_fp64", **_rhs((48, 48, 48), host=True)),
        # the smoke run's block: launches and latency count
        dict(name="step_24x20x16_fp64", **_step((24, 20, 16), 32)),
        # gauge wave, periodic (the convergence workload)
        dict(name="step_gauge_wave_48_fp64", **_step((48, 48, 48), 32, data="gauge")),
        # the single-puncture workload, mixed precision with FP64 tiles near the puncture
        dict(name="step_puncture_128_mixed", **_step((128, 128, 128), 16, "mixed", chi_fp64=0.5)),
        # the binary hierarchy on 3 small levels: small uneven blocks, in both precisions
        dict(name="hier_3level_mixed", **_hier(3, 64, 32.0, "16 24 32", (20, 100), 8)),
        dict(name="hier_3level_fp64", **_hier(3, 64, 32.0, "16 24 32", (20, 100), 8, "fp64", 0.0)),
        # the reference's own AMR semantics (whole-block prolongation around every step)
        dict(name="hier_reference_amr_mixed", **_hier(3, 64, 32.0, "16 24 32", (20, 100), 4, amr="reference", layout=7)),
        # the benchmark's binary hierarchy: 376 blocks on 4 levels
        dict(name="hier_4level_mixed", **_hier(4, 128, 64.0, "16 24 32 48 64", (80, 400), 4)),
        # the constraint monitor, printed by a run after every coarse step
        dict(name="norms_128", kind="norms", nx=128, ny=128, nz=128),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rhs", "rhs", "rhs", "step", "step", "hier", "hier", "hier", "norms"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "rhs":
        host = rng.random() < 0.2
        n = [_size(rng, 12, 64 if host else 128) for _ in range(3)]
        return _rhs(n, prec, matter=not host and rng.random() < 0.4, host=host)
    if kind == "step":
        n = [_size(rng, 12, 112) for _ in range(3)]
        if rng.random() < 0.6:
            n[0] += n[0] % 2  # most block extents are even
        steps = rng.choice([4, 8, 16])
        if rng.random() < 0.25:
            return _step([n[0]] * 3, steps, prec, data="gauge")
        return _step(n, steps, prec, chi_fp64=rng.choice([0.0, 0.5, 0.7]) if prec == "mixed" else 0.0,
                     matter=rng.random() < 0.25)
    if kind == "hier":
        levels = rng.choice([2, 3])
        coarse_n = rng.choice([48, 56, 64, 80, 96])
        sizes = rng.choice(["16 24 32", "16 24 32 48", "16 24 32 40 48 64", "24 32 40"])
        return _hier(levels, coarse_n, float(coarse_n // 2), sizes, (1, 400), rng.choice([2, 4]), prec,
                     rng.choice([0.0, 0.5, 0.7]) if prec == "mixed" else 0.0,
                     "reference" if rng.random() < 0.2 else "ghosts", rng.randrange(1 << 16))
    n = [_size(rng, 24, 128) for _ in range(3)]
    return dict(kind="norms", nx=n[0], ny=n[1], nz=n[2])


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(seed)
    return g


def _block(case):
    """The single block of a case: dx = 0.25 around the origin, or the gauge wave's unit box."""
    n = (case["nx"], case["ny"], case["nz"])
    half = [0.5] * 3 if case.get("data") == "gauge" else [0.125 * c for c in n]
    return gb.GridBlock(0, 0, n, [-h for h in half], half)


def _layout(case):
    return gb.hierarchy.make_hierarchy(case["layout"], case["levels"], case["coarse_n"], case["extent"],
                                       [int(s) for s in case["sizes"].split()],
                                       (case["min_blocks"], case["max_blocks"]))


def _blocks(case):
    if case["kind"] != "hier":
        return [_block(case)]
    return [gb.GridBlock(i, b.level, b.ncells, b.lo, b.hi) for i, b in enumerate(_layout(case).blocks)]


def _punctures(case, seed):
    """Masses and positions: one puncture near the origin, or the binary at x = +-3
    (on cell corners of every level: off them these evolutions blow up at once)."""
    u = np.random.Generator(np.random.PCG64(seed)).uniform(-0.1, 0.1, size=2)
    if case["kind"] == "hier":
        return [(0.5 * (1 + u[0]), (3.0, 0.0, 0.0)), (0.5 * (1 + u[1]), (-3.0, 0.0, 0.0))]
    return [(1.0 + u[0], (0.05, -0.1, 0.02))]


def _coords(b, dev):
    out = []
    for d in range(3):
        i = torch.arange(b.totalCells(d), dtype=torch.float64, device=dev)
        x = b.lo[d] + (i - NG + 0.5) * b.dx(d)
        out.append(x.view([-1 if e == 2 - d else 1 for e in range(3)]))
    return out


def _puncture_data(b, punctures, out):
    """Brill-Lindquist data with r floored at dx / 2: chi = psi^-4, alpha = psi^-2,
    Gamma-hat^i = 8/3 d_i psi / psi, the rest flat."""
    X = _coords(b, out.device)
    psi = torch.ones(out.shape[1:], dtype=torch.float64, device=out.device)
    dpsi = [torch.zeros_like(psi) for _ in range(3)]
    floor = 0.5 * b.dx(0)
    for m, p in punctures:
        d = [X[a] - p[a] for a in range(3)]
        r = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2]).sqrt().clamp(min=floor)
        psi += m / (2 * r)
        for a in range(3):
            dpsi[a] += -m / (2 * r ** 3) * d[a]
    out.zero_()
    for v in (GXX, GXX + 3, GXX + 5):
        out[v] = 1.0
    out[CHI] = psi ** -4
    out[ALPHA] = psi ** -2
    for a in range(3):
        out[GHX + a] = 8.0 / 3.0 * dpsi[a] / psi


def _gauge_data(b, amplitude, phase, out):
    """The gauge wave gamma_xx = 1 - A sin(2 pi x + phase), everything else flat."""
    X = _coords(b, out.device)[0]
    H = -amplitude * torch.sin(2 * math.pi * X + phase)
    chi = (1 + H) ** (-1.0 / 3.0)
    out.zero_()
    out[CHI] = chi
    out[GXX] = (1 + H) * chi
    out[GXX + 3] = chi
    out[GXX + 5] = chi
    out[ALPHA] = (1 + H).sqrt()


def _smooth(b, r, amplitude, dev):
    """A seeded smooth function of the coordinates, two plane waves."""
    X = _coords(b, dev)
    f = 0.0
    for _ in range(2):
        k = r.uniform(-1.2, 1.2, size=3)
        f = f + torch.sin(float(k[0]) * X[0] + float(k[1]) * X[1] + float(k[2]) * X[2] + float(r.uniform(0, 6.28)))
    return (0.5 * amplitude) * f


def _state(case, seed, blocks):
    """The initial state of every block, one flat tensor in block order."""
    dev = _device()
    flat = torch.empty(sum(NV * b.totalSize() for b in blocks), dtype=torch.float64, device=dev)
    gen = _generator(seed)
    r = np.random.Generator(np.random.PCG64(seed + 1))
    punctures = _punctures(case, seed)
    wave = (0.1 * r.uniform(0.9, 1.1), r.uniform(0.0, 6.28))
    at = 0
    for b in blocks:
        u = flat[at:at + NV * b.totalSize()].view(NV, b.totalCells(2), b.totalCells(1), b.totalCells(0))
        at += u.numel()
        if case.get("data") == "gauge":
            _gauge_data(b, wave[0], wave[1], u)
        else:
            _puncture_data(b, punctures, u)
            if case["kind"] in ("rhs", "norms"):  # an evolved state has every field in play
                for v in range(NV):
                    u[v] += _smooth(b, r, 0.02 if v else 0.002, dev)
        u += (torch.rand(u.shape, generator=gen, dtype=torch.float64, device=dev) * 2 - 1) * NOISE
    return flat


def _matter(case, seed, b):
    """Sources of a smooth matter distribution: rho[N], Si[N,3], Sij[N,6], S[N]."""
    dev = _device()
    r = np.random.Generator(np.random.PCG64(seed + 2))
    shape = (b.totalCells(2), b.totalCells(1), b.totalCells(0))
    N = b.totalSize()
    f = [(_smooth(b, r, 1e-3, dev).expand(shape)).reshape(N) for _ in range(11)]
    rho = 2e-3 + f[0]
    Si = torch.stack(f[1:4], 1).contiguous()
    Sij = torch.stack(f[4:10], 1).contiguous()
    return rho, Si, Sij, (Sij[:, 0] + Sij[:, 3] + Sij[:, 5]).contiguous()


def _primitives(case, seed, b):
    """A magnetised fluid at rest up to small velocities (11 fields, PrimitiveVar order)."""
    dev = _device()
    r = np.random.Generator(np.random.PCG64(seed + 3))
    shape = (b.totalCells(2), b.totalCells(1), b.totalCells(0))
    base = (2e-3, 0, 0, 0, 1e-4, 0, 0, 0, 0.1, 0.0, 0.1)
    amp = (1e-3, 0.1, 0.1, 0.1, 5e-5, 1e-2, 1e-2, 1e-2, 0.02, 0.0, 0.0)
    return torch.stack([base[q] + _smooth(b, r, amp[q], dev).expand(shape) for q in range(11)]).contiguous()


def _precision(case):
    return gb.PRECISION_MIXED if case["precision"] == "mixed" else gb.PRECISION_FP64


def prepare(case, seed):
    blocks = _blocks(case)
    flat = _state(case, seed, blocks)
    if case["kind"] == "rhs":
        b = blocks[0]
        op = gb.CCZ4Evolution(gb.CCZ4Params(), _precision(case))
        u = flat.view(NV, b.totalCells(2), b.totalCells(1), b.totalCells(0))
        if case["host"]:
            rhs = gb.GridBlock(1, 0, b.ncells, b.lo, b.hi)
            b.array[...] = u.cpu().numpy()
            return dict(kind="rhs_host", op=op, grid=b, rhs=rhs)
        sources = _matter(case, seed, b) if case["matter"] else ()
        rhs = torch.zeros_like(u)
        ptr = [ctypes.c_void_p(t.data_ptr()) for t in (u, rhs, *sources)] + [None] * (0 if sources else 4)
        return dict(kind="rhs", op=op, desc=b.desc(), ptr=ptr, keep=(u, sources), rhs=rhs)
    ev = gb.Evolver(gb.CCZ4Params())
    if case.get("matter"):
        ev.enable_matter()
    for b in blocks:
        ev.add_block(b)
    if case.get("chi_fp64"):
        ev.set_fp64_chi_threshold(case["chi_fp64"])
    ev.commit()
    if case.get("matter"):
        ev.upload_primitives(0, _primitives(case, seed, blocks[0]).cpu().numpy())
        ev.sync()
    pin = torch.cuda.is_available()
    first = torch.empty(flat.shape, dtype=torch.float64, pin_memory=pin)
    first.copy_(flat)

    def arrays(t):
        a, at = t.numpy(), 0
        out = []
        for b in blocks:
            n = NV * b.totalSize()
            out.append(a[at:at + n].reshape(NV, b.totalCells(2), b.totalCells(1), b.totalCells(0)))
            at += n
        return out

    if case["kind"] == "norms":
        ev.upload(array=arrays(first))
        ev.sync()
        return dict(kind="norms", ev=ev, keep=first)
    last = torch.empty(flat.shape, dtype=torch.float64, pin_memory=pin)
    s = dict(kind=case["kind"], ev=ev, first=arrays(first), last=arrays(last), out=last, keep=first,
             steps=case["steps"], precision=_precision(case))
    if case["kind"] == "hier":
        s["dt"] = CFL * blocks[0].dx(0)
        s["amr"] = gb.AMR_GHOSTS if case["amr"] == "ghosts" else gb.AMR_REFERENCE
    else:
        s["dt"] = CFL * min(blocks[0].dx(d) for d in range(3))
        s["bc"] = gb.BC_PERIODIC if case["data"] == "gauge" else gb.BC_REFERENCE
    return s


def run(state):
    s = state
    if s["kind"] == "rhs":
        op = s["op"]
        # the arguments after the descriptor: u, rhs, rho, Si, Sij, S, precision, stream (the context's own)
        op.ctx.check(op.ctx.lib.granite_ccz4_compute_rhs_device(op.ctx.h, ctypes.byref(s["desc"]), *s["ptr"],
                                                                op.precision, None))
        return s["rhs"]
    if s["kind"] == "rhs_host":
        s["op"].computeRHSVacuum(s["grid"], s["rhs"])
        return s["rhs"].array
    ev = s["ev"]
    if s["kind"] == "norms":
        return ev.constraint_norms()
    ev.upload(array=s["first"])
    for _ in range(s["steps"]):
        if s["kind"] == "hier":
            ev.hierarchy_step(s["dt"], s["precision"], s["amr"])
        else:
            ev.rk3_step(0, s["dt"], s["precision"], s["bc"])
    ev.download(out=s["last"])
    return s["out"]


def work(case):
    """Bytes: the operator reads the state (and sources) and writes the RHS; a
    point-update's three stages read and write 8 x 22 values (the first stage's
    two inputs are one), and a pass moves the state in and out. Flops: 10,395
    per RHS with dissipation as the reference is written, 12 per field for the
    RK3 combines; the constraints need about half of an RHS."""
    blocks = _blocks(case)
    interior = sum(math.prod(b.ncells) for b in blocks)
    cells = sum(b.totalSize() for b in blocks)
    if case["kind"] == "rhs":
        return {"bytes": 176.0 * (cells + interior) + (88.0 * interior if case["matter"] else 0.0),
                "flops": 10395.0 * interior}
    if case["kind"] == "norms":
        return {"bytes": 18 * 8.0 * cells, "flops": 5200.0 * interior}
    updates = case["steps"] * sum(math.prod(b.ncells) * 2 ** b.level for b in blocks)
    return {"bytes": 1408.0 * updates + 2 * 176.0 * cells, "flops": 31449.0 * updates}


# ---------------------------------------------------------------------------
# the same in plain FP64 torch, without the framework's kernels
# ---------------------------------------------------------------------------

SYM = ((0, 1, 2), (1, 3, 4), (2, 4, 5))
PAIRS = ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))


class _Points:
    """Interior points of a set of blocks in flat [22, cells] storage: their cell
    indices and the y and z strides of their blocks."""

    def __init__(self, blocks, offsets, dev):
        c, sy, sz = [], [], []
        for b, at in zip(blocks, offsets):
            T0, T1 = b.totalCells(0), b.totalCells(1)
            i = torch.arange(NG, NG + b.ncells[0], device=dev).view(1, 1, -1)
            j = torch.arange(NG, NG + b.ncells[1], device=dev).view(1, -1, 1)
            k = torch.arange(NG, NG + b.ncells[2], device=dev).view(-1, 1, 1)
            q = (at + i + T0 * (j + T1 * k)).reshape(-1)
            c.append(q)
            sy.append(torch.full_like(q, T0))
            sz.append(torch.full_like(q, T0 * T1))
        self.c, self.s = torch.cat(c), [torch.ones((), dtype=torch.long, device=dev), torch.cat(sy), torch.cat(sz)]

    def chunk(self, lo, hi):
        p = object.__new__(_Points)
        p.c = self.c[lo:hi]
        p.s = [self.s[0], self.s[1][lo:hi], self.s[2][lo:hi]]
        return p


class _Stencils:
    """Derivatives of every field at the points, each neighbour gathered once."""

    def __init__(self, U, p, dx, beta=None, w=None, sigma=0.0):
        self.U, self.p, self.dx = U, p, dx
        self.f0 = f0 = self.at(0)
        self.d, self.dd, self.adv, self.ko = [], [], 0.0, 0.0
        for a in range(3):
            t = p.s[a]
            lo = [self.at(-q * t) - f0 for q in (1, 2, 3)]
            hi = [self.at(q * t) - f0 for q in (1, 2, 3)]
            self.d.append((8 * (hi[0] - lo[0]) - (hi[1] - lo[1])) / (12 * dx[a]))
            self.dd.append((16 * (hi[0] + lo[0]) - (hi[1] + lo[1])) / (12 * dx[a] ** 2))
            if beta is None:
                continue
            # advection, upwind blended with centred, and dissipation
            pos = beta[a] >= 0
            x = [torch.where(pos, m, n) for m, n in zip(lo, hi)] + [self.at(torch.where(pos, -4 * t, 4 * t)) - f0]
            up = (-48 * x[0] + 36 * x[1] - 16 * x[2] + 3 * x[3]) / (12 * dx[a])
            self.adv = self.adv + w * beta[a].abs() * up + (1 - w) * beta[a] * self.d[a]
            self.ko = self.ko + sigma / (64 * dx[a]) * ((hi[2] + lo[2]) - 6 * (hi[1] + lo[1]) + 15 * (hi[0] + lo[0]))

    def at(self, o, fields=slice(None)):
        return self.U[fields].index_select(1, self.p.c + o)

    def hessian(self, fields):
        """xx xy xz yy yz zz second derivatives of a range of fields."""
        h = []
        for a, b in PAIRS:
            if a == b:
                h.append(self.dd[a][fields])
                continue
            s, t = self.p.s[a], self.p.s[b]
            h.append(((self.at(s + t, fields) - self.at(s - t, fields)) -
                      (self.at(t - s, fields) - self.at(-s - t, fields))) / (4 * self.dx[a] * self.dx[b]))
        return h


def _geometry(S):
    """Metric, Christoffels and Ricci of the conformal metric, with what they are made of."""
    chi, gt = S.f0[CHI], [S.f0[GXX + q] for q in range(6)]
    g = lambda i, j: gt[SYM[i][j]]  # noqa: E731
    det = (gt[0] * (gt[3] * gt[5] - gt[4] ** 2) - gt[1] * (gt[1] * gt[5] - gt[4] * gt[2]) +
           gt[2] * (gt[1] * gt[4] - gt[3] * gt[2]))
    inv = 1.0 / (det + 1e-30)
    up = [(gt[3] * gt[5] - gt[4] ** 2) * inv, (gt[2] * gt[4] - gt[1] * gt[5]) * inv,
          (gt[1] * gt[4] - gt[2] * gt[3]) * inv, (gt[0] * gt[5] - gt[2] ** 2) * inv,
          (gt[1] * gt[2] - gt[0] * gt[4]) * inv, (gt[0] * gt[3] - gt[1] ** 2) * inv]
    gu = lambda i, j: up[SYM[i][j]]  # noqa: E731
    trace = lambda t: sum(gu(i, j) * t[SYM[i][j]] for i in range(3) for j in range(3))  # noqa: E731
    dg = [S.d[d][GXX:GXX + 6] for d in range(3)]  # dg[d][q]
    H = S.hessian(slice(GXX, GXX + 6))
    G1 = [[0.5 * (dg[i][SYM[k][j]] + dg[j][SYM[k][i]] - dg[k][SYM[i][j]]) for i, j in PAIRS] for k in range(3)]
    ch = [[sum(gu(i, l) * G1[l][q] for l in range(3)) for q in range(6)] for i in range(3)]
    Gc = [trace(ch[k]) for k in range(3)]
    Gh = [S.f0[GHX + a] for a in range(3)]
    dGh = [S.d[d][GHX:GHX + 3] for d in range(3)]
    Ric = []
    for i, j in PAIRS:
        q = SYM[i][j]
        t = -0.5 * trace([H[r][q] for r in range(6)])
        for k in range(3):
            t = t + 0.5 * (g(k, i) * dGh[j][k] + g(k, j) * dGh[i][k]) + (Gh[k] - Gc[k]) * G1[k][q]
            for l in range(3):
                for m in range(3):
                    t = t + gu(l, m) * (ch[k][SYM[l][i]] * G1[k][SYM[j][m]] + ch[k][SYM[l][j]] * G1[k][SYM[i][m]])
        Ric.append(t)
    return chi, gt, up, gu, trace, G1, ch, Ric, Gh


def _covariant(S, v, ch):
    """Gradient and conformal covariant Hessian of the scalar field v."""
    d = [S.d[a][v] for a in range(3)]
    h = [x[0] for x in S.hessian(slice(v, v + 1))]
    return d, [h[q] - sum(ch[k][q] * d[k] for k in range(3)) for q in range(6)]


def _chi_ricci(chi, gt, up, gu, trace, dchi, DDchi, Ric):
    lap = trace(DDchi)
    d2 = sum(gu(l, m) * dchi[l] * dchi[m] for l in range(3) for m in range(3))
    return [Ric[SYM[i][j]] + 0.5 / (chi + 1e-30) * (DDchi[SYM[i][j]] + gt[SYM[i][j]] * lap) -
            0.25 / (chi * chi + 1e-30) * (dchi[i] * dchi[j] - 3 * gt[SYM[i][j]] * d2) for i, j in PAIRS]


def _rhs_points(U, p, dx, prm, matter):
    """L(u) with dissipation at the points p: [22, points]."""
    chi_raw = U[CHI, p.c]
    chi = torch.where(torch.isfinite(chi_raw) & (chi_raw >= 1e-4), chi_raw, torch.full_like(chi_raw, 1e-4))
    beta = [U[BETAX + a, p.c] for a in range(3)]
    w = 0.5 * (1 + torch.tanh((chi - prm.chi_blend_center) / prm.chi_blend_width))
    S = _Stencils(U, p, dx, beta, w, prm.ko_sigma)
    adv = S.adv
    _, gt, up, gu, trace, G1, ch, Rt, Gh = _geometry(S)
    g = lambda i, j: gt[SYM[i][j]]  # noqa: E731
    At = [S.f0[AXX + q] for q in range(6)]
    K, Th, al = S.f0[KTR], S.f0[THETA], S.f0[ALPHA]
    dchi, DDchi = _covariant(S, CHI, ch)
    Ric = _chi_ricci(chi, gt, up, gu, trace, dchi, DDchi, Rt)
    Rs = chi * trace(Ric)
    dal, DDa = _covariant(S, ALPHA, ch)
    db = [S.d[d][BETAX:BETAX + 3] for d in range(3)]  # db[j][i] = d_j beta^i
    Hb = S.hessian(slice(BETAX, BETAX + 3))
    divb = db[0][0] + db[1][1] + db[2][2]
    Am = [[sum(gu(i, k) * At[SYM[k][j]] for k in range(3)) for j in range(3)] for i in range(3)]
    AtAt = sum(Am[i][j] * Am[j][i] for i in range(3) for j in range(3))
    rho, Si, Sij, Str = (0.0, [0.0] * 3, [0.0] * 6, 0.0) if matter is None else \
        (matter[0][p.c], [matter[1][p.c, a] for a in range(3)], [matter[2][p.c, q] for q in range(6)], matter[3][p.c])
    k1, k2 = prm.kappa1, prm.kappa2
    out = torch.empty((NV, p.c.numel()), dtype=torch.float64, device=U.device)
    out[CHI] = 2.0 / 3.0 * chi * (al * K - divb) + adv[CHI]
    for i, j in PAIRS:
        q = SYM[i][j]
        out[GXX + q] = (-2 * al * At[q] + adv[GXX + q] - 2.0 / 3.0 * gt[q] * divb +
                        sum(g(i, d) * db[j][d] + g(j, d) * db[i][d] for d in range(3)))
    cross = sum(gu(a, b) * dchi[a] * dal[b] for a in range(3) for b in range(3))
    out[KTR] = (-(chi * trace(DDa) - 0.5 * cross) + al * (AtAt + K * K / 3) + 4 * math.pi * al * (rho + Str) +
                k1 * (1 - k2) * al * Th + adv[KTR])
    dK = [S.d[d][KTR] for d in range(3)]
    ddiv = [sum(Hb[SYM[a][d]][a] for a in range(3)) for d in range(3)]  # d_d d_a beta^a
    for i in range(3):
        t = 2 * al * sum(ch[i][SYM[j][k]] * At[SYM[j][k]] for j in range(3) for k in range(3))
        t = t + 3 * al / (chi + 1e-30) * sum(Am[i][d] * dchi[d] for d in range(3))
        for d in range(3):
            t = t + gu(i, d) * (-4.0 / 3.0 * al * dK[d] - 16 * math.pi * al * Si[d] + ddiv[d] / 3) - Gh[d] * db[d][i]
        t = t + trace([Hb[q][i] for q in range(6)]) + adv[GHX + i] + 2.0 / 3.0 * Gh[i] * divb - 2 * k1 * al * Gh[i]
        out[GHX + i] = t
    out[THETA] = (0.5 * al * (Rs - AtAt + 2 * K * K / 3 - 16 * math.pi * rho) - al * k1 * (2 + k2) * Th + adv[THETA])
    raw = []
    for i, j in PAIRS:
        q = SYM[i][j]
        sq = sum(At[SYM[i][k]] * Am[k][j] for k in range(3))
        raw.append(chi * (-DDa[q] + al * (Ric[q] - 8 * math.pi * Sij[q])) + al * (K * At[q] - 2 * sq) + adv[AXX + q] +
                   sum(At[SYM[i][d]] * db[j][d] + At[SYM[j][d]] * db[i][d] for d in range(3)) -
                   2.0 / 3.0 * At[q] * divb)
    tr = trace(raw)
    for q in range(6):
        out[AXX + q] = raw[q] - gt[q] * tr / 3
    out[ALPHA] = -2 * al * K + adv[ALPHA]
    for d in range(3):
        out[BETAX + d] = 0.75 * Gh[d] - prm.eta * beta[d] + adv[BETAX + d]
    return out + S.ko


CHUNK = 1 << 19


def _rhs_all(U, p, dx, prm, matter):
    n = p.c.numel()
    return torch.cat([_rhs_points(U, p.chunk(a, min(n, a + CHUNK)), dx, prm, matter) for a in range(0, n, CHUNK)], 1)


def _constraint_sums(U, p, dx):
    """Sum of H^2 and of |M|^2 over the points."""
    S = _Stencils(U, p, dx)
    chi, gt, up, gu, trace, G1, ch, Rt, Gh = _geometry(S)
    At, K = [S.f0[AXX + q] for q in range(6)], S.f0[KTR]
    dchi, DDchi = _covariant(S, CHI, ch)
    Rs = chi * trace(_chi_ricci(chi, gt, up, gu, trace, dchi, DDchi, Rt))
    Am = [[sum(gu(i, k) * At[SYM[k][j]] for k in range(3)) for j in range(3)] for i in range(3)]
    H = Rs + 2.0 / 3.0 * K * K - sum(Am[i][j] * Am[j][i] for i in range(3) for j in range(3))
    dA = [S.d[d][AXX:AXX + 6] for d in range(3)]
    M2 = 0.0
    for i in range(3):
        M = -2.0 / 3.0 * S.d[i][KTR]
        for j in range(3):
            for k in range(3):
                D = dA[j][SYM[k][i]]
                for m in range(3):
                    D = D - ch[m][SYM[j][k]] * At[SYM[m][i]] - ch[m][SYM[j][i]] * At[SYM[k][m]]
                M = M + gu(j, k) * (D - 3.0 / (2 * chi + 1e-30) * At[SYM[i][j]] * dchi[k])
        M2 = M2 + M * M
    return float((H * H).sum()), float(M2.sum())


class _Level:
    """The blocks of one level in flat storage, with the index maps of its fills."""

    def __init__(self, blocks, dev):
        self.blocks, self.dev = blocks, dev
        self.off = np.concatenate([[0], np.cumsum([b.totalSize() for b in blocks])])
        self.p = _Points(blocks, self.off, dev)
        self.dx = [blocks[0].dx(d) for d in range(3)]
        self.U = None
        self.fills = {}
        self.copy = self.pro = None  # (destination, source) and the prolongation's table

    def cells(self, b, at):
        """Per axis: index, clamped index and whether it is a ghost, over all cells of a block."""
        T = [b.totalCells(d) for d in range(3)]
        i = [torch.arange(T[d], device=self.dev).view([-1 if e == 2 - d else 1 for e in range(3)]) for d in range(3)]
        c = [x.clamp(NG, NG + b.ncells[d] - 1) for d, x in enumerate(i)]
        return T, i, c, [x != y for x, y in zip(i, c)]

    def index(self, b, at, T, i):
        return (at + i[0] + T[0] * (i[1] + T[1] * i[2])).expand(T[2], T[1], T[0]).reshape(-1)

    def local_table(self, mode, masks):
        """Ghost cells, the cells they are filled from and the radii of the falloff's three passes."""
        out = []
        for q, (b, at) in enumerate(zip(self.blocks, self.off)):
            T, i, c, gh = self.cells(b, at)
            dst = self.index(b, at, T, i)
            if mode == "periodic":
                src = [NG + (x - NG) % b.ncells[d] for d, x in enumerate(i)]
            elif masks is not None:
                src = [torch.where((x < NG) & masks[q][d][0] | (x >= NG + b.ncells[d]) & masks[q][d][1], c[d], x)
                       for d, x in enumerate(i)]
            else:
                src = c
            s = self.index(b, at, T, src)
            ghost = s != dst
            row = [dst[ghost], s[ghost]]
            if mode == "falloff":
                x = [b.lo[d] + (i[d].double() - NG + 0.5) * b.dx(d) for d in range(3)]
                y = [b.lo[d] + (c[d].double() - NG + 0.5) * b.dx(d) for d in range(3)]
                flat = lambda t: t.expand(T[2], T[1], T[0]).reshape(-1)[ghost]  # noqa: E731
                rad = lambda a, e, f: flat((a * a + e * e + f * f).sqrt() + 1e-30)  # noqa: E731
                # the x pass runs on interior rows, the y pass on the x-filled planes, then z
                for d, (ri, rg) in enumerate((((y[0], y[1], y[2]), (x[0], y[1], y[2])),
                                              ((x[0], y[1], y[2]), (x[0], x[1], y[2])),
                                              ((x[0], x[1], y[2]), (x[0], x[1], x[2])))):
                    row.append(torch.where(flat(gh[d]), rad(*ri) / rad(*rg), torch.ones((), dtype=torch.float64,
                                                                                        device=self.dev)))
            out.append(row)
        return [torch.cat(t) for t in zip(*out)]

    def local_fill(self, U, mode, masks=None):
        """Zero-gradient (on the faces of a mask), periodic or 1/r falloff in every ghost cell, block by block."""
        key = mode if masks is None else "masked"
        if key not in self.fills:
            self.fills[key] = self.local_table(mode, masks)
        dst, src, *ratios = self.fills[key]
        val = U[:, src]
        finf = torch.zeros((NV, 1), dtype=torch.float64, device=self.dev)
        finf[list(F_INF_ONE)] = 1.0
        for r in ratios:
            val = torch.where(r == 1, val, finf + (val - finf) * r)
        U[:, dst] = val

    def prolong_table(self, fine, at, cells, coarse, cat):
        """Trilinear sources of fine cells (i, j, k index tensors) in one coarse block."""
        idx, wt = [], []
        for d in range(3):
            f = ((fine.lo[d] + (cells[d].double() - NG + 0.5) * fine.dx(d)) - (coarse.lo[d] + 0.5 * coarse.dx(d))) / coarse.dx(d) + NG
            a = (f.abs() + 0.5).floor() * f.sign()
            a = a.clamp(0, coarse.totalCells(d) - 1)
            fr = f - a
            e = (a + torch.where(fr >= 0, 1.0, -1.0)).clamp(0, coarse.totalCells(d) - 1)
            idx.append((a.long(), e.long()))
            wt.append((1 - fr.abs(), fr.abs()))
        T0, T1 = coarse.totalCells(0), coarse.totalCells(1)
        src, w = [], []
        for q in range(8):
            o = [(q >> d) & 1 for d in range(3)]
            src.append(cat + idx[0][o[0]] + T0 * (idx[1][o[1]] + T1 * idx[2][o[2]]))
            w.append(wt[0][o[0]] * wt[1][o[1]] * wt[2][o[2]])
        return torch.stack(src), torch.stack(w)


def _origin(b, lo, dx):
    return [int(round((b.lo[d] - lo[d]) / dx[d])) for d in range(3)]


def _connect(lev, parent, lo, amr):
    """Ghost sources of a level (same-level neighbour, else coarse block), in GHOSTS
    mode; whole-block prolongation and the uncovered faces in REFERENCE mode; and
    the restriction map into the parent, a list of (coarse cell, 8 fine cells)."""
    dev = lev.dev
    G = [_origin(b, lo, lev.dx) for b in lev.blocks]
    PG = [_origin(b, lo, parent.dx) for b in parent.blocks] if parent else []
    dst_c, src_c, dst_p, tab = [], [], [], []
    masks = []
    for b, at, g in zip(lev.blocks, lev.off, G):
        T, i, c, gh = lev.cells(b, at)
        full = lambda t: t.expand(T[2], T[1], T[0]).reshape(-1)  # noqa: E731
        ijk = [full(x) for x in i]
        own = lev.index(b, at, T, i)
        if amr == "reference":
            if parent:
                last = len(parent.blocks) - 1
                s, w = lev.prolong_table(b, at, ijk, parent.blocks[last], int(parent.off[last]))
                dst_p.append(own)
                tab.append((s, w))
                m = []
                for d in range(3):
                    x0, x1 = b.lo[d] + 0.5 * b.dx(d), b.hi[d] - 0.5 * b.dx(d)
                    m.append((not any(q.lo[d] + 0.5 * q.dx(d) <= x0 + 0.5 * b.dx(d) for q in parent.blocks),
                              not any(q.hi[d] - 0.5 * q.dx(d) >= x1 - 0.5 * b.dx(d) for q in parent.blocks)))
                masks.append(m)
            continue
        ghost = full(gh[0] | gh[1] | gh[2])
        ijk, own = [x[ghost] for x in ijk], own[ghost]
        pos = [x - NG + g[d] for d, x in enumerate(ijk)]
        src = torch.full_like(own, -1)
        for q, qat, qg in zip(lev.blocks, lev.off, G):
            if q is b or any(qg[d] >= g[d] + b.ncells[d] + NG or qg[d] + q.ncells[d] <= g[d] - NG for d in range(3)):
                continue
            inside = True
            for d in range(3):
                inside = inside & (pos[d] >= qg[d]) & (pos[d] < qg[d] + q.ncells[d])
            at_q = int(qat) + (pos[0] - qg[0] + NG) + q.totalCells(0) * (
                (pos[1] - qg[1] + NG) + q.totalCells(1) * (pos[2] - qg[2] + NG))
            src = torch.where(inside, at_q, src)
        same = src >= 0
        dst_c.append(own[same])
        src_c.append(src[same])
        which = torch.full_like(own, -1)
        for n, (q, qg) in enumerate(zip(parent.blocks if parent else [], PG)):
            inside = ~same
            for d in range(3):
                inside = inside & (pos[d] >= 2 * qg[d]) & (pos[d] < 2 * (qg[d] + q.ncells[d]))
            which = torch.where(inside, n, which)
        for n in torch.unique(which[which >= 0]).tolist():
            m = which == n
            dst_p.append(own[m])
            tab.append(lev.prolong_table(b, at, [x[m] for x in ijk], parent.blocks[n], int(parent.off[n])))
    lev.copy = (torch.cat(dst_c), torch.cat(src_c)) if dst_c else None
    lev.pro = (torch.cat(dst_p), torch.cat([t[0] for t in tab], 1), torch.cat([t[1] for t in tab], 1)) if dst_p else None
    lev.masks = masks
    lev.restrict = []
    if not parent:
        return
    for b, at, g in zip(lev.blocks, lev.off, G):
        for q, qat, qg in zip(parent.blocks, parent.off, PG):
            if amr == "reference":
                # a coarse centre lies midway between two fine cells, the lower one at or past the first
                # interior cell; the box reaches into the upper ghost layer
                rng = [range(max(qg[d], -(-g[d] // 2)), min(qg[d] + q.ncells[d], (g[d] + b.ncells[d] + NG) // 2))
                       for d in range(3)]
            else:
                rng = [range(max(qg[d], (g[d] + 1) // 2), min(qg[d] + q.ncells[d], (g[d] + b.ncells[d]) // 2))
                       for d in range(3)]
            if any(len(r) == 0 for r in rng):
                continue
            I = [torch.arange(r.start, r.stop, device=dev).view([-1 if e == 2 - d else 1 for e in range(3)])
                 for d, r in enumerate(rng)]
            dst = int(qat) + (I[0] - qg[0] + NG) + q.totalCells(0) * (
                (I[1] - qg[1] + NG) + q.totalCells(1) * (I[2] - qg[2] + NG))
            f = [2 * x - g[d] + NG for d, x in enumerate(I)]
            src = torch.stack([(int(at) + (f[0] + o % 2) + b.totalCells(0) * (
                (f[1] + o // 2 % 2) + b.totalCells(1) * (f[2] + o // 4))).reshape(-1) for o in range(8)])
            lev.restrict.append((dst.reshape(-1), src))


def _fill(levels, L, U, level_fill, case):
    lev = levels[L]
    local = "zero" if level_fill else "falloff"
    if case["amr"] == "reference":
        if level_fill and L > 0:
            _prolong(levels, L, U)
            lev.local_fill(U, "zero", lev.masks)
        else:
            lev.local_fill(U, local)
        return
    lev.local_fill(U, local)
    if lev.copy:
        U[:, lev.copy[0]] = U[:, lev.copy[1]]
    _prolong(levels, L, U)


def _prolong(levels, L, U):
    if levels[L].pro is None:
        return
    dst, src, w = levels[L].pro
    for a in range(0, dst.numel(), CHUNK):
        val = 0.0
        for q in range(8):
            val = val + w[q, a:a + CHUNK] * levels[L - 1].U[:, src[q, a:a + CHUNK]]
        U[:, dst[a:a + CHUNK]] = val


def _rk3(lev, fill, dt, prm, matter=None):
    """SSP-RK3 with the floors after every stage and the algebraic constraints after the last."""
    c = lev.p.c
    un = lev.U[:, c]
    u = lev.U
    for s, (a1, a2, a3) in enumerate(((1.0, 0.0, 1.0), (0.75, 0.25, 0.25), (1 / 3, 2 / 3, 2 / 3))):
        r = a1 * un + a2 * u[:, c] + a3 * dt * _rhs_all(u, lev.p, lev.dx, prm, matter)
        r[CHI] = torch.where(torch.isfinite(r[CHI]), r[CHI], torch.full_like(r[CHI], 1e-4)).clamp(1e-4, 1.5)
        r[ALPHA] = torch.where(torch.isfinite(r[ALPHA]), r[ALPHA], torch.full_like(r[ALPHA], 1e-6)).clamp(min=1e-6)
        if s == 2:
            g = r[GXX:GXX + 6]
            det = (g[0] * (g[3] * g[5] - g[4] ** 2) - g[1] * (g[1] * g[5] - g[4] * g[2]) +
                   g[2] * (g[1] * g[4] - g[3] * g[2]))
            g = g * det ** (-1.0 / 3.0)
            A = r[AXX:AXX + 6].clone()
            tr = ((g[3] * g[5] - g[4] ** 2) * A[0] + (g[0] * g[5] - g[2] ** 2) * A[3] + (g[0] * g[3] - g[1] ** 2) * A[5] +
                  2 * ((g[2] * g[4] - g[1] * g[5]) * A[1] + (g[1] * g[4] - g[2] * g[3]) * A[2] +
                       (g[1] * g[2] - g[0] * g[4]) * A[4]))
            r[GXX:GXX + 6] = g
            r[AXX:AXX + 6] = A - tr / 3 * g
            lev.U[:, c] = r
            fill(lev.U, True)
            return
        u = lev.U.clone() if s == 0 else u.clone()
        u[:, c] = r
        fill(u, False)


def _subcycle(levels, L, dt, prm, case):
    lev = levels[L]
    fill = lambda U, level_fill: _fill(levels, L, U, level_fill, case)  # noqa: E731
    fill(lev.U, True)
    _rk3(lev, fill, dt, prm)
    if L + 1 < len(levels):
        for _ in range(2):
            _subcycle(levels, L + 1, dt / 2, prm, case)
        for dst, src in levels[L + 1].restrict:
            val = 0.0
            for q in range(8):
                val = val + levels[L + 1].U[:, src[q]]
            lev.U[:, dst] = val / 8


def _sources(prim):
    """Matter sources of magnetised-fluid primitives, flat over the cells."""
    q = prim.reshape(11, -1)
    rho, v, pr, B, eps = q[0], q[1:4], q[4], q[5:8], q[8]
    h = 1 + eps + pr / (rho + 1e-30)
    W2 = 1 / (1 - (v * v).sum(0)).clamp(min=1e-10)
    Bv = (B * v).sum(0)
    b2 = (B * B).sum(0) / W2 + Bv * Bv
    e = rho * h * W2 + b2
    ph = pr + 0.5 * b2
    b = B / W2 + Bv * v
    Si = torch.stack([e * v[a] - Bv * b[a] for a in range(3)], 1)
    Sij = torch.stack([e * v[i] * v[j] + (ph if i == j else 0) - b[i] * b[j] - B[i] * B[j] / W2 for i, j in PAIRS], 1)
    return rho * h * W2 - pr + 0.5 * b2, Si, Sij, Sij[:, 0] + Sij[:, 3] + Sij[:, 5]


def exact(case, seed):
    prm = gb.CCZ4Params()
    blocks = _blocks(case)
    flat = _state(case, seed, blocks)
    nlev = 1 + max(b.level for b in blocks)
    levels, at = [], 0
    for L in range(nlev):
        lev = _Level([b for b in blocks if b.level == L], flat.device)
        n = NV * int(lev.off[-1])
        part = flat[at:at + n]
        lev.U = torch.cat([part[NV * a:NV * e].view(NV, -1) for a, e in zip(lev.off[:-1].tolist(), lev.off[1:].tolist())], 1)
        at += n
        levels.append(lev)
    lev, b = levels[0], blocks[0]
    if case["kind"] == "rhs":
        matter = _matter(case, seed, b) if case["matter"] else None
        out = torch.zeros_like(lev.U)
        out[:, lev.p.c] = _rhs_all(lev.U, lev.p, lev.dx, prm, matter)
        return out.view(NV, b.totalCells(2), b.totalCells(1), b.totalCells(0))
    if case["kind"] == "norms":
        n = lev.p.c.numel()
        s = [_constraint_sums(lev.U, lev.p.chunk(a, min(n, a + CHUNK)), lev.dx) for a in range(0, n, CHUNK)]
        return tuple(math.sqrt(sum(x[q] for x in s) / n) for q in range(2))
    if case["kind"] == "step":
        matter = _sources(_primitives(case, seed, b)) if case["matter"] else None
        if case["data"] == "gauge":
            fill = lambda U, level_fill: lev.local_fill(U, "periodic")  # noqa: E731
        else:
            fill = lambda U, level_fill: lev.local_fill(U, "zero" if level_fill else "falloff")  # noqa: E731
        fill(lev.U, True)
        for _ in range(case["steps"]):
            _rk3(lev, fill, CFL * min(lev.dx), prm, matter)
    else:
        lo = [min(q.lo[d] for q in levels[0].blocks) for d in range(3)]
        for L, x in enumerate(levels):
            _connect(x, levels[L - 1] if L else None, lo, case["amr"])
        for _ in range(case["steps"]):
            _subcycle(levels, 0, CFL * levels[0].dx[0], prm, case)
    return torch.cat([lev.U[:, a:e].reshape(-1) for lev in levels
                      for a, e in zip(lev.off[:-1].tolist(), lev.off[1:].tolist())])

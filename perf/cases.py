"""What a user of this library has it do, as cases that can be timed.

Each case is one piece of work that a program gives the library through its
public entry points (the ``gop`` module): a grid advanced to the program's
next output and copied back, a whole request from admission to result, a batch
of uneven grids, the CFL step of a state that the caller holds.  ``listed``
names the measured ones, ``draw`` gives more of the same ranges, ``exact``
computes what a case returns with plain torch in 64 bits: the scheme of
GAMERA-OP (PDM reconstruction, Rusanov flux, constrained transport, AB2)
written over whole arrays, from the same initial states.
"""
from __future__ import annotations

import ctypes
import importlib
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path("gamera-op_b200").resolve()))
gop = importlib.import_module("gop")

NG = 4
DEV = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64
GAMMA, CFL, CA = 5.0 / 3.0, 0.3, 10.0
RHO_FLOOR, P_FLOOR = 0.00316227, 0.000316227
# shapes of the batched workload's uneven grids
BATCH_GRIDS = ((256, 256, 4), (128, 128, 128), (64, 64, 64), (128, 128, 4), (96, 96, 96), (64, 64, 4))
# FP64 operations of one cell-update and the bytes of its state (W and B of two
# time levels in, one out)
FLOP_CELL, BYTE_CELL = 3471, 216


def listed():
    run = dict(family="run", coord="cart", bc="pppppp")
    return [
        # a thin two-dimensional vortex, the library's smallest everyday grid: launches and latency
        dict(run, name="ot_64x64x4_fp64", problem="ot", ni=64, nj=64, nk=4, precision="fp64", steps=20),
        # the reference's Orszag-Tang configuration, plain and mixed
        dict(run, name="ot_256x256x4_fp64", problem="ot", ni=256, nj=256, nk=4, precision="fp64", steps=50),
        dict(run, name="ot_256x256x4_mixed", problem="ot", ni=256, nj=256, nk=4, precision="mixed", steps=50),
        # ragged sizes and a mix of outflow, symmetry and periodic faces
        dict(run, name="blast_77x45x21_open_fp64", problem="blast", ni=77, nj=45, nk=21, bc="eesspp",
             precision="fp64", steps=40),
        # a served request from admission to result: created, set up on the device, stepped, copied
        # back, freed
        dict(family="request", name="request_64_mixed", problem="blast", coord="cart", bc="pppppp", ni=64,
             nj=64, nk=64, precision="mixed", steps=100),
        # the blast wave at the size of a larger request, and the headline grid plain and mixed
        dict(run, name="blast_128_fp64", problem="blast", ni=128, nj=128, nk=128, precision="fp64", steps=40),
        dict(run, name="blast_256_fp64", problem="blast", ni=256, nj=256, nk=256, precision="fp64", steps=20),
        dict(run, name="blast_256_mixed", problem="blast", ni=256, nj=256, nk=256, precision="mixed", steps=20),
        # the curvilinear path: a pole-free spherical shell with outflow on every face
        dict(run, name="shell_192x128x128_fp64", problem="loop", coord="sph", ni=192, nj=128, nk=128,
             bc="eeeeee", precision="fp64", steps=20),
        dict(run, name="shell_96x64x48_mixed", problem="loop", coord="sph", ni=96, nj=64, nk=48,
             bc="eeeeee", precision="mixed", steps=40),
        # many uneven grids stepped together
        dict(family="batch", name="batch_16_uneven_mixed", members=16, precision="mixed", steps=30),
        # the CFL step and div B of a state the caller keeps on the device (restored from a
        # single-precision file)
        dict(family="cfl", name="cfl_192_device_state", problem="blast", coord="cart", bc="pppppp", ni=192,
             nj=192, nk=192, precision="fp64", steps=0),
    ]


def draw(rng):
    """One more case: grids of about 10 K to 4 M cells, odd sizes among them."""
    def size(lo, hi):
        return max(4, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))

    kind = rng.choice(["ot", "ot", "blast", "blast", "shell", "shell", "request", "batch", "cfl"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "batch":
        return dict(family="batch", members=rng.randint(4, 16), precision=precision, steps=rng.randint(10, 25))
    if kind == "ot":
        ni, nj = size(48, 320), size(48, 320)
        return dict(family="run", coord="cart", bc="pppppp", problem="ot", ni=ni, nj=nj,
                    nk=rng.choice([4, 4, 5, 8]), precision=precision, steps=rng.randint(15, 50))
    if kind == "shell":
        return dict(family="run", coord="sph", bc="eeeeee", problem="loop", ni=size(32, 192), nj=size(24, 128),
                    nk=size(20, 128), precision=precision, steps=rng.randint(10, 20))
    ni, nj, nk = size(24, 160), size(24, 160), size(24, 160)
    if kind == "request":
        return dict(family="request", problem="blast", coord="cart", bc="pppppp", ni=ni, nj=nj, nk=nk,
                    precision=precision, steps=rng.randint(20, 80))
    if kind == "cfl":
        return dict(family="cfl", problem="blast", coord="cart", bc="pppppp", ni=ni, nj=nj, nk=nk,
                    precision="fp64", steps=0)
    return dict(family="run", coord="cart", bc=rng.choice(["pppppp", "pppppp", "eesspp", "eeeeee"]), problem="blast",
                ni=ni, nj=nj, nk=nk, precision=precision, steps=rng.randint(10, 30))


# ------------------------------------------------------------- initial states

def _members(case):
    """The grids of a case, as (problem, n) pairs."""
    if case["family"] != "batch":
        return [(case["problem"], (case["ni"], case["nj"], case["nk"]))]
    grids = [BATCH_GRIDS[m % len(BATCH_GRIDS)] for m in range(case["members"])]
    return [("ot" if n[2] == 4 else "blast", n) for n in grids]


def _domain(problem, n):
    """Cubic cells: the third axis spans n_k / n_i of the first."""
    if problem == "loop":
        return (1.0, 2.0, 0.25 * math.pi, 0.75 * math.pi, -0.25 * math.pi, 0.25 * math.pi)
    if problem == "ot":
        return (0.0, 1.0, 0.0, 1.0, 0.0, n[2] / n[0])
    return (-0.5, 0.5, -0.5, 0.5, -0.5, 0.5)


def _physics(problem, rng):
    """What differs from seed to seed."""
    if problem == "ot":
        return dict(phase=tuple(rng.uniform(0.0, 1.0, 2)), amp=rng.uniform(0.8, 1.1))
    if problem == "blast":
        d = rng.normal(size=3)
        b = rng.uniform(0.4, 1.0) * d / np.linalg.norm(d)
        return dict(p_in=float(rng.uniform(4.0, 20.0)), b=tuple(float(v) for v in b),
                    center=tuple(float(v) for v in rng.uniform(-0.1, 0.1, 3)),
                    radius=float(rng.uniform(0.1, 0.16)))
    return dict(v=tuple(float(v) for v in rng.uniform(0.3, 1.0, 3)), x=float(rng.uniform(1.45, 1.55)),
                y=float(rng.uniform(-0.1, 0.1)), a0=float(rng.uniform(0.05, 0.1)))


def _coords(problem, n):
    dom = _domain(problem, n)
    return [torch.tensor([dom[2 * a] + (i - NG) * (dom[2 * a + 1] - dom[2 * a]) / n[a]
                          for i in range(n[a] + 2 * NG + 1)], dtype=F64, device=DEV) for a in range(3)]


def _initial(problem, n, ph):
    """Gas (6 fields) and face field (3) on the ghost-extended grid."""
    N = tuple(m + 2 * NG + 1 for m in n)
    x = [c.reshape([-1 if a == d else 1 for d in range(3)]) for a, c in enumerate(_coords(problem, n))]
    ctr = [0.5 * (c.narrow(a, 0, N[a] - 1) + c.narrow(a, 1, N[a] - 1)) for a, c in enumerate(x)]
    gas = torch.zeros((6,) + N, dtype=F64, device=DEV)
    fb = torch.zeros((3,) + N, dtype=F64, device=DEV)
    act = tuple(slice(NG, NG + m) for m in n)
    cell = [c.narrow(a, NG, n[a]) for a, c in enumerate(ctr)]

    def circulate(az, k_len):
        """Face B from A_z's line integrals along the edges of k (the others are zero)."""
        la = az * k_len
        d0 = la.narrow(0, 1, N[0] - 1) - la.narrow(0, 0, N[0] - 1)
        d1 = la.narrow(1, 1, N[1] - 1) - la.narrow(1, 0, N[1] - 1)
        return d0, d1

    if problem == "ot":
        tp = 2.0 * math.pi
        gas[0][act] = 25.0 / (36.0 * math.pi)
        gas[4][act] = 5.0 / (12.0 * math.pi)
        gas[1][act] = -ph["amp"] * torch.sin(tp * (cell[1] + ph["phase"][1]))
        gas[2][act] = ph["amp"] * torch.sin(tp * (cell[0] + ph["phase"][0]))
        az = (torch.cos(2 * tp * (x[0] + ph["phase"][0])) / (4 * math.pi)
              + torch.cos(tp * (x[1] + ph["phase"][1])) / (2 * math.pi)) / math.sqrt(4 * math.pi)
        az = az.expand(N[0], N[1], 1)
        d0, d1 = circulate(az, 1.0)
        fb[0][:, :N[1] - 1, :N[2] - 1] = d1 / (x[1].narrow(1, 1, N[1] - 1) - x[1].narrow(1, 0, N[1] - 1))
        fb[1][:N[0] - 1, :, :N[2] - 1] = -d0 / (x[0].narrow(0, 1, N[0] - 1) - x[0].narrow(0, 0, N[0] - 1))
    elif problem == "blast":
        r = sum((cell[a] - ph["center"][a]) ** 2 for a in range(3)).sqrt()
        gas[0][act] = 1.0
        gas[4][act] = torch.where(r < ph["radius"], ph["p_in"], 0.1).to(F64)
        for a in range(3):
            s = list(act)
            s[a] = slice(NG, NG + n[a] + 1)
            fb[a][tuple(s)] = ph["b"][a]
    else:  # a field loop carried through the shell by a uniform flow
        r, t, f = x
        gas[0, :-1, :-1, :-1] = 1.0
        gas[4, :-1, :-1, :-1] = 1.0
        tc, fc = ctr[1], ctr[2]
        vx, vy, vz = ph["v"]
        st, ct, sf, cf = tc.sin(), tc.cos(), fc.sin(), fc.cos()
        gas[1, :-1, :-1, :-1] = vx * st * cf + vy * st * sf + vz * ct
        gas[2, :-1, :-1, :-1] = vx * ct * cf + vy * ct * sf - vz * st
        gas[3, :-1, :-1, :-1] = -vx * sf + vy * cf
        # A_phi = a0 exp(-d^2 / s^2) about a point of the shell: edges along phi only
        d2 = ((r * t.sin() - ph["x"]) ** 2 + (r * t.cos() - ph["y"]) ** 2)
        aphi = ph["a0"] * torch.exp(-d2 / 0.15 ** 2)
        la = (aphi * r * t.sin()).expand(N[0], N[1], 1)
        dth = t.narrow(1, 0, N[1] - 1).cos() - t.narrow(1, 1, N[1] - 1).cos()
        fb[0][:, :N[1] - 1, :N[2] - 1] = (la.narrow(1, 1, N[1] - 1) - la.narrow(1, 0, N[1] - 1)) / (r * r * dth)
        r0, r1 = r.narrow(0, 0, N[0] - 1), r.narrow(0, 1, N[0] - 1)
        fb[1][:N[0] - 1, :, :N[2] - 1] = -(la.narrow(0, 1, N[0] - 1) - la.narrow(0, 0, N[0] - 1)) / (
            0.5 * (r1 * r1 - r0 * r0) * t.sin())
        fb[2, :N[0] - 1, :N[1] - 1, :] = 0.02 / (0.5 * (r0 + r1))
    return gas, fb


def _single(fb):
    """A face field as a single-precision file gives it back."""
    return fb.to(torch.float32).to(F64)


# ------------------------------------------------------------------ the calls

def _precision(case):
    return gop.PREC_MIXED if case["precision"] == "mixed" else gop.PREC_FP64


def _instance(case, problem, n):
    dom = _domain(problem, n)
    xs = [gop.grid_uniform(n[a], dom[2 * a], dom[2 * a + 1]) for a in range(3)]
    coord = gop.COORD_SPHERICAL if problem == "loop" else gop.COORD_CARTESIAN
    return gop.Instance(n, *xs, coord=coord, bc=case.get("bc", "pppppp"), precision=_precision(case))


def _host_buffers(n):
    N = tuple(m + 2 * NG + 1 for m in n)
    return {f: torch.zeros((nf,) + N, dtype=F64, pin_memory=DEV == "cuda").numpy()
            for f, nf in (("gas", 6), ("face_b", 3))}


def prepare(case, seed):
    rng = np.random.default_rng([seed, 20261204])
    members = [(p, n, _physics(p, rng)) for p, n in _members(case)]
    family = case["family"]
    if family == "request":
        (_, n, ph), = members
        return dict(case=case, n=n, ph=ph, out=_host_buffers(n))
    if family == "cfl":
        (p, n, ph), = members
        gas, fb = _initial(p, n, ph)
        act = tuple(slice(NG, NG + m) for m in n)
        g = torch.Generator(device=DEV).manual_seed(seed)
        gas[(slice(1, 4),) + act] = 0.3 * torch.randn((3,) + n, dtype=F64, device=DEV, generator=g)
        gas[(slice(0, 1),) + act] += 0.2 * torch.rand((1,) + n, dtype=F64, device=DEV, generator=g)
        for a in range(3):  # tilt it, so that its rounding leaves a divergence
            fb[a] *= 1.0 + 0.1 * torch.rand(fb.shape[1:], dtype=F64, device=DEV, generator=g)
        inst = _instance(case, p, n)  # for its grid descriptor
        call = gop.lib().gop_cfl_dt_noalloc
        call.argtypes = [ctypes.POINTER(gop.Desc)] + [ctypes.c_void_p] * 6
        return dict(case=case, inst=inst, gas=gas, fb=_single(fb), call=call,
                    out=torch.zeros(2, dtype=F64, device=DEV))
    insts, outs = [], []
    for p, n, ph in members:
        gas, fb = _initial(p, n, ph)
        inst = _instance(case, p, n)
        inst.upload(gas.cpu().numpy(), fb.cpu().numpy())
        inst.prepare()
        insts.append(inst)
        outs.append(_host_buffers(n))
    state = dict(case=case, insts=insts, outs=outs)
    if family == "batch":
        state["batch"] = gop.Batch(insts)
    return state


def run(state):
    case = state["case"]
    family, steps = case["family"], case["steps"]
    if family == "cfl":
        st = torch.cuda.current_stream().cuda_stream
        rc = state["call"](ctypes.byref(state["inst"].desc), state["gas"].data_ptr(), state["fb"].data_ptr(),
                           None, None, state["out"].data_ptr(), st)
        if rc:
            raise RuntimeError(gop.lib().gop_last_error().decode())
        return state["out"]
    if family == "request":
        inst = _instance(case, "blast", state["n"])
        inst.init_problem_device(gop.PROBLEM_BLAST, **state["ph"])
        inst.prepare()
        t = inst.step(steps)
        out = inst.download(("gas", "face_b"), out=state["out"])
        inst.close()
        return dict(out, time=t)
    if family == "batch":
        state["batch"].step([steps] * len(state["insts"]))
        return [i.download(("gas", "face_b"), out=o) for i, o in zip(state["insts"], state["outs"])]
    # to the next output: the steps, then the state in the host's buffers
    inst, = state["insts"]
    t = inst.step(steps)
    return dict(inst.download(("gas", "face_b"), out=state["outs"][0]), time=t)


def work(case):
    cells = sum(math.prod(n) for _, n in _members(case))
    if case["family"] == "cfl":  # 5 gas fields and 3 face fields read once
        return {"bytes": 64 * cells, "flops": 60 * cells}
    points = sum(math.prod(m + 2 * NG + 1 for m in n) for _, n in _members(case))
    # the result's copy to the host reads its 9 fields once more
    return {"bytes": case["steps"] * BYTE_CELL * cells + 72 * points, "flops": case["steps"] * FLOP_CELL * cells}


# ------------------------------------------- the same in plain torch, 64 bits

def _cut(t, lo, n):
    """t's last three axes from lo, n long; axes of length 1 stay."""
    for d in range(3):
        ax = t.dim() - 3 + d
        if t.shape[ax] != 1:
            t = t.narrow(ax, lo[d], n[d])
    return t


class _Grid:
    """Geometry and reconstruction weights of a uniform Cartesian or spherical grid."""

    def __init__(self, problem, n, bc):
        self.n, self.N, self.bc, self.sph = n, tuple(m + 2 * NG + 1 for m in n), bc, problem == "loop"
        x1d = [c.cpu().numpy() for c in _coords(problem, n)]

        def along(a, v):
            return torch.as_tensor(np.ascontiguousarray(v), device=DEV).reshape(
                [-1 if d == a else 1 for d in range(3)])

        def padded(v):  # one value per point, the last repeated
            return np.append(v, v[-1])

        dx = [padded(np.diff(c)) for c in x1d]
        mid = [c + 0.5 * d for c, d in zip(x1d, dx)]
        ctr = [m.copy() for m in mid]
        if self.sph:
            ctr[0] = mid[0] + 2.0 * mid[0] * dx[0] ** 2 / (12.0 * mid[0] ** 2 + dx[0] ** 2)
            t0, t1 = x1d[1], x1d[1] + dx[1]
            ctr[1] = (np.sin(t1) - np.sin(t0) - (t1 * np.cos(t1) - t0 * np.cos(t0))) / (np.cos(t0) - np.cos(t1))
        self.lo_w = [along(a, (x1d[a] + dx[a] - ctr[a]) / dx[a]) for a in range(3)]
        self.hi_w = [along(a, (ctr[a] - x1d[a]) / dx[a]) for a in range(3)]
        d = [along(a, dx[a]) for a in range(3)]
        self.dx = d
        if not self.sph:
            self.area = [d[1] * d[2], d[0] * d[2], d[0] * d[1]]
            self.vol = d[0] * d[1] * d[2]
            self.edge = d
            self.length = d
        else:
            r, t = along(0, x1d[0]), along(1, x1d[1])
            cost = along(1, np.cos(x1d[1]) - np.cos(x1d[1] + dx[1]))
            half = along(0, 0.5 * ((x1d[0] + dx[0]) ** 2 - x1d[0] ** 2))
            self.area = [r * r * cost * d[2], half * t.sin() * d[2], half * d[1]]
            self.vol = along(0, ((x1d[0] + dx[0]) ** 3 - x1d[0] ** 3) / 3.0) * cost * d[2]
            self.edge = [d[0], r * d[1], r * t.sin() * d[2]]
            rc, tc = along(0, mid[0]), along(1, mid[1])
            self.length = [d[0], rc * d[1], rc * tc.sin() * d[2]]
            self.rc = rc
            s0, s1 = np.sin(x1d[1]), np.sin(x1d[1] + dx[1])
            self.cot = along(1, (s1 - s0) / (s1 + s0))
        self.w = [self._weights(a, x1d[a]) for a in range(3)]

    def _weights(self, a, x):
        """Seven left and seven right taps and the four limiter coefficients of every face of axis a."""
        N, n = self.N[a], self.n[a]
        w = np.zeros((18, N))
        seven = np.array([-3.0, 25.0, -101.0, 319.0, 214.0, -38.0, 4.0]) / 420.0
        five = np.array([0.0, 2.0, -13.0, 47.0, 27.0, -3.0, 0.0]) / 60.0

        def measure(u):
            return u * u if a == 0 else np.sin(u)

        def volume(c):
            return (x[c + 1] ** 3 - x[c] ** 3) / 3.0 if a == 0 else math.cos(x[c]) - math.cos(x[c + 1])

        gn, gw = np.polynomial.legendre.leggauss(8)

        def taps(f, first):
            """Five cells from `first` whose averages give the quartic's value at face f."""
            h = x[f] - x[f - 1]
            A = np.zeros((5, 5))
            for c in range(5):
                u0 = x[0] + (first + c) * (x[1] - x[0]) if first + c < 0 else x[first + c]
                u1 = u0 + (x[1] - x[0])
                u = 0.5 * (u0 + u1) + 0.5 * (u1 - u0) * gn
                m = gw * measure(u)
                for j in range(5):
                    A[j, c] = (m * ((u - x[f]) / h) ** j).sum() / m.sum()
            return np.linalg.solve(A, np.array([1.0, 0, 0, 0, 0]))

        e = 1.0 / 3.0
        for f in range(NG, NG + n + 1):
            if not self.sph or a == 2:
                w[:7, f] = w[7:14, f] = five if self.sph else seven
                w[14:, f] = (2.0, -2.0, 2.0, -2.0)
                continue
            w[1:6, f] = taps(f, f - 3)
            w[8:13, f] = taps(f, f - 2)[::-1]
            dx = x[f] - x[f - 1]
            g = measure(x)
            q = volume(f - 1) / dx
            w[14, f], w[15, f] = (q - e * g[f]) / (e * g[f]), (e * g[f - 1] - q) / (e * g[f])
            q = volume(f) / (x[f + 1] - x[f]) if f + 1 < N else q
            w[16, f], w[17, f] = (q - e * g[f]) / (e * g[f]), (e * g[f + 1] - q) / (e * g[f])
        return torch.as_tensor(w, device=DEV).reshape([18] + [-1 if d == a else 1 for d in range(3)])

    def states(self, half, lim, a, lo, n):
        """Left and right states at the faces of axis a in the box (lo, n)."""
        def tap(t, o):
            at = list(lo)
            at[a] += o
            return _cut(t, at, n)

        w = _cut(self.w[a], lo, n)
        l0, l1, l2, l3 = (tap(lim, o) for o in (-2, -1, 0, 1))
        dm, d1, dp = l1 - l0, l2 - l1, l3 - l2
        s = d1.sign()
        hi, low = torch.maximum(l1, l2), torch.minimum(l1, l2)

        def side(cells, wt, near, far, c1, c2, dside, sgn):
            f = sum(tap(half, o) * wt[t] for t, o in enumerate(cells))
            f = torch.maximum(low, torch.minimum(f, hi))
            dc = 0.25 * (c1 * near + c2 * far).abs() + 0.5 * dside.abs()
            return f - sgn * ((f - near).abs() - (dside.sign() + s).abs() * dc).clamp_min(0.0)

        return (side(range(-4, 3), w[:7], l1, l0, w[14], w[15], dm, s),
                side(range(3, -4, -1), w[7:14], l2, l3, w[16], w[17], dp, -s))

    def center_b(self, B):
        """Cell-centred field from the faces (ghost cells too)."""
        out = []
        for a in range(3):
            up = torch.cat([B[a].narrow(a, 1, self.N[a] - 1), B[a].narrow(a, self.N[a] - 1, 1)], a)
            out.append(B[a] * self.lo_w[a] + up * self.hi_w[a])
        return torch.stack(out)

    def ghosts(self, W, B):
        n, N = self.n, self.N
        for a in range(3):
            if self.bc[2 * a] != "p":
                continue
            for t, o in [(W[m], 0) for m in range(5)] + [(B[c], int(c == a)) for c in range(3)]:
                low, high = t.narrow(a, n[a], NG).clone(), t.narrow(a, NG + o, NG).clone()
                t.narrow(a, 0, NG).copy_(low)
                t.narrow(a, n[a] + NG + o, NG).copy_(high)
        for face in range(6):
            a, up, kind = face // 2, face % 2, self.bc[face]
            if kind == "p":
                continue
            for t, o in [(W[m], 0) for m in range(5)] + [(B[c], int(c == a)) for c in range(3)]:
                for l in range(NG):
                    dst = l if not up else n[a] + NG + l + o
                    if kind == "e":
                        src = NG if not up else n[a] + NG - 1 + o
                    else:  # symmetric
                        src = 2 * NG - 1 - l + o if not up else n[a] + NG - 1 - l
                    t.narrow(a, dst, 1).copy_(t.narrow(a, src, 1).clone())

    def dt(self, W, B):
        lo = (NG,) * 3
        r, u, v, w, p = (_cut(W[m], lo, self.n) for m in range(5))
        b2 = _cut(self.center_b(B), lo, self.n).square().sum(0)
        va2 = b2 / r
        va2 = va2 * CA ** 2 / (va2 + CA ** 2)
        vc = (u * u + v * v + w * w).sqrt() + (GAMMA * p / r + va2).sqrt()
        return float((CFL / sum(vc / _cut(self.length[a], lo, self.n) for a in range(3))).min())

    def fluxes(self, a, Wh, W, Mh, M, B):
        """Fluxes of mass, momentum, energy and the stress at the active faces of axis a; the averaged
        velocity states along a."""
        lo, n = (NG,) * 3, [m + (d == a) for d, m in enumerate(self.n)]
        st = [self.states(Wh[m], W[m], a, lo, n) for m in range(5)]
        mg = [self.states(Mh[c], M[c], a, lo, n) for c in range(3)]
        bn = _cut(B[a], lo, n)
        side = []
        for s in range(2):
            r, p, v = st[0][s], st[4][s], [st[1 + c][s] for c in range(3)]
            b = [mg[c][s] for c in range(3)]
            b2 = b[0] ** 2 + b[1] ** 2 + b[2] ** 2
            va2 = b2 / r
            va2 = va2 * CA ** 2 / (va2 + CA ** 2)
            speed = v[a].abs() + (GAMMA * p / r + va2).sqrt()
            e = 0.5 * r * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2) + p / (GAMMA - 1.0)
            side.append((r, v, p, b, b2, e, speed))
        (rl, vl, pl, bl, b2l, el, cl), (rr, vr, pr, br, b2r, er, cr) = side
        vf = torch.maximum(cl, cr)
        F = [0.5 * (rl * vl[a] + rr * vr[a] - vf * (rr - rl))]
        for c in range(3):
            f = rl * vl[c] * vl[a] + rr * vr[c] * vr[a] - vf * (rr * vr[c] - rl * vl[c])
            F.append(0.5 * (f + pl + pr if c == a else f))
        F.append(0.5 * ((el + pl) * vl[a] + (er + pr) * vr[a] - vf * (er - el)))
        q = (b2l + b2r) / (4.0 * CA)
        for c in range(3):
            t = -0.5 * (bl[c] + br[c]) * bn
            if c == a:
                t = t + 0.25 * (b2l + b2r)
            F.append(t - q * (vr[c] - vl[c]))
        return F

    def emf(self, D, Wh, W, Bh, B):
        """E along axis D at its active edges."""
        p, q = (D + 1) % 3, (D + 2) % 3
        lo, n = [NG] * 3, [m + (d != D) for d, m in enumerate(self.n)]
        wide, wn = list(lo), list(n)
        wide[q], wn[q] = 0, self.N[q] - 1  # every cell along q
        v = []
        for comp in (p, q):
            full = torch.zeros(self.N, dtype=F64, device=DEV)
            L, R = self.states(Wh[1 + comp], W[1 + comp], p, wide, wn)
            _cut(full, wide, wn).copy_(0.5 * (L + R))
            L, R = self.states(full, full, q, lo, n)
            v.append(0.5 * (L + R))
        bpl, bpr = self.states(Bh[p], B[p], q, lo, n)
        bql, bqr = self.states(Bh[q], B[q], p, lo, n)
        rho4 = 0.0
        for dp in (-1, 0):
            for dq in (-1, 0):
                at = list(lo)
                at[p] += dp
                at[q] += dq
                rho4 = rho4 + _cut(Wh[0], at, n)
        bp, bq = 0.5 * (bpl + bpr), 0.5 * (bql + bqr)
        va = ((bp * bp + bq * bq) / (0.25 * rho4)).sqrt()
        vz = va * CA / (va * va + CA * CA).sqrt() + (v[0] ** 2 + v[1] ** 2).sqrt()
        e = torch.zeros(self.N, dtype=F64, device=DEV)
        _cut(e, lo, n).copy_(v[1] * bp - v[0] * bq + 0.5 * vz * (bpl + bqr - bpr - bql))
        return e

    def step(self, W, Wo, B, Bo, dt, dt0):
        n, lo = self.n, (NG,) * 3
        c = 0.5 * dt / dt0
        Wh, Bh = W + c * (W - Wo), B + c * (B - Bo)
        M, Mo = self.center_b(B), self.center_b(Bo)
        Mh = M + c * (M - Mo)
        E = [self.emf(D, Wh, W, Bh, B) * self.edge[D] for D in range(3)]
        Bn = B.clone()
        for a in range(3):  # constrained transport
            p, q = (a + 1) % 3, (a + 2) % 3
            m = [k + (d == a) for d, k in enumerate(n)]
            up, uq = list(lo), list(lo)
            up[p] += 1
            uq[q] += 1
            curl = _cut(E[q], up, m) - _cut(E[q], lo, m) - (_cut(E[p], uq, m) - _cut(E[p], lo, m))
            _cut(Bn[a], lo, m).sub_(dt * curl / _cut(self.area[a], lo, m))
        del E
        vol = _cut(self.vol, lo, n)
        dU, src = [0.0] * 8, [0.0] * 6
        for a in range(3):
            F = self.fluxes(a, Wh, W, Mh, M, B)
            m = [k + (d == a) for d, k in enumerate(n)]
            area = _cut(self.area[a], lo, m)
            al, au = (area, area) if area.shape[a] == 1 else (area.narrow(a, 0, n[a]), area.narrow(a, 1, n[a]))
            low = [f.narrow(a, 0, n[a]) * al for f in F]
            top = [f.narrow(a, 1, n[a]) * au for f in F]
            for k in range(8):
                dU[k] = dU[k] + (top[k] - low[k]) / vol
            if not self.sph:
                continue
            r, v2, v3, p = (_cut(Wh[k], lo, n) for k in (0, 2, 3, 4))
            h2, h3 = p + r * v2 * v2, p + r * v3 * v3
            b = _cut(Mh, lo, n)
            b2 = b.square().sum(0)
            m2, m3 = 0.5 * b2 - b[1] ** 2, 0.5 * b2 - b[2] ** 2
            if a == 0:
                g = 0.5 * _cut(self.dx[0] / self.rc, lo, n) / vol
                for k, (t2, t3) in ((0, (h2, h3)), (3, (m2, m3))):
                    f = 1 if k == 0 else 5
                    src[k] = src[k] + 0.5 * (t2 + t3) * (au - al) / vol
                    src[k + 1] = src[k + 1] - (low[f + 1] + top[f + 1]) * g
                    src[k + 2] = src[k + 2] - (low[f + 2] + top[f + 2]) * g
            elif a == 1:
                s = _cut(self.cot, lo, n) / vol
                for k, t3 in ((0, h3), (3, m3)):
                    f = 1 if k == 0 else 5
                    src[k + 1] = src[k + 1] + (au - al) / vol * t3
                    src[k + 2] = src[k + 2] - (low[f + 2] + top[f + 2]) * s
        r0, p0 = _cut(W[0], lo, n), _cut(W[4], lo, n)
        v0 = [_cut(W[1 + k], lo, n) for k in range(3)]
        ke = v0[0] ** 2 + v0[1] ** 2 + v0[2] ** 2
        rho_u = r0 - dt * dU[0]
        mom = [r0 * v0[k] - dt * dU[1 + k] + dt * src[k] for k in range(3)]
        en = 0.5 * r0 * ke + p0 / (GAMMA - 1.0) - dt * dU[4]
        p = (en - 0.5 * (mom[0] ** 2 + mom[1] ** 2 + mom[2] ** 2) / rho_u) * (GAMMA - 1.0)
        low_rho = rho_u < RHO_FLOOR
        rho = torch.where(low_rho, RHO_FLOOR, rho_u)
        p = torch.where(low_rho, P_FLOOR, p).clamp_min(P_FLOOR)
        mt = 0.5 * (_cut(self.center_b(Bn), lo, n) + _cut(M, lo, n))
        b2 = mt.square().sum(0)
        alf = b2 / rho / CA ** 2
        drho = -dt * dU[0]
        hyd = [-dt * dU[1 + k] + dt * src[k] for k in range(3)]
        tv = [alf * (hyd[k] - drho * v0[k]) for k in range(3)]
        along = (mt[0] * tv[0] + mt[1] * tv[1] + mt[2] * tv[2]) / (b2 + 1e-10)
        Wn = W.clone()
        _cut(Wn[0], lo, n).copy_(rho)
        _cut(Wn[4], lo, n).copy_(p)
        for k in range(3):
            mag = -dt * dU[5 + k] + dt * src[3 + k]
            inc = (hyd[k] + mag + alf * drho * v0[k] + mt[k] * along) / (1.0 + alf)
            _cut(Wn[1 + k], lo, n).copy_((r0 * v0[k] + inc) / rho_u)
        self.ghosts(Wn, Bn)
        return Wn, Bn


def _exact_run(problem, n, bc, steps, gas, fb):
    g = _Grid(problem, n, bc)
    W, B = gas[:5].clone(), fb.clone()
    g.ghosts(W, B)
    Wo, Bo, time = W, B, 0.0
    dt0 = dt = g.dt(W, B)
    for _ in range(steps):
        time += dt
        Wn, Bn = g.step(W, Wo, B, Bo, dt, dt0)
        Wo, Bo, W, B, dt0 = W, B, Wn, Bn, dt
        dt = g.dt(W, B)
    return dict(gas=torch.cat([W, gas[5:]]), face_b=B, time=time)


def exact(case, seed):
    rng = np.random.default_rng([seed, 20261204])
    members = [(p, n, _physics(p, rng)) for p, n in _members(case)]
    if case["family"] == "cfl":
        s = prepare(case, seed)
        (p, n, _), = members
        g = _Grid(p, n, case["bc"])
        lo = (NG,) * 3
        div = 0.0
        for a in range(3):
            f = s["fb"][a].narrow(a, NG, n[a] + 1)
            for d in range(3):
                f = f if d == a else f.narrow(d, NG, n[d])
            div = div + (f.narrow(a, 1, n[a]) - f.narrow(a, 0, n[a])) / _cut(g.dx[a], lo, n)
        return torch.tensor([g.dt(s["gas"], s["fb"]), float(div.abs().max())], dtype=F64)
    out = [_exact_run(p, n, case.get("bc", "pppppp"), case["steps"], *_initial(p, n, ph)) for p, n, ph in members]
    if case["family"] == "batch":
        return [{k: o[k] for k in ("gas", "face_b")} for o in out]
    return out[0]

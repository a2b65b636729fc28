"""Representative calls of the library, for timing and for checking results.

A case is one call (or the few calls that a host program makes together) on
the GPU: `listed()` names the fixed ones, `draw(rng)` gives others of the same
ranges.  `prepare` makes the inputs and the context that a program keeps,
`run` makes the calls, `work` counts the bytes and operations that the result
cannot do without, and `exact` recomputes the outputs in 64 bits with plain
torch and numpy.

Kinds of case:
  step       sg_step: interpolation, membrane force and spreading in one call,
             once per time step (the library's main path)
  graph      the same step replayed from the CUDA graph captured on its buffers
  subs       the reference's three subroutines called one after the other
             (eulr2lagr, complagrforces, lagr2eulr), as a host code does that
             replaces them one by one
  flow       sg_flow_step: the FFT flow solver's step
  indicator  sg_indicator with the viscosity and the centrifugal terms
  loop       one step of the coupled solver (IBSolver): all of the above

Keys: itot, jtot, ktot: interior cells; ncap: capsules; lmin, lmax: their SH
degrees, uniform in that range; fp64: FP64 or mixed precision; bend: the
reference's default bending (cbend = 0.3); law: 0 Skalak, 1 neo-Hookean;
host: arrays in pinned host memory, copied in and out by the call.
"""
import math

import numpy as np
import torch

from suguru_b200 import workloads
from suguru_b200.coupling import CouplingStep
from suguru_b200.ib_solver import IBSolver

CBEND = 0.3       # param.f90:90-91
CELL = 32         # one capsule at most per block of CELL^3 cells
FLOW = dict(dt=0.01 / 32, rep=0.0016, vb2=0.0, vt2=0.0)
IND = dict(visc0=1.0 / 0.0016, lam=5.0, thetainc=70.0 * math.pi / 180.0, ta=1160000.0, rep=0.0016)
BASE = dict(ncap=1, lmin=15, lmax=15, fp64=True, bend=False, law=0, host=False)


def _case(kind, itot, jtot, ktot, **kw):
    return {"kind": kind, "itot": itot, "jtot": jtot, "ktot": ktot, **BASE, **kw}


def listed():
    named = {
        # one capsule in a channel, the smallest run: the call's latency counts
        "step_single": _case("step", 128, 64, 64),
        # the same, mixed precision, as the time loop replays it
        "graph_single_mixed": _case("graph", 128, 64, 64, fp64=False),
        # a dense suspension (the benchmark's workload) in both precisions
        "step_dense": _case("step", 256, 256, 128, ncap=256),
        "step_dense_mixed": _case("step", 256, 256, 128, ncap=256, fp64=False),
        # the same with the reference's default membrane, which bends
        "step_dense_bend_mixed": _case("step", 256, 256, 128, ncap=256, fp64=False, bend=True),
        # capsules of uneven size and degree, the largest workload of the benchmark
        "step_uneven_mixed": _case("step", 512, 256, 256, ncap=1024, lmin=7, lmax=23, fp64=False),
        # host arrays: a host code whose arrays stay in its own memory
        "step_host_mixed": _case("step", 128, 128, 64, ncap=24, lmin=12, lmax=16, fp64=False, host=True),
        # three calls on a ragged grid, neo-Hookean membranes of low and high degree
        "subs_ragged": _case("subs", 250, 182, 101, ncap=60, lmin=5, lmax=31, law=1),
        # the flow solver on the dense suspension's grid, and on lengths that are no powers of two
        "flow_dense": _case("flow", 256, 256, 128),
        "flow_ragged": _case("flow", 180, 150, 99),
        # the indicator of the dense suspension
        "indicator_dense": _case("indicator", 256, 256, 128, ncap=256),
        # a whole coupled step of the dense suspension, every stage
        "loop_dense": _case("loop", 256, 256, 128, ncap=256),
    }
    return [{"name": n, **c} for n, c in named.items()]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _extent(rng, blocks, even=False):
    """Cells of `blocks` blocks and some more: multiples of 32 as often as odd lengths.  The
    spreading tiles leave no remainder of 1 or 2 in x and y; the FFT wants small prime factors."""
    n = CELL * blocks
    if rng.random() < 0.5:
        return n
    smooth = {n + r for r in range(3, 30) if (n + r) % 8 not in (1, 2) and not (even and (n + r) % 2)
              and _largest_prime(n + r) <= 31}
    return rng.choice(sorted(smooth)) if smooth else n


def _largest_prime(n):
    p, best = 2, 1
    while n > 1:
        while n % p == 0:
            n, best = n // p, p
        p += 1
    return best


def draw(rng):
    kind = rng.choice(["step", "step", "step", "graph", "subs", "flow", "flow", "indicator", "loop"])
    mixed = kind in ("step", "graph", "subs") and rng.random() < 0.6
    host = kind == "step" and rng.random() < 0.15
    even = kind in ("flow", "indicator", "loop")  # the real transform's length
    cells = 2 << 20 if host else 4 << 20 if even else 30 << 20 if mixed else 8 << 20
    while True:
        b = [_log_int(rng, 1.6, 12) for _ in range(3)]
        ext = [_extent(rng, b[0], even), _extent(rng, b[1]), CELL * b[2] + rng.choice([0, 0, 4, 7, 13])]
        if ext[0] >= 64 and ext[0] * ext[1] * ext[2] <= cells and ext[0] <= 512 and ext[1] <= 384:
            break
    room = b[0] * b[1] * b[2]
    lmin = rng.randint(5, 20)
    lmax = lmin if rng.random() < 0.4 else min(31, lmin + rng.randint(1, 12))
    ncap = max(1, min(room, _log_int(rng, 1, 1024)))
    while ncap * 8 * (lmax + 1) ** 2 > (1 << 20 if mixed else 1 << 19):
        ncap = max(1, ncap // 2)
    return _case(kind, *ext, ncap=ncap, lmin=lmin, lmax=lmax, fp64=not mixed,
                 bend=kind in ("step", "graph", "subs") and rng.random() < 0.25,
                 law=int(kind in ("step", "graph", "subs") and rng.random() < 0.2),
                 host=host)


# ------------------------------------------------------------------ inputs
def _grid(case):
    d = 1.0 / 32
    return case["itot"], case["jtot"], case["ktot"], d, d, d


def _degrees(case):
    """The capsules' degrees: part of the case, not of the seeded inputs."""
    return np.random.default_rng(7).integers(case["lmin"], case["lmax"] + 1, case["ncap"]).astype(np.int32)


def _capsules(case, rng):
    """Degrees, radii and centres: one capsule at most per block of CELL^3 cells."""
    itot, jtot, ktot, dx, _, _ = _grid(case)
    nb = [itot // CELL, jtot // CELL, ktot // CELL]
    degree = _degrees(case)
    radius = np.minimum(degree / 1.875, 12.0) * dx
    block = rng.choice(nb[0] * nb[1] * nb[2], case["ncap"], replace=False)
    corner = np.stack([block % nb[0], block // nb[0] % nb[1], block // (nb[0] * nb[1])], 1) * CELL
    free = CELL / 2 - 1.2 * radius[:, None] / dx - 1.0
    centre = (corner + CELL / 2 + rng.uniform(-1, 1, (case["ncap"], 3)) * np.maximum(free, 0.0)) * dx
    # move the whole suspension in x and y, so that capsules cross the periodic faces
    centre[:, 0] += rng.uniform(0, itot * dx)
    centre[:, 1] += rng.uniform(0, jtot * dx)
    centre[:, 0] %= itot * dx
    centre[:, 1] %= jtot * dx
    return degree, radius, centre


def _points(case, rng):
    """Force points of every capsule: spheres with a seeded perturbation of 5 % falling as 1/l^2."""
    degree, radius, centre = _capsules(case, rng)
    xyz = [None] * len(degree)
    for L in np.unique(degree):
        caps = np.flatnonzero(degree == L)
        N = int(L) + 1
        sh = _Harmonics(N, 2 * N, 4 * N, "cpu", 0)
        l = np.arange(N)
        l2 = np.where(l > 0, 1.0 / np.maximum(l, 1) ** 2, 0.0)
        low = l[:, None] <= l[None, :]  # m <= n
        co = rng.normal(size=(2, caps.size, N, N)) * (0.05 * l2 * low) * radius[caps, None, None]
        r = sh.synth(torch.from_numpy(co[0]), torch.from_numpy(co[1])).numpy() + radius[caps, None, None]
        th, ph = sh.theta.numpy()[:, None], sh.phi.numpy()[None, :]
        unit = [np.sin(th) * np.sin(ph), np.sin(th) * np.cos(ph), np.cos(th) + 0 * ph]
        p = np.stack([centre[caps, c, None, None] + r * unit[c] for c in range(3)], 1).reshape(caps.size, 3, -1)
        for q, c in enumerate(caps):
            xyz[c] = p[q]
    return degree, radius, np.ascontiguousarray(np.concatenate(xyz, 1))


def _fields(case, rng, count, dtype, amp=1.0, wall=True):
    """`count` smooth random fields with periodic halos (x fastest); wall: zero at the walls in z."""
    itot, jtot, ktot = case["itot"], case["jtot"], case["ktot"]
    f64 = dict(dtype=torch.float64, device="cuda")
    x, y, z = (torch.arange(n + 2, **f64) / n for n in (itot, jtot, ktot))
    s = torch.sin(math.pi * z) if wall else torch.cos(math.pi * z)
    out = []
    for _ in range(count):
        nx, ny = rng.integers(-4, 5, 12), rng.integers(-4, 5, 12)
        ph, a = rng.uniform(0, 2 * math.pi, 12), amp * rng.normal(size=12)
        plane = sum(a[q] * torch.cos(2 * math.pi * (nx[q] * x[None, :] + ny[q] * y[:, None]) + ph[q])
                    for q in range(12))
        f = s[:, None, None] * plane[None]
        out.append(_periodic(f).to(dtype))
    return out


def _periodic(f):
    f[:, :, -1], f[:, :, 0] = f[:, :, 1].clone(), f[:, :, -2].clone()
    f[:, -1, :], f[:, 0, :] = f[:, 1, :].clone(), f[:, -2, :].clone()
    return f


def _pinned(a):
    t = torch.empty(a.shape, dtype=a.dtype, pin_memory=True)
    t.copy_(a)
    return t.numpy()


def _inputs(case, seed):
    """What a case's calls read, from the seed alone, on the GPU in 64 bits (or as the call takes it)."""
    rng = np.random.default_rng([seed, 11])
    kind = case["kind"]
    v = {}
    if kind != "flow":
        v["degree"], v["radius"], xyz = _points(case, rng)
        v["xyz"] = xyz
        v["X"] = [torch.from_numpy(a).cuda() for a in xyz]
    td = torch.float64 if case["fp64"] else torch.float32
    if kind in ("step", "graph", "subs"):
        v["u"] = _fields(case, rng, 3, td)
    if kind == "indicator":
        v["F"] = _fields(case, rng, 2, torch.float64)  # the forces that the centrifugal terms join
        v["nrm"] = _radial_normals(case, v)
    if kind in ("flow", "loop"):
        u = _fields(case, rng, 3, torch.float64)
        _walls(u)
        v["u0"] = u
    if kind == "flow":
        old = [0.98 * f for f in u]
        v["u1"] = old
        v["p0"] = _boundp(_fields(case, rng, 1, torch.float64, wall=False)[0])
        v["F"] = _fields(case, rng, 3, torch.float64, amp=0.5, wall=False)
    return v


def _radial_normals(case, v):
    """Inward unit normals and areas of the points, as the sphere of the same centre has them."""
    n, off = [], 0
    for L, R in zip(v["degree"], v["radius"]):
        m = 8 * (int(L) + 1) ** 2
        p = v["xyz"][:, off:off + m]
        d = p - p.mean(1, keepdims=True)
        r = np.sqrt((d * d).sum(0))
        _, w = _gauss(2 * (int(L) + 1))
        area = r * r * np.repeat(w, 4 * (int(L) + 1)) * (2 * math.pi / (4 * (int(L) + 1)))
        n.append(np.concatenate([-d / r, area[None]], 0))
        off += m
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in np.concatenate(n, 1)]


def prepare(case, seed):
    kind, grid = case["kind"], _grid(case)
    v = _inputs(case, seed)
    if kind == "loop":
        deg, rad, xyz = v["degree"], v["radius"], v["xyz"]
        wl = workloads.Workload("loop", grid, deg, rad, np.zeros((deg.size, 3)), *xyz, modes={}, shear=0.0)
        # a step this short leaves the suspension in place over many passes
        solver = IBSolver(wl, 1e-6, FLOW["rep"], [f.cpu().numpy() for f in v["u0"]], indicator=IND)
        torch.cuda.synchronize()
        return {"case": case, "solver": solver}
    st = torch.cuda.Stream()
    degree = v.get("degree", np.zeros(0, np.int32))
    cs = CouplingStep(grid, degree, v.get("radius", np.zeros(0)), 1.0, 1.0,
                      precision="fp64" if case["fp64"] else "mixed", mem="host" if case["host"] else "device",
                      stream=st.cuda_stream, async_=not case["host"])
    s = {"case": case, "cs": cs, "stream": st}
    if kind in ("step", "graph", "subs"):
        if case["law"]:
            cs.set_capsule_law([case["law"]] * degree.size)
        if case["bend"]:
            cs.set_capsule_bending(CBEND * v["radius"] ** 2)
        td = v["u"][0].dtype
        lag = [torch.zeros(v["X"][0].numel(), dtype=td, device="cuda") for _ in range(10)]
        eul = [torch.zeros_like(v["u"][0]) for _ in range(3)]
        s.update(X=v["X"], u=v["u"], lag=lag, eul=eul)
        if case["host"]:
            for k in ("X", "u", "lag", "eul"):
                s[k] = [_pinned(a) for a in s[k]]
        torch.cuda.synchronize()
        if kind == "graph":
            cs.step(*s["u"], *s["X"], lag_out=s["lag"], eul_out=s["eul"])
            cs.synchronize()
            cs.graph_capture(*s["u"], *s["X"], s["lag"], s["eul"])
    elif kind == "indicator":
        cs.set_indicator_params(**IND)
        s.update(X=v["X"], nrm=v["nrm"], F=v["F"], fyz=[torch.empty_like(f) for f in v["F"]],
                 out=[torch.empty_like(v["F"][0]) for _ in range(2)])
    else:
        cs.set_flow_params(FLOW["rep"], FLOW["vb2"], FLOW["vt2"])
        s.update(uo=v["u0"], uoo=v["u1"], p0=v["p0"], p=torch.empty_like(v["p0"]), F=v["F"],
                 out=[torch.zeros_like(v["p0"]) for _ in range(3)])
    torch.cuda.synchronize()
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind == "loop":
        o = s["solver"]
        o.step()
        return {"X": o.X, "u": o.u, "p": o.p, "force": o.force, "lag": o.lag, "ind": o.ind}
    cs = s["cs"]
    if kind == "step":
        return cs.step(*s["u"], *s["X"], lag_out=s["lag"], eul_out=s["eul"])
    if kind == "graph":
        cs.graph_launch()
        L = s["lag"]
        return dict(u=L[0:3], f=L[3:6], n=L[6:9], area=L[9], fgrid=s["eul"])
    if kind == "subs":
        L = s["lag"]
        cs.eulr2lagr(*s["u"], *s["X"], out=L[0:3])
        cs.complagrforces(*s["X"], out=L[3:10])
        cs.lagr2eulr(*s["X"], *L[3:6], L[9], out=s["eul"])
        return dict(u=L[0:3], f=L[3:6], n=L[6:9], area=L[9], fgrid=s["eul"])
    with torch.cuda.stream(s["stream"]):
        if kind == "indicator":
            for a, b in zip(s["fyz"], s["F"]):  # the spread's forces, which the call adds to
                a.copy_(b)
            cs.indicator(*s["X"], *s["nrm"], fy=s["fyz"][0], fz=s["fyz"][1], out=s["out"])
            return {"ind": s["out"], "fyz": s["fyz"]}
        s["p"].copy_(s["p0"])  # the call updates the pressure in place
        cs.flow_step(FLOW["dt"], *s["uo"], *s["uoo"], s["p"], *s["F"], out=s["out"])
        return {"u": s["out"], "p": s["p"]}


# ------------------------------------------------------------------ work
def work(case):
    kind = case["kind"]
    cells = (case["itot"] + 2) * (case["jtot"] + 2) * (case["ktot"] + 2)
    e = 8 if case["fp64"] else 4
    N = _degrees(case).astype(float) + 1
    pts = float((8 * N * N).sum()) if kind != "flow" else 0.0
    fft = 2.5 * cells * math.log2(case["itot"] * case["jtot"])  # real 2-D transform, one direction
    # one Legendre transform of one field of one capsule; 6 in, 18 + 12 (bending) out, 6 + 8 + 6 + 4 + 14 after
    leg = float((4 * N ** 3).sum())
    step = {"bytes": pts * (24 + 10 * e) + 3 * e * (cells + min(cells, 27 * pts)),
            "flops": pts * (2 * 3 * 27 * 2 + 800) + leg * (56 + (12 if case["bend"] else 0))}
    flow = {"bytes": 8 * cells * 14, "flops": 8 * fft + cells * 150}
    ind = {"bytes": pts * 56 + 8 * cells * 6, "flops": 2 * fft + pts * 3 * 27 * 2 + cells * 20}
    if kind == "flow":
        return flow
    if kind == "indicator":
        return ind
    if kind == "loop":
        return {k: step[k] + flow[k] + ind[k] for k in step}
    return step


# ------------------------------------------------------------------ 64-bit results
def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return np.arccos(x)[::-1].copy(), w[::-1].copy()


class _Harmonics:
    """Spherical-harmonic series of degree < N on nlat Gauss latitudes x nlon longitudes, with the
    first `nder` theta derivatives; f = sum' P (a cos m phi - b sin m phi), half weight on m = 0."""

    def __init__(self, N, nlat, nlon, dev, nder):
        th, w = _gauss(nlat)
        x, s = np.cos(th), np.sin(th)
        M = N + nder + 1
        P = np.zeros((M, N, nlat))
        pmm = np.full(nlat, math.sqrt(0.5))
        for m in range(N):
            if m:
                pmm = pmm * math.sqrt((2 * m + 1) / (2 * m)) * s
            P[m, m] = pmm
            if m + 1 < N:
                P[m, m + 1] = math.sqrt(2 * m + 3) * x * pmm
            for n in range(m + 2, N):
                a = math.sqrt((4 * n * n - 1) / (n * n - m * m))
                b = math.sqrt(((n - 1) ** 2 - m * m) / (4 * (n - 1) ** 2 - 1))
                P[m, n] = a * (x * P[m, n - 1] - b * P[m, n - 2])
        m, n = np.arange(M)[:, None, None], np.arange(N)[None, :, None]
        up = np.sqrt(np.maximum((n + m + 1) * (n - m), 0.0))
        dn = np.sqrt(np.maximum((n + m) * (n - m + 1), 0.0))
        D = [P]
        for _ in range(nder):  # dP_m = (dn P_{m-1} - up P_{m+1}) / 2, -sqrt(n(n+1)) P_1 for m = 0
            q = np.zeros_like(P)
            f = D[-1]
            q[1:-1] = 0.5 * (dn[1:-1] * f[:-2] - up[1:-1] * f[2:])
            q[0] = -up[0] * f[1]
            D.append(q)
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
        self.N, self.nlat, self.nlon = N, nlat, nlon
        self.D = [t(d[:N]) for d in D]
        self.theta, self.w = t(th), t(w)
        self.phi = torch.arange(nlon, dtype=torch.float64, device=dev) * (2 * math.pi / nlon)
        mm = torch.arange(N, dtype=torch.float64, device=dev)
        self.half = torch.ones(N, dtype=torch.float64, device=dev)
        self.half[0] = 0.5
        self.m = mm
        self.cos, self.sin = torch.cos(mm[:, None] * self.phi), torch.sin(mm[:, None] * self.phi)

    def analyse(self, f):
        P = self.D[0] * self.w
        fc, fs = f @ self.cos.T * (2 / self.nlon), f @ self.sin.T * (-2 / self.nlon)
        return torch.einsum("...im,mni->...mn", fc, P), torch.einsum("...im,mni->...mn", fs, P)

    def synth(self, a, b, dt=0, dp=0):
        """The series with dt theta and dp phi derivatives."""
        ga = torch.einsum("...mn,mni->...im", a, self.D[dt]) * self.half
        gb = torch.einsum("...mn,mni->...im", b, self.D[dt]) * self.half
        c, s = self.cos, self.sin
        k = self.m[:, None]
        for _ in range(dp):
            c, s = -k * s, k * c
        return ga @ c - gb @ s


class _Jet:
    """A function of (theta, phi) with its derivatives (f, t, p, tt, tp, pp) at every point."""

    def __init__(self, d):
        self.d = list(d)

    def __add__(self, o):
        return _Jet([a + b for a, b in zip(self.d, o.d)])

    def __sub__(self, o):
        return _Jet([a - b for a, b in zip(self.d, o.d)])

    def __mul__(self, o):
        if not isinstance(o, _Jet):
            return _Jet([a * o for a in self.d])
        f, ft, fp, ftt, ftp, fpp = self.d
        g, gt, gp, gtt, gtp, gpp = o.d
        return _Jet([f * g, ft * g + f * gt, fp * g + f * gp, ftt * g + 2 * ft * gt + f * gtt,
                     ftp * g + ft * gp + fp * gt + f * gtp, fpp * g + 2 * fp * gp + f * gpp])

    def chain(self, h, h1, h2):
        """h(self) from h and its first two derivatives at self."""
        f, ft, fp, ftt, ftp, fpp = self.d
        return _Jet([h, h1 * ft, h1 * fp, h1 * ftt + h2 * ft * ft, h1 * ftp + h2 * ft * fp, h1 * fpp + h2 * fp * fp])

    def power(self, e):
        f = self.d[0]
        return self.chain(f ** e, e * f ** (e - 1), e * (e - 1) * f ** (e - 2))


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _cross(a, b):
    return [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]


def _surface_force(x, th, R, gs, csk, law, eb):
    """Force per area and unit normal from the derivatives x(dt, dp) (lists of 3) of the surface:
    f = (T^ab_,a + G^c_ca T^ab) a_b + T^ab x_ab with the membrane tension T of the law, and with a
    bending modulus eb the transverse shear of the moment M^ba = eb a^bg (A^ga B_gg - a^ga b_gg)."""
    top = 4 if eb is not None else 2
    zero = torch.zeros_like(x(0, 0)[0])
    get = lambda i, j: x(i, j) if i + j <= top else [zero] * 3
    jet = lambda i, j: [_Jet(v) for v in zip(get(i, j), get(i + 1, j), get(i, j + 1), get(i + 2, j),
                                             get(i + 1, j + 1), get(i, j + 2))]
    a = [jet(1, 0), jet(0, 1)]
    xab = [[jet(2, 0), jet(1, 1)], [jet(1, 1), jet(0, 2)]]
    g = [[_dot(a[i], a[j]) for j in range(2)] for i in range(2)]
    det = g[0][0] * g[1][1] - g[0][1] * g[0][1]
    inv = det.power(-1.0)
    con = [[g[1][1] * inv, g[0][1] * inv * -1.0], [g[0][1] * inv * -1.0, g[0][0] * inv]]
    up = [[con[i][0] * a[0][c] + con[i][1] * a[1][c] for c in range(3)] for i in range(2)]
    isq = det.power(-0.5)
    n = [c * isq for c in _cross(a[0], a[1])]
    b = [[_dot(n, xab[i][j]) for j in range(2)] for i in range(2)]
    # the reference sphere: A^11 = 1/R^2, A^22 = 1/(R sin t)^2, B_11 = R, B_22 = R sin^2 t
    s, c = torch.sin(th)[:, None] + zero, torch.cos(th)[:, None] + zero
    sin = _Jet([s, c, zero, -s, zero, zero])
    one = _Jet([zero + 1.0] + [zero] * 5)
    A = [one * (1 / R ** 2), (sin * sin).power(-1.0) * (1 / R ** 2)]
    B = [one * R, sin * sin * R]
    J2 = A[0] * A[1] * det
    J = J2.power(0.5)
    I1 = A[0] * g[0][0] + A[1] * g[1][1] - one * 2.0
    hf = 0.5 * gs
    if law:  # neo-Hookean
        W1, W2 = one * hf, J2.power(-2.0) * -hf
    else:
        W1, W2 = (one + I1) * hf, ((J2 - one) * csk - one) * hf
    t1, t2 = W1 * J.power(-1.0) * 2.0, J * W2 * 2.0
    T = [[t1 * A[i] + t2 * con[i][j] if i == j else t2 * con[i][j] for j in range(2)] for i in range(2)]
    V = lambda q: q.d[0]
    D = lambda q, i: q.d[1 + i]
    gam = [D(det, i) / (2 * V(det)) for i in range(2)]  # G^c_ci
    f = [zero] * 3
    for i in range(2):
        for j in range(2):
            for k in range(3):
                f[k] = f[k] + (D(T[i][j], i) + gam[i] * V(T[i][j])) * V(a[j][k]) + V(T[i][j]) * V(xab[i][j][k])
    normal = [V(q) for q in n]
    if eb is None:
        return f, normal
    G = [[[_dot(xab[i][j], up[k]) for j in range(2)] for i in range(2)] for k in range(2)]  # G[k][i][j] = G^k_ij
    raw = [[sum((con[be][q] * ((A[al] * B[al] if q == al else one * 0.0)
                               - (con[0][al] * b[q][0] + con[1][al] * b[q][1])) for q in range(2)), one * 0.0)
            for al in range(2)] for be in range(2)]
    raw = [[q * eb for q in r] for r in raw]
    second = sum(raw[be][al].d[(3, 4, 5)[be + al]] for be in range(2) for al in range(2))
    M = [[raw[0][0], raw[1][0]], [raw[1][0], raw[1][1]]]
    Q = [zero, zero]
    div = second
    for be in range(2):
        for al in range(2):
            Q[be] = Q[be] + D(M[be][al], al)
            for lm in range(2):
                for gm, mm in ((G[al][al][lm], M[be][lm]), (G[be][al][lm], M[lm][al])):
                    Q[be] = Q[be] + V(gm) * V(mm)
                    div = div + D(gm, be) * V(mm) + V(gm) * D(mm, be)
    for be in range(2):
        for lm in range(2):
            div = div + Q[lm] * V(G[be][be][lm])
    mixed = [[V(con[0][al]) * V(b[be][0]) + V(con[1][al]) * V(b[be][1]) for al in range(2)] for be in range(2)]
    for k in range(3):
        for al in range(2):
            f[k] = f[k] - (mixed[0][al] * Q[0] + mixed[1][al] * Q[1]) * V(a[al][k])
        f[k] = f[k] + div * normal[k]
    return f, normal


def _membrane(degree, radius, X, law, bend):
    """complagrforces: force, normals and area of every point, 64 bits."""
    dev = X[0].device
    out = torch.zeros(7, X[0].numel(), dtype=torch.float64, device=dev)
    off = np.concatenate([[0], np.cumsum(8 * (degree.astype(np.int64) + 1) ** 2)])
    for L in np.unique(degree):
        N = int(L) + 1
        caps = np.flatnonzero(degree == L)
        big, small = _Harmonics(N, 2 * N, 4 * N, dev, 4 if bend else 2), _Harmonics(N, N, 2 * N, dev, 1)
        idx = torch.from_numpy(off[caps][:, None] + np.arange(8 * N * N)[None]).to(dev)
        R = torch.from_numpy(radius[caps]).to(dev)[:, None, None]

        def sphere(sh, dt, dp):
            t, p = sh.theta[:, None] + dt * math.pi / 2, sh.phi[None, :] + dp * math.pi / 2
            flat = torch.cos(t) + 0 * p if dp == 0 else torch.zeros_like(t + p)
            return [R * q for q in (torch.sin(t) * torch.sin(p), torch.sin(t) * torch.cos(p), flat)]

        ref = sphere(big, 0, 0)
        co = []
        for c in range(3):
            x = X[c][idx]
            x = (x - x.mean(1, keepdim=True)).reshape(-1, 2 * N, 4 * N)
            co.append(big.analyse(x - ref[c]))
        shape = lambda sh, i, j: [sh.synth(*co[c], i, j) + q for c, q in enumerate(sphere(sh, i, j))]
        seen = {}

        def deriv(i, j):
            if (i, j) not in seen:
                seen[i, j] = shape(big, i, j)
            return seen[i, j]

        eb = CBEND * R ** 2 if bend else None
        f, n = _surface_force(deriv, big.theta, R, 1.0, 1.0, law, eb)
        res = [big.synth(*big.analyse(q)) for q in f]
        # normals and surface metric pass through the coarser grid of 2N longitudes
        nv = [small.synth(*big.analyse(q)) for q in n]
        r = torch.sqrt(_dot(nv, nv))
        cr = _cross(shape(small, 1, 0), shape(small, 0, 1))
        for q in [nv[0] / r, nv[1] / r, nv[2] / r, torch.sqrt(_dot(cr, cr))]:
            res.append(big.synth(*small.analyse(q)))
        res[6] = res[6] * (big.w / torch.sin(big.theta) * (2 * math.pi / (4 * N)))[:, None]
        for q in range(7):
            out[q][idx.reshape(-1)] = res[q].reshape(-1)
    return list(out)


def _delta(r):
    r = r.abs()
    inner = (1 + torch.sqrt(torch.clamp(1 - 3 * r * r, min=0.0))) / 3
    outer = (5 - 3 * r - torch.sqrt(torch.clamp(1 - 3 * (1 - r) ** 2, min=0.0))) / 6
    return torch.where(r <= 0.5, inner, torch.where(r <= 1.5, outer, torch.zeros_like(r)))


def _stencil(grid, X, comp, halo=False):
    """Indices and weights [npts, 3, 3, 3] of component comp's nodes (comp < 0: cell centres);
    halo: the z window reaches the wall halo planes."""
    n, d = grid[:3], grid[3:]
    idx, wgt = [], []
    for q in range(3):
        s = X[q] / d[q] + (0.0 if q == comp else 0.5)  # node i sits at i (face) or i - 1/2 (centre)
        near = torch.floor(s + 0.5)
        i = near[:, None] + torch.arange(-1, 2, dtype=torch.float64, device=s.device)
        w = _delta(i - s[:, None])
        i = i.long()
        if q < 2:
            i = (i - 1) % n[q] + 1
        else:
            lo, hi = (0, n[2] + 1) if halo else (1, n[2])
            w = torch.where((i >= lo) & (i <= hi), w, torch.zeros_like(w))
            i = i.clamp(lo, hi)
        idx.append(i)
        wgt.append(w)
    flat = (idx[2][:, :, None, None] * (n[1] + 2) + idx[1][:, None, :, None]) * (n[0] + 2) + idx[0][:, None, None, :]
    return flat, wgt[2][:, :, None, None] * wgt[1][:, None, :, None] * wgt[0][:, None, None, :]


def _spread(grid, X, F, area, centred=False):
    out = []
    s = area / (grid[3] * grid[4] * grid[5])
    for c in range(3):
        g = torch.zeros((grid[2] + 2, grid[1] + 2, grid[0] + 2), dtype=torch.float64, device=area.device)
        flat, w = _stencil(grid, X, -1 if centred else c, halo=centred)
        g.view(-1).index_add_(0, flat.reshape(-1), (w * (F[c] * s)[:, None, None, None]).reshape(-1))
        out.append(_periodic(g))
    return out


def _walls(u, vb2=0.0, vt2=0.0):
    """bounduvw: no-slip walls (v: wall values), then the periodic copies."""
    u[0][0], u[0][-1] = -u[0][1], -u[0][-2]
    u[1][0], u[1][-1] = vb2 - u[1][1], vt2 - u[1][-2]
    u[2][0] = 0.0
    u[2][-2] = 0.0
    u[2][-1] = u[2][-3]
    for f in u:
        _periodic(f)


def _boundp(f):
    f[0], f[-1] = f[1].clone(), f[-2].clone()
    return _periodic(f)


def _poisson(rhs, d, rows, shift):
    """(Laplacian - shift) x = rhs, periodic x and y, z rows: 1 Neumann, 2 no-slip cell values, 3 w."""
    nz, ny, nx = rhs.shape
    dev = rhs.device
    kx = torch.arange(nx // 2 + 1, dtype=torch.float64, device=dev)
    ky = torch.arange(ny, dtype=torch.float64, device=dev)
    lam = (-4 / d[1] ** 2 * torch.sin(math.pi * ky / ny) ** 2)[:, None] - 4 / d[0] ** 2 * torch.sin(math.pi * kx / nx) ** 2
    p = torch.fft.rfft2(rhs)
    e = 1 / d[2] ** 2
    lower, upper, diag = [e] * nz, [e] * nz, [lam - 2 * e - shift] * nz
    lower[0] = upper[-1] = 0.0
    if rows == 3:
        lower[-1], diag[-1] = 0.0, torch.ones_like(lam)
    else:
        diag[0] = diag[0] + (e if rows == 1 else -e)
        diag[-1] = diag[-1] + (e if rows == 1 else -e)
    cp = [upper[0] / diag[0]]
    q = [p[0] / diag[0]]
    for k in range(1, nz):
        piv = diag[k] - lower[k] * cp[-1]
        if rows == 1 and k == nz - 1:  # the mean's free constant: zero in the top row
            piv[0, 0] = 1.0
        cp.append(upper[k] / piv)
        q.append((p[k] - lower[k] * q[-1]) / piv)
    if rows == 1:
        q[-1][0, 0] = 0.0
    for k in range(nz - 2, -1, -1):
        q[k] = q[k] - cp[k] * q[k + 1]
    return torch.fft.irfft2(torch.stack(q), s=(ny, nx))


def _flow(case, v):
    d = _grid(case)[3:]
    dt, rep = FLOW["dt"], FLOW["rep"]

    def at(f, dx=0, dy=0, dz=0):
        z, y, x = f.shape
        return f[1 + dz:z - 1 + dz, 1 + dy:y - 1 + dy, 1 + dx:x - 1 + dx]

    step = [dict(dx=1), dict(dy=1), dict(dz=1)]
    axis = ("dx", "dy", "dz")

    def advect(u, c):
        """Divergence of the face fluxes of component c: mean of u_c across each face times the mean
        of the carrying velocity."""
        total = 0
        for q in range(3):
            for side in (0, -1):  # the upper and the lower face in direction q
                at_side = lambda f, **o: at(f, **{**dict.fromkeys(axis, 0), **o})
                if q == c:
                    far = {axis[q]: 1 if side == 0 else -1}
                    m = 0.5 * (at_side(u[c]) + at_side(u[c], **far))
                    flux = m * m
                else:
                    o = {axis[q]: side}
                    near = {axis[q]: 1 if side == 0 else -1}
                    carried = 0.5 * (at_side(u[c]) + at_side(u[c], **near))
                    carrier = 0.5 * (at_side(u[q], **o) + at_side(u[q], **o, **step[c]))
                    flux = carried * carrier
                total = total + (flux if side == 0 else -flux) / d[q]
        return total

    u, p = [], v["p0"].clone()
    for c in range(3):
        r = (at(p, **step[c]) - at(p)) / d[c] - at(v["F"][c])
        r = r + 1.5 * advect(v["u0"], c) - 0.5 * advect(v["u1"], c) - at(v["u0"][c]) / dt
        r = r * rep
        if c == 2:
            r[-1] = 0.0
        f = torch.zeros_like(p)
        f[1:-1, 1:-1, 1:-1] = _poisson(r, d, 3 if c == 2 else 2, rep / dt)
        u.append(f)
    _walls(u)
    div = sum((at(u[c]) - at(u[c], **{axis[c]: -1})) / d[c] for c in range(3)) / dt
    q = torch.zeros_like(p)
    q[1:-1, 1:-1, 1:-1] = _poisson(div, d, 1, 0.0)
    _boundp(q)
    for c in range(3):
        u[c][1:-1, 1:-1, 1:-1] -= dt / d[c] * (at(q, **step[c]) - at(q))
    _walls(u)
    return {"u": u, "p": _boundp(p + q)}


def _indicator(case, v):
    grid = _grid(case)
    d, nz = grid[3:], grid[2]
    q = nz // 4
    X = [v["X"][0], v["X"][1], v["X"][2] + q * d[2]]
    g = _spread(grid, X, v["nrm"][:3], v["nrm"][3], centred=True)
    div = ((g[0][1:-1, 1:-1, 2:] - g[0][1:-1, 1:-1, :-2]) / (2 * d[0])
           + (g[1][1:-1, 2:, 1:-1] - g[1][1:-1, :-2, 1:-1]) / (2 * d[1])
           + (g[2][2:, 1:-1, 1:-1] - g[2][:-2, 1:-1, 1:-1]) / (2 * d[2]))
    sol = _poisson(div, d, 1, 0.0)
    ind = torch.zeros_like(g[0])
    ind[1:nz - q + 1, 1:-1, 1:-1] = sol[q:]
    _boundp(ind)
    inner = ind[1:-1, 1:-1, 1:-1]
    inner[inner < 0.01] = 0.0
    inner[inner >= 0.9] = 1.0
    visc = torch.zeros_like(ind)
    visc[1:-1, 1:-1, 1:-1] = IND["visc0"] * (1 + (IND["lam"] - 1) * inner)
    _boundp(visc)
    amp = (IND["ta"] / IND["rep"] ** 2) ** 0.25
    fy, fz = v["F"][0].clone(), v["F"][1].clone()
    fy[1:-1, 1:-1, 1:-1] += 0.5 * (inner + ind[1:-1, 2:, 1:-1]) * math.sin(IND["thetainc"]) * amp
    fz[1:-1, 1:-1, 1:-1] += 0.5 * (inner + ind[2:, 1:-1, 1:-1]) * -math.cos(IND["thetainc"]) * amp
    return {"ind": [ind, visc], "fyz": [fy, fz]}


def exact(case, seed):
    """The outputs of one pass in 64 bits; None for the coupled loop, whose state a pass moves on."""
    if case["kind"] == "loop":
        return None
    v = _inputs(case, seed)
    if case["kind"] == "flow":
        return _flow(case, v)
    if case["kind"] == "indicator":
        return _indicator(case, v)
    grid = _grid(case)
    u = []
    for c in range(3):
        flat, w = _stencil(grid, v["X"], c)
        u.append((v["u"][c].double().reshape(-1)[flat.reshape(-1)].reshape(w.shape) * w).sum((1, 2, 3)))
    m = _membrane(v["degree"], v["radius"], v["X"], case["law"], case["bend"])
    return dict(u=u, f=m[0:3], n=m[3:6], area=m[6], fgrid=_spread(grid, v["X"], m[0:3], m[6]))

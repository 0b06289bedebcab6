"""Performance cases: the work a user of the library has it do, through its
public Python classes (nlmech_gb300.gpu), over the range of sizes that the
benchmark workloads, the decks and the tests span.

A case is a dict of plain values; listed() gives the fixed ones, draw() gives
others of the same ranges.  prepare() builds the specimen and the model handle
a program keeps, run() makes one pass, work() counts the bytes and operations
a pass cannot do without, exact() computes the pass in 64 bits with plain
torch, straight from the peridynamic formulas.

An explicit pass is a run of some hundred to some thousand time steps followed
by the read-back of the fields, as between two outputs of a simulation.  Loads
are slow and initial velocities small enough that no bond breaks beyond the
pre-crack, so that a pass costs the same however often it is repeated.
Compensated-FP32 models hold forces in FP32; a program that picks them stores
its output fields in single precision, and so does run().
"""
import math

import numpy as np
import torch

from nlmech_gb300 import abi, configs, gpu
from nlmech_gb300.decks import BC, MaterialDeck, Problem

FP32C, FP64 = "fp32c", "fp64"


def listed():
    return [
        # 2-D RNPBond plate of 10,000 nodes at horizon 4h, 1000 Verlet steps: the
        # smallest run in daily use (parameter studies); bound by per-step latency
        dict(name="plate_100_fp32c", kind="plate", precision=FP32C, nx=100, ny=100, ratio=4,
             steps=1000, scheme="verlet", loads=False, damage=False),
        # the headline workload: 1000 x 1000 plate at horizon 3h, its whole run
        dict(name="plate_1000_fp32c", kind="plate", precision=FP32C, nx=1000, ny=1000, ratio=3,
             steps=5000, scheme="verlet", loads=False, damage=False),
        # a plate of odd sides, central differences, a force load and a no-fail rim
        dict(name="plate_ragged_fp32c_cd", kind="plate", precision=FP32C, nx=613, ny=347,
             ratio=4, steps=800, scheme="central", loads=True, damage=False),
        # FP64, the default precision, with the damage field of an output step
        dict(name="plate_320_fp64", kind="plate", precision=FP64, nx=320, ny=250, ratio=3,
             steps=100, scheme="verlet", loads=False, damage=True),
        # 3-D ElasticState cube with a notch, one million nodes
        dict(name="cube_100_fp32c", kind="cube", precision=FP32C, nx=100, ny=100, nz=100,
             steps=300, damage=False),
        # 3-D ElasticState block of odd sides in FP64
        dict(name="cube_31_fp64", kind="cube", precision=FP64, nx=31, ny=29, nz=27, steps=40,
             damage=True),
        # an ensemble of plates of uneven size stepped together
        dict(name="ensemble_16", kind="ensemble", plates=16, nmin=5000, nmax=100000, ratio=4,
             steps=1000),
        # host-resident step: u, v, f copied in and out of pinned memory every step
        dict(name="host_step_1000", kind="host_step", nx=1000, ny=1000, ratio=3),
        # one quasi-static load step of the 200 x 200 RNPBond plate (Newton + PCG)
        dict(name="qs_plate_200", kind="qs", nx=200),
        # one quasi-static load step of an ElasticState plate (Newton, difference
        # Jacobian, BiCGSTAB)
        dict(name="esqs_plate_40", kind="esqs", nx=40, ny=36),
        # the horizon neighbour search on its own: host coordinates in, rows out
        dict(name="neighbors_700x500", kind="neighbors", dim=2, nx=700, ny=500, nz=1,
             ratio=4.36),
        # start prediction of the learned quasi-static solver for a 200 x 200 plate
        dict(name="mlp_forward_40k", kind="mlp", rows=40000, hidden=128, layers=3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _even(v):
    return max(2, int(v) // 2 * 2)


def draw(rng):
    kind = rng.choice(["plate", "plate", "plate64", "cube", "cube64", "ensemble", "host_step",
                       "qs", "esqs", "neighbors", "mlp"])
    if kind == "plate":
        nx, ny = _log_int(rng, 48, 950), _log_int(rng, 48, 950)
        steps = _even(min(2000, 1.5e9 / (nx * ny), rng.uniform(200, 2000)))
        return dict(kind="plate", precision=FP32C, nx=nx, ny=ny, ratio=rng.choice([3, 4]),
                    steps=steps, scheme=rng.choice(["verlet", "verlet", "central"]),
                    loads=rng.random() < 0.4, damage=rng.random() < 0.3)
    if kind == "plate64":
        nx, ny = _log_int(rng, 40, 600), _log_int(rng, 40, 600)
        return dict(kind="plate", precision=FP64, nx=nx, ny=ny, ratio=rng.choice([3, 4]),
                    steps=_even(max(10, min(200, 8e6 / (nx * ny)))),
                    scheme=rng.choice(["verlet", "verlet", "central"]),
                    loads=rng.random() < 0.4, damage=rng.random() < 0.5)
    if kind == "cube":
        n = [_log_int(rng, 20, 100) for _ in range(3)]
        return dict(kind="cube", precision=FP32C, nx=n[0], ny=n[1], nz=n[2],
                    steps=_even(max(20, min(300, 1e8 / (n[0] * n[1] * n[2])))),
                    damage=rng.random() < 0.3)
    if kind == "cube64":
        n = [_log_int(rng, 12, 44) for _ in range(3)]
        return dict(kind="cube", precision=FP64, nx=n[0], ny=n[1], nz=n[2],
                    steps=_even(max(10, min(100, 1e6 / (n[0] * n[1] * n[2])))),
                    damage=rng.random() < 0.5)
    if kind == "ensemble":
        nmin = _log_int(rng, 2000, 8000)
        return dict(kind="ensemble", plates=rng.randint(4, 18), nmin=nmin,
                    nmax=_log_int(rng, 20000, 100000), ratio=rng.choice([3, 4]),
                    steps=_even(rng.uniform(100, 800)))
    if kind == "host_step":
        return dict(kind="host_step", nx=_log_int(rng, 100, 1000), ny=_log_int(rng, 100, 1000),
                    ratio=rng.choice([3, 4]))
    if kind == "qs":
        return dict(kind="qs", nx=_log_int(rng, 60, 240))
    if kind == "esqs":
        return dict(kind="esqs", nx=rng.randint(12, 40), ny=rng.randint(10, 36))
    if kind == "neighbors":
        if rng.random() < 0.5:
            return dict(kind="neighbors", dim=2, nx=_log_int(rng, 60, 700),
                        ny=_log_int(rng, 60, 500), nz=1, ratio=rng.choice([3.4, 4.36]))
        return dict(kind="neighbors", dim=3, nx=_log_int(rng, 12, 48), ny=_log_int(rng, 12, 48),
                    nz=_log_int(rng, 12, 48), ratio=3.39)
    return dict(kind="mlp", rows=_log_int(rng, 500, 120000), hidden=rng.choice([64, 128]),
                layers=rng.choice([2, 3]))


# ---- specimens -------------------------------------------------------------

def _waves(x, rng, amp, dim):
    """A seeded smooth velocity field: four sine modes per component."""
    L = x.max(axis=0) + 1e-30
    v = np.zeros_like(x)
    for d in range(dim):
        for _ in range(4):
            k = rng.integers(1, 5, size=dim)
            ph = rng.uniform(0, 2 * math.pi)
            arg = sum(math.pi * int(k[c]) * x[:, c] / L[c] for c in range(dim)) + ph
            v[:, d] += amp / 4 * np.sin(arg)
    return v


def _plate(nx, ny, ratio, h, dt, seed, loads=False):
    rng = np.random.default_rng(seed + 77)
    crack = float(rng.uniform(0.1, 0.3)) * nx * h
    p = configs.rnp_plate(nx, h, ratio, crack, 2e-4, dt, 1, seed=seed, ny=ny)
    p.v0 = _waves(p.x, rng, 0.01, 2)
    if loads:
        H = ny * h
        p.fbc = [BC(region="rectangle", x1=-h, x2=nx // 10 * h, y1=-h, y2=H + h, direction=[1],
                    time_fn="linear", time_params=[-1e11], spatial_fn="constant",
                    spatial_params=[1.0])]
        p.no_fail = abi.NOFAIL_COMPUTE
        p.no_fail_tol = (2 * ratio + 0.25) * h
    return p


def _problem(case, seed):
    k = case["kind"]
    if k == "plate":
        return _plate(case["nx"], case["ny"], case["ratio"], 0.1 / max(case["nx"], case["ny"]),
                      2e-6 / max(case["nx"], case["ny"]), seed, case["loads"])
    if k == "host_step":
        return _plate(case["nx"], case["ny"], case["ratio"], 0.1 / max(case["nx"], case["ny"]),
                      2e-6 / max(case["nx"], case["ny"]), seed)
    if k == "cube":
        h = 1e-3
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        p = configs.elastic_state_cube(2, h, seed=seed)  # material, dt
        p.x, p.volume = configs.grid3d(nx, ny, nz, h, 0.05, seed)
        rng = np.random.default_rng(seed + 1)
        p.v0 = _waves(p.x, rng, 0.02, 3)
        ck = p.cracks[0]
        ck.z0, ck.lo, ck.hi = 0.5 * nz * h, (-h, -h), (0.5 * nx * h, ny * h + h)
        return p
    if k == "qs":
        rng = np.random.default_rng(seed + 5)
        c = (float(rng.uniform(0.35, 0.65)), float(rng.uniform(0.35, 0.65)))
        return configs.qs_plate(case["nx"], crack_frac=float(rng.uniform(0.1, 0.3)),
                                crack_center=c, du=1e-8, jitter=0.05, seed=seed)
    if k == "esqs":
        h, nx, ny = 0.1, case["nx"], case["ny"]
        x, vol = configs.grid2d(nx, ny, h, jitter=0.05, seed=seed)
        W, H = nx * h, ny * h
        mat = MaterialDeck(kind="ElasticState", density=1200.0, K=4000.0, G=1500.0)
        left = dict(region="rectangle", x1=-0.1 * h, x2=1.2 * h, y1=-0.1 * h, y2=H + h)
        right = dict(region="rectangle", x1=W - 1.2 * h, x2=W + 0.1 * h, y1=-0.1 * h, y2=H + h)
        one = dict(spatial_fn="constant", spatial_params=[1.0])
        ubc = [BC(direction=[1, 2], time_fn="constant", time_params=[0.0], **one, **left),
               BC(direction=[2], time_fn="linear", time_params=[0.05], **one, **right)]
        fbc = [BC(direction=[1], time_fn="linear", time_params=[1.0], spatial_fn="constant",
                  spatial_params=[-2.0], **right)]
        return Problem(dim=2, x=x, volume=vol, horizon=3 * h, mesh_size=h, material=mat,
                       ubc=ubc, fbc=fbc)
    raise ValueError(k)


def _ensemble(case, seed):
    rng = np.random.default_rng(seed)
    sizes = np.random.default_rng(case["plates"])  # the sizes belong to the case
    out = []
    for s in range(case["plates"]):
        n = int(sizes.integers(case["nmin"], case["nmax"] + 1))
        nx = max(8, int(round(math.sqrt(n))))
        out.append(_plate(nx, nx, case["ratio"], 0.1 / nx, 6e-9, int(rng.integers(1 << 30))))
    return out


def _esqs_dt():
    return 0.1


def _mlp_params(case, seed):
    """He-initialised weights in the nlm_mlp layout, zero padding."""
    rng = np.random.default_rng(seed + 9)
    n_in, n_h, n_l, n_out = 10, case["hidden"], case["layers"], 2
    lay = gpu.mlp_layout(n_in, n_h, n_l, n_out)
    live = [n_in] + [n_h] * n_l + [n_out]
    p = np.zeros(lay[-1][3] + lay[-1][1], dtype=np.float32)
    for l, (di, do, wo, bo) in enumerate(lay):
        w = np.zeros((di, do), dtype=np.float32)
        w[:live[l], :live[l + 1]] = rng.normal(0, math.sqrt(2 / live[l]),
                                               (live[l], live[l + 1]))
        p[wo:wo + di * do] = w.ravel()
        p[bo:bo + live[l + 1]] = rng.normal(0, 0.1, live[l + 1])
    return p, lay


def _mlp_rows(case, seed):
    rng = np.random.default_rng(seed)
    return rng.normal(0, 1, (case["rows"], 10)).astype(np.float32)


# ---- a pass ------------------------------------------------------------------

def prepare(case, seed):
    k = case["kind"]
    st = {"case": case}
    if k in ("plate", "cube"):
        p = _problem(case, seed)
        fp32 = case["precision"] == FP32C
        central = case.get("scheme") == "central"
        m = gpu.FDModel(p, precision=abi.FP32C if fp32 else abi.FP64,
                        scheme=abi.CENTRAL_DIFFERENCE if central else abi.VELOCITY_VERLET)
        m.set_graph(20)
        st["model"] = m
        if fp32:
            st["out"] = [np.zeros((p.n, 3), dtype=np.float32) for _ in range(3)]
    elif k == "ensemble":
        ps = _ensemble(case, seed)
        b = gpu.Batch(ps)
        b.set_graph(20)
        st["model"] = b
        st["out"] = [[np.zeros((p.n, 3), dtype=np.float32) for _ in range(3)] for p in ps]
    elif k == "host_step":
        p = _problem(case, seed)
        st["model"] = gpu.FDModel(p, precision=abi.FP32C)
        st["uvf"] = [torch.zeros((p.n, 3), dtype=torch.float64).pin_memory() for _ in range(3)]
        st["uvf"][1].copy_(torch.from_numpy(p.v0))
    elif k == "qs":
        # tolerance far below the benchmark's 1e-8, so that the converged state
        # is defined to the last digits whatever the Krylov iterates were
        st["model"] = gpu.QSModel(_problem(case, seed), gpu.qs_params(tol=1e-13))
    elif k == "esqs":
        prm = gpu.esqs_params(max_iters=50, tol=1e-9, tol_relative=True, jacobian=1,
                              dt=_esqs_dt())
        st["model"] = gpu.ESQSModel(_problem(case, seed), prm)
    elif k == "neighbors":
        # jitter and horizon leave the number of bonds fixed; the numbering
        # starts at a seeded node
        h = 1e-3
        if case["dim"] == 2:
            x, _ = configs.grid2d(case["nx"], case["ny"], h, 0.01, seed)
        else:
            x, _ = configs.grid3d(case["nx"], case["ny"], case["nz"], h, 0.01, seed)
        x = np.roll(x, int(np.random.default_rng(seed).integers(1, len(x))), axis=0)
        st.update(x=np.ascontiguousarray(x), horizon=case["ratio"] * h)
    elif k == "mlp":
        p, _ = _mlp_params(case, seed)
        m = gpu.MLP(10, case["hidden"], case["layers"], 2)
        m.set_params(p)
        st.update(model=m, x=_mlp_rows(case, seed))
    return st


def _single(fields, out):
    for a, o in zip(fields, out):
        np.copyto(o, a, casting="same_kind")
    return out


def run(state):
    case = state["case"]
    k = case["kind"]
    m = state.get("model")
    if k in ("plate", "cube"):
        m.run(case["steps"])
        f = m.state()
        if case["precision"] == FP32C:
            f = _single(f, state["out"])
        r = {"u": f[0], "v": f[1], "f": f[2], "broken": m.count_broken()}
        if case["damage"]:
            r["phi"], r["Z"] = m.damage()
        return r
    if k == "ensemble":
        m.run(case["steps"])
        return [_single(m.state(s), o) for s, o in enumerate(state["out"])]
    if k == "host_step":
        m.step_host_ptr(*[t.data_ptr() for t in state["uvf"]])
        return state["uvf"]
    if k == "qs":
        m.load_step()
        return m.state()
    if k == "esqs":
        m.solve(1)
        return list(m.get())
    if k == "neighbors":
        return list(gpu.neighbor_search(state["x"], state["horizon"], case["dim"]))
    return m.forward(state["x"])


# ---- compulsory work ---------------------------------------------------------

def _offsets(ratio, dim):
    """Lattice offsets within the horizon (jitter can reach a little past it)."""
    r = int(ratio)
    rng = range(-r, r + 1)
    lim = (ratio + 0.1 * math.sqrt(dim)) ** 2
    return [(a, b, c) for c in (rng if dim == 3 else (0,)) for b in rng for a in rng
            if (a, b, c) != (0, 0, 0) and a * a + b * b + c * c <= lim]


def _bonds(nx, ny, nz, ratio, dim):
    """Directed bonds of the lattice (half of those at the horizon itself)."""
    s = 0.0
    for a, b, c in _offsets(ratio, dim):
        w = 1.0 if a * a + b * b + c * c < ratio * ratio else 0.5
        if a * a + b * b + c * c > ratio * ratio:
            continue
        s += w * max(0, nx - abs(a)) * max(0, ny - abs(b)) * max(0, nz - abs(c))
    return s


def work(case):
    """Per explicit step: a neighbour id (4 B) and a bond bit per bond, and per
    node the position, volume and flags read and u, v, f read and written in
    the precision's own storage; about 30 operations per 2-D bond (plus one
    exponential) and 70 per ElasticState bond over both passes."""
    k = case["kind"]
    if k in ("plate", "host_step", "cube"):
        dim = 3 if k == "cube" else 2
        n = case["nx"] * case["ny"] * case.get("nz", 1)
        nb = _bonds(case["nx"], case["ny"], case.get("nz", 1), case.get("ratio", 3), dim)
        steps = case.get("steps", 1)
        w = 16.0 if case.get("precision") == FP64 else 8.0  # bytes per component: u + v
        f = 8.0 if case.get("precision") == FP64 else 4.0
        node = dim * 8 + 9 + 2 * dim * (w + f)
        host = 24.0 * n * 3  # u, v, f read back (or in and out)
        host *= 2 if k == "host_step" else 1
        return {"bytes": steps * (4.25 * nb * (2 if dim == 3 else 1) + node * n) + host,
                "flops": steps * nb * (70.0 if dim == 3 else 30.0)}
    if k == "ensemble":
        sizes = np.random.default_rng(case["plates"])
        b = f = 0.0
        for _ in range(case["plates"]):
            nx = max(8, int(round(math.sqrt(int(sizes.integers(case["nmin"],
                                                               case["nmax"] + 1))))))
            nb = _bonds(nx, nx, 1, case["ratio"], 2)
            b += case["steps"] * (4.25 * nb + 73.0 * nx * nx) + 72.0 * nx * nx
            f += case["steps"] * nb * 30.0
        return {"bytes": b, "flops": f}
    if k == "qs":
        # 4 Newton systems of about 2 nx PCG iterations: tangent block and id
        # per bond, five vectors per node
        n = case["nx"] ** 2
        nb = _bonds(case["nx"], case["nx"], 1, 3, 2)
        it = 4 * 2 * case["nx"]
        return {"bytes": it * (16.0 * nb + 40.0 * n), "flops": it * (8.0 * nb + 30.0 * n)}
    if k == "esqs":
        # 3 Newton systems: Jacobian blocks written once and read twice in each
        # of about 2 max(nx, ny) BiCGSTAB iterations
        n = case["nx"] * case["ny"]
        nb = _bonds(case["nx"], case["ny"], 1, 3, 2)
        it = 3 * 2 * max(case["nx"], case["ny"])
        return {"bytes": it * 2 * 36.0 * (nb + n), "flops": it * 2 * 8.0 * (nb + n)}
    if k == "neighbors":
        n = case["nx"] * case["ny"] * case["nz"]
        nb = _bonds(case["nx"], case["ny"], case["nz"], case["ratio"], case["dim"])
        return {"bytes": 24.0 * n + 8.0 * n + 4.0 * nb, "flops": 9.0 * nb}
    h, l = case["hidden"], case["layers"]
    par = 10 * h + (l - 1) * h * h + 2 * h
    return {"bytes": case["rows"] * 48.0 + 4.0 * par, "flops": 2.0 * par * case["rows"]}


# ---- the same in 64 bits, in plain torch ------------------------------------

def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _gt(a, b):
    """The reference's definitelyGreaterThan: a - b > 1e-5 max(|a|, |b|)."""
    return (a - b) > 1e-5 * torch.maximum(a.abs(), torch.as_tensor(b, dtype=a.dtype,
                                                                   device=a.device).abs())


class _Bonds:
    """Bonds of a jittered lattice as [offset, node] tables: neighbour index,
    whether the bond exists, bond vector, length and corrected volume."""

    def __init__(self, p, nx, ny, nz=1):
        dev = _dev()
        self.dim = dim = p.dim
        n = p.n
        x = torch.from_numpy(p.x).to(dev)
        self.x = [x[:, d].contiguous() for d in range(dim)]
        idn = torch.arange(n, device=dev)
        ix, iy, iz = idn % nx, (idn // nx) % ny, idn // (nx * ny)
        off = _offsets(round(p.horizon / p.mesh_size), dim)
        idx, ok = [], []
        for a, b, c in off:
            jx, jy, jz = ix + a, iy + b, iz + c
            o = (jx >= 0) & (jx < nx) & (jy >= 0) & (jy < ny) & (jz >= 0) & (jz < nz)
            idx.append(torch.where(o, (jz * ny + jy) * nx + jx, idn))
            ok.append(o)
        self.idx, ok = torch.stack(idx), torch.stack(ok)
        self.d = [xd[self.idx] - xd for xd in self.x]
        self.r = torch.sqrt(sum(d * d for d in self.d))
        rad = p.horizon + 1e-10
        self.mask = ok & ((rad - self.r) > 1e-5 * rad)
        self.r = torch.where(self.mask, self.r, torch.ones_like(self.r))
        self.vol = torch.from_numpy(p.volume).to(dev)
        self.h, self.delta = p.mesh_size, p.horizon
        corr = torch.where(_gt(self.r, torch.full_like(self.r, self.delta - 0.5 * self.h)),
                           (self.delta + 0.5 * self.h - self.r) / self.h,
                           torch.ones_like(self.r))
        self.w = torch.where(self.mask, self.vol[self.idx] * corr, torch.zeros_like(corr))
        self.alive = self.mask.clone()
        for c in p.cracks:
            if c.kind == "edge":  # horizontal: x within its span, y on either side
                X = self.x[0]
                inside = ~(_gt(torch.full_like(X, c.pb[0]), X) | _gt(X, c.pt[0]))
                up = self.x[1] >= c.pb[1]
                cut = inside & inside[self.idx] & (up != up[self.idx])
            else:
                z = self.x[2]
                t = (c.z0 - z) / torch.where(self.d[2] == 0, torch.ones_like(self.d[2]),
                                             self.d[2])
                px, py = self.x[0] + t * self.d[0], self.x[1] + t * self.d[1]
                cut = (((z < c.z0) != (z[self.idx] < c.z0)) & (px >= c.lo[0]) &
                       (px <= c.hi[0]) & (py >= c.lo[1]) & (py <= c.hi[1]))
            self.alive &= ~cut

    def diff(self, a):
        return [q[self.idx] - q for q in a]


class _RNP(_Bonds):
    """RNPBond with J = 1, plane stress: F = 4 J S C beta exp(-beta r S^2) /
    (pi delta^3) V e, broken where |S| exceeds sqrt(0.5 / (beta r))."""

    def __init__(self, p, *grid):
        super().__init__(p, *grid)
        m = p.material
        nu, J = 1.0 / 3.0, m.influence_params[0]
        lam = m.E * nu / ((1 + nu) * (1 - 2 * nu))
        M = J / (self.dim + 1)
        self.C = math.pi * m.Gc / (4 * M)
        self.beta = 4 * lam / (self.C * M)
        self.k = 4 * J * self.C * self.beta / (math.pi * self.delta ** 3) * self.w
        self.sc = math.sqrt(0.5 / self.beta) / torch.sqrt(self.r)
        self.rr = self.r * self.r
        self.e = [d / self.r for d in self.d]
        rim = torch.zeros_like(self.x[0], dtype=torch.bool)
        if p.no_fail:  # nodes near the bounding box, whose lower corner is the origin
            for d in range(2):
                q = self.x[d]
                rim |= (q < p.no_fail_tol) | (q > float(q.max()) - p.no_fail_tol)
        self.tough = rim | rim[self.idx]

    def strain(self, u):
        return sum(a * b for a, b in zip(self.d, self.diff(u))) / self.rr

    def force(self, u):
        S = self.strain(u)
        self.alive &= ~(_gt(S.abs(), self.sc) & ~self.tough)
        s = self.k * S
        s = torch.where(self.tough, s, s * torch.exp(-self.beta * self.r * S * S))
        s = torch.where(self.alive | (self.tough & self.mask), s, torch.zeros_like(s))
        return [(s * e).sum(0) for e in self.e]

    def damage(self, u):
        z = torch.where(self.mask, self.strain(u).abs() / self.sc, torch.zeros_like(self.r))
        return z.max(0).values


class _ES(_Bonds):
    """ElasticState in 3-D: t = (9 K / m) theta X / 3 + (15 G / m) (e - theta
    X / 3), f_i = sum (t_ij + t_ji) Y / |Y| V, broken where e / X > es_sc."""

    def __init__(self, p, *grid):
        super().__init__(p, *grid)
        m = p.material
        self.K, self.G, self.sc = m.K, m.G, m.es_sc
        self.m = (self.r * self.r * self.w).sum(0)
        if self.dim == 2:
            nu = (3 * m.K - 2 * m.G) / (2 * (3 * m.K + m.G))
            self.f2 = (2 * nu - 1) / (nu - 1)
            q = (nu + 1) / (2 * nu - 1)
            self.as_ = 9 / self.m * (m.K + q * q * m.G / 9)
            self.ad = 8 / self.m * m.G

    def stretch(self, u):
        Y = [a + b for a, b in zip(self.d, self.diff(u))]
        Yl = torch.sqrt(sum(y * y for y in Y))
        Yl = torch.where(self.mask, Yl, torch.ones_like(Yl))
        return Y, Yl, torch.where(self.mask, Yl - self.r, torch.zeros_like(Yl))

    def force(self, u):
        Y, Yl, e = self.stretch(u)
        if self.sc > 0:
            self.alive &= ~_gt(e / self.r, torch.full_like(e, self.sc))
        w = torch.where(self.alive, self.w, torch.zeros_like(self.w))
        if self.dim == 3:
            th = 3 / self.m * (self.r * e * w).sum(0)
            cs, cd, ct = 9 * self.K / self.m, 15 * self.G / self.m, 1.0
        else:
            th = 2 / self.m * self.f2 * (self.r * e * w).sum(0)
            cs = (2 * self.f2 * self.as_ - (3 - 2 * self.f2) * self.ad) / 3
            cd, ct = self.ad, 1.0
        es_i, es_j = th * self.r / 3, th[self.idx] * self.r / 3
        t = cs * ct * es_i + cd * (e - es_i) + cs[self.idx] * ct * es_j + \
            cd[self.idx] * (e - es_j)
        s = t * w / Yl
        return [(s * y).sum(0) for y in Y]

    def damage(self, u):
        z = self.stretch(u)[2].abs() / self.r / self.sc
        return torch.where(self.mask, z, torch.zeros_like(z)).max(0).values


def _loads(p, x):
    """[(node mask, dof, value(t), rate)] of the Displacement_BC sets, and
    [(node mask, dof, value(t))] of the Force_BC sets (all rectangles)."""
    def mask(b):
        return ((x[0] >= b.x1) & (x[0] <= b.x2) & (x[1] >= b.y1) & (x[1] <= b.y2))

    ub, fb = [], []
    for b in p.ubc:
        a, lin = b.time_params[0] * b.spatial_params[0], b.time_fn == "linear"
        for d in b.direction:
            ub.append((mask(b), d - 1, a, lin))
    for b in p.fbc:
        for d in b.direction:
            fb.append((mask(b), d - 1, b.time_params[0] * b.spatial_params[0]))
    return ub, fb


def _explicit(p, B, steps, central, damage):
    dim, dev = p.dim, _dev()
    ub, fb = _loads(p, B.x)
    zero = torch.zeros(p.n, dtype=torch.float64, device=dev)
    u = [zero.clone() for _ in range(dim)]
    v = [torch.from_numpy(np.ascontiguousarray(p.v0[:, d])).to(dev) for d in range(dim)]

    def fix(a, t, rate):
        for msk, d, amp, lin in ub:
            val = (amp if lin else 0.0) if rate else (amp * t if lin else amp)
            a[d] = torch.where(msk, torch.full_like(a[d], val), a[d])

    def force(t):
        f = B.force(u)
        for msk, d, amp in fb:
            f[d] = f[d] + torch.where(msk, torch.full_like(f[d], amp * t),
                                      torch.zeros_like(f[d]))
        return f

    t, dt, rho = 0.0, p.dt, p.material.density
    fix(u, t, False)
    fix(v, t, True)
    f = force(t)
    for _ in range(steps):
        t += dt
        if central:
            un = [a + (dt * dt / rho * c + dt * b) for a, b, c in zip(u, v, f)]
            fix(un, t, False)
            v = [(a - b) / dt for a, b in zip(un, u)]
            fix(v, t, True)
            u = un
            f = force(t)
        else:
            v = [b + 0.5 * dt / rho * c for b, c in zip(v, f)]
            u = [a + dt * b for a, b in zip(u, v)]
            fix(u, t, False)
            f = force(t)
            v = [b + 0.5 * dt / rho * c for b, c in zip(v, f)]
            fix(v, t, True)

    def full(a):
        a = list(a) + [zero] * (3 - dim)
        return torch.stack(a, 1).cpu().numpy()

    r = {"u": full(u), "v": full(v), "f": full(f), "broken": None}
    if damage:
        w = B.w.sum(0)
        r["phi"] = (1 - torch.where(B.alive, B.w, torch.zeros_like(B.w)).sum(0) / w).cpu().numpy()
        r["Z"] = B.damage(u).cpu().numpy()
    return r


def _exact_qs(p, nx):
    """Equilibrium of the free dofs after the first load step."""
    B = _RNP(p, nx, nx)
    ub, _ = _loads(p, B.x)
    u = torch.zeros((2, p.n), dtype=torch.float64, device=_dev())
    free = torch.ones_like(u)
    for msk, d, amp, lin in ub:
        u[d] = torch.where(msk, torch.full_like(u[d], amp if lin else 0.0), u[d])
        free[d] = torch.where(msk, torch.zeros_like(u[d]), free[d])
    du0 = u.clone()

    def tangent(u):
        S = B.strain(u)
        g = B.k * torch.clamp(1 - 2 * B.beta * B.r * S * S, min=0) * \
            torch.exp(-B.beta * B.r * S * S) / B.r
        return torch.where(B.alive, g, torch.zeros_like(g))

    def mul(g, y):  # (-K y) on the free dofs
        q = g * sum(e * d for e, d in zip(B.e, B.diff(y)))
        return -torch.stack([(q * e).sum(0) for e in B.e]) * free

    u = torch.zeros_like(u)
    rhs, add = None, du0
    for it in range(6):
        g = tangent(u)
        if it == 0:  # predictor: the boundary increment through the tangent
            rhs = -mul(g, du0)
        else:
            rhs = torch.stack(B.force(list(u))) * free
        diag = torch.stack([(g * e * e).sum(0) for e in B.e])
        diag = torch.where(diag > 0, diag, torch.ones_like(diag))
        x, r = torch.zeros_like(u), rhs.clone()
        z = r / diag * free
        q, rz = z.clone(), (r * z).sum()
        stop = 1e-9 * float(rhs.norm())
        for k in range(20 * nx):
            a = mul(g, q)
            al = rz / (q * a).sum()
            x += al * q
            r -= al * a
            if k % 32 == 31 and float(r.norm()) <= stop:
                break
            z = r / diag * free
            rz, old = (r * z).sum(), rz
            q = z + rz / old * q
        u = u + x + add
        add = 0.0
    return torch.cat([u, torch.zeros_like(u[:1])]).t().cpu().numpy()


def _exact_esqs(p, nx, ny):
    """Equilibrium after the first load step: corrections with the linear
    elastic stiffness until they stop shrinking."""
    B = _ES(p, nx, ny)
    t = _esqs_dt()
    ub, fb = _loads(p, B.x)
    n, dev = p.n, _dev()
    u = torch.zeros((2, n), dtype=torch.float64, device=dev)
    free = torch.ones_like(u, dtype=torch.bool)
    body = torch.zeros_like(u)
    for msk, d, amp, lin in ub:
        u[d] = torch.where(msk, torch.full_like(u[d], amp * t if lin else amp), u[d])
        free[d] &= ~msk
    for msk, d, amp in fb:
        body[d] += torch.where(msk, torch.full_like(u[d], amp * t), torch.zeros_like(u[d]))
    M = [d / B.r for d in B.d]

    def linear(y):  # y: [batch, 2, n]
        e = sum(M[d] * (y[:, d][:, B.idx] - y[:, d][:, None]) for d in range(2))
        e = torch.where(B.mask, e, torch.zeros_like(e))
        th = 2 / B.m * B.f2 * (B.r * e * B.w).sum(1)
        cs = (2 * B.f2 * B.as_ - (3 - 2 * B.f2) * B.ad) / 3
        ei, ej = th[:, None] * B.r / 3, th[:, B.idx] * B.r / 3
        s = (cs * ei + B.ad * (e - ei) + cs[B.idx] * ej + B.ad[B.idx] * (e - ej)) * B.w
        return torch.stack([(s * M[d]).sum(1) for d in range(2)], 1)

    dof = free.reshape(-1).nonzero().squeeze(1)
    K = torch.empty((dof.numel(), dof.numel()), dtype=torch.float64, device=dev)
    step = max(1, int(4e7 / (n * B.r.shape[0])))
    for a in range(0, dof.numel(), step):
        c = dof[a:a + step]
        y = torch.zeros((c.numel(), 2 * n), dtype=torch.float64, device=dev)
        y[torch.arange(c.numel(), device=dev), c] = 1.0
        K[:, a:a + step] = linear(y.view(-1, 2, n)).reshape(c.numel(), -1)[:, dof].t()
    lu = torch.linalg.lu_factor(K)
    for _ in range(40):
        r = (torch.stack(B.force(list(u))) + body).reshape(-1)[dof]
        du = torch.linalg.lu_solve(*lu, -r[:, None]).squeeze(1)
        u.view(-1)[dof] += du
        if float(du.norm()) <= 1e-15 * float(u.norm()):
            break
    f = torch.stack(B.force(list(u))) * B.vol
    pad = torch.zeros_like(u[:1])
    return [torch.cat([u, pad]).t().cpu().numpy(), torch.cat([f, pad]).t().cpu().numpy()]


def _exact_mlp(case, seed):
    """Operands of every product rounded to bf16, as the network defines them;
    products, sums and biases in 64 bits."""
    p, lay = _mlp_params(case, seed)
    p = torch.from_numpy(p)
    a = torch.from_numpy(_mlp_rows(case, seed)).to(torch.bfloat16)
    for l, (di, do, wo, bo) in enumerate(lay):
        w = p[wo:wo + di * do].view(di, do).to(torch.bfloat16).double()
        if a.shape[1] < di:
            a = torch.nn.functional.pad(a, (0, di - a.shape[1]))
        y = a.double() @ w + p[bo:bo + do].double()
        a = torch.relu(y).float().to(torch.bfloat16)
    return y[:, :2].numpy()


def exact(case, seed):
    k = case["kind"]
    if k == "plate":
        if case["nx"] * case["ny"] * case["steps"] > 5e8:
            return None  # minutes in 64 bits
        p = _problem(case, seed)
        return _explicit(p, _RNP(p, case["nx"], case["ny"]), case["steps"],
                         case["scheme"] == "central", case["damage"])
    if k == "cube":
        if case["nx"] * case["ny"] * case["nz"] * case["steps"] > 5e7:
            return None
        p = _problem(case, seed)
        return _explicit(p, _ES(p, case["nx"], case["ny"], case["nz"]), case["steps"], False,
                         case["damage"])
    if k == "host_step":
        p = _problem(case, seed)
        r = _explicit(p, _RNP(p, case["nx"], case["ny"]), 1, False, False)
        return [r["u"], r["v"], r["f"]]
    if k == "ensemble":
        if case["plates"] * case["nmax"] * case["steps"] > 4e8:
            return None
        out = []
        for p in _ensemble(case, seed):
            nx = int(round(math.sqrt(p.n)))
            r = _explicit(p, _RNP(p, nx, nx), case["steps"], False, False)
            out.append([r["u"], r["v"], r["f"]])
        return out
    if k == "qs":
        return _exact_qs(_problem(case, seed), case["nx"])
    if k == "esqs":
        return _exact_esqs(_problem(case, seed), case["nx"], case["ny"])
    if k == "mlp":
        return _exact_mlp(case, seed)
    return None

"""The work that programs have this framework do, as cases to be timed.

Five kinds, all through the public Python entry points:

  apply   y = K x with epsilon = x^T y on device vectors (Solver.inprod_dev, or
          abi.inprod_eps_noalloc for callers that may not allocate): the
          operator inside somebody else's Krylov method
  solve   the drop-in for aphid_serial on host arrays: gen_k2, gen_diag, qmr,
          gen_fields
  sweep   one forward model of a survey or of an inversion: set_model with a new
          conductivity, one batched sweep over frequencies and sources,
          sweep_receivers (or the whole solutions)
  train   one forward and back-propagation pass of the initial-guess network
  guess   its inference on a whole mesh

Meshes follow the benchmark models' rule (graded axes, Gaussian-random-field
earth with blocks, air on top, seawater for the seafloor ones).  Solves stop at
a relative residual of 1e-12, as the reference's shipped serial/aphid.input
asks.
"""
import math

import numpy as np
import torch

from aphid_git_b200 import Solver, abi, learn, model, unet

MU0, EPS0 = 4.0e-7 * 3.141592653589793, 8.8541878176e-12
TARGET, MAX_IT = 1e-12, 20000


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the operator on a training-size mesh: launch latency counts
        dict(name="apply-65x65x49", kind="apply", cx=64, cy=64, cz=48, eps=True, entry="context"),
        # the operator on the largest mesh of the evaluation set: 13.3 M unknowns
        dict(name="apply-161x161x129", kind="apply", cx=160, cy=160, cz=128, eps=False, entry="context"),
        # aphid_serial's program with the GPU behind `call qmr`: 32^3 cells, one frequency
        dict(name="solve-33", kind="solve", cx=32, cy=32, cz=32, nair=8, freq=1.0),
        # the smallest sweep, whose solutions the caller wants: latency of the rounds
        dict(name="sweep-25x23x21-x3", kind="sweep", cx=24, cy=22, cz=20, nair=6, nsea=0, csig="R", source="dipole",
             nsrc=1, fmin=1e-2, fmax=1e2, nfreq=3, precision="auto", result="solutions"),
        # magnetotellurics over a polarisable (Cole-Cole) earth, odd sizes, both polarisations
        dict(name="sweep-41x37x34-mt-colecole", kind="sweep", cx=40, cy=36, cz=33, nair=8, nsea=0, csig="D",
             source="mt", nsrc=2, fmin=1e-1, fmax=1e2, nfreq=4, precision="auto", result="receivers"),
        # controlled source, 24 frequencies of one small model: the ordinary batch
        dict(name="sweep-65x65x49-x24", kind="sweep", cx=64, cy=64, cz=48, nair=8, nsea=0, csig="R", source="dipole",
             nsrc=1, fmin=1e-2, fmax=1e2, nfreq=24, precision="auto", result="receivers"),
        # one heterogeneous system in mixed precision, permittivity given (model C)
        dict(name="sweep-97-modelc", kind="sweep", cx=96, cy=96, cz=96, nair=8, nsea=0, csig="C", source="dipole",
             nsrc=1, fmin=1.0, fmax=1.0, nfreq=1, precision="mixed", result="receivers"),
        # seafloor layering: systems that finish in the complex128 pass
        dict(name="sweep-97-seafloor-x2", kind="sweep", cx=96, cy=96, cz=96, nair=10, nsea=15, csig="R",
             source="dipole", nsrc=1, fmin=0.272, fmax=1.35, nfreq=2, precision="auto", result="receivers"),
        # the reference's own recurrence on the heterogeneous model
        dict(name="sweep-97-fp64", kind="sweep", cx=96, cy=96, cz=96, nair=8, nsea=0, csig="R", source="dipole",
             nsrc=1, fmin=1.0, fmax=1.0, nfreq=1, precision="fp64", result="receivers"),
        # the largest mesh, two frequencies
        dict(name="sweep-161x161x129-x2", kind="sweep", cx=160, cy=160, cz=128, nair=8, nsea=0, csig="R",
             source="dipole", nsrc=1, fmin=30.0, fmax=100.0, nfreq=2, precision="auto", result="receivers"),
        # the initial-guess network: a training pass at the training mesh, inference at the evaluation mesh
        dict(name="train-65x65x49", kind="train", cx=64, cy=64, cz=48),
        dict(name="guess-161x161x129", kind="guess", cx=160, cy=160, cz=128),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choices(["apply", "solve", "sweep", "train", "guess"], [3, 2, 9, 1, 1])[0]
    if kind == "sweep":
        sea = rng.random() < 0.2
        prec = rng.choices(["auto", "mixed", "fused64", "fp64"], [6, 2, 1, 2])[0]
        csig = "R" if sea else rng.choice(["R", "R", "C", "D"])
        source = "dipole" if sea else rng.choice(["dipole", "dipole", "mt"])
        lo = 40 if sea else 16
        cx, cy, cz = (int(_log(rng, lo, 140)) for _ in range(3))
        nodes = cx * cy * cz
        most = max(1, int((4e5 if prec == "fp64" else 2.5e6) / nodes))
        nsrc = 2 if source == "mt" else (2 if most >= 4 and rng.random() < 0.4 else 1)
        nfreq = max(1, min(24, int(_log(rng, 1, max(1.01, min(24, most / nsrc))))))
        top = 1.5 if sea else 100.0
        f0 = _log(rng, 0.25 if sea else 0.1, top)
        f1 = f0 if nfreq == 1 else _log(rng, f0, top)
        return dict(kind=kind, cx=cx, cy=cy, cz=cz, nair=10 if sea else max(2, cz // 6), nsea=15 if sea else 0,
                    csig=csig, source=source, nsrc=nsrc, fmin=f0, fmax=f1, nfreq=nfreq,
                    precision="auto" if sea and prec == "mixed" else prec,
                    result="receivers" if nodes * nfreq * nsrc > 3e5 else rng.choice(["receivers", "solutions"]))
    if kind == "solve":
        cx, cy, cz = (int(_log(rng, 16, 72)) for _ in range(3))
        return dict(kind=kind, cx=cx, cy=cy, cz=cz, nair=max(2, cz // 6), freq=_log(rng, 0.1, 100.0))
    lo, hi = {"apply": (16, 140), "train": (24, 60), "guess": (24, 140)}[kind]
    case = dict(kind=kind, cx=int(_log(rng, lo, hi)), cy=int(_log(rng, lo, hi)), cz=int(_log(rng, lo, hi)))
    if kind == "apply":
        case["entry"] = rng.choice(["context", "context", "noalloc"])
        case["eps"] = case["entry"] == "noalloc" or rng.random() < 0.5
    return case


def _freqs(c):
    return np.logspace(math.log10(c["fmin"]), math.log10(c["fmax"]), c["nfreq"])


def _unknowns(c):
    return model.nunk(c["cx"] + 1, c["cy"] + 1, c["cz"] + 1)


# ------------------------------------------------------------------ the inputs
def _mesh(c):
    """Node coordinates: 1 km core cells, six stretched cells per side, z = 0 under the air."""
    return (model.graded_axis(c["cx"]), model.graded_axis(c["cy"]),
            model.depth_axis(c["cz"], c.get("nair", max(2, c["cz"] // 6))))


def _cells(c, rng):
    """real(4) cell conductivity: air, seawater, 10^(Gaussian random field) earth with blocks."""
    cx, cy, cz = c["cx"], c["cy"], c["cz"]
    nair, nsea = c.get("nair", max(2, cz // 6)), c.get("nsea", 0)
    top = nair + nsea
    sig = np.full((cx, cy, cz), 1e-8)
    sig[:, :, nair:top] = 3.3
    earth = 10.0 ** np.clip(-2.0 + model.grf((cx, cy, cz - top), 8.0, rng), -4.0, 1.0)
    for _ in range(20):
        at = [int(rng.integers(0, max(1, n - 4))) for n in earth.shape]
        n = [int(rng.integers(2, 13)) for _ in range(3)]
        earth[at[0]:at[0] + n[0], at[1]:at[1] + n[1], at[2]:at[2] + n[2]] = 10.0 ** rng.uniform(-4, 1)
    sig[:, :, top:] = earth
    return sig.astype(np.float32)


def _rng(c, seed):
    return np.random.default_rng([seed, c["cx"], c["cy"], c["cz"]])


def _dipoles(c, nsrc):
    """+X at the centre of the ground (or sea floor), then +Y beside it."""
    i, j, k = c["cx"] // 2, (c["cy"] + 2) // 2, c.get("nair", max(2, c["cz"] // 6)) + c.get("nsea", 0) + 1
    return [[("+X", i, j, k)], [("+Y", i + 1, j - 1, k)]][:nsrc]


def _sweep_input(c, seed):
    """Cell arrays, angular frequencies, sources and the source of each system."""
    rng = _rng(c, seed)
    cells = {"sig": _cells(c, rng)}
    shape = cells["sig"].shape
    if c["csig"] == "C":
        cells["epsr"] = rng.uniform(1, 30, shape).astype(np.float32)
    elif c["csig"] == "D":
        cells["eta"] = rng.uniform(0.05, 0.6, shape).astype(np.float32)
        cells["tau"] = (10.0 ** rng.uniform(-3, 1, shape)).astype(np.float32)
        cells["cee"] = rng.uniform(0.2, 0.8, shape).astype(np.float32)
    cells = {k: np.ascontiguousarray(v.ravel(order="F")) for k, v in cells.items()}
    sources = [2, 3] if c["source"] == "mt" else _dipoles(c, c["nsrc"])
    om = 2 * math.pi * _freqs(c)
    return cells, np.tile(om, len(sources)), sources, np.repeat(np.arange(len(sources)), len(om))


def _receivers(c):
    """A grid of up to 16 x 16 nodes on the ground (sea floor)."""
    k = c["nair"] + c["nsea"] + 1
    xs, ys = (np.unique(np.linspace(3, n - 1, 16).astype(int)) for n in (c["cx"], c["cy"]))
    return np.array([(i, j, k) for j in ys for i in xs], np.int32)


def _sigma_hat(csig, omega, cells):
    """Complex cell conductivity of read_mesh, models R, C and D."""
    s = cells["sig"].astype(np.float64)
    if csig == "D":
        eta, tau, cee = (cells[k].astype(np.float64) for k in ("eta", "tau", "cee"))
        return s * (1.0 - eta / (1.0 + (1j * omega * tau) ** cee))
    return s + 1j * omega * EPS0 * (cells["epsr"].astype(np.float64) if csig == "C" else 1.0)


def _apply_input(c, seed):
    """The cell conductivity at 1 Hz and a Krylov vector's stand-in."""
    rng = _rng(c, seed)
    sig = _sigma_hat("R", 2 * math.pi, {"sig": _cells(c, rng).ravel(order="F")})
    x = rng.standard_normal(2 * _unknowns(c)).view(np.complex128)
    return sig, x


def _net_params(seed):
    """He-normal weights and small biases in the network's parameter layout."""
    rng = np.random.default_rng(seed)
    out = []
    for ci, co in _LAYERS:
        out += [rng.standard_normal(27 * ci * co) * math.sqrt(2.0 / (27 * ci)), 0.01 * rng.standard_normal(co)]
    return np.concatenate(out).astype(np.float32)


def _net_input(c, seed):
    rng = _rng(c, seed)
    dims = (c["cx"] + 1, c["cy"] + 1, c["cz"] + 1)
    x = learn.features(_cells(c, rng), 10.0 ** rng.uniform(-3, 4), _dipoles(c, 1)[0], dims)
    t = 0.3 * rng.standard_normal((x.shape[0], 8)) if c["kind"] == "train" else np.zeros((0, 8))
    return x, t.astype(np.float32)


def prepare(case, seed):
    c, s = case, {"case": case}
    if c["kind"] in ("train", "guess"):
        x, t = _net_input(c, seed)
        s["net"] = unet.UNet(c["cx"] + 1, c["cy"] + 1, c["cz"] + 1, train=c["kind"] == "train")
        s["net"].set_params(_net_params(seed))
        s["x"], s["t"] = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
        s["y"] = torch.empty(x.shape[0], 8, device="cuda")
        return s
    xn, yn, zn = _mesh(c)
    if c["kind"] == "apply":
        sig, x = _apply_input(c, seed)
        s["stream"] = torch.cuda.Stream()
        s["solver"] = Solver(stream=s["stream"].cuda_stream)
        s["solver"].set_nodes(xn, yn, zn)
        s["k2"] = torch.from_numpy(s["solver"].gen_k2(sig, 2 * math.pi)).cuda()
        s["x"] = torch.from_numpy(x).cuda()
        s["y"], s["eps"] = torch.empty_like(s["x"]), torch.zeros(1, dtype=torch.complex128, device="cuda")
        s["spacing"] = [torch.from_numpy(a).cuda() for p in zip(*map(model.spacings, (xn, yn, zn))) for a in p]
        s["stream"].wait_stream(torch.cuda.current_stream())
        return s
    s["solver"] = Solver()
    s["solver"].set_nodes(xn, yn, zn)
    if c["kind"] == "solve":
        s["omega"] = 2 * math.pi * c["freq"]
        cells = {"sig": _cells(c, _rng(c, seed)).ravel(order="F")}
        s["sig"] = _sigma_hat("R", s["omega"], cells)
        s["b"] = model.gen_rhs(xn, yn, zn, 5, _dipoles(c, 1)[0])[0]
        return s
    s["cells"], s["om"], s["sources"], s["sos"] = _sweep_input(c, seed)
    s["rec"] = _receivers(c)
    return s


# ------------------------------------------------------------------ one pass
def run(state):
    s, c = state, state["case"]
    if c["kind"] == "guess":
        s["net"].forward(s["x"], s["y"])
        return s["y"]
    if c["kind"] == "train":
        loss = s["net"].train_step(s["x"], s["t"], update=False)
        return {"loss": loss, "grads": s["net"].grads()}
    if c["kind"] == "apply":
        k2, x, y, eps = (s[k].data_ptr() for k in ("k2", "x", "y", "eps"))
        if c["entry"] == "noalloc":
            abi.inprod_eps_noalloc(c["cx"] + 1, c["cy"] + 1, c["cz"] + 1, [a.data_ptr() for a in s["spacing"]], k2,
                                   x, y, eps, s["stream"].cuda_stream)
        else:
            s["solver"].inprod_dev(k2, x, y, eps if c["eps"] else None)
        return {"y": s["y"], "eps": s["eps"]} if c["eps"] else {"y": s["y"]}
    sv = s["solver"]
    if c["kind"] == "solve":
        k2 = sv.gen_k2(s["sig"], s["omega"])
        x, info, _ = sv.qmr(k2, sv.gen_diag(k2), s["b"], TARGET, MAX_IT)
        B, E = sv.gen_fields(s["omega"], x)
        return {"x": x, "B": B, "E": E}
    m = s["cells"]
    if c["csig"] == "D":
        sv.set_model_cole_cole(m["sig"], m["eta"], m["tau"], m["cee"])
    else:
        sv.set_model(c["csig"], m["sig"], m.get("epsr"))
    whole = c["result"] == "solutions"
    x, _ = sv.sweep(s["om"], s["sources"], s["sos"], precision=c["precision"], target=TARGET, max_it=MAX_IT,
                    fetch=whole)
    if whole:
        return {"x": x}
    e, h = sv.sweep_receivers(s["rec"])
    return {"E": e, "H": h}


# ------------------------------------------------------------------ what a pass cannot do without
#: Iterations that a Jacobi-preconditioned solve to 1e-12 takes on these models, for work().
_ITERATIONS = 1500
#: Real operations of one operator row set per unknown, and of one QMR iteration's vector updates.
_ROW_FLOPS, _ITER_FLOPS = 40, 60


def work(case):
    c, n = case, _unknowns(case)
    if c["kind"] == "apply":
        return {"bytes": 48.0 * n, "flops": float(_ROW_FLOPS * n)}  # k^2 and x in, y out
    if c["kind"] in ("train", "guess"):
        v = (c["cx"] + 1) * (c["cy"] + 1) * (c["cz"] + 1)
        level = [0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0, 0]
        act = sum(2.0 * (ci + co) * v / 8 ** q for (ci, co), q in zip(_LAYERS, level))
        flops = sum(2.0 * 27 * ci * co * v / 8 ** q for (ci, co), q in zip(_LAYERS, level))
        k = 3 if c["kind"] == "train" else 1  # forward; data and weight gradients
        return {"bytes": k * act + 44.0 * v, "flops": k * flops}
    nsys = 1 if c["kind"] == "solve" else c["nfreq"] * (2 if c["source"] == "mt" else c["nsrc"])
    # Krylov vectors in and out once per iteration: q, v, p in complex64, or
    # in complex128 where the precision asks for it
    per = 96.0 if c["kind"] == "solve" or c["precision"] in ("fp64", "fused64") else 48.0
    return {"bytes": per * n * nsys * _ITERATIONS, "flops": float((_ROW_FLOPS + _ITER_FLOPS) * n * nsys * _ITERATIONS)}


# ------------------------------------------------------------------ 64-bit answers in plain torch
def _axis(x):
    """Of one axis: primary lengths d(0:n), dual lengths, edge and node coefficients (e2, e3, n4, n5)."""
    d = np.concatenate([[x[1] - x[0]], np.diff(x), [x[-1] - x[-2]]])
    n = len(x)
    dc = np.empty(n)
    dc[1:-1] = 0.5 * (d[1:n - 1] + d[2:n])
    dc[0], dc[-1] = dc[1], dc[-2]
    up, lo = -np.ones(n), -np.ones(n)
    up[-1], lo[0] = 0.0, 0.0
    eu, el = up[1:], lo[:-1]
    return dict(n=n, d=d, dc=dc, e2=eu / dc[1:] / d[1:n], e3=el / dc[:-1] / d[1:n], n4=up / d[1:] / dc,
                n5=lo / d[:n] / dc)


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _shapes(n):
    return [(n[0] - 1, n[1], n[2]), (n[0], n[1] - 1, n[2]), (n[0], n[1], n[2] - 1), tuple(n)]


class _Operator:
    """K of the staggered-grid A-Phi equations as a sparse complex128 matrix,
    and its diagonal (1 where a row is empty)."""

    def __init__(self, nodes, sig, omega):
        self.ax = [_axis(np.asarray(x, np.float64)) for x in nodes]
        n = [a["n"] for a in self.ax]
        dev = _device()
        shapes = _shapes(n)
        off = np.concatenate([[0], np.cumsum([a * b * c for a, b, c in shapes])])
        self.n, self.shapes, self.off = int(off[-1]), shapes, off
        k2 = self._k2(np.asarray(sig).reshape([m - 1 for m in n], order="F"), omega)
        k2 = [torch.from_numpy(np.ascontiguousarray(k.transpose(2, 1, 0))).to(dev) for k in k2]
        idx = [torch.arange(int(off[q]), int(off[q + 1]), device=dev).reshape(s[::-1]) for q, s in enumerate(shapes)]
        rows, cols, vals = [], [], []

        def view(v, axis):  # a 1-D table along an axis of a (k, j, i) array
            sh = [1, 1, 1]
            sh[2 - axis] = -1
            return torch.from_numpy(np.ascontiguousarray(v)).to(dev).reshape(sh)

        def cut(t, axis, lo, hi):
            return t.narrow(2 - axis, lo, t.shape[2 - axis] - lo - hi)

        def put(r, c_, v):
            r, c_, v = torch.broadcast_tensors(r, c_, v)
            rows.append(r.reshape(-1)), cols.append(c_.reshape(-1)), vals.append(v.reshape(-1).to(torch.complex128))

        def both(r, ci, v, axis, cp, cm, vol):  # the two neighbours along an axis: coefficients cp, cm
            w = torch.broadcast_to(v * vol, r.shape)
            put(cut(r, axis, 0, 1), cut(ci, axis, 1, 0), cut(torch.broadcast_to(w * cp, r.shape), axis, 0, 1))
            put(cut(r, axis, 1, 0), cut(ci, axis, 0, 1), cut(torch.broadcast_to(w * cm, r.shape), axis, 1, 0))

        diag = []
        for a in range(3):
            A, r = self.ax[a], idx[a]
            o = [q for q in range(3) if q != a]
            vol = view(A["d"][1:A["n"]], a) * view(self.ax[o[0]]["dc"], o[0]) * view(self.ax[o[1]]["dc"], o[1])
            co = {a: (view(A["e2"], a), view(A["e3"], a))}
            for q in o:
                co[q] = (view(self.ax[q]["n4"], q), view(self.ax[q]["n5"], q))
            dg = vol * (k2[a] - sum(x for p in co.values() for x in p))
            put(r, r, dg)
            diag.append(dg)
            one = torch.ones(1, dtype=torch.float64, device=dev)
            for q, (cp, cm) in co.items():
                both(r, r, one, q, cp, cm, vol)
            s = vol / view(A["d"][1:A["n"]], a)
            put(r, cut(idx[3], a, 1, 0), s * (cut(k2[3], a, 1, 0) - k2[a]))
            put(r, cut(idx[3], a, 0, 1), -s * (cut(k2[3], a, 0, 1) - k2[a]))

        def inner(t, but=None):  # interior nodes along every axis (but one)
            for q in range(3):
                t = t if q == but else cut(t, q, 1, 1)
            return t

        def at(v, q):
            return view(v[1:-1], q)

        r, kp, p = inner(idx[3]), inner(k2[3]), idx[3]
        vol = at(self.ax[0]["dc"], 0) * at(self.ax[1]["dc"], 1) * at(self.ax[2]["dc"], 2)
        total = 0
        for a in range(3):
            e, ke = inner(idx[a], a), inner(k2[a], a)
            kplus, kminus = cut(ke, a, 1, 0), cut(ke, a, 0, 1)
            cp, cm = at(self.ax[a]["n4"], a) * kplus, at(self.ax[a]["n5"], a) * kminus
            total = total + cp + cm
            side = inner(p, a)
            put(r, cut(side, a, 2, 0), vol * cp)
            put(r, cut(side, a, 0, 2), vol * cm)
            put(r, cut(e, a, 1, 0), vol / at(self.ax[a]["dc"], a) * (kplus - kp))
            put(r, cut(e, a, 0, 1), -vol / at(self.ax[a]["dc"], a) * (kminus - kp))
        dphi = vol * (kp * kp - total)
        put(r, r, dphi)
        full = torch.ones(shapes[3][::-1], dtype=torch.complex128, device=dev)
        full[1:-1, 1:-1, 1:-1] = dphi
        self.diag = torch.cat([d.reshape(-1) for d in diag + [full]])
        i = torch.stack([torch.cat(rows), torch.cat(cols)])
        rows.clear(), cols.clear()
        m = torch.sparse_coo_tensor(i, torch.cat(vals), (self.n, self.n), check_invariants=False)
        del i
        vals.clear()
        self.K = m.coalesce().to_sparse_csr()

    def _k2(self, sig, omega):
        """i omega mu0 times the area- and volume-weighted averages of the cells around edges and nodes."""

        def mean(v, axis):  # width-weighted mean over the two cells at each node, ends clamped
            d = self.ax[axis]["d"][1:-1]
            sh = [1, 1, 1]
            sh[axis] = -1
            a, b = v.take(range(len(d) - 1), axis), v.take(range(1, len(d)), axis)
            wa, wb = d[:-1].reshape(sh), d[1:].reshape(sh)
            t = (a * wa + b * wb) / (wa + wb)
            return np.concatenate([t.take([0], axis), t, t.take([-1], axis)], axis)

        xy, xz, yz = mean(mean(sig, 0), 1), mean(mean(sig, 0), 2), mean(mean(sig, 1), 2)
        return [1j * omega * MU0 * t for t in (yz, xz, xy, mean(xy, 2))]

    def __call__(self, x):
        return torch.mv(self.K, x)

    def rhs(self, source):
        """A dipole (direction +X or +Y, one-based tail node) or an MT sheet (2 or 3)."""
        b = [np.zeros(s) for s in self.shapes]
        d = [a["d"] for a in self.ax]
        n = [a["n"] for a in self.ax]
        if source in (2, 3):
            a, o = (0, 1) if source == 2 else (1, 0)
            half = 0.5 * (d[o][:n[o]] + d[o][1:n[o] + 1])
            w = MU0 * np.outer(d[a][1:n[a]], half)
            b[a][:, :, 1] = w if a == 0 else w.T
        else:
            (dr, i, j, k), = source
            a, t = "XYZ".index(dr[1]), [i - 1, j - 1, k - 1]
            h = list(t)
            h[a] += 1
            b[a][tuple(t)] = MU0 * d[a][t[a] + 1]
            b[3][tuple(t)], b[3][tuple(h)] = MU0, -MU0
        return torch.from_numpy(np.concatenate([x.ravel(order="F") for x in b])).to(_device(), torch.complex128)

    def solve(self, b):
        """Jacobi-preconditioned QMR in complex128, restarted from the true residual until it stops falling."""
        x, r = torch.zeros_like(b), b.clone()
        inv, norm = 1.0 / self.diag, float(torch.linalg.vector_norm(b))
        at = norm
        for _ in range(6):
            tol = max(1e-3 * at, 2e-15 * norm) if at < 1e-6 * norm else max(1e-13 * norm, 1e-7 * at)
            e = self._qmr(r, inv, tol)
            r2 = b - self(x + e)
            now = float(torch.linalg.vector_norm(r2))
            if not now < at:
                break
            x, r, stalled, at = x + e, r2, now > 0.5 * at, now
            if stalled or at < 3e-14 * norm:
                break
        return x

    def _qmr(self, b, inv, tol):
        x, d, s, p = (torch.zeros_like(b) for _ in range(4))
        r, v = b.clone(), b.clone()
        rho, eps, eta, theta, c = torch.linalg.vector_norm(v), 1.0, -1.0, 0.0, 1.0
        for it in range(8000):
            v /= rho
            z = inv * v
            delta = torch.dot(v, z)
            p = z if it == 0 else z - (rho * delta / eps) * p
            q = self(p)
            eps = torch.dot(p, q)
            beta = eps / delta
            v = q - beta * v
            rho1 = torch.linalg.vector_norm(v)
            theta1 = rho1 / (c * torch.abs(beta))
            c1 = 1.0 / torch.sqrt(1.0 + theta1 * theta1)
            eta = -eta * rho * c1 * c1 / (beta * c * c)
            k = (theta * c1) ** 2
            d = eta * p + k * d
            s = eta * q + k * s
            x += d
            r -= s
            rho, theta, c = rho1, theta1, c1
            if it % 8 == 0 and not float(torch.linalg.vector_norm(r)) > tol:
                break
        return x

    def fields(self, x, omega):
        """(B on faces, E on edges): curl A and -i omega (A - grad Phi), (k, j, i) arrays."""
        p = [x[int(self.off[q]):int(self.off[q + 1])].reshape(s[::-1]) for q, s in enumerate(self.shapes)]
        d = []
        for a in range(3):
            sh = [1, 1, 1]
            sh[2 - a] = -1
            d.append(torch.from_numpy(self.ax[a]["d"][1:-1].copy()).to(x.device).reshape(sh))

        def diff(t, a):
            return torch.diff(t, dim=2 - a) / d[a]

        B = [diff(p[2], 1) - diff(p[1], 2), diff(p[0], 2) - diff(p[2], 0), diff(p[1], 0) - diff(p[0], 1)]
        E = [-1j * omega * (p[a] - diff(p[3], a)) for a in range(3)]
        return B, E


def _at_nodes(B, E, rec):
    """E and H at nodes: means of the two edges, and of the four faces, around each."""
    i, j, k = (torch.from_numpy(rec[:, q].astype(np.int64) - 1).to(E[0].device) for q in range(3))
    e = [0.5 * (E[0][k, j, i] + E[0][k, j, i - 1]), 0.5 * (E[1][k, j, i] + E[1][k, j - 1, i]),
         0.5 * (E[2][k, j, i] + E[2][k - 1, j, i])]
    h = [sum(B_[k - dk, j - dj, i - di] for dk in kk for dj in jj for di in ii) / (4.0 * MU0)
         for B_, kk, jj, ii in ((B[0], (0, 1), (0, 1), (0,)), (B[1], (0, 1), (0,), (0, 1)), (B[2], (0,), (0, 1), (0, 1)))]
    return torch.stack(e, 1), torch.stack(h, 1)


#: (input, output) channels of the network's 3 x 3 x 3 convolutions
_LAYERS = [(3, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (64, 128), (128, 128), (192, 64), (64, 64),
           (96, 32), (32, 32), (48, 16), (16, 16), (16, 8)]


def _net(params, x, dims):
    """The U-Net in 64 bits: x [V][3] -> [V][8] on the mesh nodes."""
    layers, at = [], 0
    for ci, co in _LAYERS:
        w = params[at:at + 27 * ci * co].reshape(co, 27, ci)
        at += 27 * ci * co
        layers.append((w, params[at:at + co]))
        at += co
    X, Y, Z = dims
    full = [-(-m // 8) * 8 for m in (Z, Y, X)]
    a = torch.zeros(*full, 3, dtype=torch.float64, device=x.device)
    a[:Z, :Y, :X] = x.reshape(Z, Y, X, 3)

    def conv(t, q, relu=True):
        w, bias = layers[q]
        z, y, x_, ci = t.shape
        f = torch.nn.functional.pad(t, (0, 0, 1, 1, 1, 1, 1, 1))
        out = bias.expand(z * y * x_, -1)
        for tap in range(27):
            dz, dy, dx = tap // 9, tap // 3 % 3, tap % 3
            out = out + f[dz:dz + z, dy:dy + y, dx:dx + x_].reshape(-1, ci) @ w[:, tap].T
        out = torch.relu(out) if relu else out
        return out.reshape(z, y, x_, -1)

    def pool(t):
        z, y, x_, ch = t.shape
        return t.reshape(z // 2, 2, y // 2, 2, x_ // 2, 2, ch).mean((1, 3, 5))

    def up(t):
        return t.repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2)

    s1 = conv(conv(a, 0), 1)
    s2 = conv(conv(pool(s1), 2), 3)
    s3 = conv(conv(pool(s2), 4), 5)
    a = conv(conv(pool(s3), 6), 7)
    for q, skip in ((8, s3), (10, s2), (12, s1)):
        a = conv(conv(torch.cat([up(a), skip], -1), q), q + 1)
    return conv(a, 14, relu=False)[:Z, :Y, :X].reshape(-1, 8)


def exact(case, seed):
    c, dev = case, _device()
    if c["kind"] in ("train", "guess"):
        x, t = (torch.from_numpy(a).to(dev, torch.float64) for a in _net_input(c, seed))
        p = torch.from_numpy(_net_params(seed)).to(dev, torch.float64)
        dims = (c["cx"] + 1, c["cy"] + 1, c["cz"] + 1)
        if c["kind"] == "guess":
            with torch.no_grad():
                return _net(p, x, dims)
        p.requires_grad_(True)
        loss = ((_net(p, x, dims) - t) ** 2).mean()
        loss.backward()
        return {"loss": float(loss.detach()), "grads": p.grad}
    nodes = _mesh(c)
    if c["kind"] == "apply":
        sig, x = _apply_input(c, seed)
        x = torch.from_numpy(x).to(dev)
        y = _Operator(nodes, sig, 2 * math.pi)(x)
        return {"y": y, "eps": torch.dot(x, y).reshape(1)} if c["eps"] else {"y": y}
    if c["kind"] == "solve":
        w = 2 * math.pi * c["freq"]
        K = _Operator(nodes, _sigma_hat("R", w, {"sig": _cells(c, _rng(c, seed)).ravel(order="F")}), w)
        x = K.solve(K.rhs(_dipoles(c, 1)[0]))
        B, E = K.fields(x, w)
        return {"x": x, "B": torch.cat([t.reshape(-1) for t in B]), "E": torch.cat([t.reshape(-1) for t in E])}
    cells, om, sources, sos = _sweep_input(c, seed)
    if _unknowns(c) * len(om) > 2.5e7:
        return None  # more than about 20 seconds
    xs, es, hs = [], [], []
    for w, q in zip(om, sos):
        K = _Operator(nodes, _sigma_hat(c["csig"], w, cells), w)
        x = K.solve(K.rhs(sources[q]))
        if c["result"] == "solutions":
            xs.append(x)
        else:
            e, h = _at_nodes(*K.fields(x, w), _receivers(c))
            es.append(e), hs.append(h)
    return {"x": torch.stack(xs)} if xs else {"E": torch.stack(es), "H": torch.stack(hs)}

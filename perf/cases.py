"""Measured cases: what a user of this framework has it do, through its
public entry points.

Kinds, each over the range of sizes it is used at:

  step     a new permeability field to its pressure and face fluxes: TPFA
           assembly, AMG setup, CG, flux reconstruction (gpu.Solver)
  guess    the same from the learned initial guess (guess.solve_from_guess)
  resolve  another right-hand side on a hierarchy that is kept
  picard   the coupled reservoir / conduit run (karst.picard), host arrays
  bridge   the reference application's own call, solve_linsys, on host
           arrays, twice per matrix as its reservoir loop makes it
  batch    many uneven grids solved together (batch.solve_batch_graph),
           host arrays
  trunk    the guess network's inference up to its last activation
  layer    one of the network's 3x3x3 convolutions in training: forward,
           data gradient, weight gradient, bias gradient

Options: "fp64" is the default solver (FP64 V-cycle, the reference's
hierarchy), "fast" the reduced-precision V-cycle with the exact level-0
reduction; both in FP64 CG.  Solves run to a true residual of 1e-12, where
the pressure is the discrete system's to ~1e-10 (the batch, whose small
grids reach FP64's limit sooner, to 1e-11); the bridge stops where the
reference does.  Every field is generated: log10 K = -14 + std g with g a
Gaussian field of the given correlation length (cells), plus random-walk
conduits.
"""
import math
import os

import numpy as np
import torch

from hmfem_b200 import batch, gpu, guess, karst
from hmfem_b200.problem import Problem, random_walk_conduit

TOL = 1e-12
FAST = dict(precision=1, schur0=1, bf16_from=1)
MODEL = os.path.join(os.path.dirname(guess.__file__), "models", "unet_config4.npz")


def listed():
    return [
        # the smallest grid of the configurations: launch and host latency
        {"name": "step_32_fp64", "kind": "step", "nx": 32, "ny": 32, "nz": 32,
         "opt": "fp64", "std": 1.0, "corr": 4.0, "conduits": 0},
        # an uneven grid with odd edges (the batched instances' range), where
        # no even-nx form applies
        {"name": "step_87x61x75_fp64", "kind": "step", "nx": 87, "ny": 61, "nz": 75,
         "opt": "fp64", "std": 1.5, "corr": 4.0, "conduits": 3},
        # the karst benchmark grid, reduced precision
        {"name": "step_128_fast", "kind": "step", "nx": 128, "ny": 128, "nz": 128,
         "opt": "fast", "std": 1.5, "corr": 8.0, "conduits": 4},
        # the headline grid with the default solver
        {"name": "step_256_fp64", "kind": "step", "nx": 256, "ny": 256, "nz": 256,
         "opt": "fp64", "std": 1.5, "corr": 8.0, "conduits": 8},
        # the headline step: reduced precision from the learned guess
        {"name": "guess_256_fast", "kind": "guess", "nx": 256, "ny": 256, "nz": 256,
         "opt": "fast", "std": 1.5, "corr": 8.0, "conduits": 8},
        # sources changed on a kept hierarchy, an oblong grid
        {"name": "resolve_160x96x64_fast", "kind": "resolve", "nx": 160, "ny": 96, "nz": 64,
         "opt": "fast", "std": 1.5, "corr": 6.0, "conduits": 2},
        # the coupled run on the reference run script's grid and conduit
        {"name": "picard_210x42x20_fast", "kind": "picard", "nx": 210, "ny": 42, "nz": 20,
         "opt": "fast", "std": 0.3},
        # the unmodified application's solves on that grid
        {"name": "bridge_210x42x20", "kind": "bridge", "nx": 210, "ny": 42, "nz": 20,
         "std": 0.5, "corr": 2.0},
        # uncertainty sampling: instances of 24..96 cells a side
        {"name": "batch_16_fast", "kind": "batch", "m": 16, "lo": 24, "hi": 96, "opt": "fast"},
        # the learned guess's inference at its training size
        {"name": "trunk_128", "kind": "trunk", "nx": 128, "ny": 128, "nz": 128},
        # training: a full-resolution layer and a coarse, wide one
        {"name": "layer_16_16_128", "kind": "layer", "nx": 128, "ny": 128, "nz": 128,
         "cin": 16, "cout": 16},
        {"name": "layer_96_32_64", "kind": "layer", "nx": 64, "ny": 64, "nz": 64,
         "cin": 96, "cout": 32},
    ]


def _edge(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "guess", "resolve", "resolve", "picard",
                       "bridge", "batch", "trunk", "layer", "layer"])
    opt = rng.choice(["fp64", "fast"])
    if kind in ("step", "resolve"):
        hi = 256 if kind == "step" else 192
        return {"kind": kind, "nx": _edge(rng, 20, hi), "ny": _edge(rng, 20, hi),
                "nz": _edge(rng, 12, hi), "opt": opt, "std": round(rng.uniform(0.5, 1.5), 3),
                "corr": round(rng.uniform(2.0, 8.0), 2), "conduits": rng.randint(0, 8)}
    if kind == "guess":  # the network pools twice: multiples of four
        nx, ny, nz = (4 * _edge(rng, 8, 48) for _ in range(3))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "opt": opt,
                "std": round(rng.uniform(0.5, 1.5), 3), "corr": round(rng.uniform(4.0, 8.0), 2),
                "conduits": rng.randint(0, 8)}
    if kind == "picard":
        return {"kind": kind, "nx": rng.randint(60, 210), "ny": rng.randint(12, 42),
                "nz": rng.randint(8, 20), "opt": opt, "std": round(rng.uniform(0.1, 0.5), 3)}
    if kind == "bridge":
        return {"kind": kind, "nx": _edge(rng, 24, 210), "ny": _edge(rng, 16, 64),
                "nz": _edge(rng, 10, 48), "std": round(rng.uniform(0.2, 1.5), 3),
                "corr": round(rng.uniform(1.0, 4.0), 2)}
    if kind == "batch":
        return {"kind": kind, "m": rng.randint(4, 16), "lo": 24, "hi": rng.randint(40, 96),
                "opt": opt}
    if kind == "trunk":
        nx, ny, nz = (4 * _edge(rng, 8, 48) for _ in range(3))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz}
    cin, cout = rng.choice([(c, d) for _, c, d in guess.UNet.SPEC])
    nx, ny, nz = (_edge(rng, 20, 128) for _ in range(3))
    return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "cin": cin, "cout": cout}


# ---- inputs -------------------------------------------------------------------

def _field(seed, nx, ny, nz, std, corr, base=-14.0):
    """10 ** (base + std g), (nz, ny, nx) FP64 on the GPU."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    g = torch.randn(nz, ny, nx, generator=gen, device="cuda", dtype=torch.float64)
    if corr > 0:
        f = [torch.fft.fftfreq(m, device="cuda", dtype=torch.float64) for m in (nz, ny)]
        fx = torch.fft.rfftfreq(nx, device="cuda", dtype=torch.float64)
        ker = torch.exp(-2.0 * (math.pi * corr) ** 2 *
                        (f[0][:, None, None] ** 2 + f[1][None, :, None] ** 2 +
                         fx[None, None, :] ** 2))
        g = torch.fft.irfftn(torch.fft.rfftn(g) * ker, s=(nz, ny, nx))
    g = g - g.mean()
    return 10.0 ** (base + std * g / g.std())


def _conduits(K, seed, count, value=1e-10):
    """Marks `count` random walks in K; returns the mask of their cells."""
    nz, ny, nx = K.shape
    rng = np.random.default_rng(seed)
    mask = torch.zeros(K.numel(), dtype=torch.uint8, device=K.device)
    for _ in range(count):
        c = torch.as_tensor(random_walk_conduit(rng, nx, ny, nz), device=K.device)
        K.view(-1)[c] = value
        mask[c] = 1
    return mask


def _grid(case, seed):
    """(Problem with device K, conduit mask) of a step-like case."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    K = _field(seed, nx, ny, nz, case["std"], case["corr"])
    mask = _conduits(K, seed + 1, case.get("conduits", 0))
    K = K.reshape(-1).contiguous()
    m = float(max(nx, ny, nz))
    return Problem(nx, ny, nz, 1.0 / m, 1.0 / m, 1.0 / m, K, K, K), mask


def _options(case):
    return dict(FAST if case["opt"] == "fast" else {}, tol=TOL)


def _sources(b, K, h, seed):
    """A right-hand side of another time: boundary inflow scaled cell by
    cell, and eight injection and eight production wells whose rates follow
    their cells' permeability."""
    rng = np.random.default_rng(seed + 2)
    out = b * torch.as_tensor(rng.uniform(0.5, 1.5, b.numel()), device=b.device)
    cells = torch.as_tensor(rng.choice(b.numel(), 16, replace=False), device=b.device)
    rate = torch.as_tensor(rng.uniform(0.1, 1.0, 16), device=b.device)
    rate[1::2] *= -1.0
    out[cells] += rate * K.reshape(-1)[cells] / h ** 2
    return out.contiguous()


def _batch_grids(case, seed):
    """The instances: edges in [lo, hi], std in [1, 1.3], 0-4 conduits."""
    rng = np.random.default_rng(seed)
    # the sizes are the case's own, the fields the seed's
    shape = np.random.default_rng(case["m"] * 1000 + case["hi"])
    out = []
    for i in range(case["m"]):
        nx, ny, nz = (int(v) for v in shape.integers(case["lo"], case["hi"] + 1, size=3))
        K = _field(seed + 10 * i, nx, ny, nz, float(rng.uniform(1.0, 1.3)), 4.0)
        _conduits(K, seed + 10 * i + 1, int(rng.integers(0, 5)))
        out.append(K)
    return out


def _picard_problem(case, seed):
    """The reference run script's layout on this grid: lateral faces at
    60 MPa, a conduit along x over 0.6 of the grid with nonlinear Robin ends
    and two fractures, a well column at 10 MPa above it."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    K = _field(seed, nx, ny, nz, case["std"], 0.0, base=-13.0).reshape(-1).cpu().numpy()
    prob = Problem(nx, ny, nz, 1.0, 5.0, 5.0, K, K, K, bc_type=(0, 0, 0, 0, 1, 1),
                   bc_value=(60e6, 60e6, 60e6, 60e6, 0.0, 0.0), visc=1e-3)
    ln = int(0.6 * nx)
    k = karst.Karst([ln], [(nx - ln) // 2], [ny // 2], [nz // 2 - 1], [1], [1e-11], [3], [3],
                    [[1.0], [1.0]], [[1.0], [1.0]], [1.01686094e-12], [3.1415], [2],
                    [[1e8 - 1.0], [1e8 - 1.0]], [[1.0], [1.0]],
                    [[max(1, ln // 5)], [(3 * ln) // 4]])
    wi, pw = np.zeros(prob.n), np.zeros(prob.n)
    for z in range(nz // 2, nz):
        c = nx // 2 + nx * (ny // 2 + ny * z)
        wi[c], pw[c] = 7.64352339e-13, 10e6
    return prob, k, wi, pw


def _bridge_arrays(case, seed):
    """solve_linsys's arguments on the host: per cell the seven coefficients
    (u, d, l, r, c, t, b), their cells (c, u, d, l, r, t, b; -1 outside) and
    two right-hand sides."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    h = 1.0 / max(nx, ny, nz)
    K = _field(seed, nx, ny, nz, case["std"], case["corr"])
    tx, ty, tz, lo, hi = _transmissibilities(K, K, K, h, h, h)
    diag = _diagonal(K.shape, tx, ty, tz, lo, hi)
    shape = (nz, ny, nx)
    E = torch.zeros(7, *shape, dtype=torch.float64, device="cuda")
    E[0, :, :-1], E[1, :, 1:] = ty, ty
    E[2, :, :, 1:], E[2, :, :, 0] = tx, lo
    E[3, :, :, :-1], E[3, :, :, -1] = tx, hi
    E[4] = diag
    E[5, :-1], E[6, 1:] = tz, tz
    s = torch.arange(nx * ny * nz, device="cuda", dtype=torch.int32).reshape(shape)
    I = torch.full((7, *shape), -1, dtype=torch.int32, device="cuda")
    I[0] = s
    I[1, :, :-1], I[2, :, 1:] = s[:, 1:], s[:, :-1]
    I[3, :, :, 1:], I[4, :, :, :-1] = s[:, :, :-1], s[:, :, 1:]
    I[5, :-1], I[6, 1:] = s[1:], s[:-1]
    b = torch.zeros(shape, dtype=torch.float64, device="cuda")
    b[:, :, 0] = lo
    b = b.reshape(-1)
    b2 = _sources(b, K, h, seed)
    host = lambda t: t.cpu().numpy()  # noqa: E731
    return (host(E.reshape(7, -1).t().contiguous()), host(I.reshape(7, -1).t().contiguous()),
            host(b), host(b2))


def _on_grid(x, step, top):
    """x rounded to multiples of `step`, at most `top` in size."""
    return (x / step).round().mul_(step).clamp_(-top, top)


def _layer_inputs(case, seed):
    """Activations after a ReLU (half of them zero), He-scaled weights, a
    small output gradient.  Activations and weights lie on binary grids (1/16
    and 1/1024) on which a layer's sums are exact in 32 bits in any order:
    whether a cell passes the ReLU, and with it every gradient, then never
    hangs on the rounding of a value next to zero."""
    n = case["nx"] * case["ny"] * case["nz"]
    cin, cout = case["cin"], case["cout"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(cin // 8, n, 8, generator=gen, device="cuda").relu()
    x = _on_grid(x, 1.0 / 16, 4.0).to(torch.bfloat16)
    w = torch.randn(27, cout, cin, generator=gen, device="cuda") * math.sqrt(2.0 / (27 * cin))
    w = _on_grid(w, 1.0 / 1024, 0.25)
    b = _on_grid(torch.randn(cout, generator=gen, device="cuda") * 0.1, 1.0 / 1024, 0.5)
    g = (torch.randn(cout // 8, n, 8, generator=gen, device="cuda") * 1e-2).to(torch.bfloat16)
    return x, w, b, g


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "guess", "resolve"):
        prob, mask = _grid(case, seed)
        st = {"kind": kind, "prob": prob, "mask": mask, "solver": gpu.Solver(**_options(case)),
              "x": torch.zeros(prob.n, dtype=torch.float64, device="cuda"),
              "v": torch.zeros(prob.n, 7, dtype=torch.float64, device="cuda")}
        if kind == "guess":
            st["model"] = guess.load(MODEL)
        if kind == "resolve":
            st["solver"].assemble(prob)
            st["solver"].setup()
            b = torch.as_tensor(st["solver"].rhs(), device="cuda")
            st["b"] = _sources(b, prob.KX, prob.hx, seed)
        return st
    if kind == "picard":
        return {"kind": kind, "run": _picard_problem(case, seed),
                "solver": gpu.Solver(**_options(case))}
    if kind == "bridge":
        return {"kind": kind, "args": _bridge_arrays(case, seed),
                "dims": (case["nx"], case["ny"], case["nz"])}
    if kind == "batch":
        probs = []
        for K in _batch_grids(case, seed):
            nz, ny, nx = K.shape
            k = K.reshape(-1).cpu().numpy()
            probs.append(Problem(nx, ny, nz, 1.0 / 64, 1.0 / 64, 1.0 / 64, k, k, k))
        return {"kind": kind, "probs": probs, "opt": case["opt"]}
    dims = (case["nx"], case["ny"], case["nz"])
    if kind == "trunk":
        K = _field(seed, *dims, 1.5, 8.0)
        mask = _conduits(K, seed + 1, 4)
        return {"kind": kind, "dims": dims, "K": K.reshape(-1).contiguous(), "mask": mask,
                "model": guess.load(MODEL)}
    x, w, b, g = _layer_inputs(case, seed)
    return {"kind": kind, "dims": dims, "g": g,
            "in": [t.requires_grad_(True) for t in (x, w, b)]}


# ---- one pass -----------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "step":
        s, prob, x = state["solver"], state["prob"], state["x"]
        s.assemble(prob)
        s.setup()
        s.solve(x=x.zero_())
        return {"p": x, "v": s.fluxes(x, state["v"])[0]}
    if kind == "guess":
        s, prob, x = state["solver"], state["prob"], state["x"]
        guess.solve_from_guess(s, prob, state["model"], prob.KX, mask=state["mask"], x=x)
        return {"p": x, "v": s.fluxes(x, state["v"])[0]}
    if kind == "resolve":
        s, x = state["solver"], state["x"]
        s.solve(b=state["b"], x=x.zero_())
        return {"p": x}
    if kind == "picard":
        prob, k, wi, pw = state["run"]
        r = karst.picard(state["solver"], k, prob, wi, pw)
        return {f: r[f] for f in ("p", "pc", "ucl", "ucr", "qk", "v")}
    if kind == "bridge":
        perm, ind, b, b2 = state["args"]
        out = []
        x = np.zeros(len(b))
        for rhs in (b, b2):
            gpu.solve_linsys(perm, ind, rhs, x, *state["dims"])
            out.append(x.copy())
        return out
    if kind == "batch":
        o = dict(FAST) if state["opt"] == "fast" else {}
        prec = o.pop("precision", 0)
        r = batch.solve_batch_graph(state["probs"], precision=prec, tol=10 * TOL, options=o)
        return [x for x, _, _ in r]
    if kind == "trunk":
        with torch.no_grad():
            f = guess.features(state["K"], state["mask"], state["dims"])
            return state["model"].trunk(f, state["dims"])
    x, w, b = state["in"]
    out = guess.conv(x, w, b, state["dims"])
    gx, gw, gb = torch.autograd.grad(out, (x, w, b), state["g"])
    return {"out": out.detach(), "gx": gx, "gw": gw, "gb": gb}


# ---- what a pass cannot do without ---------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "batch":
        n = sum(int(K[0] * K[1] * K[2]) for K in _batch_sizes(case))
        return {"bytes": 16.0 * n, "flops": 0}
    n = float(case["nx"]) * case["ny"] * case["nz"]
    if kind in ("step", "guess"):       # K in; p and seven flux fields out
        return {"bytes": (8 + 8 + 56) * n, "flops": 0}
    if kind == "resolve":               # four coefficients and b in, x out
        return {"bytes": (32 + 8 + 8) * n, "flops": 0}
    if kind == "picard":                # K, well index and pressure in; p and fluxes out
        return {"bytes": (24 + 8 + 56) * n, "flops": 0}
    if kind == "bridge":                # the seven coefficients and cells, two b and x
        return {"bytes": 2 * (56 + 28 + 8 + 8) * n, "flops": 0}
    if kind == "trunk":                 # K and the mask in, 16 channels out
        f = 0.0
        for (name, cin, cout) in guess.UNet.SPEC:
            f += 2.0 * 27 * cin * cout * n / {"e0": 1, "d0": 1, "e1": 8, "d1": 8, "bn": 64}[name[:2]]
        return {"bytes": (9 + 32) * n, "flops": f}
    ci, co = case["cin"], case["cout"]  # x, gout in; out, gx out; three products
    return {"bytes": 4.0 * (ci + co) * n + 8.0 * 27 * ci * co, "flops": 3 * 2.0 * 27 * ci * co * n}


def _batch_sizes(case):
    shape = np.random.default_rng(case["m"] * 1000 + case["hi"])
    return [shape.integers(case["lo"], case["hi"] + 1, size=3) for _ in range(case["m"])]


# ---- the same in 64 bits, plain torch --------------------------------------------

def _transmissibilities(KX, KY, KZ, hx, hy, hz):
    """Interior face coefficients along x, y, z and the Dirichlet ones of
    the two x faces (two-point fluxes, harmonic means)."""
    hm = lambda a, b: 2.0 * a * b / (a + b)  # noqa: E731
    return (hm(KX[:, :, :-1], KX[:, :, 1:]) / hx ** 2, hm(KY[:, :-1], KY[:, 1:]) / hy ** 2,
            hm(KZ[:-1], KZ[1:]) / hz ** 2, 2.0 * KX[:, :, 0] / hx ** 2,
            2.0 * KX[:, :, -1] / hx ** 2)


def _diagonal(shape, tx, ty, tz, lo, hi):
    d = torch.zeros(shape, dtype=torch.float64, device=tx.device)
    d[:, :, 1:] += tx
    d[:, :, :-1] += tx
    d[:, 1:] += ty
    d[:, :-1] += ty
    d[1:] += tz
    d[:-1] += tz
    d[:, :, 0] += lo
    d[:, :, -1] += hi
    return d


def _solve(K, h, rhs):
    """Jacobi-preconditioned CG with residual replacement for each b of
    `rhs` (None: the boundary values'), to the accuracy FP64 allows."""
    tx, ty, tz, lo, hi = _transmissibilities(K, K, K, h, h, h)
    d = _diagonal(K.shape, tx, ty, tz, lo, hi)

    def apply(x):
        y = d * x
        y[:, :, :-1] -= tx * x[:, :, 1:]
        y[:, :, 1:] -= tx * x[:, :, :-1]
        y[:, :-1] -= ty * x[:, 1:]
        y[:, 1:] -= ty * x[:, :-1]
        y[:-1] -= tz * x[1:]
        y[1:] -= tz * x[:-1]
        return y

    out = []
    for b in rhs:
        if b is None:
            b = torch.zeros_like(K)
            b[:, :, 0] = lo
        b = b.reshape(K.shape)
        x = torch.zeros_like(K)
        bb = (b * b).sum()
        for _ in range(3):
            r = b - apply(x)
            z = r / d
            s = z.clone()
            rz = (r * z).sum()
            for it in range(20000):
                q = apply(s)
                a = rz / (s * q).sum()
                x += a * s
                r -= a * q
                z = r / d
                rz, old = (r * z).sum(), rz
                s = z + (rz / old) * s
                if it % 32 == 31 and float((r * r).sum() / bb) < 1e-29:
                    break
        out.append(x)
    return out, (tx, ty, tz, lo, hi)


def _fluxes(x, coeff, h):
    """(n, 7) face fluxes in the order u, d, l, r, c, t, b; c zero.  The
    outer faces: Dirichlet 1 at x = 0, 0 at x = 1, no flow elsewhere."""
    tx, ty, tz, lo, hi = coeff
    v = torch.zeros(7, *x.shape, dtype=torch.float64, device=x.device)
    f = h * ty * (x[:, :-1] - x[:, 1:])
    v[0, :, :-1], v[1, :, 1:] = f, -f
    f = h * tx * (x[:, :, :-1] - x[:, :, 1:])
    v[3, :, :, :-1], v[2, :, :, 1:] = f, -f
    v[2, :, :, 0] = h * lo * (x[:, :, 0] - 1.0)
    v[3, :, :, -1] = h * hi * x[:, :, -1]
    f = h * tz * (x[:-1] - x[1:])
    v[5, :-1], v[6, 1:] = f, -f
    return v.reshape(7, -1).t().contiguous()


def _taps(x, dims):
    """x (n, c) shifted by each of the 27 taps, zero outside, in tap order."""
    nx, ny, nz = dims
    g = torch.nn.functional.pad(x.reshape(nz, ny, nx, -1), (0, 0, 1, 1, 1, 1, 1, 1))
    for t in range(27):
        dz, dy, dx = t // 9, (t // 3) % 3, t % 3
        yield t, g[dz:dz + nz, dy:dy + ny, dx:dx + nx].reshape(nx * ny * nz, -1)


def _conv64(x, w, dims):
    out = 0.0
    for t, xs in _taps(x, dims):
        out = out + xs @ w[t].t()
    return out


def _rows(x):   # channel-blocked (c/8, n, 8) -> (n, c) in 64 bits
    return x.detach().double().permute(1, 0, 2).reshape(x.shape[1], -1)


def _blocked(x):
    return x.reshape(x.shape[0], -1, 8).permute(1, 0, 2).contiguous()


def _trunk64(model, f, dims):
    def conv(x, name, d):
        w = model.w[name].detach().to(torch.bfloat16).double()
        return (_conv64(x, w, d) + model.b[name].detach().double()).relu()

    def block(x, a, d):
        return conv(conv(x, a + "a", d), a + "b", d)

    def pool(x, d):
        nx, ny, nz = d
        g = x.reshape(nz // 2, 2, ny // 2, 2, nx // 2, 2, -1).mean((1, 3, 5))
        return g.reshape(-1, x.shape[1]), (nx // 2, ny // 2, nz // 2)

    def up(x, skip, d):
        nx, ny, nz = d
        g = x.reshape(nz // 2, 1, ny // 2, 1, nx // 2, 1, -1)
        g = g.expand(-1, 2, -1, 2, -1, 2, -1).reshape(nx * ny * nz, -1)
        return torch.cat([g, skip], 1)

    e0 = block(f, "e0", dims)
    x, d1 = pool(e0, dims)
    e1 = block(x, "e1", d1)
    x, d2 = pool(e1, d1)
    x = block(x, "bn", d2)
    x = block(up(x, e1, d1), "d1", d1)
    return block(up(x, e0, dims), "d0", dims)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "guess", "resolve"):
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        n = nx * ny * nz
        if n > 6_000_000:  # tens of thousands of plain CG steps: minutes
            return None
        K = _field(seed, nx, ny, nz, case["std"], case["corr"])
        _conduits(K, seed + 1, case["conduits"])
        h = 1.0 / float(max(nx, ny, nz))
        if kind == "resolve":
            b = torch.zeros_like(K)
            b[:, :, 0] = 2.0 * K[:, :, 0] / h ** 2
            (x,), _ = _solve(K, h, [_sources(b.reshape(-1), K, h, seed)])
            return {"p": x.reshape(-1)}
        (x,), coeff = _solve(K, h, [None])
        return {"p": x.reshape(-1), "v": _fluxes(x, coeff, h)}
    if kind == "picard":  # a nonlinear fixed point of eighty reservoir solves
        return None
    if kind == "bridge":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        h = 1.0 / max(nx, ny, nz)
        K = _field(seed, nx, ny, nz, case["std"], case["corr"])
        b = torch.zeros_like(K)
        b[:, :, 0] = 2.0 * K[:, :, 0] / h ** 2
        (x, x2), _ = _solve(K, h, [b, _sources(b.reshape(-1), K, h, seed)])
        return [x.reshape(-1), x2.reshape(-1)]
    if kind == "batch":  # as many plain solves as instances: the smaller batches
        grids = _batch_grids(case, seed)
        if sum(K.numel() for K in grids) > 1_000_000:
            return None
        return [_solve(K, 1.0 / 64, [None])[0][0].reshape(-1) for K in grids]
    dims = (case["nx"], case["ny"], case["nz"])
    if kind == "trunk":
        nx, ny, nz = dims
        K = _field(seed, *dims, 1.5, 8.0)
        mask = _conduits(K, seed + 1, 4)
        f = torch.zeros(nx * ny * nz, guess.IN_CH, dtype=torch.float64, device="cuda")
        f[:, 0] = (torch.log10(K.reshape(-1)) + 14.0) / 2.0
        f[:, 1] = mask.double()
        i = torch.arange(nx * ny * nz, device="cuda") % nx
        f[:, 2] = (i == 0).double() - (i == nx - 1).double()
        return _blocked(_trunk64(guess.load(MODEL), f, dims))
    x, w, b, g = _layer_inputs(case, seed)
    xr, gr = _rows(x), _rows(g)
    wr = w.to(torch.bfloat16).double()  # the products take 16-bit operands
    y = _conv64(xr, wr, dims) + b.double()
    gr = gr * (y > 0)
    gx = _conv64(gr, wr.flip(0).transpose(1, 2), dims)
    gw = torch.stack([gr.t() @ xs for _, xs in _taps(xr, dims)])
    return {"out": _blocked(y.relu()), "gx": _blocked(gx), "gw": gw, "gb": gr.sum(0)}

"""The work that a user of this package has it do, as cases that can be timed and compared.

Each case goes through the public entry points (dictIn.Run, RunBatch, BatchSolver,
EikonalValues, a solved Interface, Selling.Decomposition, WarmStart's UNet) on synthetic
fields of the distributions that the package's benchmark and tests use: Isotropic costs
exp(0.5 g), Riemannian metrics R(theta) diag(1, lambda) R(theta)^T with smoothed theta
and lambda uniform in [1, 100], and in 3D eigenvalues log-uniform in [1, 25] with
smoothed rotations.  All inputs come from the seed alone and are made on the GPU.

`exact` solves the same discrete scheme in 64 bits with plain torch operations: Selling's
decomposition, then value iteration to its fixed point, and for the sensitivities
iteration of the transposed linear system.
"""
import math

import numpy as np
import torch

from adaptivegriddiscretizations_b200 import Eikonal, Selling
from adaptivegriddiscretizations_b200.Eikonal.HFM_CUDA import Interface
from adaptivegriddiscretizations_b200.WarmStart.unet import UNet
from adaptivegriddiscretizations_b200.autograd import eikonal_values

INF = math.inf


# ----------------------------------------------------------------------------- cases --
def listed():
    return [
        # the smallest call: one Isotropic2 solve of the 256 x 256 configuration, tolerance 1e-6
        {"name": "run_iso2_256", "kind": "run", "model": "Isotropic2", "n0": 256, "n1": 256, "nseeds": 1, "tol": 1e-6},
        # one ordinary anisotropic solve, default tolerances, several seeds
        {"name": "run_riem2_512", "kind": "run", "model": "Riemann2", "n0": 512, "n1": 512, "nseeds": 4},
        # a large ragged grid, float64 values by the multiprecision scheme
        {"name": "run_iso2_f64_1203x1501", "kind": "run", "model": "Isotropic2", "n0": 1203, "n1": 1501, "nseeds": 1,
         "float64": True},
        # a large 3D solve with a variable cost, odd sides
        {"name": "run_iso3_201", "kind": "run", "model": "Isotropic3", "n0": 201, "n1": 201, "n2": 201, "nseeds": 1},
        # a large 3D solve with reverse sensitivity of the arrival times at 128 receivers
        {"name": "run_riem3_200_reverse", "kind": "run", "model": "Riemann3", "n0": 200, "n1": 200, "n2": 200,
         "nseeds": 1, "receivers": 128},
        # inversion of a cost field by autograd: values and gradient, obstacles, ragged sides
        {"name": "grad_riem2_walls_301x413", "kind": "grad", "model": "Riemann2", "n0": 301, "n1": 413, "nseeds": 2,
         "receivers": 64, "walls": True},
        # minimal paths from 64 tips on a solved 1024 x 1024 problem, each followed for 1200 steps
        {"name": "geodesics_riem2_1024", "kind": "geodesics", "n0": 1024, "n1": 1024, "tips": 64, "steps": 1200},
        # serving: repeated batches of one configuration (the benchmark's workload)
        {"name": "batch_riem2_512x128", "kind": "batch", "model": "Riemann2", "n0": 512, "n1": 512, "batch": 128,
         "nseeds": 4},
        # many solves of uneven sizes and source sets in one launch, both models
        {"name": "uneven_48", "kind": "uneven", "count": 48},
        # the learned warm start's prediction for a serving batch: 128 problems of 512 x 512
        {"name": "unet_forward_128", "kind": "unet_forward", "batch": 128, "side": 128},
        # one training step of that network at its training batch
        {"name": "unet_train_32", "kind": "unet_train", "batch": 32, "side": 128},
        # the standalone decomposition of a 3D tensor field
        {"name": "selling3_110", "kind": "selling", "ndim": 3, "count": 110 ** 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "grad", "geodesics", "batch", "uneven", "unet_forward", "unet_train",
                       "selling"])
    if kind in ("run", "grad"):
        model = rng.choice(["Isotropic2", "Riemann2", "Isotropic3", "Riemann3"])
        if model.endswith("2"):
            hi = {"run": 1400, "grad": 700}[kind]
            c = {"kind": kind, "model": model, "n0": _log_int(rng, 64, hi), "n1": _log_int(rng, 64, hi)}
        else:
            hi = {"run": 200, "grad": 100}[kind]
            c = {"kind": kind, "model": model, **{k: _log_int(rng, 24, hi) for k in ("n0", "n1", "n2")}}
        c["nseeds"] = rng.randint(1, 8)
        if kind == "grad":
            c["receivers"] = _log_int(rng, 8, 256)
            c["walls"] = rng.random() < 0.4
        elif rng.random() < 0.3:
            c["receivers"] = _log_int(rng, 8, 256)
        elif rng.random() < 0.3:
            c["float64"] = True
        return c
    if kind == "geodesics":
        n = _log_int(rng, 96, 1100)
        return {"kind": kind, "n0": n, "n1": n + rng.randint(0, n // 8), "tips": _log_int(rng, 1, 64),
                "steps": rng.randint(n // 2, n)}
    if kind == "batch":
        model = rng.choice(["Isotropic2", "Riemann2"])
        n0, n1 = _log_int(rng, 64, 512), _log_int(rng, 64, 512)
        return {"kind": kind, "model": model, "n0": n0, "n1": n1, "nseeds": rng.randint(1, 8),
                "batch": _log_int(rng, 4, min(256, 128 * 512 * 512 // (n0 * n1)))}
    if kind == "uneven":
        return {"kind": kind, "count": _log_int(rng, 4, 60)}
    if kind == "unet_forward":
        return {"kind": kind, "batch": _log_int(rng, 1, 127), "side": rng.choice([64, 128])}
    if kind == "unet_train":
        return {"kind": kind, "batch": _log_int(rng, 4, 31), "side": rng.choice([64, 128])}
    return {"kind": kind, "ndim": rng.choice([2, 3]), "count": _log_int(rng, 1000, 1300000)}


# ---------------------------------------------------------------------------- inputs --
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _smooth(shape, sigma, gen, fields=1):
    """Periodic Gaussian-smoothed white noise, unit variance, (fields, *shape)."""
    if fields > 32:
        return torch.cat([_smooth(shape, sigma, gen, min(32, fields - k)) for k in range(0, fields, 32)])
    g = torch.randn((fields,) + shape, generator=gen, device="cuda")
    filt = torch.ones((), device="cuda")
    for k, n in enumerate(shape):
        f = torch.fft.fftfreq(n, device="cuda") if k < len(shape) - 1 else torch.fft.rfftfreq(n, device="cuda")
        e = torch.exp(-2.0 * math.pi ** 2 * sigma ** 2 * f ** 2)
        filt = filt * e.reshape((-1,) + (1,) * (len(shape) - 1 - k))
    dims = tuple(range(1, len(shape) + 1))
    g = torch.fft.irfftn(torch.fft.rfftn(g, dim=dims) * filt, s=shape, dim=dims)
    return g / g.std()


def _cost(shape, gen, count=1):
    """(count, *shape)."""
    return torch.exp(0.5 * _smooth(shape, 8.0 if len(shape) == 2 else 6.0, gen, count)).contiguous()


def _metric(shape, gen, count=1):
    """HFM layout (count, *shape, symdim), (*shape, symdim) in 3D."""
    if len(shape) == 2:
        th = torch.atan2(_smooth(shape, 8.0, gen, count), _smooth(shape, 8.0, gen, count))
        lam = 1.0 + 99.0 * torch.rand((count,) + shape, generator=gen, device="cuda")
        c, s = torch.cos(th), torch.sin(th)
        return torch.stack([c * c + lam * s * s, c * s * (1 - lam), s * s + lam * c * c], -1).contiguous()
    w, x, y, z = torch.nn.functional.normalize(_smooth(shape, 6.0, gen, 4), dim=0)
    rows = [[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
            [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
            [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]]
    ev = torch.exp(math.log(25.0) * torch.rand((3,) + shape, generator=gen, device="cuda"))
    return torch.stack([sum(rows[i][k] * ev[k] * rows[j][k] for k in range(3)) for i in range(3)
                        for j in range(i + 1)], -1).contiguous()


def _points(shape, h, count, gen, margin=0.05):
    """Indices (count, ndim) and coordinates of grid points, distinct, host float32."""
    seen, out = set(), []
    while len(out) < count:
        r = torch.rand(len(shape), generator=gen, device="cuda").cpu().numpy()
        i = tuple(int((margin + (1 - 2 * margin) * r[k]) * n) for k, n in enumerate(shape))
        if i not in seen:
            seen.add(i)
            out.append(i)
    idx = np.array(out, np.int64)
    return idx, ((idx + 0.5) * h).astype(np.float32)


def _shape(case):
    return tuple(case[k] for k in ("n0", "n1", "n2") if k in case)


def _problem(case, gen):
    """One eikonal problem: dictIn keys, and what `exact` needs."""
    shape = _shape(case)
    h = np.float32(1.0 / max(shape))
    seeds_i, seeds = _points(shape, h, case["nseeds"], gen)
    d = {"model": case["model"], "mode": "gpu", "verbosity": 0, "dims": list(shape), "gridScale": float(h),
         "origin": [0.0] * len(shape), "seeds": seeds, "exportValues": True}
    p = {"shape": shape, "h": float(h), "seeds": seeds_i, "metric": None, "cost": None}
    if case["model"].startswith("Isotropic") or case["kind"] == "grad":
        d["cost"] = p["cost"] = _cost(shape, gen)[0]
    if case["model"].startswith("Riemann"):
        d["metric"] = p["metric"] = _metric(shape, gen).reshape(shape + (-1,))
    if "tol" in case:
        d["tol"] = case["tol"]
    if case.get("float64"):
        d["values_float64"] = True
    if case.get("walls"):  # a straight wall with a gap across the middle of the domain
        w = torch.zeros(shape, dtype=torch.bool, device="cuda")
        w[shape[0] // 2, : (3 * shape[1]) // 4] = True
        w[tuple(seeds_i.T)] = False
        d["walls"] = w
    if case.get("receivers"):
        r_i, _ = _points(shape, h, case["receivers"], gen, 0.02)
        sens = torch.zeros(shape, device="cuda")
        sens[tuple(torch.as_tensor(r_i.T, device="cuda"))] = 1.0
        p["sens"] = sens
        if case["kind"] == "run":
            d["sensitivity"] = sens[..., None].contiguous()
    return d, p


def _uneven_side(k):
    return (64, 128, 256, 384, 512)[(3 * k + k // 5) % 5]


def _uneven(case, seed):
    """Both models in turn, 1 to 8 seeds."""
    gen, out = _generator(seed), []
    for k in range(case["count"]):
        n = _uneven_side(k)
        c = {"kind": "run", "model": ("Isotropic2", "Riemann2")[k % 2], "n0": n, "n1": n, "nseeds": 1 + 5 * k % 8}
        out.append(_problem(c, gen))
    return out


def _batch_inputs(case, seed):
    gen = _generator(seed)
    shape, B = _shape(case), case["batch"]
    h = np.float32(1.0 / max(shape))
    riem = case["model"] == "Riemann2"
    data = _metric(shape, gen, B) if riem else _cost(shape, gen, B)
    idx = torch.stack([torch.randint(0, n, (B, case["nseeds"]), generator=gen, device="cuda") for n in shape], -1)
    seeds = ((idx + 0.5) * float(h)).float().contiguous()
    return shape, float(h), data, idx, seeds


def _smooth_values(shape, gen):
    """A metric pulled back from the Euclidean one by a smooth map x -> y(x), its exact distance
    to a seed (a solution whose geodesics are smooth curves), and tips at least 0.31 away from it."""
    h = 1.0 / max(shape)
    ax = [(torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) * h for n in shape]
    X = torch.meshgrid(*ax, indexing="ij")
    a, b, c, e = (0.2 + 0.8 * torch.rand(4, generator=gen, device="cuda")).tolist()
    s0, s1 = 0.05 * a, 0.05 * b
    y0 = X[0] + s0 * torch.sin(2 * math.pi * (X[1] + c))
    y1 = 1.5 * X[1] + s1 * torch.sin(2 * math.pi * (X[0] + e))
    j01 = 2 * math.pi * s0 * torch.cos(2 * math.pi * (X[1] + c))
    j10 = 2 * math.pi * s1 * torch.cos(2 * math.pi * (X[0] + e))
    one = torch.ones_like(j01)
    m = torch.stack([one + j10 * j10, j01 * one + 1.5 * j10, j01 * j01 + 2.25 * one], -1).float().contiguous()
    seeds_i, seeds = _points(shape, np.float32(h), 1, gen, 0.3)
    i, j = seeds_i[0]
    u = torch.sqrt((y0 - y0[i, j]) ** 2 + (y1 - y1[i, j]) ** 2).float().contiguous()
    tips = (0.12 + 0.76 * torch.rand((1024, 2), generator=gen, device="cuda").cpu().numpy()) * np.array(shape) * h
    tips = tips[np.linalg.norm(tips - seeds[0], axis=1) > 0.31]
    return h, m, u, seeds, tips[:64].astype(np.float32)


def prepare(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    if kind == "run":
        return {"kind": kind, "d": _problem(case, gen)[0]}
    if kind == "grad":
        d, p = _problem(case, gen)
        cost = d.pop("cost")
        return {"kind": kind, "h": Eikonal.dictIn(d), "cost": cost.requires_grad_(True), "cotangent": p["sens"]}
    if kind == "uneven":
        return {"kind": kind, "ds": [d for d, _ in _uneven(case, seed)]}
    if kind == "batch":
        shape, h, data, _, seeds = _batch_inputs(case, seed)
        template = Eikonal.dictIn({"model": case["model"], "mode": "gpu", "verbosity": 0, "dims": list(shape),
                                   "gridScale": h, "origin": [0.0, 0.0]})
        key = "metric" if case["model"] == "Riemann2" else "cost"
        return {"kind": kind, "solver": Eikonal.BatchSolver(template, case["batch"]), "in": {key: data, "seeds": seeds}}
    if kind == "geodesics":  # a solved problem, as Run(retself=True) hands it back
        h, m, u, seeds, tips = _smooth_values(_shape(case), gen)
        itf = Interface(Eikonal.dictIn({
            "model": "Riemann2", "mode": "gpu", "verbosity": -2, "dims": list(_shape(case)), "gridScale": h,
            "origin": [0.0, 0.0], "metric": m, "seeds": seeds, "values": u, "tips": tips[: case["tips"]],
            "geodesic_max_length": case["steps"] + 1, "geodesic_typical_length": case["steps"] + 1}))
        itf.SetKernelTraits()
        itf.SetGeometry()
        itf.SetArgs()
        itf.PostProcess()
        return {"kind": kind, "itf": itf, "read": {k: list(v) if isinstance(v, list) else dict(v)
                                                   for k, v in itf.hfmOut["keys"].items()}}
    if kind == "unet_forward":
        x = torch.randn((case["batch"], case["side"], case["side"], 8), generator=gen, device="cuda").bfloat16()
        return {"kind": kind, "net": UNet(seed=seed % (1 << 31)), "x": x}
    if kind == "unet_train":
        n, s = case["batch"], case["side"]
        x = torch.randn((n, s, s, 8), generator=gen, device="cuda").bfloat16()
        t = 0.2 * _smooth((s, s), 8.0, gen, n)
        net = UNet(seed=seed % (1 << 31))
        for b in [l.b for l in net.layers()] + [net.hb]:  # as in the course of a training
            b.copy_(0.05 * torch.randn(b.shape, generator=gen, device="cuda"))
        return {"kind": kind, "net": net, "x": x, "t": t.contiguous()}
    # selling: symmetric positive definite matrices (ndim, ndim, count)
    nd = case["ndim"]
    f = torch.randn((nd, nd, case["count"]), generator=gen, device="cuda")
    m = 0.2 * torch.eye(nd, device="cuda")[:, :, None] + torch.einsum("ikn,jkn->ijn", f, f)
    return {"kind": kind, "m": m.contiguous()}


# ------------------------------------------------------------------------------- run --
def run(state):
    kind = state["kind"]
    if kind == "run":
        out = Eikonal.dictIn(state["d"]).Run()
        return {k: out[k] for k in ("values", "costSensitivity", "seedValueSensitivity") if k in out.keys()}
    if kind == "grad":
        v = eikonal_values(state["h"], state["cost"])
        (g,) = torch.autograd.grad(v, state["cost"], state["cotangent"])
        return {"values": v.detach(), "gradient": g}
    if kind == "uneven":
        outs = Eikonal.RunBatch([Eikonal.dictIn(d) for d in state["ds"]])
        return [o["values"] for o in outs]
    if kind == "batch":
        return state["solver"].submit(**state["in"]).result()
    if kind == "geodesics":
        itf = state["itf"]  # each key is read once per call: the record of an earlier call is put back
        itf.hfmOut["keys"].update({k: list(v) if isinstance(v, list) else dict(v) for k, v in state["read"].items()})
        itf.GetGeodesics()
        return itf.hfmOut["geodesics"]
    if kind == "unet_forward":
        return state["net"].forward(state["x"])
    if kind == "unet_train":
        net = state["net"]
        r = net.forward(state["x"])
        net.backward(state["t"], state["t"].numel())
        net.step(1e-4)
        return {"r": r, "w": [x for l in net.layers() for x in (l.w, l.b)], "head": [net.hw, net.hb],
                "moments": [x for l in net.layers() for x in (l.mw, l.mb)], "head_moments": [net.mhw, net.mhb]}
    return Selling.Decomposition(state["m"])


# ------------------------------------------------------------------------------ work --
def _solve_work(shape, model, receivers):
    n = math.prod(shape)
    sd = {"Isotropic2": 0, "Isotropic3": 0, "Riemann2": 3, "Riemann3": 6}[model]
    k = sd or len(shape)
    # the metric and/or cost read, the values written; one update a point
    b, f = n * 4 * ((sd or 1) + 1), n * 12 * k
    if receivers:  # the sensitivity read, the cost's sensitivity written; a product and a sum per active neighbour
        b, f = b + 8 * n, f + 2 * k * n
    return b, f


def _unet_flops(side):
    px = [side * side >> (2 * k) for k in range(4)]
    c = (32, 64, 128, 256)
    f = px[0] * (8 * c[0] + c[0] * c[0]) + px[1] * (c[0] * c[1] + c[1] ** 2) + px[2] * (c[1] * c[2] + c[2] ** 2)
    f += px[3] * (c[2] * c[3] + c[3] ** 2) + px[2] * ((c[3] + c[2]) * c[2] + c[2] ** 2)
    f += px[1] * ((c[2] + c[1]) * c[1] + c[1] ** 2) + px[0] * ((c[1] + c[0]) * c[0] + c[0] ** 2)
    return 18.0 * f


def work(case):
    kind = case["kind"]
    if kind in ("run", "grad"):
        b, f = _solve_work(_shape(case), case["model"], case.get("receivers"))
    elif kind == "uneven":
        b, f = 0, 0
        for k in range(case["count"]):
            x, y = _solve_work((_uneven_side(k),) * 2, ("Isotropic2", "Riemann2")[k % 2], 0)
            b, f = b + x, f + y
    elif kind == "batch":
        b, f = (case["batch"] * x for x in _solve_work(_shape(case), case["model"], 0))
    elif kind == "geodesics":  # a point written, and four cells' flow read every fourth step
        steps = case["tips"] * case["steps"]
        b, f = steps * (8 + 16), steps * 100
    elif kind == "unet_forward":
        b, f = case["batch"] * case["side"] ** 2 * (16 + 4), case["batch"] * _unet_flops(case["side"])
    elif kind == "unet_train":
        b, f = case["batch"] * case["side"] ** 2 * (16 + 8) + 28 * 1.9e6, 3 * case["batch"] * _unet_flops(case["side"])
    else:
        nd, sd = case["ndim"], case["ndim"] * (case["ndim"] + 1) // 2
        b, f = case["count"] * 4 * (sd + sd + nd * sd), case["count"] * 60 * sd
    return {"bytes": float(b), "flops": float(f)}


def tolerance(case):
    kind = case["kind"]
    if kind in ("run", "grad") and case.get("receivers"):
        # sensitivities: the flow weights are differences of values known to the stopping tolerance
        # (5e-6 of the values; 3.3e-5 off the 64-bit solution, 1.2e-6 between two runs)
        return {"rel": 2e-4, "max": 2e-2}
    if kind in ("run", "grad", "uneven", "batch"):
        # two solves that stop within a few times 5e-6 of the same fixed point, 5e-7 off it in
        # the mean; single points differ by up to 6e-5 between two runs
        return {"rel": 1e-5, "max": 4e-4}
    if kind == "geodesics":  # 1200 steps in float32 along smooth curves
        return {"rel": 1e-5, "max": 1e-4}
    if kind == "unet_forward":  # bf16 activations: 6.5e-3 off 64 bits
        return {"rel": 2e-2, "max": 0.5}
    if kind == "unet_train":  # gradients to 2e-3; an Adam step turns on a gradient's sign where it is small
        return {"rel": 1e-2, "max": 0.5}
    return {"rel": 1e-6, "max": 1e-5, "differ": 0.0}


# ----------------------------------------------------------------------------- exact --
def _perp(b, nd):
    if nd == 2:
        return [torch.stack([-b[k][1], b[k][0]]) for k in (2, 0, 1)]
    c = torch.linalg.cross
    pairs = ((2, 3), (1, 3), (1, 2), (0, 3), (0, 2), (0, 1))
    return [c(b[i], b[j], dim=0) for i, j in pairs]


def _selling(D):
    """Weights (symdim, N) and offsets (symdim, ndim, N) of the matrices D (ndim, ndim, N)."""
    nd, N = D.shape[0], D.shape[2]
    eye = torch.eye(nd, dtype=torch.float64, device="cuda")
    b = [eye[k][:, None].expand(nd, N).clone() for k in range(nd)]
    b.append(-torch.ones((nd, N), dtype=torch.float64, device="cuda"))
    pairs = [(0, 1), (1, 2), (2, 0)] if nd == 2 else [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]

    def dot(i, j):
        return torch.einsum("in,ijn,jn->n", b[i], D, b[j])

    still = True
    for it in range(100):
        if it % 4 == 0 and not still:
            break
        still = False
        for i, j in pairs:
            pos = dot(i, j) > 0
            still = still or bool(pos.any())
            if nd == 2:
                k = 3 - i - j
                b[k] = torch.where(pos, b[i] - b[j], b[k])
            else:
                for k in set(range(4)) - {i, j}:
                    b[k] = torch.where(pos, b[k] + b[i], b[k])
            b[i] = torch.where(pos, -b[i], b[i])
    w = torch.stack([(-dot(i, j)).clamp_min(0) for i, j in pairs])
    return w, torch.stack(_perp(b, nd))


def _stencil(p, model):
    """Weights (K, N) and neighbour indices (K, 2, N), N outside the domain."""
    shape, h = p["shape"], p["h"]
    nd, N = len(shape), math.prod(shape)
    if model.startswith("Isotropic"):
        w = torch.full((nd, N), h ** -2, dtype=torch.float64, device="cuda")
        e = torch.eye(nd, dtype=torch.int64, device="cuda")[:, :, None]
    else:
        m = p["metric"].double().reshape(N, -1).T * h * h
        M, k = torch.empty((nd, nd, N), dtype=torch.float64, device="cuda"), 0
        for i in range(nd):
            for j in range(i + 1):
                M[i, j] = M[j, i] = m[k]
                k += 1
        w, e = _selling(torch.linalg.inv(M.permute(2, 0, 1)).permute(1, 2, 0))
        e = e.round().long()
    grid = torch.stack(torch.meshgrid(*[torch.arange(n, device="cuda") for n in shape], indexing="ij")).reshape(nd, N)
    idx = torch.empty((len(w), 2, N), dtype=torch.int64, device="cuda")
    for k in range(len(w)):
        for s in range(2):
            y = grid + (2 * s - 1) * e[k]
            ok, flat = torch.ones(N, dtype=torch.bool, device="cuda"), torch.zeros(N, dtype=torch.int64, device="cuda")
            for a, n in enumerate(shape):
                ok &= (y[a] >= 0) & (y[a] < n)
                flat = flat * n + y[a]
            idx[k, s] = torch.where(ok, flat, N)
    return w, idx


def _update(w, v, rhs):
    """The root u of sum_k w_k (u - v_k)_+^2 = rhs^2."""
    v, w = list(v), list(w)
    for i in range(len(v)):  # odd-even transposition sort of the (value, weight) pairs
        for j in range(i % 2, len(v) - 1, 2):
            keep = v[j] <= v[j + 1]
            v[j], v[j + 1] = torch.minimum(v[j], v[j + 1]), torch.maximum(v[j], v[j + 1])
            w[j], w[j + 1] = torch.where(keep, w[j], w[j + 1]), torch.where(keep, w[j + 1], w[j])
    v0 = v[0]
    a, b, c = w[0].clone(), torch.zeros_like(v0), -rhs * rhs
    stop = torch.zeros_like(v0, dtype=torch.bool)
    for q in range(1, len(v)):
        t = v[q] - v0
        stop |= ~torch.isfinite(t) | ((a * t - 2 * b) * t + c > 0)
        t = torch.where(stop, torch.zeros_like(t), t)
        wq = torch.where(stop, torch.zeros_like(t), w[q])
        a, b, c = a + wq, b + wq * t, c + wq * t * t
    r = (b + torch.sqrt((b * b - a * c).clamp_min(0))) / a
    return torch.where((a == 0) | ~torch.isfinite(v0), torch.full_like(v0, INF), v0 + r)


def _values64(w, idx, rhs, fixed):
    """The fixed point of the scheme by value iteration; fixed (N,): the seed values, NaN elsewhere."""
    N = rhs.numel()
    seed = ~torch.isnan(fixed)
    u = torch.full((N + 1,), INF, dtype=torch.float64, device="cuda")
    u[:N][seed] = fixed[seed]
    for it in range(1, 20001):
        v = torch.minimum(u[idx[:, 0]], u[idx[:, 1]])
        new = torch.where(seed, u[:N], torch.minimum(u[:N], _update(w, v, rhs)))
        if it % 32 == 0 and bool(((u[:N] - new) <= 1e-13 * new).logical_or(new == u[:N]).all()):
            u[:N] = new
            break
        u[:N] = new
    return u


def _adjoint64(w, idx, rhs, seed, u, s):
    """lam of diag lam - W^T lam = s, W the upwind weights at the solution u (N + 1,)."""
    N = rhs.numel()
    a, b = u[idx[:, 0]], u[idx[:, 1]]
    v = torch.minimum(a, b)
    val = _update(w, v, rhs)
    fw = (w * (val - v).clamp_min(0)).nan_to_num(0.0, 0.0, 0.0)
    fw[:, seed] = 0
    to = torch.where(a > b, idx[:, 1], idx[:, 0]).reshape(-1)
    diag = fw.sum(0)
    diag = torch.where(diag == 0, torch.ones_like(diag), diag)
    lam = torch.zeros_like(s)
    for it in range(1, 20001):
        acc = torch.zeros(N + 1, dtype=torch.float64, device="cuda").index_add_(0, to, (fw * lam).reshape(-1))[:N]
        new = (s + acc) / diag
        if it % 32 == 0 and bool(((new - lam).abs() <= 1e-13 * new.abs()).all()):
            return new
        lam = new
    return lam


def _exact_solve(problems, models):
    """Values of several problems, one iteration over all of their points."""
    K = max(len(p["shape"]) if m.startswith("Iso") else len(p["shape"]) * (len(p["shape"]) + 1) // 2
            for p, m in zip(problems, models))
    N = sum(math.prod(p["shape"]) for p in problems)
    w = torch.zeros((K, N), dtype=torch.float64, device="cuda")
    idx = torch.full((K, 2, N), N, dtype=torch.int64, device="cuda")
    rhs = torch.ones(N, dtype=torch.float64, device="cuda")
    fixed = torch.full((N,), math.nan, dtype=torch.float64, device="cuda")
    at, spans = 0, []
    for p, m in zip(problems, models):
        n = math.prod(p["shape"])
        pw, pi = _stencil(p, m)
        w[: len(pw), at:at + n] = pw
        idx[: len(pw), :, at:at + n] = torch.where(pi == n, N, pi + at)
        if p["cost"] is not None:
            rhs[at:at + n] = p["cost"].detach().double().reshape(-1)
        seeds = torch.as_tensor(np.ravel_multi_index(np.asarray(p["seeds"]).T, p["shape"]), device="cuda")
        fixed[at + seeds] = 0.0
        spans.append((at, n))
        at += n
    u = _values64(w, idx, rhs, fixed)
    return w, idx, rhs, ~torch.isnan(fixed), u, [u[a:a + n].reshape(p["shape"]) for (a, n), p in zip(spans, problems)]


def _exact_unet(net, x, t=None):
    """The network in 64 bits on its bf16 weights; with t, the gradients of the mean squared error."""
    F = torch.nn.functional
    ws = [l.wb[:, : 9 * l.cin].double().reshape(l.cout, 3, 3, l.cin).permute(0, 3, 1, 2).contiguous()
          for l in net.layers()]
    bs = [l.b.double() for l in net.layers()]
    hw, hb = net.hw.double(), net.hb.double()
    params = ws + bs + [hw, hb]
    grads = [torch.zeros_like(q) for q in params]
    outs = []

    def conv(k, y):
        return F.relu(F.conv2d(y, ws[k], bs[k], padding=1))

    for part, tp in zip(x.split(8), (t if t is not None else x).split(8)):
        for q in params:
            q.requires_grad_(t is not None)
        y = part.double().permute(0, 3, 1, 2)
        skips = []
        for lev in range(4):
            y = conv(2 * lev + 1, conv(2 * lev, y))
            if lev < 3:
                skips.append(y)
                y = F.avg_pool2d(y, 2)
        for lev in range(3):
            y = torch.cat([F.interpolate(y, scale_factor=2, mode="nearest"), skips[2 - lev]], 1)
            y = conv(9 + 2 * lev, conv(8 + 2 * lev, y))
        r = (y * hw[:, None, None]).sum(1) + hb
        outs.append(r.detach())
        if t is not None:
            g = torch.autograd.grad(((r - tp.double()) ** 2).sum() / t.numel(), params)
            grads = [a + b for a, b in zip(grads, g)]
    return torch.cat(outs), grads


def _exact_train(net, x, t):
    r, g = _exact_unet(net, x, t)
    L, w, mom = net.layers(), [], []

    def adam(p, gr, lr=1e-4):  # the first step
        m, v = 0.1 * gr, 0.001 * gr * gr
        return p.double() - lr * (m / 0.1) / (torch.sqrt(v / 0.001) + 1e-8), m

    for k, l in enumerate(L):
        gw = torch.zeros_like(l.w, dtype=torch.float64)
        gw[:, : 9 * l.cin] = g[k].permute(0, 2, 3, 1).reshape(l.cout, -1)
        for p, gr in ((l.w, gw), (l.b, g[len(L) + k])):
            a, m = adam(p, gr)
            w.append(a)
            mom.append(m)
    heads = [adam(net.hw, g[-2]), adam(net.hb, g[-1])]
    return {"r": r, "w": w, "head": [a for a, _ in heads], "moments": mom, "head_moments": [m for _, m in heads]}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("geodesics", "selling") or case.get("walls"):
        return None  # whole numbers and piecewise choices beside the numbers; visibility around walls
    if kind in ("run", "grad"):
        _, p = _problem(case, _generator(seed))
        w, idx, rhs, is_seed, u, (v,) = _exact_solve([p], [case["model"]])
        if not case.get("receivers"):
            return {"values": v}
        lam = _adjoint64(w, idx, rhs, is_seed, u, p["sens"].double().reshape(-1))
        on_seeds = lam[torch.as_tensor(np.ravel_multi_index(p["seeds"].T, p["shape"]), device="cuda")].clone()
        lam[is_seed] = 0
        if kind == "grad":
            return {"values": v, "gradient": (lam * rhs).reshape(p["shape"])}
        return {"values": v, "costSensitivity": lam.reshape(p["shape"] + (1,)), "seedValueSensitivity": on_seeds[:, None]}
    if kind == "uneven":
        ps = [p for _, p in _uneven(case, seed)]
        return _exact_solve(ps, [("Isotropic2", "Riemann2")[k % 2] for k in range(len(ps))])[5]
    if kind == "batch":
        shape, h, data, seeds, _ = _batch_inputs(case, seed)
        key = "metric" if case["model"] == "Riemann2" else "cost"
        vs = []
        for k in range(0, case["batch"], 32):
            ps = [{"shape": shape, "h": h, "metric": None, "cost": None, "seeds": s.cpu().numpy(), key: d}
                  for d, s in zip(data[k:k + 32], seeds[k:k + 32])]
            vs += _exact_solve(ps, [case["model"]] * len(ps))[5]
        return torch.stack(vs)
    s = prepare(case, seed)
    if kind == "unet_forward":
        return _exact_unet(s["net"], s["x"])[0]
    return _exact_train(s["net"], s["x"], s["t"])

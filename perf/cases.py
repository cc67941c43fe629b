"""The workloads that speed is measured on, through the package's public entry points.

Kinds (a case's "kind"):
  single   darcy.solve: one field, host arrays in and out, as the reference's
           users call it
  batch    darcy.solve_batch: a stack of fields of one side
  uneven   darcy.solve_batch_uneven: fields of many sides in one call
  predict  capi.Net.predict_device: starts for a stack of fields already on
           the GPU, as the learned solve and a device-resident pipeline call it
  train    WarmStartNet.train_more: Adam steps on loaded pairs, from given weights
  learned  learn.solve_batch_learned: predicted starts, then the batched solve

The solutions come back whole, with the convergence flags. Iteration counts
and the last recursive residual are left out: they follow the rounding of the
dot products (the batched engine's launch shape is autotuned, and the last
iterations sit on a plateau near tol at high contrast), as the reference's own
follow its thread count.

Fields are thresholded Gaussian random fields (spectrum tau^(alpha-1)
(pi^2 |k|^2 + tau^2)^(-alpha/2), alpha 2, tau 3, two phases), made here on the
GPU in FP64 from the seed alone.
"""

from __future__ import annotations

import math

import numpy as np
import torch

TOL = 1e-10

# Two-phase permeabilities by contrast: the generator's defaults (4), a soft
# medium (100) and the hard medium of the combined workload (1e4). (At 1e6 the
# same kernels run, but a solution stopped at TOL moves by up to 3e-9 with the
# rounding of the dot products, the reference's own included, so two builds'
# solutions cannot be compared there.)
PHASES = {4: (12.0, 3.0), 100: (10.0, 0.1), 10_000: (1e2, 1e-2)}

# MG-PCG iterations to TOL to count operations with (rounded from solves of
# side 64 .. 2048; the count grows slowly with the side).
ITERATIONS = {4: 22, 100: 28, 10_000: 50}

# FP64 or FP32 operations of one iteration per cell: the operator (9), three
# dot products (6), three vector updates (6), and a W-cycle of two smoothing
# sweeps (18 each), a residual (10) and the transfers (4) per visit, levels
# summing to 2 fine visits.
OPS_PER_CELL = 21 + 2 * (2 * 18 + 10 + 4)

NET_WEIGHTS = [(32, 2), (32, 32), (32, 32), (32, 32), (32, 32), (1, 32)]  # (out, in) channels of the 3 x 3 layers
NET_MACS = 9 * sum(o * i for o, i in NET_WEIGHTS)  # per pixel, forward
NET_PARAMS = sum(9 * o * i + o for o, i in NET_WEIGHTS)


def listed():
    return [
        # the smallest call: the reference's own first example (64^2, default phases)
        {"name": "single 64 fp64", "kind": "single", "n": 64, "contrast": 4, "form": "fp64", "f": "one"},
        # an odd grid with a forcing field, at the contrast the reference quotes for odd sizes
        {"name": "single 511 fp64", "kind": "single", "n": 511, "contrast": 10_000, "form": "fp64", "f": "field"},
        # the headline field size, one solve at a time
        {"name": "single 1024 mixed", "kind": "single", "n": 1024, "contrast": 10_000, "form": "mixed", "f": "one"},
        # the largest single grid, drop-in form
        {"name": "single 2048 fp64", "kind": "single", "n": 2048, "contrast": 4, "form": "fp64", "f": "one"},
        # the headline benchmark: 8 large fields as one batch
        {"name": "batch 8x1024 mixed", "kind": "batch", "count": 8, "n": 1024, "contrast": 10_000, "form": "mixed"},
        # the other half of the metric: many small problems (operator-learning data sets)
        {"name": "batch 4096x64 mixed", "kind": "batch", "count": 4096, "n": 64, "contrast": 4, "form": "mixed"},
        # the same in the drop-in form, a smaller data set
        {"name": "batch 1024x64 fp64", "kind": "batch", "count": 1024, "n": 64, "contrast": 4, "form": "fp64"},
        # mid-size fields at mid contrast (the bulk of the combined workload)
        {"name": "batch 512x128 fp64", "kind": "batch", "count": 512, "n": 128, "contrast": 10_000, "form": "fp64"},
        # uneven sides in one call
        {"name": "uneven 640 mixed", "kind": "uneven", "count": 640, "low": 32, "high": 256, "contrast": 4,
         "form": "mixed"},
        # the warm-start network: prediction, training, and the solve that uses it
        {"name": "predict 2000x64", "kind": "predict", "count": 2000, "n": 64, "contrast": 4},
        {"name": "train 64 b256", "kind": "train", "count": 512, "n": 64, "contrast": 4, "batch": 256, "steps": 12},
        {"name": "learned 2048x64 mixed", "kind": "learned", "count": 2048, "n": 64, "contrast": 4, "form": "mixed"},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["single", "single", "single", "batch", "batch", "batch", "uneven", "predict", "train", "learned"])
    contrast = rng.choice([4, 100, 10_000])
    form = rng.choice(["fp64", "mixed"])
    if kind == "single":
        n = _log_int(rng, 40, 1600)
        return {"kind": kind, "n": n, "contrast": contrast, "form": form, "f": rng.choice(["one", "field"])}
    if kind == "batch":
        if rng.random() < 0.25:  # large fields: concurrent grid solves
            return {"kind": kind, "count": rng.randint(2, 6), "n": _log_int(rng, 384, 900),
                    "contrast": contrast, "form": form}
        n = _log_int(rng, 20, 200)
        return {"kind": kind, "count": max(8, min(6000, int(rng.uniform(0.1, 0.6) * (1 << 23) / n**2))), "n": n,
                "contrast": contrast, "form": form}
    if kind == "uneven":
        low = _log_int(rng, 12, 64)
        return {"kind": kind, "count": rng.randint(100, 600), "low": low, "high": rng.randint(low + 20, 220),
                "contrast": 4, "form": form}
    n = 2 * _log_int(rng, 12, 56)
    cells = 1 << 23
    if kind == "train":
        batch = max(4, min(256, int(rng.uniform(0.1, 0.8) * (1 << 20) / n**2)))
        return {"kind": kind, "count": 2 * batch + rng.randint(0, 40), "n": n, "contrast": 4, "batch": batch,
                "steps": rng.randint(2, 12)}
    count = max(4, int(rng.uniform(0.1, 0.9) * cells / n**2))
    case = {"kind": kind, "count": count, "n": n, "contrast": 4}
    return case if kind == "predict" else {**case, "form": form}


# ------------------------------------------------------------------ inputs


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _fields(count, n, contrast, g):
    """(count, n, n) two-phase fields, FP64 on the GPU."""
    k = torch.arange(n, device="cuda", dtype=torch.float64)
    cosine = torch.cos(math.pi * k[:, None] * (2 * k[None, :] + 1) / (2 * n)) * math.sqrt(2.0 / n)
    cosine[0] /= math.sqrt(2.0)
    amplitude = 3.0 / (math.pi**2 * (k[:, None] ** 2 + k[None, :] ** 2) + 9.0)
    amplitude[0, 0] = 0.0
    hi, lo = PHASES[contrast]
    out = torch.empty((count, n, n), device="cuda", dtype=torch.float64)
    step = max(1, (1 << 24) // (n * n))
    for at in range(0, count, step):
        c = min(step, count - at)
        noise = torch.randn((c, n, n), device="cuda", dtype=torch.float64, generator=g) * amplitude
        grf = cosine.T @ noise @ cosine
        out[at:at + c] = torch.where(grf >= 0, hi, lo)
    return out


def _sides(case):
    r = np.random.default_rng([case["count"], case["low"], case["high"]])  # the mix of sides belongs to the case
    return [int(round(math.exp(v))) for v in r.uniform(math.log(case["low"]), math.log(case["high"]), case["count"])]


def _forcing(case, g):
    """A smooth positive forcing field, or None for f = 1."""
    if case.get("f", "one") == "one":
        return None
    n = case["n"]
    x = (torch.arange(n, device="cuda", dtype=torch.float64) + 1) / (n + 1)
    c = torch.rand((3,), device="cuda", dtype=torch.float64, generator=g)
    return 1.0 + c[0] * torch.sin(3 * x)[:, None] * torch.cos(2 * x)[None, :] + 0.5 * c[1] * x[:, None] + 0.1 * c[2]


def _inputs(case, seed):
    """What a pass computes from, on the GPU: a (list of (count, n, n) stacks for uneven), f, weights."""
    g = _generator(seed)
    made = {}
    if case["kind"] == "uneven":
        made["sides"] = _sides(case)
        made["a"] = {n: _fields(made["sides"].count(n), n, case["contrast"], g) for n in sorted(set(made["sides"]))}
        return made
    made["a"] = _fields(case.get("count", 1), case["n"], case["contrast"], g)
    made["f"] = _forcing(case, g)
    if case["kind"] in ("predict", "train", "learned"):
        # He-uniform weights, the output layer scaled down, small biases
        parts = []
        for layer, (out, inp) in enumerate(NET_WEIGHTS):
            limit = math.sqrt(6.0 / (9 * inp)) * (0.1 if layer == len(NET_WEIGHTS) - 1 else 1.0)
            w = torch.rand((out, 9 * inp), device="cuda", dtype=torch.float64, generator=g)
            parts.append(((2 * w - 1) * limit).reshape(-1))
            parts.append(0.02 * torch.randn((out,), device="cuda", dtype=torch.float64, generator=g))
        made["weights"] = torch.cat(parts).float()
        # mean and spread of log a of such fields, RMS of u, reference forcing
        hi, lo = (math.log(v) for v in PHASES[case["contrast"]])
        made["scaling"] = [0.5 * (hi + lo), 0.5 * (hi - lo), 7e-3, 1.0]
    return made


def prepare(case, seed):
    import darcy_cpp_gb300 as darcy

    made = _inputs(case, seed)
    kind = case["kind"]
    state = {"kind": kind, "darcy": darcy, "form": case.get("form", "fp64")}
    if kind == "single":
        state["a"] = made["a"][0].cpu().numpy()
        state["f"] = 1.0 if made["f"] is None else made["f"].cpu().numpy()
    elif kind == "uneven":
        left = {n: list(v.cpu().numpy()) for n, v in made["a"].items()}
        state["a"] = [np.ascontiguousarray(left[n].pop()) for n in made["sides"]]
    elif kind != "predict":
        state["a"] = made["a"].cpu().numpy()
    if kind in ("predict", "train", "learned"):
        from darcy_cpp_gb300 import learn

        net = learn.WarmStartNet(case["n"], seed=1)
        state["weights"] = made["weights"].cpu().numpy()
        net.set_params(state["weights"])
        net.set_scaling(made["scaling"])
        state["net"], state["learn"] = net, learn
    if kind == "predict":
        state["a"] = made["a"]
        state["u0"] = torch.empty_like(made["a"])
    if kind == "train":
        u = _direct(made["a"], 1.0).cpu().numpy()
        net.handle.load_pairs(state.pop("a"), u)
        state["steps"], state["batch"] = case["steps"], case["batch"]
    return state


def run(state):
    kind = state["kind"]
    if kind == "single":
        res = state["darcy"].solve(state["a"], state["f"], tol=TOL, form=state["form"])
        return {"u": res.u, "converged": res.converged, "levels": res.levels}
    if kind == "batch":
        res = state["darcy"].solve_batch(state["a"], 1.0, tol=TOL, form=state["form"])
        return {"u": res.u, "converged": res.converged}
    if kind == "uneven":
        res = state["darcy"].solve_batch_uneven(state["a"], 1.0, tol=TOL, form=state["form"])
        # the solutions are views of one array, in order
        return {"u": res.u[0].base, "converged": res.converged, "levels": res.levels}
    if kind == "predict":
        a, u0 = state["a"], state["u0"]
        state["net"].handle.predict_device(a.data_ptr(), a.shape[0], u0.data_ptr(),
                                           stream=torch.cuda.current_stream().cuda_stream)
        return {"u0": u0}
    if kind == "train":
        state["net"].set_params(state["weights"])
        losses = state["net"].train_more(state["steps"], batch=state["batch"], lr=1e-3, seed=1)
        return {"losses": losses, "params": state["net"].params()}
    res = state["learn"].solve_batch_learned(state["net"], state["a"], 1.0, tol=TOL, form=state["form"])
    return {"u": res.u, "converged": res.converged}


def work(case):
    kind = case["kind"]
    if kind == "uneven":
        # sides spread evenly over their logarithm: the mean of n^2
        low, high = case["low"], case["high"]
        cells = case["count"] * (high**2 - low**2) / (2 * math.log(high / low))
    else:
        cells = case.get("count", 1) * case["n"] ** 2
    if kind == "predict":
        return {"bytes": 16 * cells + 4 * NET_PARAMS, "flops": 2 * NET_MACS * cells}
    if kind == "train":
        pixels = case["steps"] * case["batch"] * case["n"] ** 2
        # features (two BF16 channels), target and permeability read once a step; weights and moments updated
        return {"bytes": 12 * pixels + case["steps"] * 24 * NET_PARAMS, "flops": 6 * NET_MACS * pixels}
    flops = cells * ITERATIONS[case["contrast"]] * OPS_PER_CELL
    if kind == "learned":
        flops += 2 * NET_MACS * cells
    # the permeability in, the solution out (the forcing field too, where there is one)
    return {"bytes": (24 if case.get("f") == "field" else 16) * cells, "flops": flops}


# -------------------------------------------------------- 64-bit references


def _direct(a, f):
    """u of -div(a grad u) = f for a stack of fields (same side), FP64, by block
    elimination over grid rows: harmonic-mean faces, the cell's own value on
    the boundary faces, right-hand side f h^2."""
    count, n, _ = a.shape
    east = 2 * a[:, :, :-1] * a[:, :, 1:] / (a[:, :, :-1] + a[:, :, 1:])
    north = 2 * a[:, :-1] * a[:, 1:] / (a[:, :-1] + a[:, 1:])
    diag = torch.zeros_like(a)
    diag[:, :, :-1] += east
    diag[:, :, 1:] += east
    diag[:, :-1] += north
    diag[:, 1:] += north
    diag[:, :, 0] += a[:, :, 0]
    diag[:, :, -1] += a[:, :, -1]
    diag[:, 0] += a[:, 0]
    diag[:, -1] += a[:, -1]
    b = torch.as_tensor(f, device=a.device, dtype=a.dtype).expand(n, n) / (n + 1) ** 2
    step = max(1, (24 << 30) // (8 * n**3))
    u = torch.empty_like(a)
    for at in range(0, count, step):
        sl = slice(at, min(count, at + step))
        inverses, right = [], []
        for i in range(n):
            rows = torch.diag_embed(diag[sl, i])
            if n > 1:
                rows -= torch.diag_embed(east[sl, i], 1) + torch.diag_embed(east[sl, i], -1)
            r = b[i].expand(rows.shape[0], n).clone()
            if i:
                s = north[sl, i - 1]
                rows -= s[:, :, None] * inverses[-1] * s[:, None, :]
                r += s * (inverses[-1] @ right[-1][:, :, None])[:, :, 0]
            inverses.append(torch.linalg.inv(rows))
            right.append(r)
        x = (inverses[-1] @ right[-1][:, :, None])[:, :, 0]
        u[sl, n - 1] = x
        for i in range(n - 2, -1, -1):
            x = (inverses[i] @ (right[i] + north[sl, i] * x)[:, :, None])[:, :, 0]
            u[sl, i] = x
    return u


def _network(a, weights, scaling, n):
    """The warm-start network in FP64: inputs (log a - mean) / spread and the
    unit-RMS solution of the grid for a = f = 1; six 3 x 3 convolutions, GELU
    after the first five."""
    mean, spread, uscale, _ = scaling
    unit = _direct(torch.ones((1, n, n), device="cuda", dtype=torch.float64), 1.0)[0]
    unit = unit / unit.square().mean().sqrt()
    w = weights.double()
    layers, at = [], 0
    for out, inp in NET_WEIGHTS:
        k = w[at:at + 9 * out * inp].reshape(out, 3, 3, inp).permute(0, 3, 1, 2).contiguous()
        at += 9 * out * inp
        layers.append((k, w[at:at + out]))
        at += out
    u0 = torch.empty_like(a)
    step = max(1, (1 << 21) // (n * n))
    for lo in range(0, a.shape[0], step):
        x = torch.stack([(a[lo:lo + step].log() - mean) / spread, unit.expand_as(a[lo:lo + step])], 1)
        for q, (k, bias) in enumerate(layers):
            pad = torch.nn.functional.pad(x, (1, 1, 1, 1))
            x = bias[None, :, None, None].expand(x.shape[0], -1, n, n).clone()
            for dy in range(3):
                for dx in range(3):
                    x += torch.einsum("oc,bchw->bohw", k[:, :, dy, dx], pad[:, :, dy:dy + n, dx:dx + n])
            if q + 1 < len(layers):
                x = 0.5 * x * (1 + torch.erf(x / math.sqrt(2.0)))
        u0[lo:lo + step] = x[:, 0] * uscale
    return u0


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return None  # weights after Adam steps in BF16 are no function of FP64 ones
    if kind in ("single", "batch") and case.get("count", 1) * case["n"] ** 4 > 1.2e12:
        return None  # block elimination of these would take over 20 seconds
    made = _inputs(case, seed)
    if kind == "predict":
        return {"u0": _network(made["a"], made["weights"], made["scaling"], case["n"]).cpu().numpy()}
    if kind == "uneven":
        left = {n: list(_direct(v, 1.0).cpu().numpy()) for n, v in made["a"].items()}
        return {"u": np.concatenate([left[n].pop().ravel() for n in made["sides"]]), "converged": None,
                "levels": None}
    u = _direct(made["a"], 1.0 if made.get("f") is None else made["f"]).cpu().numpy()
    if kind == "single":
        return {"u": u[0], "converged": None, "levels": None}
    return {"u": u, "converged": None}

"""The work that users of this framework have it do, as cases that can be timed.

A case is a dict of plain values.  ``listed()`` gives the twelve standing ones
and ``draw(rng)`` another of the same ranges; ``prepare`` builds what a
training script holds (decomposition, engine with parameters and Adam moments
of a run under way, points, step object), ``run`` is one pass through the
public entry points, ``work`` the bytes and operations that the pass cannot do
without, and ``exact`` the same results in 64 bits from plain torch.

Kinds of pass:

* ``step``     one training step of a built-in problem (``FusedStep.step``):
               on fixed points under a scheduler mask, on points redrawn on
               the device, or on batches from pinned host memory;
* ``generic``  one training step of a problem without a fused residual
               (``GenericStep.step``): torch evaluates constraint and loss;
* ``predict``  the solution at test points (``FBPINNTrainer.predict``);
* ``lists``    the interaction lists of a point set (``takes.get_inputs``).

The loss leaves ``run`` as float32, the type of the residuals that it is the
mean of (the step keeps its FP64 sum on the device).
"""

import math

import numpy as np
import torch

from fbpinns_gb300 import _lib
from fbpinns_gb300.constants import get_subdomain_ws
from fbpinns_gb300.decompositions import MultilevelRectangularDecompositionND, RectangularDecompositionND
from fbpinns_gb300.engine import FBPINNEngine, d2mask_of
from fbpinns_gb300.optim import adam
from fbpinns_gb300.problems import (BurgersEquation2D, HarmonicOscillator1DHardBC, Helmholtz2D, Poisson2D,
                                    WaveEquationConstantVelocity3D, WaveEquationGaussianVelocity3D, seeded_gaussians)
from fbpinns_gb300.takes import get_inputs
from fbpinns_gb300.trainers import FBPINNTrainer, FusedStep, GenericStep

LR, B1, B2, EPS = 1e-3, 0.9, 0.999, 1e-8

# per problem: domain, dims of the second derivatives, and the size of a gradient
# entry in a run under way (the Adam moments are drawn at it)
PROBLEMS = {
    "ho": dict(lo=(0.0,), hi=(1.0,), d2=(0,), grad=4e5),
    "burgers": dict(lo=(-1.0, 0.0), hi=(1.0, 1.0), d2=(0,), grad=5e-2),
    "poisson": dict(lo=(0.0, 0.0), hi=(1.0, 1.0), d2=(0, 1), grad=3e1),
    "wave": dict(lo=(-1.0, -1.0, 0.0), hi=(1.0, 1.0, 1.0), d2=(0, 1, 2), grad=1e0),
    "helmholtz": dict(lo=(0.0, 0.0), hi=(1.0, 1.0), d2=(0, 1), grad=1e3),
}


def _case(name, kind, problem, boxes, points, layers, width=2.9, levels=False, mode="fixed", act="tanh", mask="all"):
    """boxes / points: counts per dim ("15x15x4"); levels: boxes are the counts per
    side of each level of a multilevel decomposition ("1,2,4")."""
    c = dict(kind=kind, problem=problem, boxes=boxes, points=points, layers=layers, width=width, levels=levels,
             mode=mode, act=act, mask=mask)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the 1D oscillator run: 200 points, 15 networks -- the smallest step, all latency
        _case("ho_step", "step", "ho", "15", "200", "32-32", width=2.0),
        # space-time Burgers with its line scheduler part-way through the time slabs
        _case("burgers_step", "step", "burgers", "16x8", "200x200", "16-16", mask="line"),
        # a coarse multilevel Poisson run with a small redrawn batch (odd size)
        _case("poisson_small_step", "step", "poisson", "1,2,4,8", "16381", "16-16", levels=True, mode="resample"),
        # the headline workload: six levels, 1365 networks, 2^18 points redrawn every step
        _case("poisson_step", "step", "poisson", "1,2,4,8,16,32", "262144", "16-16", levels=True, mode="resample"),
        # the same networks fed from a host data pipeline (pinned batches)
        _case("poisson_host_step", "step", "poisson", "1,2,4,8,16,32", "100003", "16-16", levels=True, mode="host"),
        # the (2+1)D wave run: 900 networks of width 32, a 58^3 grid
        _case("wave_step", "step", "wave", "15x15x4", "58x58x58", "32-32"),
        # the largest: 4096 networks of width 32 and about two million redrawn points
        _case("helmholtz_step", "step", "helmholtz", "64x64", "2097143", "32-32", mode="resample"),
        # sine networks on the multilevel Poisson problem
        _case("siren_step", "step", "poisson", "1,2,4,8,16", "65537", "16-16", levels=True, mode="resample",
              act="sin"),
        # adaptive activations (one more trainable parameter per neuron)
        _case("adaptive_step", "step", "poisson", "1,2,4,8,16", "65537", "16-16", levels=True, mode="resample",
              act="adaptive_tanh"),
        # a user's own problem through autograd: the wave equation with a variable velocity
        _case("generic_step", "generic", "wave", "7x7x4", "30x30x30", "32-32"),
        # test-step inference of the headline model on its 100 x 100 test grid
        _case("predict", "predict", "poisson", "1,2,4,8,16,32", "100x100", "16-16", levels=True),
        # interaction lists of a new batch for the headline decomposition
        _case("lists", "lists", "poisson", "1,2,4,8,16,32", "150001", "16-16", levels=True),
    ]


def _log_int(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def _split(rng, n, xd):
    """About n grid points over xd dims, the counts unequal."""
    side = n ** (1.0 / xd)
    return "x".join(str(max(3, int(side * math.exp(rng.uniform(-0.3, 0.3))))) for _ in range(xd))


def draw(rng):
    kind = rng.choice(["step"] * 7 + ["generic", "predict", "lists"])
    width = round(rng.uniform(1.9, 3.0), 2)
    if kind == "generic":
        return _case(None, "generic", "wave", f"{rng.randint(3, 9)}x{rng.randint(3, 9)}x{rng.randint(2, 5)}",
                     _split(rng, _log_int(rng, 500, 40000), 3), "32-32", width=width)
    if kind in ("predict", "lists"):
        top = rng.randint(2, 6)
        n = _log_int(rng, 100, 300000)
        return _case(None, kind, "poisson", ",".join(str(2 ** k) for k in range(top)),
                     _split(rng, n, 2) if kind == "predict" else str(n), "16-16", width=width, levels=True)
    problem = rng.choice(["ho", "burgers", "poisson", "poisson", "wave", "helmholtz"])
    if problem == "ho":
        return _case(None, kind, problem, str(rng.randint(3, 60)), str(_log_int(rng, 30, 20000)),
                     rng.choice(["32", "32-32"]), width=width)
    if problem == "burgers":
        return _case(None, kind, problem, f"{rng.randint(4, 24)}x{rng.randint(3, 12)}",
                     _split(rng, _log_int(rng, 900, 160000), 2), "16-16", width=width,
                     act=rng.choice(["tanh", "tanh", "tanh", "sin", "adaptive_tanh", "adaptive_sin"]),
                     mask=rng.choice(["all", "line"]))
    if problem == "poisson":
        top = rng.randint(3, 6)
        return _case(None, kind, problem, ",".join(str(2 ** k) for k in range(top)), str(_log_int(rng, 1000, 260000)),
                     "16-16", width=width, levels=True, mode=rng.choice(["fixed", "resample", "resample", "host"]),
                     act=rng.choice(["tanh", "tanh", "tanh", "sin", "adaptive_tanh", "adaptive_sin"]))
    if problem == "wave":
        return _case(None, kind, problem, f"{rng.randint(3, 15)}x{rng.randint(3, 15)}x{rng.randint(2, 5)}",
                     _split(rng, _log_int(rng, 1000, 120000), 3), "32-32", width=width)
    k = rng.randint(6, 64)
    return _case(None, kind, problem, f"{k}x{rng.randint(6, 64)}", str(_log_int(rng, 4000, 1000000)), "32-32",
                 width=width, mode=rng.choice(["fixed", "resample", "resample"]))


# ---------------------------------------------------------------------------
# the pieces of a run
# ---------------------------------------------------------------------------

def _counts(text):
    return [int(v) for v in text.replace(",", "x").split("x")]


def _n_points(c):
    return int(np.prod(_counts(c["points"])))


def _linspace(lo, hi, k):
    return np.linspace(lo, hi, k) if k > 1 else np.array([(lo + hi) / 2])


def _decomposition(c):
    """Static decomposition params, built as a configuration file does."""
    p, counts = PROBLEMS[c["problem"]], _counts(c["boxes"])
    if not c["levels"]:
        xs = [_linspace(a, b, k) for a, b, k in zip(p["lo"], p["hi"], counts)]
        return RectangularDecompositionND.init_params(xs, get_subdomain_ws(xs, c["width"]), (0., 1.))[0]
    xss, wss = [], []
    for k in counts:
        xs = [_linspace(a, b, k) for a, b in zip(p["lo"], p["hi"])]
        xss.append(xs)
        wss.append(get_subdomain_ws(xs, c["width"]) if k > 1 else [np.array([b - a]) for a, b in zip(p["lo"], p["hi"])])
    return MultilevelRectangularDecompositionND.init_params(xss, wss, (0., 1.))[0]


def _problem(c):
    """(problem class, static problem params)."""
    if c["problem"] == "ho":
        return HarmonicOscillator1DHardBC, HarmonicOscillator1DHardBC.init_params(d=2, w0=80, sd=0.1)[0]
    if c["problem"] == "burgers":
        return BurgersEquation2D, BurgersEquation2D.init_params()[0]
    if c["problem"] == "poisson":
        return Poisson2D, Poisson2D.init_params(n_freq=6, sd=0.1)[0]
    if c["problem"] == "helmholtz":
        return Helmholtz2D, Helmholtz2D.init_params(k=40 * math.pi, n_sources=64, seed=0)[0]
    source = seeded_gaussians(12, 0, centre=(-0.5, 0.5), width=(0.1, 0.2), amp=(1.0, 1.0))
    if c["kind"] == "generic":
        return WaveEquationGaussianVelocity3D, WaveEquationGaussianVelocity3D.init_params(c0=1.0, source=source)[0]
    return WaveEquationConstantVelocity3D, WaveEquationConstantVelocity3D.init_params(c0=1.0, source=source)[0]


def _layer_sizes(c):
    return [len(PROBLEMS[c["problem"]]["lo"])] + [int(v) for v in c["layers"].split("-")] + [1]


def _extra(c):
    return {"tanh": 0, "sin": 0, "adaptive_tanh": 1, "adaptive_sin": 2}[c["act"]]


def _n_param(c):
    ls = _layer_sizes(c)
    return sum(fo * (fi + 1 + _extra(c)) for fi, fo in zip(ls[:-1], ls[1:]))


def _theta(c, m, seed):
    """Initial networks as the FCN / SIREN init draws them, per layer W, b and
    the activation parameters around 1; one row per network."""
    g = torch.Generator().manual_seed(1000 + seed)
    ls, cols = _layer_sizes(c), []
    for fi, fo in zip(ls[:-1], ls[1:]):
        v = math.sqrt((6.0 if c["act"].endswith("sin") else 1.0) / fi)
        cols.append((torch.rand((m, fo * (fi + 1)), generator=g) * 2 - 1) * v)
        cols.append(1 + 0.1 * (torch.rand((m, fo * _extra(c)), generator=g) * 2 - 1))
    return torch.cat(cols, 1).float()


def _moments(c, m, seed):
    """Adam's moments and step count of a run under way."""
    g = torch.Generator().manual_seed(2000 + seed)
    s, n = PROBLEMS[c["problem"]]["grad"], (m, _n_param(c))
    return torch.randn(n, generator=g) * (0.3 * s), (0.5 + torch.rand(n, generator=g)) * s * s, 1000 + seed % 1000


def _points(c, seed):
    """Fixed points: a grid, jittered by the seed where it has one point per count."""
    p, counts = PROBLEMS[c["problem"]], _counts(c["points"])
    g = torch.Generator().manual_seed(3000 + seed)
    lo, hi = torch.tensor(p["lo"]), torch.tensor(p["hi"])
    if len(counts) < len(p["lo"]):
        return lo + (hi - lo) * torch.rand((counts[0], len(p["lo"])), generator=g)
    axes = [torch.linspace(a, b, k, dtype=torch.float64) for a, b, k in zip(p["lo"], p["hi"], counts)]
    x = torch.stack(torch.meshgrid(*axes, indexing="ij"), -1).reshape(-1, len(axes)).float()
    step = (hi - lo) / torch.tensor(counts)
    x = x + 0.2 * step * (torch.rand(x.shape, generator=g) * 2 - 1)
    return torch.minimum(torch.maximum(x, lo), hi)


def _host_batches(c, seed):
    return [_points(c, 7 * seed + k) for k in range(4)]


def _mask(c, static, seed):
    """Scheduler mask: all active, or a line scheduler part-way along the last
    dim (fixed behind the front, active at it, inactive ahead)."""
    m = static["m"]
    if c["mask"] == "all":
        return np.ones(m, dtype=int)
    a, b = static["xmins0"][:, -1], static["xmaxs0"][:, -1]
    t = 0.45 + 0.02 * (seed % 5)
    return np.where(b <= t, 2, np.where(a <= t, 1, 0)).astype(int)


def _required(c):
    d2 = PROBLEMS[c["problem"]]["d2"]
    return ((0, ()),) + tuple((0, (d,)) for d in range(len(PROBLEMS[c["problem"]]["lo"]))) + \
        tuple((0, (d, d)) for d in d2)


def _engine(c, static, spec, seed):
    """The engine as the trainer builds it: one jet slot for second derivatives
    that the residual only uses summed, where that kernel is compiled."""
    ls = _layer_sizes(c)
    d2 = d2mask_of([_required(c)], ls[0])
    group = (spec or {}).get("d2_group", 0)
    if group:
        d2 |= _lib.D2_LAPLACIAN if group == (d2 & 7) else _lib.D2_GROUP(group)
    eng = FBPINNEngine(static, ls, d2, activation=c["act"])
    eng.set_theta(_theta(c, static["m"], seed))
    m1, m2, count = _moments(c, static["m"], seed)
    eng.m1.copy_(m1)
    eng.m2.copy_(m2)
    eng.count.fill_(count)
    return eng


def prepare(case, seed):
    c = case
    static = _decomposition(c)
    p = PROBLEMS[c["problem"]]
    if c["kind"] == "lists":
        # the same cloud in another order for every seed: as many pairs, other lists
        order = torch.randperm(_n_points(c), generator=torch.Generator().manual_seed(seed))
        return dict(kind="lists", x=_points(c, 0)[order].cuda(), active=_mask(c, static, seed),
                    all_params={"static": {"decomposition": static}})
    problem, static_problem = _problem(c)
    all_params = {"static": {"decomposition": static, "problem": static_problem}, "trainable": {}}
    opt = adam(LR, B1, B2, EPS)
    if c["kind"] == "generic":
        all_params["static"]["problem"] = {k: v.cuda() if torch.is_tensor(v) else v for k, v in static_problem.items()}
        eng = _engine(c, static, None, seed)
        req = problem.sample_constraints(all_params, _Interior, None, None, [None])[0][-1]
        return dict(kind="generic", eng=eng, opt=opt,
                    step=GenericStep(eng, problem, all_params, [[_points(c, seed)]], [req]))
    spec = problem.fused_spec(all_params)
    eng = _engine(c, static, spec, seed)
    if c["kind"] == "predict":
        return dict(kind="predict", eng=eng, problem=problem, all_params=all_params, x=_points(c, seed).cuda())
    state = dict(kind="step", eng=eng, host=None, k=0)
    if c["mode"] == "resample":
        step = FusedStep(eng, spec, opt, resample=(_n_points(c), list(p["lo"]), list(p["hi"]), seed))
        eng.set_state(np.ones(static["m"], dtype=int))
    elif c["mode"] == "host":
        batches = _host_batches(c, seed)
        step = FusedStep(eng, spec, opt, host_points=_n_points(c), x_probe=batches[0], pipeline=True)
        eng.set_state(np.ones(static["m"], dtype=int))
        state["host"] = [b.pin_memory() for b in batches]
    else:
        step = FusedStep(eng, spec, opt, x=_points(c, seed), scheduled=True)
        step.set_state(_mask(c, static, seed))
    state["step"] = step
    return state


class _Interior:
    """Stands in for the domain where only a constraint's derivative list is asked for."""

    @staticmethod
    def sample_interior(all_params, key, sampler, batch_shape):
        return None


def run(state):
    s = state
    if s["kind"] == "lists":
        takes, all_ims, (active, _, _) = get_inputs(s["x"], s["active"], s["all_params"])
        return list(takes) + [all_ims, active]
    if s["kind"] == "predict":
        return FBPINNTrainer.predict(s["eng"], s["all_params"], s["problem"], s["x"])
    eng = s["eng"]
    if s["kind"] == "generic":
        loss = s["step"].step(s["opt"])
        return {"loss": loss, "theta": eng.theta, "m1": eng.m1, "m2": eng.m2}
    if s["host"] is None:
        loss = s["step"].step()
    else:  # the data pipeline is one batch ahead
        loss = s["step"].step(s["host"][s["k"] % 4], s["host"][(s["k"] + 1) % 4])
        s["k"] += 1
    return {"loss": loss.float(), "grad": eng.grad, "theta": eng.theta}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _expected_pairs(c):
    """Mean number of (point, box) pairs of points spread over the domain."""
    static = _decomposition(c)
    p = PROBLEMS[c["problem"]]
    lo, hi = np.array(p["lo"]), np.array(p["hi"])
    a, b = (static["subdomain"]["params"][k].double().numpy() for k in (0, 1))
    frac = np.clip(np.minimum(b, hi) - np.maximum(a, lo), 0, None) / (hi - lo)
    return float(frac.prod(1).sum() * _n_points(c)), static["m"]


def work(case):
    c = case
    s, m = _expected_pairs(c)
    n, ls = _n_points(c), _layer_sizes(c)
    if c["kind"] == "lists":  # points in; box, point and slot of each pair and the point of each slot out
        return {"bytes": 4.0 * n * ls[0] + 12.0 * s + 4.0 * n * len(_counts(c["boxes"])), "flops": 0}
    macs = sum(a * b for a, b in zip(ls[:-1], ls[1:]))
    theta = 4.0 * m * _n_param(c)
    if c["kind"] == "predict":
        return {"bytes": theta + 4.0 * n * (ls[0] + 1), "flops": 2.0 * macs * s}
    grouped = c["kind"] == "step" and c["problem"] in ("poisson", "helmholtz", "wave")
    jet = 1 + ls[0] + len(PROBLEMS[c["problem"]]["d2"]) - (1 if grouped else 0)
    # forward 2, reverse 4 operations per weight and jet component; parameters and moments
    # read and written, the gradient written, the points read
    return {"bytes": 7 * theta + 4.0 * n * ls[0], "flops": 6.0 * macs * jet * s}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------

def _philox(n, seed, offset):
    """The four words of Philox-4x32-10 with counter (i, offset) and the seed as key."""
    i = np.arange(n, dtype=np.uint64)
    low = np.uint64(0xFFFFFFFF)
    c = [i & low, i >> np.uint64(32), np.full(n, offset & 0xFFFFFFFF, np.uint64), np.full(n, offset >> 32, np.uint64)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        a, b = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(b >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), b & low, (a >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), a & low]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _exact_points(c, seed):
    if c["mode"] != "resample":
        return (_host_batches(c, seed)[0] if c["mode"] == "host" else _points(c, seed)).cuda()
    p = PROBLEMS[c["problem"]]
    words = _philox(_n_points(c), seed, 1000 + seed % 1000)
    u = np.stack([(words[d] >> np.uint64(8)).astype(np.float32) / np.float32(1 << 24) for d in range(len(p["lo"]))], 1)
    lo, hi = np.array(p["lo"], np.float32), np.array(p["hi"], np.float32)
    return torch.from_numpy(lo + (hi - lo) * u).cuda()


def _sigma(act, z, extra, tanh=torch.tanh):
    """The activation and its first two derivatives, differentiable in z and the parameters."""
    if act in ("tanh", "adaptive_tanh"):
        a = extra[0] if extra else None
        t = tanh(z) if a is None else tanh(z / a)
        d = 1 - t * t
        return (t, d, -2 * t * d) if a is None else (a * t, d, -2 * t * d / a)
    cc, o = extra if extra else (1.0, 1.0)
    sn, cs = torch.sin(o * z), torch.cos(o * z)
    return cc * sn, cc * o * cs, -cc * o * o * sn


def _layers(c, theta):
    """theta (B, P) -> per layer (W (B, fo, fi), b, activation parameters), each with a point axis."""
    ls, o, out = _layer_sizes(c), 0, []
    for fi, fo in zip(ls[:-1], ls[1:]):
        W = theta[:, o:o + fo * fi].reshape(-1, fo, fi)
        o += fo * fi
        vec = []
        for _ in range(1 + _extra(c)):
            vec.append(theta[:, o:o + fo].unsqueeze(1))
            o += fo
        out.append((W, vec[0], vec[1:]))
    return out


def _pair_jets(c, theta, box, x, flag):
    """Jets of u w and of w at points x (B, C, xd) of boxes ``box`` = (lo, hi) (B, xd):
    two lists [value, d/dx_d ..., d2/dx_d2 for the problem's dims], each (B, C)."""
    xd, d2 = x.shape[2], PROBLEMS[c["problem"]]["d2"]
    sd = ((box[1] - box[0]) / 2).unsqueeze(1)
    xn = (x - ((box[1] + box[0]) / 2).unsqueeze(1)) / sd
    layers = _layers(c, theta)
    v, dv, ddv = xn, [None] * xd, [None] * len(d2)
    for li, (W, b, extra) in enumerate(layers):
        Wt = W.transpose(1, 2)
        z = torch.bmm(v, Wt) + b
        if li == 0:  # the normalised point's derivatives: one column of W / sd, no second derivatives
            dz = [Wt[:, d:d + 1] / sd[:, :, d:d + 1] for d in range(xd)]
            ddz = [torch.zeros_like(dz[0]) for _ in d2]
        else:
            dz, ddz = [torch.bmm(t, Wt) for t in dv], [torch.bmm(t, Wt) for t in ddv]
        if li == len(layers) - 1:
            u = [t[..., 0] for t in [z] + dz + ddz]
            break
        a, t1, t2 = _sigma(c["act"], z, extra)
        v, dv = a, [t1 * t for t in dz]
        ddv = [t1 * ddz[s] + t2 * dz[d] * dz[d] for s, d in enumerate(d2)]
    ph = math.pi * xn
    k = math.pi / sd
    w0 = ((1 + torch.cos(ph)) / 2) ** 2
    w1 = -(1 + torch.cos(ph)) * torch.sin(ph) / 2 * k
    w2 = (torch.sin(ph) ** 2 - torch.cos(ph) - torch.cos(ph) ** 2) / 2 * k * k

    def product(skip, factor):
        for d in range(xd):
            if d != skip:
                factor = factor * w0[..., d]
        return flag.unsqueeze(1) * factor

    one = torch.ones_like(w0[..., 0])
    w = [product(-1, one) + (1 - flag.unsqueeze(1))]
    w += [product(d, w1[..., d]) for d in range(xd)] + [product(d, w2[..., d]) for d in d2]
    uw = [u[0] * w[0]] + [u[1 + d] * w[0] + u[0] * w[1 + d] for d in range(xd)]
    uw += [u[1 + xd + s] * w[0] + 2 * u[1 + d] * w[1 + d] + u[0] * w[1 + xd + s] for s, d in enumerate(d2)]
    return uw, w


def _function_jets(f, x, d2):
    """[f, df/dx_d, d2f/dx_d2] of a pointwise function by autograd."""
    x = x.clone().requires_grad_(True)
    y = f(x)
    if not y.requires_grad:
        z = torch.zeros_like(y)
        return [y.detach()] + [z] * (x.shape[1] + len(d2))
    g, = torch.autograd.grad(y.sum(), x, create_graph=True)
    out = [y] + [g[:, d] for d in range(x.shape[1])]
    for d in d2:
        h = torch.autograd.grad(g[:, d].sum(), x, retain_graph=True, allow_unused=True)[0] if g.requires_grad else None
        out.append(torch.zeros_like(y) if h is None else h[:, d])
    return [t.detach() for t in out]


def _gaussians(table, x):
    p = torch.as_tensor(table, dtype=torch.float32).double().cuda()
    out = torch.zeros_like(x[:, 0])
    for mx, my, sd, amp in p.tolist():
        out = out + amp * torch.exp(-0.5 * ((x[:, 0] - mx) ** 2 + (x[:, 1] - my) ** 2) / sd ** 2)
    return out


def _constraint(c):
    """(A, B) of the constrained solution A(x) + B(x) u(x)."""
    tanh = torch.tanh
    if c["problem"] == "ho":
        return lambda x: 1 + 0 * x[:, 0], lambda x: tanh(x[:, 0] / 0.1) ** 2
    if c["problem"] == "burgers":
        return (lambda x: -torch.sin(math.pi * x[:, 0]),
                lambda x: tanh((x[:, 0] + 1) / 0.1) * tanh((1 - x[:, 0]) / 0.1) * tanh(x[:, 1] / 0.1))
    if c["problem"] == "wave":
        src = _problem(c)[1]["source"]
        t1 = float(src[:, 2].min())
        return (lambda x: torch.exp(-0.5 * (1.5 * x[:, 2] / t1) ** 2) * _gaussians(src, x),
                lambda x: tanh(2.5 * x[:, 2] / t1) ** 2)
    return (lambda x: 0 * x[:, 0],
            lambda x: tanh(x[:, 0] / 0.1) * tanh((1 - x[:, 0]) / 0.1) * tanh(x[:, 1] / 0.1) * tanh((1 - x[:, 1]) / 0.1))


def _residual(c, x, u):
    """PDE residual from the constrained jets u = [u, u_d ..., u_dd ...]."""
    if c["problem"] == "ho":
        return u[2] + 4 * u[1] + 6400 * u[0]
    if c["problem"] == "burgers":
        return u[2] + u[0] * u[1] - 0.01 / math.pi * u[3]
    if c["problem"] == "wave":
        v = 1.0
        if c["kind"] == "generic":
            v = 1.0 + _gaussians(_problem(c)[1]["mixture"], x)
        return u[4] + u[5] - u[6] / v ** 2
    if c["problem"] == "helmholtz":
        return u[3] + u[4] + (40 * math.pi) ** 2 * u[0] + _gaussians(_problem(c)[1]["source"], x)
    f = torch.zeros_like(x[:, 0])
    for k in range(1, 7):
        a = 2 ** k * math.pi
        f = f + 2.0 ** (k + 1) * math.pi ** 2 * torch.sin(a * x[:, 0]) * torch.sin(a * x[:, 1])
    return u[3] + u[4] + f


def _blocks(c, static, x, pairs=200000):
    """Runs of boxes of one level with about ``pairs`` pairs: (level, boxes, point index (B, C), inside (B, C))."""
    lo, hi = (static["subdomain"]["params"][k].float().cuda() for k in (0, 1))
    pou = static["subdomain"]["pou"].reshape(-1).long().tolist()

    def inside(j, e):
        return ((x[None] >= lo[j:e, None]) & (x[None] <= hi[j:e, None])).all(2)

    counts = torch.cat([inside(j, j + 16).sum(1) for j in range(0, len(pou), 16)]).tolist()
    j = 0
    while j < len(pou):
        e, widest = j + 1, counts[j]
        while e < len(pou) and pou[e] == pou[j] and (e + 1 - j) * max(widest, counts[e]) <= pairs:
            widest, e = max(widest, counts[e]), e + 1
        if widest:
            row, point = inside(j, e).nonzero(as_tuple=True)
            first = torch.as_tensor(np.cumsum([0] + counts[j:e - 1]), device=x.device)
            place = torch.arange(len(row), device=x.device) - first[row]
            idx = torch.zeros((e - j, widest), dtype=torch.long, device=x.device)
            real = torch.zeros((e - j, widest), dtype=torch.bool, device=x.device)
            idx[row, place], real[row, place] = point, True
            yield pou[j], list(range(j, e)), idx, real
        j = e


def exact(case, seed):
    c = case
    if c["kind"] == "lists":
        return None
    static = _decomposition(c)
    p, m = PROBLEMS[c["problem"]], static["m"]
    xd, d2, P = len(p["lo"]), p["d2"], _n_param(c)
    x32 = _exact_points(c, seed)
    theta = _theta(c, m, seed).double().cuda()
    box = [static["subdomain"]["params"][k].double().cuda() for k in (0, 1)]
    flag = static["subdomain"]["params"][4].double().reshape(-1).cuda()
    raw = torch.as_tensor(_mask(c, static, seed)).cuda()
    state = torch.ones(m, dtype=torch.long, device="cuda")
    if c["kind"] == "step" and c["mask"] != "all":  # only the points inside active boxes train
        keep = torch.zeros(len(x32), dtype=torch.bool, device="cuda")
        for _, js, idx, inside in _blocks(c, static, x32):
            keep[idx[(raw[js] == 1)[:, None] & inside]] = True
        x32 = x32[keep]
        state = torch.zeros(m, dtype=torch.long, device="cuda")
        for _, js, _, inside in _blocks(c, static, x32):
            state[js] = torch.where(inside.any(1), torch.where(raw[js] == 2, 2, 1), 0)
    x, n, J = x32.double(), len(x32), 1 + xd + len(d2)
    levels = len(set(static["subdomain"]["pou"].reshape(-1).tolist()))
    blocks = list(_blocks(c, static, x32))
    sums = torch.zeros((2, levels, J, n), dtype=torch.float64, device="cuda")
    with torch.no_grad():
        for lv, js, idx, inside in blocks:
            uw, w = _pair_jets(c, theta[js], [b[js] for b in box], x[idx], flag[js])
            for q, jets in enumerate((uw, w)):
                for k in range(J):
                    sums[q, lv, k].index_add_(0, idx.reshape(-1), (jets[k] * inside).reshape(-1))
    A, B = _constraint(c)
    A, B = _function_jets(A, x, d2), _function_jets(B, x, d2)
    N, W = sums[0].requires_grad_(True), sums[1]
    U = [0] * J
    for lv in range(levels):
        have = W[lv, 0] > 0
        w0 = torch.where(have, W[lv, 0], torch.ones_like(x[:, 0]))
        q = [N[lv, 0] / w0]
        q += [(N[lv, 1 + d] - q[0] * W[lv, 1 + d]) / w0 for d in range(xd)]
        q += [(N[lv, 1 + xd + s] - 2 * q[1 + d] * W[lv, 1 + d] - q[0] * W[lv, 1 + xd + s]) / w0
              for s, d in enumerate(d2)]
        U = [a + torch.where(have, b, torch.zeros_like(b)) / levels for a, b in zip(U, q)]
    uc = [A[0] + B[0] * U[0]] + [A[1 + d] + B[1 + d] * U[0] + B[0] * U[1 + d] for d in range(xd)]
    uc += [A[1 + xd + s] + B[1 + xd + s] * U[0] + 2 * B[1 + d] * U[1 + d] + B[0] * U[1 + xd + s]
           for s, d in enumerate(d2)]
    if c["kind"] == "predict":
        return uc[0].detach().reshape(-1, 1)
    loss = (_residual(c, x, uc) ** 2).mean()
    seeds, = torch.autograd.grad(loss, N)
    grad = torch.zeros((m, P), dtype=torch.float64, device="cuda")
    for lv, js, idx, inside in blocks:
        th = theta[js].requires_grad_(True)
        uw, _ = _pair_jets(c, th, [b[js] for b in box], x[idx], flag[js])
        total = sum((uw[k] * (seeds[lv, k][idx] * inside)).sum() for k in range(J))
        grad[js] = torch.autograd.grad(total, th)[0]
    grad = grad * (state == 1)[:, None]
    m1, m2, count = _moments(c, m, seed)
    m1, m2 = m1.double().cuda(), m2.double().cuda()
    n1, n2 = (1 - B1) * grad + B1 * m1, (1 - B2) * grad * grad + B2 * m2
    step = LR * (n1 / (1 - B1 ** (count + 1))) / (torch.sqrt(n2 / (1 - B2 ** (count + 1))) + EPS)
    theta = torch.where((state == 1)[:, None], theta - step, theta)
    if c["kind"] == "generic":
        return {"loss": loss.detach(), "theta": theta, "m1": n1, "m2": n2}
    return {"loss": loss.detach().reshape(1), "grad": grad, "theta": theta}

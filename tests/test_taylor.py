"""The Taylor rules of constrained_jets against its nested-jvp route (float64,
CPU): the jets and their gradient, for the built-in constraints and for
functions that use every rule, other shapes, or a call without a rule."""

import math

import numpy as np
import pytest
import torch
import torch.utils.checkpoint

from fbpinns_gb300 import engine, problems as PR, taylor


def _static(p):
    return {"static": {"problem": {k: v.double() if torch.is_tensor(v) else v for k, v in p.items()}}}


WAVE = np.array([[0.1, -0.2, 0.3, 1.0], [0.4, 0.3, 0.2, -0.7]])
W = torch.linspace(-1, 1, 6, dtype=torch.float64).reshape(2, 3)


def _rules(p, x, u):
    """Every rule, with scalars, constants and jets on either side."""
    a, b = x[:, 0:1], x[..., 1:2]
    c = torch.tanh(2 * a + 1) - torch.exp(-b) / 3 + 1 / (2 + a * a)
    c = c + torch.sin(b) * torch.cos(a) - torch.neg(b) ** 3 + (3 - a) / (b + 4)
    c = torch.sub(c, 0.5) + torch.square(a).mul(0.1) + 2.0 - torch.reciprocal(a + 5) * torch.full_like(p, 1.5)
    return c * u + (u * u - torch.add(a, b)) ** 1


def _broadcast(p, x, u):
    """(k, n, 2) intermediates, sums over one and two dims, None and int indices."""
    d = x[None] - W[:, None, :x.shape[1]]
    s = torch.exp(-(d ** 2).sum(2, keepdim=True)).sum(0)
    t = (d * x).sum((0, -1))[:, None]
    return s * u + t + x[:, 0].mul(2)[:, None]


CASES = {
    "ho": (1, 1, PR.HarmonicOscillator1DHardBC.constraining_fn, _static({"sd": 0.1})),
    "burgers": (2, 1, PR.BurgersEquation2D.constraining_fn, _static({"sd": 0.1})),
    "poisson": (2, 3, PR.Poisson2D.constraining_fn, _static({"sd": 0.1})),
    "wave": (3, 7, PR.WaveEquationGaussianVelocity3D.constraining_fn,
             _static({"c0": 1.0, "source": torch.as_tensor(WAVE)})),
    "rules": (2, 3, _rules, torch.zeros((17, 1), dtype=torch.float64)),
    "rules_1d_second": (2, 2, _rules, torch.zeros((17, 1), dtype=torch.float64)),
    "broadcast": (3, 5, _broadcast, None),
    "all_points": (2, 3, lambda p, x, u: u * x[:, 0:1] + (u * u).sum(0, keepdim=True), None),
    "no_u": (2, 3, lambda p, x, u: torch.sin(x[:, 1:2]), None),
    "constant": (2, 3, lambda p, x, u: torch.ones_like(u), None),
    "scaled": (2, 3, lambda p, x, u: u * 2, None),
    "no_rule": (2, 3, lambda p, x, u: torch.atan(x[:, 0:1]) * u + torch.where(x[:, 1:2] > 0.5, u, 2 * u), None),
    "power": (2, 3, lambda p, x, u: (x[:, 0:1] + 2) ** 0.5 * u, None),
    "in_place": (2, 3, lambda p, x, u: (x[:, 0:1] * u).add_(u), None),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_taylor_rules_match_nested_jvp(name, monkeypatch):
    xd, d2, fn, p = CASES[name]
    J = engine.jet_size(xd, d2)
    g = torch.Generator().manual_seed(3)
    x = torch.rand((17, xd), generator=g, dtype=torch.float64)
    U = torch.randn((17, J), generator=g, dtype=torch.float64, requires_grad=True)
    seed = torch.randn((17, J), generator=g, dtype=torch.float64)
    for need in (None, [1], [J - 1]):
        got = engine.constrained_jets(fn, p, x, U, xd, d2, need)
        with monkeypatch.context() as m:
            m.setattr(taylor, "RULES", {})
            m.setattr(taylor, "PLAIN", set())
            ref = engine.constrained_jets(fn, p, x, U, xd, d2, need)
        torch.testing.assert_close(got, ref, rtol=1e-11, atol=1e-11 * ref.abs().max().item())
        assert got.requires_grad == ref.requires_grad
        if ref.requires_grad:
            dg, dr = (torch.autograd.grad((v * seed).sum(), U)[0] for v in (got, ref))
            torch.testing.assert_close(dg, dr, rtol=1e-11, atol=1e-11 * dr.abs().max().item())


def test_every_builtin_constraint_has_rules():
    for name in ("ho", "burgers", "poisson", "wave"):
        xd, d2, fn, p = CASES[name]
        x = torch.rand((5, xd), dtype=torch.float64)
        z = torch.zeros((xd, 5, 1), dtype=torch.float64)
        _, _, d, dd = taylor.jets(lambda a, b: fn(p, a, b), x, list(range(xd)), x[:, 0:1] * 1, z + 1, z)
        assert d.shape == dd.shape == (xd, 5, 1) and torch.isfinite(d).all() and math.isfinite(dd.sum().item())


class _Square(torch.autograd.Function):
    """u^2 with its own derivatives, usable under torch.func."""

    @staticmethod
    def forward(u):
        return u * u

    @staticmethod
    def setup_context(ctx, inputs, output):
        ctx.save_for_backward(*inputs)
        ctx.save_for_forward(*inputs)

    @staticmethod
    def backward(ctx, g):
        return 2 * ctx.saved_tensors[0] * g

    @staticmethod
    def jvp(ctx, t):
        return 2 * ctx.saved_tensors[0] * t


class _Through(torch.autograd.Function):
    """Returns its input, with another derivative than the identity's."""

    @staticmethod
    def forward(u):
        return u

    @staticmethod
    def setup_context(ctx, inputs, output):
        pass

    @staticmethod
    def backward(ctx, g):
        return 3 * g

    @staticmethod
    def jvp(ctx, t):
        return 3 * t


@torch.jit.script
def _scripted(x, u):
    return torch.tanh(x[:, 0:1]) * u


_traced = torch.jit.trace(lambda x, u: torch.tanh(x[:, 0:1]) * u, (W[:, :2], W[:, :1]))


def _caught(x, u):
    try:
        return torch.atan(x[:, 0:1]) * u
    except BaseException:
        return 0 * u


def _partly_no_grad(x, u):
    with torch.no_grad():
        a = torch.tanh(x[:, 0:1]) * u
    return a + u * x[:, 0:1]


_T = torch.func
PAST_THE_RULES = {  # calls that do not come (only) through __torch_function__
    "vmap": lambda p, x, u: torch.vmap(lambda a, b: torch.tanh(a[0:1]) * b)(x, u),
    "vmap_closure": lambda p, x, u: torch.vmap(lambda b: b * 2)(u) * torch.tanh(x[:, 0:1]),
    "script": lambda p, x, u: _scripted(x, u),
    "trace": lambda p, x, u: _traced(x, u),
    "func_vjp": lambda p, x, u: _T.vjp(lambda a: a * a * x[:, 0:1], u)[1](torch.ones_like(u))[0] * u,
    "func_vjp_value": lambda p, x, u: _T.vjp(lambda a: a * a, u)[0] * x[:, 0:1],
    "func_grad": lambda p, x, u: _T.grad(lambda a: (a * a * a).sum())(u) * x[:, 0:1],
    "func_grad_closure": lambda p, x, u: _T.grad(lambda a: (a * x[:, 0:1]).sum())(torch.zeros_like(u)) * u,
    "func_jvp": lambda p, x, u: _T.jvp(lambda a: a * a, (u,), (torch.ones_like(u),))[1] * x[:, 0:1],
    "function": lambda p, x, u: _Square.apply(u) * x[:, 0:1],
    "function_and_u": lambda p, x, u: _Square.apply(u) * x[:, 0:1] + u,
    "function_through": lambda p, x, u: _Through.apply(u) * x[:, 0:1],
    "function_through_alone": lambda p, x, u: _Through.apply(u),
    "caught": lambda p, x, u: _caught(x, u),
    "partly_no_grad": lambda p, x, u: _partly_no_grad(x, u),
}


def _jets_and_grad(fn, x, U, d2, seed, grad=True):
    with torch.set_grad_enabled(grad):
        y = engine.constrained_jets(fn, None, x, U, x.shape[1], d2)
    assert y.requires_grad or not grad
    return y.detach(), torch.autograd.grad((y * seed).sum(), U)[0] if grad else None


@pytest.mark.parametrize("grad", [True, False])
@pytest.mark.parametrize("name", sorted(PAST_THE_RULES))
def test_constraints_that_reach_past_the_rules(name, grad, monkeypatch):
    """Jets and gradient are those of the nested jvp, with gradients on and off."""
    fn, (x, U, seed) = PAST_THE_RULES[name], _xu()
    y, dy = _jets_and_grad(fn, x, U, 3, seed, grad)
    with monkeypatch.context() as m:
        m.setattr(taylor, "RULES", {})
        m.setattr(taylor, "PLAIN", set())
        ref, dref = _jets_and_grad(fn, x, U, 3, seed, grad)
    assert ref[:, 1:].abs().max() > 0.1
    torch.testing.assert_close(y, ref, rtol=1e-11, atol=1e-11)
    if grad:
        torch.testing.assert_close(dy, dref, rtol=1e-11, atol=1e-11)


def _xu():
    g = torch.Generator().manual_seed(3)
    return (torch.rand((17, 2), generator=g, dtype=torch.float64),
            torch.randn((17, 5), generator=g, dtype=torch.float64, requires_grad=True),
            torch.randn((17, 5), generator=g, dtype=torch.float64))


@pytest.mark.parametrize("outer", ["vmap", "grad", "jvp", "dual", "hooks", "checkpoint"])
def test_jets_under_outer_transforms(outer):
    """constrained_jets itself inside a transform gives what it gives outside."""
    fn = CASES["rules"][2]
    p = torch.zeros((17, 1), dtype=torch.float64)
    x, U, seed = _xu()

    def jets(V):
        return engine.constrained_jets(fn, p, x, V, 2, 3)

    y, dy = jets(U).detach(), torch.autograd.grad((jets(U) * seed).sum(), U)[0]
    V = U.detach()
    if outer == "vmap":
        got, want = torch.vmap(jets)(torch.stack([V, 2 * V])), torch.stack([y, jets(2 * V)])
    elif outer == "grad":
        got, want = _T.grad(lambda v: (jets(v) * seed).sum())(V), dy
    elif outer == "jvp":
        got, want = (_T.jvp(jets, (V,), (seed,))[1] * seed).sum(), None
    elif outer == "dual":
        with torch.autograd.forward_ad.dual_level():
            t = torch.autograd.forward_ad.unpack_dual(jets(torch.autograd.forward_ad.make_dual(V, seed))).tangent
        got, want = (t * seed).sum(), None
    elif outer == "hooks":
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t.clone(), lambda t: t):
            z = jets(U)
        got, want = torch.autograd.grad((z * seed).sum(), U)[0], dy
    else:
        z = torch.utils.checkpoint.checkpoint(jets, U, use_reentrant=False)
        got, want = torch.autograd.grad((z * seed).sum(), U)[0], dy
    if want is None:  # seed . J seed from the reverse mode
        W2 = U.detach().requires_grad_(True)
        h = torch.zeros_like(y, requires_grad=True)
        g, = torch.autograd.grad((jets(W2) * h).sum(), W2, create_graph=True)
        want = (torch.autograd.grad((g * seed).sum(), h)[0] * seed).sum()
    torch.testing.assert_close(got, want, rtol=1e-11, atol=1e-11)


def test_quotient_of_jets_where_the_reciprocal_overflows():
    """u / v of jets with v below the reciprocal of the largest number: the
    value and the derivatives along u of the direct quotient."""
    x, U, _ = _xu()
    U = U.detach()[:, :4]
    s = 2.0 ** -1040

    def fn(p, x, u):
        return (u * s) / (torch.exp(x[:, 1:2]) * s)
    y = engine.constrained_jets(fn, None, x, U, 2, 1)
    u, v = U[:, 0] * s, torch.exp(x[:, 1]) * s
    assert torch.equal(y[:, 0], u / v) and torch.isfinite(y).all()
    torch.testing.assert_close(y[:, 1], (U[:, 1] * s) / v, rtol=1e-9, atol=0)


def _quotient(p, x, u):
    return (u * (x[:, 0:1] + 1)) / (x[:, 1:2] * 3 + 1)


def test_quotient_of_jets_rounds_once():
    """The value in float32 is the one that the function itself gives."""
    x, U, _ = _xu()
    x, U = x.float(), U.detach().float()[:, :4]
    y = engine.constrained_jets(_quotient, None, x, U, 2, 1)
    assert torch.equal(y[:, 0:1], _quotient(None, x, U[:, 0:1]))


@pytest.mark.parametrize("call", [lambda x, u: (x * u).sum(2, keepdim=True), lambda x, u: (x * u).sum((0, -3))[:, None],
                                  lambda x, u: torch.sum(x * u, (1, -1), keepdim=True)])
def test_wrong_dims_of_a_sum_are_refused(call):
    """As the plain call does: an IndexError out of range, a RuntimeError for a dim given twice."""
    x, U, _ = _xu()
    with pytest.raises((IndexError, RuntimeError)) as plain:
        call(x, U[:, 0:1])
    with pytest.raises(plain.type):
        engine.constrained_jets(lambda p, x, u: call(x, u) * u, None, x, U, 2, 3)


@pytest.mark.parametrize("p", [float("inf"), 2.0 ** 40])
def test_powers_beyond_the_rule_go_to_the_jvp(p, monkeypatch):
    x, U, _ = _xu()
    y = engine.constrained_jets(lambda q, x, u: u + torch.tanh(x[:, 0:1]) ** p, None, x, U, 2, 3)
    with monkeypatch.context() as m:
        m.setattr(taylor, "RULES", {})
        ref = engine.constrained_jets(lambda q, x, u: u + torch.tanh(x[:, 0:1]) ** p, None, x, U, 2, 3)
    torch.testing.assert_close(y, ref, rtol=1e-11, atol=1e-11, equal_nan=True)


@pytest.mark.parametrize("name", ["burgers", "no_rule", "vmap", "function"])
def test_jets_in_inference_mode(name):
    """Where forward mode is off, by the rules and by the jvp, as outside."""
    fn, p = (CASES[name][2:] if name in CASES else (PAST_THE_RULES[name], None))
    x, U, _ = _xu()
    ref = engine.constrained_jets(fn, p, x, U.detach(), 2, 3)
    assert ref[:, 1:].abs().max() > 0.1
    with torch.inference_mode():
        y = engine.constrained_jets(fn, p, x * 1, U * 1, 2, 3)
    torch.testing.assert_close(y, ref, rtol=1e-11, atol=1e-11)

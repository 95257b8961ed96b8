"""Which constraining functions predict evaluates in the kernels."""

import ctypes as C

import numpy as np
import pytest
import torch

from fbpinns_gb300 import _lib, problems as PR

BUILTIN = {"ho": (PR.HarmonicOscillator1DHardBC, 1), "burgers": (PR.BurgersEquation2D, 2),
           "wave": (PR.WaveEquationConstantVelocity3D, 3), "wave_gaussian": (PR.WaveEquationGaussianVelocity3D, 3),
           "poisson": (PR.Poisson2D, 2), "helmholtz": (PR.Helmholtz2D, 2)}


def _params(cls, **kw):
    return {"static": {"problem": dict(cls.init_params()[0], **kw)}, "trainable": {}}


@pytest.mark.parametrize("name", sorted(BUILTIN))
def test_only_at_the_ansatz_number_of_dims(name):
    """A problem with a parameter as one more input keeps a constraint that
    reads its first columns; the kernels have it for its own dims only."""
    cls, xd = BUILTIN[name]

    class Parametrised(cls):
        pass

    assert PR.ansatz_spec(Parametrised, _params(cls), xd) is not None
    u, x = torch.ones((5, 1)), torch.rand((5, xd + 1))
    assert torch.isfinite(cls.constraining_fn(_params(cls), x, u)).all()
    assert PR.ansatz_spec(Parametrised, _params(cls), xd + 1) is None


@pytest.mark.parametrize("name", sorted(BUILTIN))
def test_the_library_refuses_a_problem_kind_at_other_dims(name):
    """(No points, so that nothing could be launched.)"""
    cls, xd = BUILTIN[name]
    pr = _lib.Problem()
    pr.kind = int(PR.ansatz_spec(cls, _params(cls))["kind"])
    lib, some = _lib.load(), C.c_void_p(16)
    for dims in {1, 2, 3} - {xd}:
        assert lib.fbp_pou_solution(dims, 0, C.byref(pr), 0, 1, some, some, some, some, some, 0, some, None) == -3
        assert lib.fbp_pou_loss(dims, 0, C.byref(pr), 0, 1, some, some, some, some, some, some, None, 0, 0, some, 1,
                                some, None) == -3
    assert lib.fbp_pou_solution(xd, 0, C.byref(pr), 0, 1, some, some, some, some, some, 0, some, None) == 0


class _Unhashable:
    """A callable that compares by value, so that it has no hash."""

    def __eq__(self, other):
        return isinstance(other, _Unhashable)

    def __call__(self, all_params, x, u):
        return u


@pytest.mark.parametrize("name,kw", [
    ("helmholtz", dict(k=np.linspace(1.0, 2.0, 5))), ("burgers", dict(nu=np.ones(3))), ("ho", dict(mu=[1, 2])),
    ("ho", dict(k=torch.ones(2))), ("poisson", dict(n_freq=np.arange(3))), ("poisson", dict(sd=torch.ones(5, 1))),
    ("burgers", dict(sd=torch.ones(5, 1))), ("wave", dict(source=torch.ones(2, 5))), ("helmholtz", dict(source=None)),
    ("poisson", dict(sd=1j))])
def test_parameters_that_the_kernels_cannot_take(name, kw):
    """Arrays for numbers (of the residual alone, or of the constraint per
    point) and wider tables: constraining_fn evaluates or refuses them, unless
    the ansatz does not depend on them."""
    cls, xd = BUILTIN[name]
    spec = PR.ansatz_spec(cls, _params(cls, **kw), xd)
    if kw.keys() & {"n_freq"} or (name == "helmholtz" and "source" in kw):
        assert spec["n_int"] == 0 and spec["gauss"] is None and all(type(v) is float for v in spec["p"])
    else:
        assert spec is None


def test_a_constraining_fn_without_a_hash():
    class Own(PR.Poisson2D):
        constraining_fn = _Unhashable()
    assert PR.ansatz_spec(Own, _params(Own), 2) is None


@pytest.mark.gpu
def test_predict_of_a_parametrised_problem(cuda):
    """Burgers with a third input: the solution is constraining_fn of the networks' sum."""
    from helpers import decomposition, random_layers
    from fbpinns_gb300.engine import FBPINNEngine
    from fbpinns_gb300.networks import pack_layers
    from fbpinns_gb300.trainers import FBPINNTrainer

    class Parametrised(PR.BurgersEquation2D):
        pass

    static = decomposition("wave")
    eng = FBPINNEngine(static, [3, 32, 32, 1], 7)
    eng.set_theta(pack_layers([(w.float(), b.float()) for w, b in random_layers([3, 32, 32, 1], static["m"], seed=3)]))
    x = (torch.rand((700, 3), generator=torch.Generator().manual_seed(1)) * 2 - 1).abs().cuda()
    ps = eng.points(x)
    eng.forward_pairs(ps, z2=False)
    ref = Parametrised.constraining_fn(_params(Parametrised), x, eng.pou_forward(ps)[:, 0:1])
    assert ref.abs().max() > 0.1
    assert torch.equal(FBPINNTrainer.predict(eng, _params(Parametrised), Parametrised, x), ref)

"""Which constraining functions predict evaluates in the kernels."""

import ctypes as C

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

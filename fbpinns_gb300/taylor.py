"""Second-order Taylor arithmetic on tensors, for the jets of a problem's
``constraining_fn``.

``Jet`` is a tensor that also carries its first and second derivatives along
several directions at once, stacked in front: ``d`` and ``dd`` of shape
(directions, *shape), or None for zero.  A torch call on it is answered by the
rule of that call (the chain rule on plain tensors, which autograd records), so
one evaluation of a function gives what a nested ``torch.func.jvp`` per
direction gives.  The jvp's ops on zero tangents go through Python meta
kernels, about 0.3 ms each: 72 ms a step for the wave equation's constraint,
where the rules take 4.  A call without a rule raises ``NoRule`` and the
caller uses the jvp.

A ``Jet`` holds no data of its own, so whatever reaches past the rules (vmap,
torch.func, TorchScript, C++ extensions) has nothing to compute on and ends up
in ``Jet.__torch_dispatch__``, which refuses as well; a refusal that the
function or TorchScript turns into something else is still on the trace.
"""

import torch


class NoRule(BaseException):
    """A torch call that ``Jet`` has no rule for (not an Exception, so that a
    function's own ``except Exception`` does not take it)."""


def _pad(s, ndim):
    """A stack (D, *shape) as (D, 1, ..., *shape) with ndim dims after the first."""
    k = ndim - (s.dim() - 1)
    return s if k <= 0 else s.reshape((s.shape[0],) + (1,) * k + tuple(s.shape[1:]))


def _sum(*terms):
    """Sum of the terms that are not None (None if there is none)."""
    out = None
    for t in terms:
        if t is not None:
            out = t if out is None else out + t
    return out


def _mul(s, f, ndim):
    """Stack s times the plain factor f (a tensor or a number)."""
    return None if s is None else _pad(s, ndim) * f


def _parts(a):
    return (a.v, a.d, a.dd) if isinstance(a, Jet) else (a, None, None)


def _full(s, v):
    """Stack s broadcast to the shape of the value v."""
    if s is None:
        return None
    s = _pad(s, v.dim())
    return s if tuple(s.shape[1:]) == tuple(v.shape) else s.expand((s.shape[0],) + tuple(v.shape))


def _add(a, b, sign=1):
    (u, ud, udd), (v, vd, vdd) = _parts(a), _parts(b)
    w = u + v if sign > 0 else u - v
    n = w.dim()

    def both(p, q):
        p, q = (None if s is None else _pad(s, n) for s in (p, q))
        if q is not None and sign < 0:
            return -q if p is None else p - q
        return _sum(p, q)
    return Jet.make(w, _full(both(ud, vd), w), _full(both(udd, vdd), w))


def _times(a, b):
    (u, ud, udd), (v, vd, vdd) = _parts(a), _parts(b)
    w = u * v
    n = w.dim()
    cross = None
    if ud is not None and vd is not None:
        cross = 2.0 * (_pad(ud, n) * _pad(vd, n))
    return Jet.make(w, _full(_sum(_mul(ud, v, n), _mul(vd, u, n)), w),
                    _full(_sum(_mul(udd, v, n), cross, _mul(vdd, u, n)), w))


def _chain(a, f, f1, f2):
    """f(a) from the value f and the derivatives f1, f2 at a.v."""
    n = f.dim()
    second = None if a.d is None else f2 * (a.d * a.d)
    return Jet.make(f, _mul(a.d, f1, n), _sum(_mul(a.dd, f1, n), second))


def _tanh(a):
    t = torch.tanh(a.v)
    s = 1.0 - t * t
    return _chain(a, t, s, -2.0 * t * s)


def _exp(a):
    e = torch.exp(a.v)
    return _chain(a, e, e, e)


def _sin(a):
    s, c = torch.sin(a.v), torch.cos(a.v)
    return _chain(a, s, c, -s)


def _cos(a):
    s, c = torch.sin(a.v), torch.cos(a.v)
    return _chain(a, c, -s, -c)


def _reciprocal(a):
    r = torch.reciprocal(a.v)
    r2 = r * r
    return _chain(a, r, -r2, 2.0 * r2 * r)


def _div(a, b):
    if not isinstance(b, Jet):
        v, d, dd = _parts(a)
        w = v / b
        return Jet.make(w, _full(None if d is None else _pad(d, w.dim()) / b, w),
                        _full(None if dd is None else _pad(dd, w.dim()) / b, w))
    # from w v = u: the quotient itself, not u (1 / v), which overflows where v is
    # tiny and rounds twice
    (u, ud, udd), (v, vd, vdd) = _parts(a), _parts(b)
    w = u / v
    n = w.dim()

    def over_v(s):
        return None if s is None else _full(_pad(s, n) / v, w)

    def minus(s, t):
        return _sum(None if s is None else _pad(s, n), None if t is None else -t)
    d = over_v(minus(ud, _mul(vd, w, n)))
    cross = None if d is None or vd is None else 2.0 * (d * _pad(vd, n))
    return Jet.make(w, d, over_v(minus(udd, _sum(cross, _mul(vdd, w, n)))))


def _pow(a, p):
    """a ** p for an integer p >= 1 (other powers: the jvp)."""
    if not isinstance(a, Jet) or isinstance(p, bool) or not isinstance(p, (int, float)) or not 1 <= p < 2 ** 31 \
            or p != int(p):
        raise NoRule
    p = int(p)
    if p == 1:
        return a
    v, m = a.v, a.v if p == 2 else a.v ** (p - 1)
    f2 = float(p * (p - 1)) if p == 2 else p * (p - 1) * v ** (p - 2)
    return _chain(a, v ** p, float(p) * m, f2)


def _neg(a):
    return Jet.make(-a.v, None if a.d is None else -a.d, None if a.dd is None else -a.dd)


def _getitem(a, idx):
    items = idx if isinstance(idx, tuple) else (idx,)
    if not all(i is None or i is Ellipsis or type(i) in (int, slice) for i in items):
        raise NoRule
    at = (slice(None),) + items
    return Jet.make(a.v[idx], None if a.d is None else a.d[at], None if a.dd is None else a.dd[at])


def _reduce(a, dim=None, keepdim=False):
    if dim is None or not isinstance(a, Jet):
        raise NoRule
    dims = dim if isinstance(dim, (tuple, list)) else (dim,)
    n = a.v.dim()
    if not dims or not all(type(i) is int and -n <= i < n for i in dims):
        raise NoRule
    dims = [i % n for i in dims]
    up = [i + 1 for i in dims]
    return Jet.make(a.v.sum(dims, keepdim=keepdim), None if a.d is None else a.d.sum(up, keepdim=keepdim),
                    None if a.dd is None else a.dd.sum(up, keepdim=keepdim))


T = torch.Tensor
RULES = {}
for _fns, _rule in [
        ((torch.add, T.add, T.__add__, T.__radd__), lambda a, b: _add(a, b)),
        ((torch.sub, T.sub, T.__sub__), lambda a, b: _add(a, b, -1)),
        ((T.__rsub__, torch.rsub), lambda a, b: _add(b, a, -1)),
        ((torch.mul, T.mul, T.__mul__, T.__rmul__, torch.multiply, T.multiply), _times),
        ((torch.div, T.div, T.__truediv__, torch.true_divide, T.true_divide), _div),
        ((T.__rtruediv__, T.__rdiv__), lambda a, b: _div(b, a)),
        ((torch.pow, T.pow, T.__pow__), _pow),
        ((torch.square, T.square), lambda a: _pow(a, 2)),
        ((torch.neg, T.neg, T.__neg__, torch.negative, T.negative), _neg),
        ((torch.tanh, T.tanh), _tanh),
        ((torch.exp, T.exp), _exp),
        ((torch.sin, T.sin), _sin),
        ((torch.cos, T.cos), _cos),
        ((torch.reciprocal, T.reciprocal), _reciprocal),
        ((T.__getitem__,), _getitem),
        ((torch.sum, T.sum), _reduce)]:
    for _f in _fns:
        RULES[_f] = _rule

# properties and calls that say nothing about the values' derivatives
PLAIN = {getattr(T, k).__get__ for k in ("shape", "dtype", "device", "ndim", "is_cuda", "requires_grad", "layout")} | \
    {T.size, T.dim, T.numel, T.__len__, T.is_floating_point, T.is_contiguous,
     torch.zeros_like, torch.ones_like, T.new_zeros, T.new_ones}


class _Trace:
    """One evaluation of a function on Jets: the grad mode that it began in, and
    whether it made a call that has no rule."""

    def __init__(self):
        self.grad, self.refused = torch.is_grad_enabled(), False

    def refuse(self):
        self.refused = True
        raise NoRule

    def same_modes(self):
        """False inside a custom autograd.Function (which turns forward mode off,
        and its own derivatives are then wanted) and under another grad mode."""
        return torch.is_grad_enabled() == self.grad and torch._C._is_fwd_grad_enabled()


def _trace_in(args):
    """The trace of a Jet among the arguments (nested ones too), or None."""
    for a in args.values() if isinstance(args, dict) else args:
        t = a.trace if isinstance(a, Jet) else _trace_in(a) if isinstance(a, (tuple, list, dict)) else None
        if t is not None:
            return t
    return None


def _refuse(*args):
    t = _trace_in(args)
    if t is not None:
        t.refuse()
    raise NoRule


_wrapper = torch.Tensor._make_wrapper_subclass


class Jet(torch.Tensor):
    """A tensor with derivative stacks; made by ``Jet.make``."""

    @staticmethod
    def make(v, d, dd, trace=None):
        j = _wrapper(Jet, v.shape, dtype=v.dtype, device=v.device)
        j.v, j.d, j.dd, j.trace = v, d, dd, trace
        return j

    @classmethod
    def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
        _refuse(args, kwargs or {})

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        kwargs = kwargs or {}
        for a in args:
            if type(a) is Jet:
                trace = a.trace
                break
        else:
            _refuse(args, kwargs)
        if not trace.same_modes() or not _TYPES.issuperset(types):
            trace.refuse()
        with torch._C.DisableTorchFunctionSubclass():
            if func in PLAIN:
                return func(*(a.v if type(a) is Jet else a for a in args), **kwargs)
            rule = RULES.get(func)
            if rule is None:
                trace.refuse()
            try:
                out = rule(*args, **kwargs)
            except NoRule:
                trace.refuse()
            except (TypeError, AttributeError):  # an argument that the rule does not take (alpha=, out=, dtype=)
                trace.refuse()
            out.trace = trace
            return out


_TYPES = {Jet, torch.Tensor, torch.nn.Parameter}


def jets(fn, x, dims, u, ud, udd):
    """(same, value, d, dd) of fn(x, u) along the unit directions ``dims`` of x
    (n, xd), where u has the derivatives ud, udd (directions, n, 1): whether fn
    returned its u itself, and its value, d and dd as (n, 1) and (directions, n,
    1), or None for zero.  Raises NoRule where fn makes a call without a rule."""
    e = torch.zeros((len(dims), 1, x.shape[1]), dtype=x.dtype, device=x.device)
    for i, d in enumerate(dims):
        e[i, 0, d] = 1.0
    trace = _Trace()
    if not trace.same_modes():
        raise NoRule
    uj = Jet.make(u, ud, udd, trace)
    try:
        y = fn(Jet.make(x, e.expand(-1, x.shape[0], -1), None, trace), uj)
    except Exception:
        if trace.refused:  # what TorchScript makes of a refusal, or fn's answer to one
            raise NoRule from None
        raise
    if trace.refused or not isinstance(y, torch.Tensor) or y.dtype != u.dtype:
        raise NoRule
    return (y is uj,) + ((y.v, y.d, y.dd) if isinstance(y, Jet) else (y, None, None))

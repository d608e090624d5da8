"""Directional derivatives of the oracle in extended precision (no test functions
here): dual numbers over NumPy arrays, and the array operations oracle.ref uses,
on them.  ``jacobian(rhs, q)`` gives d rhs / d q column by column."""
import numpy as np

from oracle.ref import _NumpyOps

LD = np.longdouble


class Dual:
    """Value v and derivative d."""
    __array_priority__ = 1000

    def __init__(self, v, d):
        self.v, self.d = v, d

    shape = property(lambda self: self.v.shape)
    ndim = property(lambda self: self.v.ndim)

    def __add__(self, o):
        if isinstance(o, Dual):
            return Dual(self.v + o.v, self.d + o.d)
        return Dual(self.v + o, self.d + np.zeros_like(self.v + o))

    __radd__ = __add__

    def __neg__(self):
        return Dual(-self.v, -self.d)

    def __sub__(self, o):
        return self + (-o)

    def __rsub__(self, o):
        return (-self) + o

    def __mul__(self, o):
        if isinstance(o, Dual):
            return Dual(self.v * o.v, self.d * o.v + self.v * o.d)
        return Dual(self.v * o, self.d * o)

    __rmul__ = __mul__

    def __truediv__(self, o):
        if isinstance(o, Dual):
            r = self.v / o.v
            return Dual(r, (self.d - r * o.d) / o.v)
        return Dual(self.v / o, self.d / o)

    def __pow__(self, e):
        return Dual(self.v ** e, e * self.v ** (e - 1) * self.d)

    def __getitem__(self, i):
        return Dual(self.v[i], self.d[i])

    def __gt__(self, o):
        return self.v > (o.v if isinstance(o, Dual) else o)

    def __ge__(self, o):
        return self.v >= (o.v if isinstance(o, Dual) else o)


def _dual(x):
    if isinstance(x, Dual):
        return x
    x = np.asarray(x, LD)
    return Dual(x, np.zeros_like(x))


class DualOps(_NumpyOps):
    name = "dual"

    def roll(self, a, shift, axis):
        return Dual(np.roll(a.v, shift, axis), np.roll(a.d, shift, axis))

    def stack(self, xs, axis=0):
        xs = [_dual(x) for x in xs]
        s = np.broadcast_shapes(*[x.shape for x in xs])
        return Dual(*[np.stack([np.broadcast_to(getattr(x, f), s) for x in xs], axis) for f in "vd"])

    def where(self, c, a, b):
        a, b = _dual(a), _dual(b)
        return Dual(np.where(c, a.v, b.v), np.where(c, a.d, b.d))

    def maximum(self, a, b):
        if not isinstance(a, Dual) and not isinstance(b, Dual):
            return np.maximum(a, b)
        a, b = _dual(a), _dual(b)
        return self.where(a.v >= b.v, a, b)

    def minimum(self, a, b):
        a, b = _dual(a), _dual(b)
        return self.where(a.v <= b.v, a, b)

    def abs(self, a):
        return Dual(np.abs(a.v), np.sign(a.v) * a.d)

    def sign(self, a):
        return np.sign(a.v)

    def sqrt(self, a):
        if not isinstance(a, Dual):
            return np.sqrt(a)
        r = np.sqrt(a.v)
        return Dual(r, a.d / (2 * r))

    def einsum(self, spec, a, b):
        return Dual(np.einsum(spec, a.v, b), np.einsum(spec, a.d, b))

    def zeros_like(self, a):
        return Dual(np.zeros_like(a.v), np.zeros_like(a.v))

    def ones_like(self, a):
        return Dual(np.ones_like(a.v), np.zeros_like(a.v))

    def sum0(self, a):
        return Dual(a.v.sum(0), a.d.sum(0)) if isinstance(a, Dual) else a.sum(0)

    def add_at(self, arr, idx, val):
        v, d = arr.v.copy(), arr.d.copy()
        v[idx] += val.v
        d[idx] += val.d
        return Dual(v, d)


def jacobian(rhs, q):
    """Row n: d rhs / d q.flat[n], in extended precision."""
    q = q.astype(LD)
    rows = []
    for n in range(q.size):
        d = np.zeros_like(q)
        d.flat[n] = 1
        rows.append(rhs(Dual(q, d)).d.ravel())
    return np.stack(rows)

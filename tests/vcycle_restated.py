"""The GB300 solver's V-cycle restated in numpy with its vectors and records
rounded where the kernels store them, so that a comparison is bound by the
rounding of the arithmetic between two stores and not by the stores.

Levels, finest first: `fused` ones run three half-steps per pass with every
value between two stores in FP32; then levels that store the correction after
each half-step; then the bottom sub-cycle, FP32 from its right-hand side to its
result."""
import numpy as np

SOR_BLACK = 1.2
WEIGHT = 2.0


def to_bf16(v):
    b = np.asarray(v, np.float32).view(np.uint32).astype(np.uint64)
    b = (b + 0x7FFF + ((b >> 16) & 1)) & 0xFFFF0000
    return b.astype(np.uint32).view(np.float32)


def to_half(v):
    return np.asarray(v, np.float32).astype(np.float16).astype(np.float32)


ROUND = {"fp16": to_half, "bf16": to_bf16, "fp32": lambda v: np.asarray(v, np.float32)}


def round_up(v, precision):
    """The record's diagonal: the FP32 sum rounded up to the record precision."""
    v = np.asarray(v, np.float32)
    if precision == "fp32":
        return v
    if precision == "fp16":
        h = v.astype(np.float16)
        return np.where(h.astype(np.float32) < v, np.nextafter(h, np.float16(np.inf)), h).astype(np.float32)
    b = (v.view(np.uint32).astype(np.uint64) + 0xFFFF) & 0xFFFF0000  # positive values
    return b.astype(np.uint32).view(np.float32)


def shift(v, axis, step, wrap):
    """The value of the neighbour `step` cells along grid axis x, y, z; 0 outside."""
    ax = 2 - axis
    out = np.roll(v, -step, ax)
    if not wrap:
        edge = [slice(None)] * 3
        edge[ax] = -1 if step > 0 else 0
        out[tuple(edge)] = 0
    return out


def pad_sum8(v):
    p = np.pad(v, [(0, n % 2) for n in v.shape])
    return p.reshape(p.shape[0] // 2, 2, p.shape[1] // 2, 2, p.shape[2] // 2, 2).sum((1, 3, 5))


def expand(ec, shape):
    return np.repeat(np.repeat(np.repeat(ec, 2, 0), 2, 1), 2, 2)[tuple(slice(0, k) for k in shape)]


class Level:
    def __init__(self, betas, react, periodic, precision, fused, dtype):
        self.master, self.react, self.periodic = betas, react, periodic
        lo = ROUND[precision]
        self.b = [lo(b).astype(dtype) for b in betas]
        self.high = [shift(b, a, 1, periodic >> a & 1) for a, b in enumerate(self.b)]
        d = sum(b + h for b, h in zip(self.b, self.high)) + lo(react).astype(dtype)
        self.diag = round_up(d, precision).astype(dtype) if fused else d
        self.inv = np.divide(1.0, self.diag, out=np.zeros_like(self.diag), where=self.diag > 0)
        z, y, x = np.indices(react.shape)
        self.red = (x + y + z) % 2 == 0
        self.fused = fused

    def neighbours(self, e):
        return sum(b * shift(e, a, -1, self.periodic >> a & 1) + h * shift(e, a, 1, self.periodic >> a & 1)
                   for a, (b, h) in enumerate(zip(self.b, self.high)))

    def half(self, e, r, red, omega=1.0):
        new = (r + self.neighbours(e)) * self.inv
        m = (self.red if red else ~self.red)
        e = np.where(m, e + omega * (new - e), e)
        e[self.diag <= 0] = 0.0
        return e

    def residual(self, e, r):
        return r - (self.diag * e - self.neighbours(e))

    def coarse(self):
        out = []
        for a, b in enumerate(self.master):  # faces between aggregates: low faces of even children
            k = b.copy()
            sel = [slice(None)] * 3
            sel[2 - a] = slice(1, None, 2)
            k[tuple(sel)] = 0.0
            out.append(0.25 * pad_sum8(k))
        return out, 0.25 * pad_sum8(self.react)


def cycle(coef, r, precision, periodic=0, dtype=np.float64, fault=None):
    """z = B r for finest-level records coef[..., (beta_x, beta_y, beta_z, reaction)].  `fault(stage, level, value)` may
    change a value on its way, to plant a mistake."""
    fault = fault or (lambda stage, l, v: v)
    store = lambda v: ROUND[precision](v).astype(dtype)
    shapes = [coef.shape[:3]]
    while max(shapes[-1]) > 4:
        shapes.append(tuple((n + 1) // 2 for n in shapes[-1]))
    last = len(shapes) - 1
    even = lambda s: all(not periodic >> a & 1 or s[2 - a] % 2 == 0 for a in range(3))
    fused = 0
    while fused < last and shapes[fused][2] % 4 == 0 and even(shapes[fused]) and (fused == 0 or np.prod(shapes[fused]) > 4096):
        fused += 1
    bottom = next(k for k in range(1, last + 1) if np.prod(shapes[k]) <= 4096)
    levels, betas, react = [], [coef[..., k].astype(np.float64) for k in range(3)], coef[..., 3].astype(np.float64)
    for l in range(last + 1):
        levels.append(Level(betas, react, periodic, precision, l < fused, dtype))
        if l < last:
            betas, react = levels[-1].coarse()

    def coarsest(r):
        lv = Level(levels[last].master, levels[last].react, periodic, "fp32", False, np.float64)
        on = lv.diag.reshape(-1) > 0
        A = np.stack([(lv.diag * u - lv.neighbours(u)).reshape(-1) for u in np.eye(r.size).reshape(-1, *r.shape)], 1)
        e = np.zeros(r.size)
        e[on] = np.linalg.solve(A[np.ix_(on, on)], r.astype(np.float64).reshape(-1)[on])
        return e.reshape(r.shape).astype(dtype)

    def solve(l, r, keep):
        """keep: whether the right-hand side and the result are stored in the level precision."""
        lv = levels[l]
        keep_half = store if keep and not lv.fused else (lambda v: v)  # after each half-step
        if l == last:
            e = coarsest(r)
            return store(e) if keep else e
        steps = [(True, 1.0), (False, SOR_BLACK), (True, 1.0)] if lv.fused else [(True, 1.0), (False, 1.0)]
        e = np.zeros_like(r)
        for k, (red, om) in enumerate(steps):
            e = keep_half(fault("down%d" % k, l, lv.half(e, r, red, om)))
        rc = fault("restrict", l, 0.25 * pad_sum8(lv.residual(e, r)))
        ec = solve(l + 1, store(rc) if l + 1 <= bottom else rc, l + 1 < bottom)
        if l + 1 == bottom:
            ec = store(ec)
        if lv.fused and l > 0:
            e = store(e)  # the black half; the red one is overwritten before it is read
        e = keep_half(e + dtype(WEIGHT) * expand(ec, r.shape))
        for k, (red, om) in enumerate(reversed(steps)):
            e = keep_half(fault("up%d" % k, l, lv.half(e, r, red, om)))
        return store(e) if lv.fused and l > 0 else e

    return fault("out", 0, solve(0, np.asarray(r).astype(dtype), fused == 0))


def one_liquid(dims, periodic=0, seed=0):
    """Records of one liquid with a solid block and an outlet above, and a random residual whose sum over every 2x2x2
    aggregate is zero: the smooth part of a correction, and with it the rounding of large values, stays small against what
    the half-steps do locally."""
    nx, ny, nz = dims
    solid = np.zeros((nz, ny, nx), np.uint8)
    solid[: nz // 3, ny // 3, nx // 4: nx // 2] = 1
    fluid = solid == 0
    coef = np.zeros((nz, ny, nx, 4), np.float32)
    for a in range(3):
        coef[..., a] = fluid & shift(fluid, a, -1, periodic >> a & 1)
    if not periodic & 4:
        coef[-1, ..., 3] = 2.0 * fluid[-1]
    r = np.where(fluid, np.random.default_rng(seed + nx + ny + nz).standard_normal((nz, ny, nx)), 0.0)
    mean = pad_sum8(r) / np.maximum(pad_sum8(fluid.astype(np.float64)), 1)
    r -= expand(mean, r.shape) * fluid
    return solid, coef, r.astype(np.float32)

"""The GB300 solver's V-cycle against an FP64 restatement in numpy, at sizes
where a tile, a quad or a run ends inside the grid."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOR_BLACK = 1.2
WEIGHT = 2.0


class Level:
    """One level: low-face mobilities, diagonal (FP64), the colour masks."""

    def __init__(self, bx, by, bz, react, periodic=0):
        self.b = (bx, by, bz)
        self.periodic = periodic
        self.react = react
        z, y, x = np.indices(bx.shape)
        self.red = (x + y + z) % 2 == 0
        self.diag = react + sum(b + self._high(b, a) for a, b in enumerate(self.b))
        self.inv = np.divide(1.0, self.diag, out=np.zeros_like(self.diag), where=self.diag > 0)

    def _high(self, v, a):  # value of the high neighbour along x, y, z (0 outside)
        out = np.zeros_like(v)
        ax = 2 - a
        if self.periodic >> a & 1:
            return np.roll(v, -1, ax)
        src = [slice(None)] * 3
        dst = [slice(None)] * 3
        src[ax], dst[ax] = slice(1, None), slice(None, -1)
        out[tuple(dst)] = v[tuple(src)]
        return out

    def _low(self, v, a):
        out = np.zeros_like(v)
        ax = 2 - a
        if self.periodic >> a & 1:
            return np.roll(v, 1, ax)
        src = [slice(None)] * 3
        dst = [slice(None)] * 3
        src[ax], dst[ax] = slice(None, -1), slice(1, None)
        out[tuple(dst)] = v[tuple(src)]
        return out

    def neighbours(self, e):
        s = np.zeros_like(e)
        for a, b in enumerate(self.b):
            s += b * self._low(e, a) + self._high(b * 1.0, a) * self._high(e, a)
        return s

    def half(self, e, r, red, omega=1.0):
        m = self.red if red else ~self.red
        new = (r + self.neighbours(e)) * self.inv
        e[m] += omega * (new - e)[m]
        e[self.diag <= 0] = 0.0

    def residual(self, e, r):
        return r - (self.diag * e - self.neighbours(e))

    def coarse(self):
        nz, ny, nx = self.react.shape
        pad = [(0, n % 2) for n in (nz, ny, nx)]

        def sum8(v):
            p = np.pad(v, pad)
            return p.reshape(p.shape[0] // 2, 2, p.shape[1] // 2, 2, p.shape[2] // 2, 2).sum((1, 3, 5))

        out = []
        for a, b in enumerate(self.b):  # faces between aggregates: low faces of even children
            k = b.copy()
            sel = [slice(None)] * 3
            sel[2 - a] = slice(1, None, 2)
            k[tuple(sel)] = 0.0
            out.append(0.25 * sum8(k))
        return Level(*out, 0.25 * sum8(self.react), self.periodic), sum8


def reference_cycle(coef, r, precision, periodic):
    levels, sums = [Level(*(coef[..., k].astype(np.float64) for k in range(4)), periodic)], []
    while max(levels[-1].react.shape) > 4:
        c, s = levels[-1].coarse()
        levels.append(c)
        sums.append(s)
    nx = [lv.react.shape[2] for lv in levels]
    n = [lv.react.size for lv in levels]
    last = len(levels) - 1
    fused = 0
    while fused < last and nx[fused] % 4 == 0 and (fused == 0 or n[fused] > 4096):
        fused += 1
    bottom = next(k for k in range(1, last + 1) if n[k] <= 4096)
    w = next((k for k in range(1, last) if n[k] <= 32768), 0)
    if n[0] * (16 if precision == "fp32" else 8) < 48 << 20:
        w = 0
    if fused <= w < bottom:  # levels between the fused ones and the bottom sub-cycle take one visit
        w = 0

    def pair(l):  # levels of red and black half-steps without over-relaxation
        nz, ny, _ = levels[l].react.shape
        run = -(-nx[l] // 64) * -(-ny // 8) * -(-nz // 2) <= (152 if precision == "fp32" else 304)
        return l >= fused or (precision == "fp32" and not periodic and not run)

    def cycle(l, r):
        lv = levels[l]
        if l == last:
            act = (lv.diag > 0).reshape(-1)
            m = r.size
            A = np.zeros((m, m))
            for i in range(m):
                u = np.zeros(m)
                u[i] = 1.0
                A[:, i] = (lv.diag * u.reshape(r.shape) - lv.neighbours(u.reshape(r.shape))).reshape(-1)
            e = np.zeros(m)
            e[act] = np.linalg.lstsq(A[np.ix_(act, act)], r.reshape(-1)[act], rcond=1e-10)[0]
            return e.reshape(r.shape)
        e = np.zeros_like(r)
        steps = [(True, 1.0), (False, 1.0)] if pair(l) else [(True, 1.0), (False, SOR_BLACK), (True, 1.0)]
        for red, om in steps:
            lv.half(e, r, red, om)
        rc = 0.25 * sums[l](lv.residual(e, r))
        ec = cycle(l + 1, rc)
        if l + 1 == w:
            ec = ec + cycle(l + 1, levels[l + 1].residual(ec, rc))
        up = np.repeat(np.repeat(np.repeat(ec, 2, 0), 2, 1), 2, 2)[tuple(slice(0, k) for k in r.shape)]
        e = e + WEIGHT * up
        for red, om in reversed(steps):
            lv.half(e, r, red, om)
        return e

    return cycle(0, r)


# (extents, periodic axes).  x extents that are no multiple of 8 or 64, y
# extents one off a tile of 8 or 32 rows, odd z extents, runs of one plane
# pair, a grid of one tile; periodic extents that stay even down to the bottom
# sub-cycle; FP32 records large enough for two visits of a coarse level
DIMS = [((72, 37, 41), 0), ((132, 33, 23), 0), ((64, 32, 18), 0), ((200, 9, 31), 0), ((20, 65, 27), 0),
        ((64, 48, 64), 1), ((96, 64, 72), 2), ((64, 41, 32), 4), ((68, 64, 64), 6), ((160, 140, 150), 0)]


@pytest.mark.parametrize("precision", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("dims,periodic", DIMS, ids=["x".join(map(str, d)) + f"-{p}" for d, p in DIMS])
def test_v_cycle_equals_the_fp64_restatement(gpu, dims, periodic, precision):
    """One liquid, so every mobility is exact in FP16 and BF16 on the finest
    level and the levels' vectors are all that is rounded: about ten roundings
    of 2^-24, 2^-12 or 2^-9 on the way, amplified at most a few times by the
    coarsest solve (20 roundings allowed of the largest value, times 8)."""
    import mhdproj

    torch = gpu
    nx, ny, nz = dims
    rng = np.random.default_rng(nx + ny + nz)
    solid = np.zeros((nz, ny, nx), np.uint8)
    solid[: nz // 3, ny // 3, nx // 4: nx // 2] = 1
    pr = mhdproj.PressureProjection(dims, 1e-4, outlet=not periodic & 4, periodic=[periodic >> a & 1 for a in range(3)], precision=precision)
    t = lambda a: torch.from_numpy(a).cuda()
    pr.set_coefficients(t(np.ones((nz, ny, nx), np.float32)), t(solid), 6440.0, 6440.0)
    coef = pr.coefficients().cpu().numpy()
    r = np.where(solid == 0, rng.standard_normal((nz, ny, nx)), 0.0).astype(np.float32)
    if periodic & 4:  # closed: a compatible right-hand side, answers up to a constant
        r -= np.where(solid == 0, r[solid == 0].astype(np.float64).mean(), 0.0).astype(np.float32)
    got = pr.apply_preconditioner(t(r)).cpu().numpy().astype(np.float64)
    pr.close()
    ref = reference_cycle(coef, r.astype(np.float64), precision, periodic)
    if periodic & 4:
        got, ref = (np.where(solid == 0, v - v[solid == 0].mean(), 0.0) for v in (got, ref))
    eps = {"fp32": 2.0 ** -24, "fp16": 2.0 ** -12, "bf16": 2.0 ** -9}[precision]
    assert np.abs(got - ref).max() <= 160 * eps * np.abs(ref).max()


# whole runs, TMA passes, passes of two half-steps (the correction of every cell)
@pytest.mark.parametrize("precision,dims,e", [("fp16", (64, 64, 64), 2), ("fp16", (128, 128, 128), 2), ("fp32", (128, 64, 128), 4)])
def test_profiled_bytes_of_the_passes(gpu, precision, dims, e):
    """The smoothing passes' compulsory bytes per cell: FP32 r, q and z, the
    correction as it is stored between them, records, an eighth of a coarse
    vector value."""
    import mhdproj

    torch = gpu
    shape = dims[::-1]
    pr = mhdproj.PressureProjection(dims, 1e-4, outlet=True, precision=precision)
    pr.set_coefficients(torch.ones(shape, device="cuda"), torch.zeros(shape, dtype=torch.uint8, device="cuda"), 6440.0, 6440.0)
    u = [torch.zeros(s, device="cuda") for s in ((shape[0], shape[1], shape[2] + 1), (shape[0], shape[1] + 1, shape[2]),
                                                 (shape[0] + 1, shape[1], shape[2]))]
    u[2][:, 0, 0] = 1.0
    pr.project(u, 1e-5)
    got = {k["name"]: k["bytes"] for k in pr.profile_kernels()}
    pr.close()
    n, records, coarse = dims[0] * dims[1] * dims[2], {"fp32": 16, "fp16": 8}[precision], {"fp32": 4, "fp16": 2}[precision] / 8
    assert got["presmooth_restrict"] == n * (4 + 4 + records + 4 + e + coarse)
    assert got["prolong_postsmooth"] == n * (e + coarse + 4 + records + 4)


@pytest.mark.parametrize("dims", [(24, 16, 160), (28, 16, 160), (24, 72, 35), (136, 9, 75)], ids=str)
def test_fp32_pair_passes_on_narrow_and_ragged_grids(gpu, dims):
    """The FP32 passes of two half-steps, their coarse rows copied (x extents
    that 8 divides) or loaded: coarse planes smaller than a copy's box, rows and
    planes that end inside a pair."""
    test_v_cycle_equals_the_fp64_restatement(gpu, dims, 0, "fp32")

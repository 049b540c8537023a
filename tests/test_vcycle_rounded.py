"""The V-cycle's FP16 and BF16 passes against a restatement that rounds where
they store, at extents where a tile, an octet, a run or a pair of planes ends
inside the grid."""
import numpy as np
import pytest

import vcycle_restated as V

EPS = {"fp16": 2.0 ** -11, "bf16": 2.0 ** -8}  # unit roundoff of the level vectors

# The same restatement in FP32 instead of FP64 differs by at most 0.88 EPS in the
# 2-norm and 0.75 EPS of the largest value on these grids (values that fall on the
# other side of a rounding); about three times that is allowed.
L2, MAX = 2.5, 2.5


def bound(got, ref, precision):
    d = np.abs(got - ref)
    return max(np.linalg.norm(d) / np.linalg.norm(ref) / (L2 * EPS[precision]), d.max() / np.abs(ref).max() / (MAX * EPS[precision]))


# Above one wave of whole runs on the finest level unless said otherwise.
# 132: an octet cut in half; y one row past a tile, odd z.  264: the same on the
# first coarse level too.  200x31: less than a tile of rows.  256x72: every level
# above the bottom sub-cycle fused, whole runs below the large ones.  Then periodic
# y in the marching form, periodic x and a small grid in whole runs.
DIMS = [((132, 33, 75), 0), ((264, 33, 149), 0), ((200, 31, 129), 0), ((256, 72, 131), 0), ((96, 64, 72), 2), ((64, 48, 64), 1),
        ((48, 40, 56), 0)]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp16", "bf16"])
@pytest.mark.parametrize("dims,periodic", DIMS, ids=["x".join(map(str, d)) + f"-{p}" for d, p in DIMS])
def test_v_cycle_to_its_rounding(gpu, dims, periodic, precision):
    import mhdproj

    torch = gpu
    solid, coef, r = V.one_liquid(dims, periodic)
    pr = mhdproj.PressureProjection(dims, 1e-4, outlet=True, periodic=[periodic >> a & 1 for a in range(3)], precision=precision)
    t = lambda a: torch.from_numpy(a).cuda()
    pr.set_coefficients(t(np.ones(solid.shape, np.float32)), t(solid), 6440.0, 6440.0)
    assert np.array_equal(pr.coefficients().cpu().numpy(), coef)
    rt = t(r)
    z = pr.apply_preconditioner(rt).clone()
    for _ in range(4):  # the same bits every time
        assert torch.equal(pr.apply_preconditioner(rt), z)
    s = np.where(solid == 0, np.random.default_rng(1).standard_normal(r.shape), 0.0).astype(np.float32)
    zs = pr.apply_preconditioner(t(s)).cpu().numpy().astype(np.float64)
    pr.close()
    z = z.cpu().numpy().astype(np.float64)
    assert bound(z, V.cycle(coef, r, precision, periodic), precision) <= 1
    # symmetric but for the roundings of two cycles: each changes <., B .> by at most L2 EPS |.| |B .|
    gap = abs(np.vdot(s, z) - np.vdot(r, zs))
    assert gap <= 2 * EPS[precision] * (np.linalg.norm(s) * np.linalg.norm(z) + np.linalg.norm(r) * np.linalg.norm(zs))


def _row_missing(stage, l, v):  # the first half-step left out in one halo row
    if stage == "down0" and l == 0:
        v[:, 32, :] = 0.0
    return v


def _edge_missing(stage, l, v):  # the second half-step up left out in the half octet at the x edge
    if stage == "up1" and l == 0:
        v[:, :, 128:] = 0.0
    return v


def _pair_mixed(stage, l, v):  # half of the last but one coarse plane's sums taken from the last one
    if stage == "restrict" and l == 0:
        v[-2] = 0.5 * (v[-2] + v[-1])
    return v


@pytest.mark.parametrize("precision", ["fp16", "bf16"])
@pytest.mark.parametrize("fault", [None, _row_missing, _edge_missing, _pair_mixed, "relaxation"], ids=str)
def test_the_bound_sees_mistakes(monkeypatch, fault, precision):
    """Planted in the restatement: each exceeds the bound, and FP32 arithmetic alone stays below it."""
    _, coef, r = V.one_liquid((132, 33, 75))
    ref = V.cycle(coef, r, precision)
    if fault is None:
        assert bound(V.cycle(coef, r, precision, dtype=np.float32).astype(np.float64), ref, precision) <= 0.5
        return
    if fault == "relaxation":
        monkeypatch.setattr(V, "SOR_BLACK", 1.0)
    assert bound(V.cycle(coef, r, precision, fault=fault if callable(fault) else None), ref, precision) > 2

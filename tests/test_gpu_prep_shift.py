"""FP32 preprocessing next to the dihedral shift's threshold: values around
2 pi - modFit, where the shift quotient turns from 0 to 1, with and without an
empty stretch in the occupancy histogram, NaN-free and at both ends of the range;
1D and 2D bin counts that are and are not the same. One misplaced value of 4,000
moves an entropy by more than 1e-4 nats; the oracle's are met within 1e-9."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import parent_gb300 as pg

pytestmark = pytest.mark.gpu

BS = (2 * np.pi + 5e-9) / 100


def _column(pos, gap, rng, n):
    """n float32 values; the shift histogram's longest gap (or, without one, its
    only minimum) starts at bin pos; floats around the threshold included."""
    thr = np.float32((pos + 0.5) * BS)
    near = [thr]
    for _ in range(6):
        near.append(np.nextafter(near[-1], np.float32(7)))
    low = thr
    for _ in range(6):
        low = np.nextafter(low, np.float32(0))
        near.append(low)
    if gap:  # the gap's first bin has to stay empty: its neighbours' edges instead
        near = [np.float32(pos * BS - 1e-6), np.float32((pos + gap) * BS + 1e-6)]
    bins = [b for b in range(100) if not (gap and (b - pos) % 100 < gap)]
    weight = np.array([0 if b == pos else 2 for b in bins], float)
    body = (rng.choice(bins, n - len(near) - 2 * (len(bins)), p=weight / weight.sum()) + rng.random(n - len(near) - 2 * len(bins))) * BS
    fill = (np.repeat([b for b in bins if b != pos or gap], 2) + 0.5) * BS  # every other bin occupied
    fill = np.concatenate([fill, np.full(2 * len(bins) - len(fill), (bins[-1] if bins[-1] != pos else bins[0]) * BS + 0.01)])
    x = np.concatenate([body, fill, np.array(near, np.float64)]).astype(np.float32)
    return np.clip(x, 0, np.float32(6.283185))


@pytest.mark.parametrize("b1,b2", [(50, 50), (36, 50)])
def test_shift_threshold(b1, b2):
    rng = np.random.default_rng(17)
    n = 4000
    cols = [_column(p, g, rng, n) for p, g in ((40, 0), (0, 0), (99, 0), (63, 0), (10, 30), (90, 25), (0, 7))]
    nd = len(cols)
    bonds = rng.normal(1.4, 0.03, (nd + 2, n)).astype(np.float32)
    angles = rng.uniform(0.4, 2.7, (nd + 1, n)).astype(np.float32)
    t = pg.Trajectory(bonds, angles, np.stack(cols))
    bins = (b1,) * 3 + (b2,) * 3
    with pg.Engine(0) as eng:
        body = eng.entropy(t, bins, "hist")
    ref = oracle.parent(t.bonds, t.angles, t.dihedrals, bins)
    for k in oracle.BLOCKS:
        if ref[k].size:
            assert np.max(np.abs(body.blocks[k] - ref[k])) <= 1e-9, k


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_equal_stretches_and_minima(dtype):
    """The first of equal empty stretches (inside the range, and one over its end),
    the first of equal minima, and single bins empty or occupied."""
    rng = np.random.default_rng(23)
    n = 3000

    def column(empty=(), low=()):
        bins = np.array([b for b in range(100) if b not in empty])
        each = np.where(np.isin(bins, low), 5, 20)
        b = np.concatenate([np.repeat(bins, each), np.full(n - each.sum(), next(b for b in bins if b not in low))])
        return ((b + 0.1 + 0.8 * rng.random(n)) * BS).astype(dtype)

    cols = [column(low=(20, 70)), column(low=(0, 99)), column(empty=(10, 11, 12, 60, 61, 62)), column(empty=(98, 99, 0, 40, 41, 42)),
            column(empty=(99, 0, 50, 51)), column(empty=(5,)), column(empty=range(3, 99)), column(empty=range(1, 100))]
    nd = len(cols)
    t = pg.Trajectory(rng.normal(1.4, 0.03, (nd + 2, n)).astype(dtype), rng.uniform(0.4, 2.7, (nd + 1, n)).astype(dtype),
                      np.stack(cols))
    with pg.Engine(0) as eng:
        body = eng.entropy(t, (40,) * 3 + (50,) * 3, "hist")
        shift = eng.dof_stats(3 * nd + 3)[2][2 * nd + 3:]
    ref = oracle.parent(t.bonds, t.angles, t.dihedrals, (40,) * 3 + (50,) * 3)
    starts = [20, 0, 10, 40, 50, 5, 3, 1]  # of 98-0 and 40-42, and of 99-0 and 50-51, the one that ends first
    assert np.max(np.abs(shift - [2 * np.pi - (s + 0.5) * BS for s in starts])) <= 1e-12
    for k in oracle.BLOCKS:
        if ref[k].size:
            assert np.max(np.abs(body.blocks[k] - ref[k])) <= 1e-9, k

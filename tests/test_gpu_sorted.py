"""The sorted-list histogram kernel (pg_pairs_sorted.cu) against the tiled
histogram kernels and the oracle.

Every pair's counts enter exact integer sums, and every kernel finishes with
the same expressions, so the bodies must agree bit for bit; the oracle's 2D
entropies are within 1e-9 nats (the bound of the other kernels' tests). Sizes
are the edges of its tiles: one block of 128 columns less, exact and more, rows
of 4 frames and batches of 32, counts past a 16-bit half, one frame, and the
smallest and largest bin counts."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import parent_gb300 as pg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = pg.Engine(0)
    yield e
    e.close()


def _both(eng, monkeypatch, traj, bins):
    out = []
    for on in ("1", "0"):
        monkeypatch.setenv("PG_HIST_SORTED", on)
        body = eng.entropy(traj, bins, "hist")
        edges, totals = eng.mist(traj.n_dih if isinstance(traj, pg.Trajectory) else traj.n_dihedrals)
        out.append((body.flat(), edges, totals))
    return out


# atoms, frames, 2D bins (b, a, d), double precision
SHAPES = [
    (3, 5, (50, 50, 50), 0),        # no dihedral: 3 DOFs
    (5, 1, (40, 40, 40), 1),        # one frame
    (44, 31, (50, 36, 40), 0),      # 126 DOFs: a block less 2; less than a batch of frames
    (45, 32, (51, 51, 51), 1),      # 129 DOFs: one column past a block
    (88, 997, (58, 57, 60), 0),     # 258 DOFs; two and four warps per table
    (30, 4097, (119, 120, 121), 0), # four and eight warps per table
    (12, 2049, (218, 218, 218), 1), # the largest table
    (40, 3000, (1, 2, 3), 0),       # the smallest tables
    (24, 20001, (50, 50, 50), 0),   # several items per row and block
]


@pytest.mark.parametrize("atoms,frames,b2,prec", SHAPES)
def test_sorted_equals_tiled_and_oracle(eng, monkeypatch, atoms, frames, b2, prec):
    bins = (20, 30, 40) + b2
    t = pg.synth_host(atoms, frames, double_prec=prec, seed=atoms + frames, frac_bimodal_dih=0.3)
    (a, ea, ta), (b, eb, tb) = _both(eng, monkeypatch, t, bins)
    assert np.array_equal(a, b)
    assert np.array_equal(ea, eb) and np.array_equal(ta, tb)
    r = oracle.parent(t.bonds, t.angles, t.dihedrals, bins)
    ref = np.concatenate([r[k] for k in oracle.BLOCKS])
    assert np.max(np.abs(a - ref)) <= 1e-9


# 1 to 8 warps per table and one table per CTA; odd and mixed bin counts, a
# column pair over a block's first column and over a change of type
JOINT = [(3, 5, (30, 30, 30), 0), (44, 31, (7, 8, 9), 1), (45, 997, (1, 2, 3), 0), (88, 4097, (10, 10, 10), 0),
         (30, 4096, (15, 14, 16), 1), (60, 2500, (20, 21, 19), 0), (24, 20001, (30, 29, 17), 0)]


@pytest.mark.parametrize("atoms,frames,b2,prec", JOINT)
def test_joint_counters_equal_tiled_and_oracle(eng, monkeypatch, atoms, frames, b2, prec):
    monkeypatch.setenv("PG_SORTED_JOINT", "1")
    test_sorted_equals_tiled_and_oracle(eng, monkeypatch, atoms, frames, b2, prec)


@pytest.mark.parametrize("bins,joint", [(50, "0"), (20, "1")])
@pytest.mark.parametrize("frames", [64512, 64513, 140000])
def test_sorted_counts_above_16_bits(eng, monkeypatch, frames, bins, joint):
    """Columns with one value in most frames: segments and counts around and
    past what a 16-bit half holds (pieces of 64,512 frames)."""
    monkeypatch.setenv("PG_SORTED_JOINT", joint)
    t = pg.synth_host(9, frames, double_prec=0, seed=5)
    for k, c in enumerate((t.bonds, t.angles, t.dihedrals)):
        c[:, : frames - 7 - k] = c[:, :1]
    (a, ea, _), (b, eb, _) = _both(eng, monkeypatch, t, (bins,) * 6)
    assert np.array_equal(a, b) and np.array_equal(ea, eb)


@pytest.mark.parametrize("bins", [(50, 50, 50, 50, 44, 39), (10, 10, 10, 9, 10, 8)])
def test_sorted_batch_equals_single_calls(eng, monkeypatch, bins):
    """One launch over systems of several sizes, replayed, against a call per
    system (the batch's items are split differently); 10 bins: joint counters."""
    monkeypatch.setenv("PG_HIST_SORTED", "1")
    trajs = [pg.synth_host(a, f, double_prec=p, seed=k) for k, (a, f, p) in
             enumerate([(50, 5000, 0), (4, 64600, 1), (90, 333, 1), (45, 9000, 0)])]
    single = []
    for t in trajs:
        body = eng.entropy(t, bins, "hist")
        single.append((body.flat(), eng.mist(t.n_dih)[0]))
    for _ in range(2):
        bodies, trees = eng.entropy_batch(trajs, bins, "hist")
        for (flat, edges), body, (e, _) in zip(single, bodies, trees):
            assert np.array_equal(flat, body.flat()) and np.array_equal(edges, e)


# half blocks on the diagonal: the first block wholly past its middle (pad of 64
# columns and more), one short of it, a single block; segments around the pieces
HALVES = [(66, 2000, (5, 7, 6), 0), (65, 4099, (16, 15, 14), 1), (67, 3001, (9, 8, 9), 0), (44, 13003, (50, 50, 50), 0),
          (88, 5200, (20, 3, 1), 1), (47, 66000, (36, 50, 44), 0), (4, 999, (3, 3, 3), 0)]


@pytest.mark.parametrize("atoms,frames,b2,prec", HALVES)
def test_half_blocks_equal_tiled_and_oracle(eng, monkeypatch, atoms, frames, b2, prec):
    monkeypatch.setenv("PG_SORTED_JOINT", "0")
    test_sorted_equals_tiled_and_oracle(eng, monkeypatch, atoms, frames, b2, prec)


@pytest.mark.parametrize("frames", [64512, 140000])
def test_half_blocks_counts_above_16_bits(eng, monkeypatch, frames):
    """66 DOFs (no row needs a lower column's counter), one value in most frames."""
    monkeypatch.setenv("PG_SORTED_JOINT", "0")
    t = pg.synth_host(24, frames, double_prec=0, seed=5)
    for k, c in enumerate((t.bonds, t.angles, t.dihedrals)):
        c[:, : frames - 7 - k] = c[:, :1]
    (a, ea, _), (b, eb, _) = _both(eng, monkeypatch, t, (30,) * 6)
    assert np.array_equal(a, b) and np.array_equal(ea, eb)

"""The one-hot kernel on packed FP4 operands (pg_onehot_bits.cuh) against the
FP8 one-hot kernel and the oracle.

Both feed exact counts into the same integer sums and finish with the same
expressions: the bodies agree bit for bit. Sizes are the edges of its K-blocks
(256 frames) and ring, of its tiles (256 x 448 rows of C), of the bit planes, of
the part of the n ln n table in shared memory, and of its frame limit."""
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


def _both(eng, monkeypatch, run):
    monkeypatch.setenv("PG_ONEHOT_PAIR", "1")
    fp8 = run()
    monkeypatch.delenv("PG_ONEHOT_PAIR")
    bits = run()
    assert eng.last_form() == "onehot"
    return fp8, bits


# atoms, frames, 2D bins (b, a, d), double precision
SHAPES = [
    (3, 1, (8, 8, 8), 1),            # no dihedral, one frame
    (5, 255, (10, 10, 10), 0),       # a K-block less a frame
    (10, 256, (16, 16, 16), 1),      # 432 rows: two row tiles, one column tile
    (19, 1025, (8, 8, 8), 0),        # 432 rows; the ring's first block again
    (17, 2049, (9, 10, 9), 0),       # 449 rows: one past a column tile
    (60, 1500, (31, 64, 15), 0),     # different 2D bin counts per type
    (9, 4097, (65, 127, 33), 1),     # seven bit planes
    (8, 40001, (8, 12, 9), 0),       # counts past the table's part in shared memory
]


@pytest.mark.parametrize("atoms,frames,b2,prec", SHAPES)
def test_bits_equal_fp8_and_oracle(eng, monkeypatch, atoms, frames, b2, prec):
    bins = (20, 30, 40) + b2
    t = pg.synth_host(atoms, frames, double_prec=prec, seed=atoms + frames, frac_bimodal_dih=0.3)
    a, b = _both(eng, monkeypatch, lambda: eng.entropy(t, bins, "onehot").flat())
    assert np.array_equal(a, b)
    r = oracle.parent(t.bonds, t.angles, t.dihedrals, bins)
    ref = np.concatenate([r[k] for k in oracle.BLOCKS])
    assert np.max(np.abs(b - ref)) <= 1e-9


def test_bits_batch_equals_single_calls(eng, monkeypatch):
    bins = (10, 12, 9, 10, 12, 9)
    trajs = [pg.synth_host(a, f, double_prec=p, seed=a) for a, f, p in ((20, 1500, 0), (3, 1, 1), (41, 5000, 1))]
    fp8, bits = _both(eng, monkeypatch, lambda: [b.flat() for b in eng.entropy_batch(trajs, bins, form="onehot")[0]])
    again = eng.entropy_batch(trajs, bins, form="onehot")[0]
    for t, a, b, c in zip(trajs, fp8, bits, again):
        assert np.array_equal(a, b) and np.array_equal(b, c.flat())
        assert np.array_equal(b, eng.entropy(t, bins, "onehot").flat())


@pytest.mark.parametrize("frames", [1 << 22, (1 << 22) + 1])
def test_bits_frame_limit(eng, monkeypatch, frames):
    """Counts to 2^22, one frame off a multiple of 64 apart; above it the FP8 kernel."""
    x = np.empty((6, frames), np.float32)
    rng = np.random.default_rng(5)
    for r, v in enumerate((1.5, 1.4, 1.3, 1.9, 2.0, 3.0)):
        x[r] = v
        x[r, rng.integers(0, frames, 37 + r)] += np.float32(0.1)
    t = pg.Trajectory(x[:3].copy(), x[3:5].copy(), x[5:].copy())
    bins = (10,) * 6
    a, b = _both(eng, monkeypatch, lambda: eng.entropy(t, bins, "onehot").flat())
    assert np.array_equal(a, b)

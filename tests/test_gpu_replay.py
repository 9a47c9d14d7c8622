"""The replay of the k-biggest scan at the edges of its windows (one segment
per thread, four windows read at once), of its 2048-record staging and of its
state, against the oracle's reservoir: floods of ties, scores that rise or
fall along the scan (every position a trigger, or the first ones only),
images of a few positions and of many windows, more candidates than valid
positions."""
import numpy as np
import pytest

from tests.test_gpu_pattern import make_terms, oracle_kbest

pytestmark = pytest.mark.gpu

# every size is one that the FFT padding leaves as it is (the oracle's scan has none)
SHAPES = [(5,), (128,), (2048,), (2058,), (4096,), (33, 64), (260, 260), (150000,), (64, 66, 64)]


def values(kind, shape, seed):
    n = int(np.prod(shape))
    rng = np.random.default_rng(seed)
    if kind == "constant":
        v = np.ones(n)
    elif kind == "two":
        v = (rng.random(n) < 0.4).astype(float)
    elif kind == "steps":
        v = np.floor(np.linspace(0, 12, n, endpoint=False))
    elif kind == "rising":
        v = np.linspace(0.0, 1.0, n)
    elif kind == "falling":
        v = np.linspace(1.0, 0.0, n)
    else:
        v = rng.standard_normal(n)
    return v.reshape(shape).astype(np.float32)


@pytest.mark.parametrize("kind", ["constant", "two", "steps", "rising", "falling", "noise"])
@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
def test_replay_edges_bit_exact(g2s, gpu, oracle, shape, kind):
    nd = len(shape)
    ti = values(kind, shape, 3)
    W = g2s.Worker(g2s.TrainingImage(ti, [0]))
    rng = np.random.default_rng(len(kind) + sum(shape))
    for k in (1, 2, 3, 6, 16):
        for reach in (0, 1):
            offs = np.zeros((1 + reach * nd, nd), np.int32)
            for d in range(reach * nd):
                offs[1 + d, d] = 1 if d % 2 else -1
            vals = np.full((len(offs), 1), np.float32(1.0))
            seed = float(np.float32(rng.random()))
            sc, ix, _ = W.pattern_kbest(offs, make_terms(offs, vals, [0]), k, seed)
            v, p, _, _, _, _ = oracle_kbest(oracle, ti, [0], offs, vals, k, seed)
            assert np.array_equal(sc, v), (k, reach, sc, v)
            assert np.array_equal(ix, p), (k, reach, ix, p)

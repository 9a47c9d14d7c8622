"""The FP32 map's 256-position spans at their edges: images whose scan ends
inside a span, narrow rows, a span with no valid position, and terms of one,
several and mixed operations, against the oracle bit for bit (the kernel adds
the same FP32 terms in the same order)."""
import numpy as np
import pytest

from g2s_b200 import synthetic as syn
from tests.test_gpu_pattern import make_terms, oracle_kbest, random_pattern

pytestmark = pytest.mark.gpu

SHAPES = [(129,), (257,), (2051,), (300, 1), (1, 300), (131, 2), (65, 3), (16, 16), (33, 31), (96, 257), (5, 6, 7),
          (3, 64, 65), (40, 3, 129)]


def image(shape, types, seed):
    rng = np.random.default_rng(seed)
    out = []
    for t in types:
        x = rng.standard_normal(shape).astype(np.float32)
        out.append((x > 0.3).astype(np.float32) if t == 1 else x)
    return out[0] if len(out) == 1 else np.ascontiguousarray(np.stack(out, -1))


@pytest.mark.parametrize("types", [[0], [0, 1], [1, 0]], ids=["continuous", "mixed", "mixed reversed"])
@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
def test_map_spans_bit_exact(g2s, gpu, oracle, shape, types):
    nd = len(shape)
    ti = image(shape, types, 7)
    rng = np.random.default_rng(sum(shape) + len(types))
    T = g2s.TrainingImage(ti, types)
    W = g2s.Worker(T)
    for k in (1, 3, 16):
        for radius in (0, 1, 3):
            offs, vals = random_pattern(rng, ti, types, 12, radius, nd)
            keep = np.all(np.abs(offs) < np.array(shape[::-1]), axis=1)
            offs, vals = offs[keep], vals[keep]
            vals[0] = ti.reshape(-1, len(types))[0]
            seed = float(np.float32(rng.random()))
            sc, ix, mn = W.pattern_kbest(offs, make_terms(offs, vals, types), k, seed)
            v, p, omn, m32, _, _ = oracle_kbest(oracle, ti, types, offs, vals, k, seed)
            assert np.array_equal(mn, omn)
            assert np.array_equal(sc, v), (k, radius, sc, v)
            fin = np.isfinite(sc)
            if np.array_equal(T.fft_size(), shape[::-1]):
                assert np.array_equal(ix[fin], p[fin]), (k, radius, ix, p)
            else:
                # the oracle's scan has no padding (other draws among ties, other
                # scan indices): every index names a cell of its score
                for i, score in zip(ix[fin], sc[fin]):
                    cell, at, stride = T.index_to_position(mn, int(i)), 0, 1
                    for d, size in enumerate(shape[::-1]):
                        at += (size - (cell % size + int(mn[d])) % size - 1) * stride
                        cell //= size
                        stride *= size
                    assert m32[at] == score


@pytest.mark.parametrize("ops", ["weights", "linear"])
def test_map_spans_weighted_and_linear(g2s, gpu, ops):
    """Weighted matches and linear terms (the packed and scalar forms) against
    the same sums in numpy FP32, term by term."""
    ti = image((37, 53), [1 if ops == "weights" else 0], 11)
    W = g2s.Worker(g2s.TrainingImage(ti, [1 if ops == "weights" else 0]))
    rng = np.random.default_rng(3)
    offs = np.unique(rng.integers(-4, 5, (20, 2)), axis=0).astype(np.int32)
    w = rng.uniform(0.1, 1.0, len(offs)).astype(np.float32)
    op = g2s.QSK_OP_EQ if ops == "weights" else g2s.QSK_OP_LIN
    terms = [(j, 0, op, float(w[j]), 1.0) for j in range(len(offs))]
    sc, ix, mn = W.pattern_kbest(offs, terms, 4, 0.25)
    lo, hi = np.minimum(offs.min(0), 0), np.maximum(offs.max(0), 0)
    ny, nx = ti.shape
    acc = None
    for j, (ox, oy) in enumerate(offs):
        x = ti[oy - lo[1]:oy - lo[1] + ny - (hi[1] - lo[1]), ox - lo[0]:ox - lo[0] + nx - (hi[0] - lo[0])]
        acc = np.zeros_like(x) if acc is None else acc
        # one rounding per term: the product is exact for a 0/1 match and in
        # float64 for a linear term (24 + 24 bits)
        t = np.where(x == 1.0, np.float64(w[j]), 0.0) if ops == "weights" else np.float64(w[j]) * x.astype(np.float64)
        acc = (acc.astype(np.float64) + t).astype(np.float32)
    want = np.sort(acc.ravel())[::-1][:4]
    # double rounding of the float64 sum can differ from a fused multiply-add
    # by one last place per term
    tol = 0.0 if ops == "weights" else len(offs) * np.spacing(np.abs(acc).max())
    assert np.abs(sc - want).max() <= tol

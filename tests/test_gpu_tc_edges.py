"""The shortlist's top-W at its edges against a full sort of the same exact
keys: fewer valid positions than W, every score equal (the tie hash decides
alone), scores that rise along the positions (every position enters), and the
widths on either side of the register / list split.  Small integers are exact
in BF16 and FP32, so keys and positions are equal, not close."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def tie_hash(seed, pos):
    x = (np.uint64(seed) ^ ((pos.astype(np.uint64) * np.uint64(0x9E3779B9)) & np.uint64(0xFFFFFFFF)))
    m = np.uint64(0xFFFFFFFF)
    x ^= x >> np.uint64(16)
    x = (x * np.uint64(0x7FEB352D)) & m
    x ^= x >> np.uint64(15)
    x = (x * np.uint64(0x846CA68B)) & m
    return x ^ (x >> np.uint64(16))


def bf16_bits(a):
    return (np.ascontiguousarray(a, np.float32).view(np.uint32) >> 16).astype(np.uint16)


@pytest.mark.parametrize("ranges", [1, 3])
@pytest.mark.parametrize("W", [8, 16, 32])
@pytest.mark.parametrize("kind", ["equal", "rising", "falling", "mixed", "narrow box"])
def test_shortlist_edges(g2s, gpu, W, kind, ranges):
    rng = np.random.default_rng(W + len(kind))
    X, Y, B, K = 40, 37, 130, 64
    N = X * Y
    rows = np.zeros((N, K), np.float32)
    q = np.zeros((B, K), np.float32)
    q[:, 0] = 1.0
    q[:, 1] = 16.0
    p = np.arange(N)
    if kind in ("rising", "falling"):
        o = p if kind == "rising" else p[::-1]
        rows[:, 0], rows[:, 1] = o % 16, o // 16   # at most 92: exact in BF16
    elif kind != "equal":
        rows[:, 0] = rng.integers(0, 4, N)
        q[:, 2] = rng.integers(-2, 3, B)
        rows[:, 2] = rng.integers(0, 3, N)
    box = np.tile(np.array([2, X - 3, 1, Y - 2, 0, 1], np.int32), (B, 1))
    if kind == "narrow box":
        box[:, 0] = rng.integers(0, X, B)
        box[:, 1] = np.minimum(box[:, 0] + rng.integers(0, 3, B), X)
        box[:, 3] = np.minimum(box[:, 2] + rng.integers(0, 4, B), Y)
    seeds = rng.integers(0, 2**32, B, dtype=np.uint32)
    keys, pos = g2s.tc_topk(bf16_bits(q), bf16_bits(rows), 0, X, Y, box, W=W, ranges=ranges, q_seed=seeds)
    score = (q @ rows.T).astype(np.float32)
    ordered = score.view(np.uint32).astype(np.uint64)
    ordered = np.where(score < 0, ~ordered & np.uint64(0xFFFFFFFF), ordered | np.uint64(0x80000000))
    x, y = p % X, p // X
    tiles = (N + 255) // 256
    per = (tiles + ranges - 1) // ranges * 256
    for b in range(B):
        inside = (x >= box[b, 0]) & (x < box[b, 1]) & (y >= box[b, 2]) & (y < box[b, 3])
        full = (ordered[b] << np.uint64(32)) | tie_hash(seeds[b], p)
        for r in range(ranges):
            at = p[inside & (p >= r * per) & (p < (r + 1) * per)]
            best = at[np.argsort(full[at])][-W:]
            want_k = np.concatenate([np.zeros(W - len(best), np.uint64), full[best]])
            want_p = np.concatenate([np.full(W - len(best), 0xFFFFFFFF, np.uint32), best.astype(np.uint32)])
            assert np.array_equal(keys[b, r], want_k), (b, r)
            assert np.array_equal(pos[b, r], want_p), (b, r)


@pytest.mark.parametrize("n,radius,prefix,passes", [(5, 8, 8, 1), (60, 8, 256, 1), (150, 30, 1984, 2)])
def test_level_plan_does_not_move_draws(g2s, gpu, n, radius, prefix, passes):
    """The order of a level's nodes, their K blocks (64 elements in BF16, 128
    in FP8) and the number of passes that plan them leave the draws alone:
    categorical patterns are exact in both formats, and a shortlist no wider
    than the kept candidates per range holds the exact k best."""
    rng = np.random.default_rng(n)
    ncat = 32
    ti = rng.integers(0, ncat, (64, 64)).astype(np.float32)   # wide enough for every pattern
    di = np.full((40, 40), np.nan, np.float32)
    kernel = np.ones((2 * radius + 1,) * 2, np.float32)
    got = {}
    for mode, batch in (("bf16", 0), ("fp8", 0), ("fp8", 128)):
        sim = g2s.Simulation(ti, di, [1], n=n, k=1.2, seed=7, kernel=kernel)
        sim.set_tensor(mode, prefix=prefix, width=32, shortlist=32, audit=1.0, batch=batch)
        sim.run()
        got[mode, batch] = sim.read()[1], sim.info()
        sim.close()
    idx, ref = got["bf16", 0]
    assert ref["tensor_prefix"] == prefix and ref["tensor_nodes"] + ref["plain_nodes"] == 1600
    assert (ref["levels"] * (prefix * ncat // 64 + 1) > 1 << 18) == (passes > 1)
    for out, info in got.values():
        assert np.array_equal(out, idx)
        assert info["regret"] == 0 and info["regret_near"] == 0
        for f in ("levels", "tensor_nodes", "plain_nodes", "audited"):
            assert info[f] == ref[f], f


@pytest.mark.parametrize("shortlist", [33, 48, 64, 128])
@pytest.mark.parametrize("edge,batch", [(60, 0), (260, 128)])
def test_long_shortlist_keeps_the_best(g2s, gpu, edge, batch, shortlist):
    """Shortlists longer than a list's 32 keys, whose lists are bounded by the
    16th best keys of the others: the k best are exact, so the draws are those
    of the short list (categorical patterns are exact in both formats, and
    their many ties are settled by the hash)."""
    rng = np.random.default_rng(edge)
    ti = rng.integers(0, 3, (edge, edge)).astype(np.float32)
    di = np.full((48, 48), np.nan, np.float32)
    got = []
    for mode, s in (("bf16", 32), ("fp8", shortlist)):
        sim = g2s.Simulation(ti, di, [1], n=12, k=2.5, seed=5, kernel=np.ones((21, 21), np.float32))
        sim.set_tensor(mode, prefix=256, width=32, shortlist=s, batch=batch, audit=1.0)
        sim.run()
        got.append((sim.read()[1], sim.info()))
        # all nodes in one step: 18 tiles, the last ones far wider
        sim.run_teacher(ti[:48, :48])
        got[-1] += (sim.read()[2],)
        sim.close()
    assert np.array_equal(got[0][2], got[1][2])
    assert got[0][1]["tensor_nodes"] > 1000 and got[1][1]["tensor_shortlist"] == shortlist
    assert got[1][1]["regret"] == 0 and got[1][1]["regret_near"] == 0
    assert np.array_equal(got[0][0], got[1][0])


@pytest.mark.parametrize("W", [8, 16, 32])
@pytest.mark.parametrize("fmt,share", [(0, 0.03), (0, 0.6), (0, 0.97), (1, 0.6)])
def test_nan_scores_are_no_candidates(g2s, gpu, fmt, share, W):
    """Positions whose score is NaN (a NaN layer value, or an infinite one
    times a zero coefficient) leave the other positions' shortlist alone."""
    rng = np.random.default_rng(int(100 * share) + W)
    X, Y, B, K = 50, 41, 130, 64
    N = X * Y
    rows = rng.integers(-2, 3, (N, K)).astype(np.float32)
    q = rng.integers(-1, 2, (B, K)).astype(np.float32)
    q[:, 0] = 0.0
    bad = rng.random(N) < share
    rows[bad, 0] = np.nan if fmt else np.where(rng.random(bad.sum()) < 0.5, np.nan, np.inf)
    fp8 = {0.0: 0x00, 1.0: 0x38, 2.0: 0x40, -1.0: 0xb8, -2.0: 0xc0}   # E4M3; NaN 0x7f
    bits = bf16_bits if fmt == 0 else np.vectorize(lambda x: fp8.get(float(x), 0x7f), otypes=[np.uint8])
    box = np.tile(np.array([1, X - 2, 0, Y - 1, 0, 1], np.int32), (B, 1))
    seeds = rng.integers(0, 2**32, B, dtype=np.uint32)
    keys, pos = g2s.tc_topk(bits(q), bits(rows), fmt, X, Y, box, W=W, q_seed=seeds)
    rows[bad, 0] = 0.0
    score = (q @ rows.T).astype(np.float32)
    ordered = score.view(np.uint32).astype(np.uint64)
    ordered = np.where(score < 0, ~ordered & np.uint64(0xFFFFFFFF), ordered | np.uint64(0x80000000))
    p = np.arange(N)
    x, y = p % X, p // X
    at = p[~bad & (x >= 1) & (x < X - 2) & (y < Y - 1)]
    for b in range(B):
        full = (ordered[b, at] << np.uint64(32)) | tie_hash(seeds[b], at)
        best = np.argsort(full)[-W:]
        pad = W - len(best)
        assert np.array_equal(keys[b, 0], np.concatenate([np.zeros(pad, np.uint64), full[best]])), b
        assert np.array_equal(pos[b, 0], np.concatenate([np.full(pad, 0xFFFFFFFF), at[best]]).astype(np.uint32)), b


@pytest.mark.parametrize("mode", ["bf16", "fp8"])
@pytest.mark.parametrize("edge,n", [(60, 20), (100, 40)])
def test_infinite_layers_leave_the_draws_repeatable(g2s, gpu, edge, n, mode):
    """Where the training image holds infinities, a node's scores follow from
    the K blocks of its whole tile; the tiles of a level are the same in every
    call, and so are the draws."""
    rng = np.random.default_rng(edge)
    ti = rng.standard_normal((edge, edge)).astype(np.float32)
    ti[5, 7], ti[edge - 9, edge // 2] = np.inf, -np.inf
    done = rng.standard_normal((40, 40)).astype(np.float32)
    sim = g2s.Simulation(ti, np.full((40, 40), np.nan, np.float32), [0], n=n, k=2.5, seed=5)
    sim.set_tensor(mode, audit=0.1)
    nodes = np.arange(50, 1600, dtype=np.int32)
    got = []
    for _ in range(8):
        sim.run_teacher_nodes(done, nodes)
        info = sim.info()
        got.append((sim.read()[2][nodes], [info[f] for f in ("tensor_nodes", "plain_nodes", "audited", "regret")]))
    sim.close()
    assert got[0][1][0] > 1000 and got[0][1][2] > 0
    for cells, counts in got[1:]:
        assert np.array_equal(cells, got[0][0]) and counts == got[0][1]


@pytest.mark.parametrize("k", [1.0, 2.5])
def test_compact_list_beyond_the_staged_keys(g2s, gpu, k):
    """A bounded shortlist's list may hold more keys than the select stages
    (768): patterns 195 columns wide on a 200-column image leave five valid
    columns, too few in any position range for a bound, so nearly all of their
    900 positions reach the list.  The draws are those of the longer shortlist,
    whose lists are not bounded."""
    X, Y, W = 200, 180, 8
    rng = np.random.default_rng(int(2 * k))
    ti = rng.integers(0, 3, (Y, X)).astype(np.float32)
    p = np.arange(X * Y)
    valid = np.bincount(p[(p % X >= 100) & (p % X < 105)] // 256, minlength=(X * Y + 255) // 256)
    assert len(valid) <= 148 and np.minimum(valid, W).sum() > 768   # one tile a range
    di = np.full((30, X), np.nan, np.float32)
    di[:, 2], di[:, 197] = rng.integers(0, 3, (2, 30))
    done = rng.integers(0, 3, di.shape).astype(np.float32)
    done[:, [2, 197]] = di[:, [2, 197]]
    got = []
    for shortlist in (W, 32):
        sim = g2s.Simulation(ti, di, [1], n=50, k=k, seed=3, kernel=np.ones((1, 399), np.float32))
        sim.set_tensor("bf16", prefix=512, width=W, shortlist=shortlist, audit=1.0)
        order, _, begin = sim.path()
        at = np.array([i for i in range(400) if 2 < order[begin + i] % X < 197][:100], np.int32)
        sim.run_teacher_nodes(done, at)
        info = sim.info()
        assert info["tensor_nodes"] == 100 and info["tensor_shortlist"] == shortlist and info["tensor_width"] == W
        assert info["audited"] == 100 and info["regret"] == 0 and info["regret_near"] == 0
        got.append(sim.read()[2][at])
        sim.close()
    assert np.array_equal(got[0], got[1])

"""The workers' pinned staging blocks: pieces of one allocation, lent and given
back in any order, blocks of their own once a batch outgrows a piece, and the
release while some are lent.  Every query's answer stays the one that the
oracle gives for the same pattern."""
import threading

import numpy as np
import pytest

from g2s_b200 import synthetic as syn
from test_gpu_pattern import make_terms, oracle_kbest, random_pattern

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("workers,batch", [(1, 1), (9, 1), (17, 3), (3, 400)])
def test_staging_blocks_lent_and_given_back(g2s, oracle, gpu, workers, batch):
    rng = np.random.default_rng(workers + batch)
    ti = syn.grf((40, 36), (6, 6), seed=2)
    image = g2s.TrainingImage(ti, [0])
    pats, seeds, want = [], [], []
    for q in range(4):
        offs, vals = random_pattern(rng, ti, [0], 10 + 5 * q, 6, 2)
        pats.append((offs, make_terms(offs, vals, [0])))
        seeds.append(np.float32(0.1 + 0.2 * q))
        want.append(oracle_kbest(oracle, ti, [0], offs, vals, 3, float(seeds[-1]))[:2])
    got, errors = {}, []

    def work(i, w):
        try:
            at = [(i + j) % 4 for j in range(batch)]
            got[i] = at, w.pattern_kbest_verbatim([pats[a] for a in at], 3, [seeds[a] for a in at],
                                                  np.full(batch, 0xffffffff, np.uint32))
        except Exception as e:   # noqa: BLE001 - reported by the main thread
            errors.append(e)

    for turn in range(3):
        ws = [g2s.Worker(image) for _ in range(workers)]
        threads = [threading.Thread(target=work, args=(i, w)) for i, w in enumerate(ws)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors
        for w in ws[turn % 2::2]:
            w.close()
        g2s.blocks_release()
        work(0, ws[0] if turn % 2 else g2s.Worker(image))
        for at, (score, index, _) in got.values():
            for j, a in enumerate(at):
                assert np.array_equal(index[j], want[a][1]) and np.array_equal(score[j], want[a][0])
        for w in ws:
            w.close()

"""Page-locked host memory after its workers have gone: bounded, none with a
limit of 0, none after a release; and a worker that comes after a release
answers as before.  The library's allocations are counted by a preloaded
object that forwards them, in a process of its own."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

COUNT = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static size_t held, size_of[4096];
static void *block[4096];
static void *next(const char *name) { return dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), name); }
int cudaHostAlloc(void **p, size_t n, unsigned flags) {
    int (*f)(void **, size_t, unsigned) = (int (*)(void **, size_t, unsigned))next("cudaHostAlloc");
    const int e = f(p, n, flags);
    for (int i = 0; e == 0 && i < 4096; ++i)
        if (!block[i]) { block[i] = *p; size_of[i] = n; held += n; break; }
    return e;
}
int cudaFreeHost(void *p) {
    int (*f)(void *) = (int (*)(void *))next("cudaFreeHost");
    for (int i = 0; i < 4096; ++i)
        if (block[i] && block[i] == p) { block[i] = 0; held -= size_of[i]; break; }
    return f(p);
}
size_t held_bytes(void) { return held; }
"""

USE = r"""
import ctypes, json, sys
import numpy as np
import g2s_b200 as g2s
held = ctypes.CDLL(sys.argv[1]).held_bytes
held.restype = ctypes.c_size_t
rng = np.random.default_rng(0)
image = g2s.TrainingImage(rng.integers(0, 2, (30, 30)).astype(np.float32), [1])
offs = np.array([[0, 0], [1, 0], [-1, 2]], np.int32)
terms = [(1, 0, g2s.QSK_OP_EQ, 1.0, 1.0), (2, 0, g2s.QSK_OP_EQ, 1.0, 0.0)]
def ask(w, batch):
    return w.pattern_kbest_verbatim([(offs, terms)] * batch, 2, np.full(batch, 0.3, np.float32),
                                    np.full(batch, 0xffffffff, np.uint32))
out = {}
for name, limit, batches in (("small", 8 << 30, [1] * 9), ("large", 8 << 30, [40000] * 12), ("none kept", 0, [1, 40000])):
    g2s.blocks_release()
    g2s.blocks_set_limit(limit)
    ws = [g2s.Worker(image) for _ in batches]
    first = [ask(w, b) for w, b in zip(ws, batches)]
    used = held()
    for w in ws:
        w.close()
    kept = held()
    w = g2s.Worker(image)
    g2s.blocks_release()
    lent = held()
    again = ask(w, 1)
    same = all(np.array_equal(f[k][j], again[k][0]) for f in first for k in (0, 1) for j in (0, -1))
    w.close()
    g2s.blocks_release()
    out[name] = [used, kept, lent, held(), bool(same)]
g2s.blocks_set_limit(8 << 30)
print(json.dumps(out))
"""


def test_page_locked_memory_is_bounded_and_given_back(g2s, gpu, tmp_path):
    (tmp_path / "count.c").write_text(COUNT)
    so = str(tmp_path / "count.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", str(tmp_path / "count.c"), "-o", so, "-ldl"], check=True)
    path = os.pathsep.join(x for x in (ROOT, os.environ.get("PYTHONPATH")) if x)
    env = dict(os.environ, LD_PRELOAD=so, PYTHONPATH=path)
    r = subprocess.run([sys.executable, "-c", USE, so], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    out = json.loads(r.stdout.strip().splitlines()[-1])
    slab = 512 << 10
    used, kept, lent, left, same = out["small"]
    assert used == 2 * slab and kept == slab and lent == slab and left == 0 and same
    used, kept, lent, left, same = out["large"]
    assert used > 64 << 20 and slab <= kept <= slab + (64 << 20) and lent == slab and left == 0 and same
    used, kept, lent, left, same = out["none kept"]
    assert used > slab and kept == 0 and lent == slab and left == 0 and same

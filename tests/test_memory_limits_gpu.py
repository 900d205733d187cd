"""Memory that only makes steps faster - the 16-bit storages' table of pull
sources, the words of resident steps - is never the reason for a call to fail.

The engine runs in a child process in which the allocation calls are replaced by
ones that count the pool's live bytes and return cudaErrorMemoryAllocation beyond
a given total, so the limit is met without filling the GPU."""
import json
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <pthread.h>
#include <stdlib.h>
#include <string.h>
typedef void* P;
enum { N = 4096 };
static P ptr[N]; static size_t size[N]; static size_t live, most;
static size_t limit = (size_t)-1;
static pthread_mutex_t mu = PTHREAD_MUTEX_INITIALIZER;
static P real(const char* name) {
    static P lib;
    if (!lib) lib = dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD);
    return dlsym(lib, name);
}
void shim_limit(size_t n) { limit = n; }
size_t shim_live(void) { return live; }
size_t shim_most(void) { size_t m = most; most = live; return m; }
int cudaMallocFromPoolAsync(P* p, size_t n, P pool, P stream) {
    pthread_mutex_lock(&mu);
    const int over = n > limit || live > limit - n;
    pthread_mutex_unlock(&mu);
    if (over) { *p = 0; return 2; }
    const int r = ((int (*)(P*, size_t, P, P))real("cudaMallocFromPoolAsync"))(p, n, pool, stream);
    pthread_mutex_lock(&mu);
    for (int i = 0; r == 0 && i < N; ++i)
        if (!ptr[i]) { ptr[i] = *p; size[i] = n; live += n; if (live > most) most = live; break; }
    pthread_mutex_unlock(&mu);
    return r;
}
int cudaMalloc(P* p, size_t n) {
    pthread_mutex_lock(&mu);
    const int over = n > limit || live > limit - n;
    pthread_mutex_unlock(&mu);
    if (over) { *p = 0; return 2; }
    return ((int (*)(P*, size_t))real("cudaMalloc"))(p, n);
}
int cudaFreeAsync(P p, P stream) {
    pthread_mutex_lock(&mu);
    for (int i = 0; i < N; ++i) if (p && ptr[i] == p) { ptr[i] = 0; live -= size[i]; break; }
    pthread_mutex_unlock(&mu);
    return ((int (*)(P, P))real("cudaFreeAsync"))(p, stream);
}
"""

CHILD = r"""
import ctypes, json, sys
import numpy as np
from lbflow_b200 import Engine
shim = ctypes.CDLL(sys.argv[1])
for f in (shim.shim_live, shim.shim_most): f.restype = ctypes.c_size_t
shim.shim_limit.argtypes = [ctypes.c_size_t]
storage, what = sys.argv[2], sys.argv[3]
g = np.where(np.random.default_rng(1).random((40, 56, 64)) < 0.95, 75, 255).astype(np.uint8)
if what == 'words': g = g[:16]
LABELS = {75: ('GV', 1e-5, 1, 0), 255: ('SD', 90.0, 0, 0)}

def run(limit_create, limit_after, read):
    # fields and dense populations after single steps and one call of several
    shim.shim_limit(limit_create); shim.shim_most()
    with Engine(g, LABELS, tau=(0.9,), storage=storage) as e:
        made = e.device_bytes, shim.shim_most()
        shim.shim_limit(limit_after)
        e.initialize()
        for _ in range(3): e.step(1)
        e.step(5, macros=True)
        e.check()
        rho, _, u = e.macros()
        pops = e.populations() if read else np.zeros(1)
        for _ in range(2): e.step(1)
        e.step(4, macros=True)
        e.check()
        return (rho, u, pops) + e.macros()[::2], made, e.device_bytes, e.fluid_nodes

free = (1 << 62)
want, (base, peak), after, nodes = run(free, free, True)
table = 20 * nodes if storage in ('fp16', 'bf16', 'bfp16') else 0
words = 576 * nodes if storage == 'fp64' else 288 * nodes
if what == 'create':                 # the state and the set-up scratch, but no table
    got, made, _, _ = run(peak - table // 2, free, True)
    assert made[0] <= base - table, (made, base, table)
elif what == 'table':                # the table, but then not the dense populations beside it
    got, made, end, _ = run(free, base + 19 * 8 * nodes - table // 2, True)
    assert made[0] == base and end <= base - table
elif what == 'words':                # no room for the resident steps' words
    got, made, end, _ = run(free, base + words // 2, False)
    want = want[:2] + (got[2],) + want[3:]
    assert end <= base + words // 2 and after > base + words // 2
else:                                # the words, but then not what is allocated later
    got, made, end, _ = run(free, base + words + 19 * 8 * nodes // 2, True)
for a, b in zip(want, got): assert np.array_equal(a, b)
print(json.dumps('ok'))
"""


@pytest.fixture(scope='module')
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp('shim')
    (d / 'shim.c').write_text(SHIM)
    subprocess.run(['gcc', '-shared', '-fPIC', '-O1', '-o', str(d / 'shim.so'), str(d / 'shim.c'), '-ldl', '-lpthread'],
                   check=True)
    return d / 'shim.so'


@pytest.mark.parametrize('storage, what', [
    ('fp16', 'create'), ('bf16', 'create'), ('bfp16', 'create'), ('fp16', 'table'), ('bfp16', 'table'),
    ('fp64', 'words'), ('fp16', 'words'), ('fp16', 'later'),
])
def test_limit(shim, storage, what):
    import os
    r = subprocess.run([sys.executable, '-c', CHILD, str(shim), storage, what], capture_output=True, text=True,
                       env=dict(os.environ, LD_PRELOAD=str(shim)), timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert json.loads(r.stdout.strip().splitlines()[-1]) == 'ok'

"""The options of an integral on the synthetic integrands (GPU), which every build holds: a run stopped after its checkpoint
and resumed equals an unbroken one, with and without the predictor; the predictor only leaves points out; SINCQED_GROWSKIP
at top = 0 changes which points have |.| sums and nothing else; a thread that finds no memory for full batches gives the
same level."""
import json
import math
import subprocess
import sys

import pytest

from sincfeyn_b200 import sq

pytestmark = pytest.mark.gpu
EXACT = ('S', 'Ah', 'ref', 'prune', 'trunc', 'unres', 'nev', 'nq', 'kept_top', 'es1', 'es2', 'abskipped', 'pskip')


def same(a, b):
    return a == b or (a != a and b != b)


def equal(a, b, fields=EXACT):
    for f in fields:
        assert all(map(same, a[f], b[f])) if isinstance(a[f], list) else same(a[f], b[f]), (f, a[f], b[f])


@pytest.mark.parametrize('kw', [{}, {'fma': 0}, {'predict': 0.3}, {'predict': 0.3, 'sym': '1,0,2,3,4'}])
@pytest.mark.parametrize('top', [2, 3])
def test_stop_and_resume(tmp_path, top, kw):
    run = ('syn_d5', 0.9, 69, 1e-9, top)
    full = sq.hsum(*run, **kw)
    assert sq.hsum(*run, ckpt_every=600, ckpt_dir=str(tmp_path), ckpt_stop=1, **kw) is None
    equal(sq.hsum(*run, ckpt_every=600, ckpt_dir=str(tmp_path), **kw), full)


@pytest.mark.parametrize('graph,h,eps', [('syn_d5', 1.1, 1e-8), ('syn_d8', 1.4, 1e-8)])
def test_the_predictor_only_leaves_points_out(graph, h, eps):
    run = (graph, h, 2*math.ceil(30/h) + 1, eps)
    r, u = sq.hsum(*run, fma=0, predict=0.5), sq.hsum(*run, fma=0)
    assert r['pskip'] > 0 and u['nev'] == r['nev'] + r['pskip']
    equal(r, u, ('ref', 'kept_top', 'trunc'))


def test_growskip_changes_the_skipped_points_alone():
    rs = [sq.hsum('syn_d5', 1.5, 41, 1e-6, 0, growskip=g) for g in (0, 1, 2, 5)]
    for r in rs[1:]:
        equal(r, rs[0], ('S', 'ref', 'prune', 'trunc', 'nev'))
        assert r['nq'] <= rs[0]['nq']


CHILD = r'''
import ctypes as C, json, math, sys
sys.path.insert(0, 'tests')
import numpy as np, torch
from test_gpu_axis_paths import Acc, Level, PointTestParams, library, nodes
L, d, K, h = library(), 8, 32, 1.0
L.sqb_find_graph.restype = C.c_void_p
L.sqb_dev_axis.argtypes = [C.c_void_p, C.c_int]
g = L.sqb_find_graph(b'syn_d8')
x = [math.exp(i*h) for i in range(-K, K + 1)]
X, W = (C.c_double*(2*K + 1))(*x), (C.c_double*(2*K + 1))(*[v*h for v in x])
assert L.sqb_dev_init(0) == 0 and L.sqb_dev_tables(X, W, K) == 0 and L.sqb_dev_axis(g, 1) == 0
n = (1 << 25 >> d) + 1000
p = np.zeros((n, 12), dtype=np.int8)
p[:, :d] = nodes(d, K, n, 2, 1)
cells = torch.from_numpy(p).cuda()
free = torch.cuda.mem_get_info()[0]
held = torch.empty(free - (1800 << 20), dtype=torch.uint8, device='cuda') if sys.argv[1] == '1' else None
lv = Level(g=g, cells=cells.data_ptr(), ncell=n, st=1, last=1, pw=1.0, thr=0.0, t=PointTestParams(1e-15, 1e-3, 1.0, 1, 0, 1, 0, 1, 0))
torch.cuda.synchronize()
acc, nn, ms = Acc(), C.c_long(), C.c_double()
rc = L.sqb_dev_level(C.byref(lv), C.byref(acc), C.byref(nn), C.byref(ms))
print(json.dumps([rc, torch.cuda.mem_get_info()[0] >> 20, sum(acc.S), sum(acc.A), sum(acc.u), acc.ne, acc.nq, acc.skipped, acc.overflow]))
'''


def test_a_level_short_of_memory(root):
    # 1.8 GB left: the full batch's 2.35 GB are refused, the lower size's 1.17 GB are not
    out = []
    for short in '01':
        r = subprocess.run([sys.executable, '-c', CHILD, short], cwd=root, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr
        out.append(json.loads(r.stdout))
    assert out[0][0] == 0 and out[1][0] == 0 and 0 < out[1][1] < 1800 - 1100
    assert out[0][2:] == out[1][2:]

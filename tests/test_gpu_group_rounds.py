"""A level of several integrals whose batches do not all fit one launch (GPU): five of more than a full batch of children
each and a small one.  They share launches of as many whole batches as fit, and each integral's sums, counters and kept
cells are those of its level alone, bit for bit."""
import ctypes as C
import math

import numpy as np
import pytest

from sincfeyn_b200 import sq

from test_gpu_axis_paths import Acc, Level, PointTestParams, library, nodes

pytestmark = pytest.mark.gpu
GRAPH, D, H, K = 'syn_d8', 8, 1.0, 32
BATCH, LAUNCH = 1 << 26, 1 << 28


@pytest.mark.parametrize('last', [1, 0])
def test_full_batches_share_launches(last):
    import torch
    L = library()
    L.sqb_find_graph.restype = C.c_void_p
    L.sqb_dev_axis.argtypes = [C.c_void_p, C.c_int]
    L.sqb_dev_axis_words.argtypes, L.sqb_dev_axis_words.restype = [C.c_void_p, C.c_int], C.c_long
    L.sqb_dev_axis_fill.argtypes = [C.c_void_p, C.c_int, C.c_void_p, C.c_int, C.c_void_p]
    L.sqb_launch_count.restype = C.c_ulonglong
    assert L.sqb_dev_init(0) == 0
    g = L.sqb_find_graph(GRAPH.encode())
    nt = 2*K + 1
    x = [math.exp(i*H) for i in range(-K, K + 1)]
    X, W = (C.c_double*nt)(*x), (C.c_double*nt)(*[v*H for v in x])
    assert L.sqb_dev_tables(X, W, K) == 0 and L.sqb_dev_axis(g, 1) == 0
    tab = torch.zeros(2*nt + L.sqb_dev_axis_words(g, K), dtype=torch.float64, device='cuda')
    tab[:2*nt] = torch.tensor(x + [v*H for v in x], dtype=torch.float64)
    torch.cuda.synchronize()
    assert L.sqb_dev_axis_fill(g, 1, tab.data_ptr(), K, tab.data_ptr() + 16*nt) == 0
    cells, nxt, lv = [], [], []
    for q, n in enumerate([290000, 270000, 1000, 280000, 300000, 263000]):
        rng = np.random.default_rng(q)
        p = np.zeros((n, 12), dtype=np.int8)
        p[:, :D], p[:, 11] = nodes(D, K, n, 2, q), (rng.random(n) < 0.5) + 2*rng.integers(0, 3, n)
        cells.append(torch.from_numpy(p).cuda())
        nxt.append(torch.zeros((0 if last else 1 << 24, 12), dtype=torch.int8, device='cuda'))
        lv.append(Level(g=g, cells=cells[-1].data_ptr(), ncell=n, next=None if last else nxt[-1].data_ptr(), next_cap=len(nxt[-1]), st=1, last=last,
                        pw=1.0, thr=1e-2, t=PointTestParams(1e-15, 1e-3, 1.0, 1, 0, 1, 0, 1, 0), X=tab.data_ptr(), Wt=tab.data_ptr() + 8*nt, K=K))
    torch.cuda.synchronize()
    n = len(lv)
    many = [v.ncell << D > BATCH for v in lv]
    assert sum(many) == 5 and 5*BATCH > LAUNCH

    def collect(accs, nn):
        torch.cuda.synchronize()
        return [(list(a.S), list(a.A), list(a.drop), list(a.b1), list(a.b2), list(a.u), a.ne, a.keep, a.nq, a.unres, a.skipped, a.overflow, k)
                for a, k in zip(accs, nn)], [t[:k].cpu().numpy() for t, k in zip(nxt, nn)]
    accs, nn, ms = (Acc*n)(), (C.c_long*n)(), C.c_double()
    c0 = L.sqb_launch_count()
    for q in range(n):
        assert L.sqb_dev_level(C.byref(lv[q]), C.byref(accs[q]), C.byref(nn, 8*q), C.byref(ms)) == 0
    alone, kept = collect(accs, nn)
    c1 = L.sqb_launch_count()
    for t in nxt:
        t.zero_()
    torch.cuda.synchronize()
    accs = (Acc*n)()
    assert L.sqb_dev_level_multi((Level*n)(*lv), n, accs, nn, C.byref(ms)) == 0
    group, kept1 = collect(accs, nn)
    c2 = L.sqb_launch_count()
    assert group == alone and all(np.array_equal(a, b) for a, b in zip(kept, kept1))
    assert all(a[11] == 0 and (last or a[12] > 0) for a in alone)
    # alone: a batch of the small one, two of each of the others; together: two launches for the first round, one for the second
    assert 11*(c2 - c1) == 3*(c1 - c0), (c1 - c0, c2 - c1)

"""The values that the axis form's level kernel writes (GPU), bit for bit: in a level whose step reaches below the box along
all axes but one, a cell has two children, and the double-double sum of two values is exact, so that the level's sum
tells both.  Against the point function at the same nodes (sq.eval_points), as written and contracted, along every axis,
first, middle and last."""
import ctypes as C
import math
from fractions import Fraction

import numpy as np
import pytest

from sincfeyn_b200 import sq

from test_gpu_axis_paths import Acc, Level, PointTestParams, library

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('last', [1, 0])
@pytest.mark.parametrize('fma', [0, 1])
@pytest.mark.parametrize('graph', ['syn_d5', 'syn_d8', 'syn_d11'])
def test_two_children_sum_to_the_point_functions_values(graph, fma, last):
    import torch
    L, d, K, h = library(), int(graph[5:]), 20, 0.3
    L.sqb_find_graph.restype = C.c_void_p
    L.sqb_dev_axis.argtypes = [C.c_void_p, C.c_int]
    g = L.sqb_find_graph(graph.encode())
    x = np.array([math.exp(i*h) for i in range(-K, K + 1)])
    w = x*h
    X, W = (C.c_double*(2*K + 1))(*x), (C.c_double*(2*K + 1))(*w)
    assert L.sqb_dev_init(0) == 0 and L.sqb_dev_tables(X, W, K) == 0 and L.sqb_dev_axis(g, fma) == 0
    rng = np.random.default_rng(d)
    st, per = K, 8
    # one axis with k >= st - K, so that its lower child is in the box; the others below
    k = rng.integers(-K, st - K, size=(d, per, d))
    for a in range(d):
        k[a, :, a] = rng.integers(st - K, K + 1, size=per)
    k = k.reshape(-1, d)
    low = k.copy()
    low[np.arange(len(k)), np.repeat(np.arange(d), per)] -= st
    v = []
    for n in (k, low):
        f, _ = sq.eval_points(graph, x[n + K], 2 if fma else 0, 0)
        p = np.ones(len(n))
        for i in range(d):
            p = p*w[n[:, i] + K]
        v.append(f*p)
    pts = np.zeros((len(k), 12), dtype=np.int8)
    pts[:, :d], pts[:, 11] = k, 1                  # no |.| sums: the value as it is
    cells = torch.from_numpy(pts).cuda()
    nxt = torch.zeros((4, 12), dtype=torch.int8, device='cuda')
    torch.cuda.synchronize()
    for i in range(len(k)):
        lv = Level(g=g, cells=cells.data_ptr() + 12*i, ncell=1, next=None if last else nxt.data_ptr(), next_cap=4, st=st, last=last, pw=1.0, thr=1e300,
                   t=PointTestParams(1e300, 1e-3, 1.0, 1, 0, 1, 0, fma, 0), max_children=0)
        acc, nn, ms = Acc(), C.c_long(), C.c_double()
        assert L.sqb_dev_level(C.byref(lv), C.byref(acc), C.byref(nn), C.byref(ms)) == 0 and acc.ne == 2
        assert sum(map(Fraction, acc.S)) == Fraction(v[0][i]) + Fraction(v[1][i]), (i, list(acc.S), v[0][i], v[1][i])

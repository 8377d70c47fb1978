"""A level's sums by batches of two sizes (GPU), the full one and the lower one that a thread short of memory takes, where
the smaller batches leave a short last one: the same counters, and the same sums to the rounding of the few double-double
additions that join the batches (2^-104 each, under 32 of them)."""
import ctypes as C
import math

import numpy as np
import pytest

from sincfeyn_b200 import sq

from test_gpu_axis_paths import Acc, Level, PointTestParams, library, nodes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('last', [1, 0])
@pytest.mark.parametrize('graph,axis', [('syn_d8', 1), ('syn_d8', 0), ('syn_d11', 1)])
def test_sums_do_not_depend_on_the_batches(graph, axis, last):
    import torch
    L, d, K, h = library(), int(graph[5:]), 32, 1.0
    L.sqb_find_graph.restype = C.c_void_p
    L.sqb_dev_axis.argtypes = [C.c_void_p, C.c_int]
    g = L.sqb_find_graph(graph.encode())
    X = (C.c_double*(2*K + 1))(*[math.exp(i*h) for i in range(-K, K + 1)])
    W = (C.c_double*(2*K + 1))(*[x*h for x in X])
    assert L.sqb_dev_init(0) == 0 and L.sqb_dev_tables(X, W, K) == 0 and (not axis or L.sqb_dev_axis(g, 1) == 0)
    n = (1 << 25 >> d) + 1000                     # a second batch of 1000 cells or a little more with the lower size
    rng = np.random.default_rng(d)
    p = np.zeros((n, 12), dtype=np.int8)
    p[:, :d], p[:, 11] = nodes(d, K, n, 2, d), (rng.random(n) < 0.5) + 2*rng.integers(0, 3, n)
    cells = torch.from_numpy(p).cuda()
    nxt = torch.zeros((1 << 24, 12), dtype=torch.int8, device='cuda')
    torch.cuda.synchronize()
    got = []
    for size in (1 << 26, 1 << 25):
        lv = Level(g=g, cells=cells.data_ptr(), ncell=n, next=None if last else nxt.data_ptr(), next_cap=len(nxt), st=1, last=last, pw=1.0, thr=1e-2,
                   t=PointTestParams(1e-15, 1e-3, 1.0, 1, 0, 1, 0, 1, 0), max_children=size)
        acc, nn, ms = Acc(), C.c_long(), C.c_double()
        assert L.sqb_dev_level(C.byref(lv), C.byref(acc), C.byref(nn), C.byref(ms)) == 0 and acc.overflow == 0
        got.append(([np.array(x) for x in (acc.S, acc.A, acc.drop, acc.b1, acc.b2, acc.u)], (acc.ne, acc.keep, acc.nq, acc.unres, acc.skipped, nn.value)))
    (s, c), (s1, c1) = got
    assert c == c1
    for x, y in zip(s, s1):
        assert abs((x - y)[0] + (x - y)[1]) <= 32*2.0**-104*s[1][0], (x, y)

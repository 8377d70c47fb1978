"""The sizes at which a call of an integrand with an axis form changes its route (GPU), against the same work by the other
route:

  * a raw launch of the plug-in of 2^17 points or more fills an axis table per CTA; the same cells or nodes in launches
    below that take the general kernel: equal bits;
  * a level batch takes the axis form's kernels when its lattice has their tables, with the fallback points in place up to
    2^18 children and queued beyond: against the general kernels (no tables), equal counters and kept cells, and the
    sums;
  * the last level and an inner one, one integral and several, are separate kernels: a group and a batch equal their
    integrals alone;
  * pointwise values pass through two staging buffers of 512 KB in turn: equal bits to calls of a few points;
  * the dilation orders its cells by a bitmap while the grid has at most 2^29 nodes, else by a sort: the same integral
    on a grid either side of that, with a support well inside both."""
import ctypes as C
import math

import numpy as np
import pytest

from sincfeyn_b200 import sq

pytestmark = pytest.mark.gpu
EPS = 2.0**-52
FIELDS = ('S', 'Ah', 'ref', 'prune', 'trunc', 'unres', 'nev', 'nq', 'kept_top', 'abskipped', 'unresdrop', 'es1', 'es2')


def library():
    L = sq.lib()
    p = C.c_void_p
    L.sqb_level_noalloc.argtypes = [C.c_char_p, C.c_double, C.c_int, p, C.c_long, C.c_int, C.c_int] + [C.c_double]*5 + \
        [C.c_int]*3 + [p, C.c_long, p, p, p]
    L.sqb_plugin_launch.argtypes = [C.c_char_p, C.c_int, p, C.c_long, p, p, p, C.c_int, C.c_double, p, p, C.c_int, C.c_int]
    return L


def nodes(d, K, n, step, seed):
    """nodes about the origin, some at the lattice's edges"""
    g = np.random.default_rng(seed)
    k = step*np.rint(g.laplace(0, 6/d**0.5, size=(n, d))/step).astype(np.int64)
    edge = g.random((n, d)) < 0.01
    k[edge] = K*g.choice([-1, 1], edge.sum())
    return np.clip(k, -K, K)


def launch(graph, form, k, skip, K, h, cells, d, st):
    import torch
    n = len(k) << d if cells else len(k)
    pts, sk = torch.from_numpy(k.astype(np.int16)).cuda(), torch.from_numpy(skip.astype(np.uint8)).cuda()
    X = torch.from_numpy(np.exp(np.arange(-K, K + 1)*h)).cuda()
    out = torch.full((2, n), -7.0, dtype=torch.float64, device='cuda')
    torch.cuda.synchronize()
    rc = library().sqb_plugin_launch(graph.encode(), form, torch.cuda.current_stream().cuda_stream, n, pts.data_ptr(), sk.data_ptr(),
                                     X.data_ptr(), K, h, out[0].data_ptr(), out[1].data_ptr(), cells, st)
    assert rc == 0, sq.lib().sqb_error()
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize('cells,st', [(0, 1), (1, 1), (1, 2)])
@pytest.mark.parametrize('form', [0, 2])
@pytest.mark.parametrize('graph', ['syn_d5', 'syn_d8', 'syn_d11'])
def test_raw_launch_is_the_same_either_side_of_the_table(graph, form, cells, st):
    d, K, h = int(graph[5:]), 44, 0.7
    edge = 1 << 17 - (d if cells else 0)
    for n in (edge - 1, edge, edge + 3):
        k = nodes(d, K, n, 2 if cells else 1, n)
        skip = np.random.default_rng(n + 1).random(n) < 0.3
        whole = launch(graph, form, k, skip, K, h, cells, d, st)
        step = max(1, edge//3)
        parts = [launch(graph, form, k[i:i + step], skip[i:i + step], K, h, cells, d, st) for i in range(0, n, step)]
        assert np.array_equal(whole.view(np.int64), np.concatenate(parts, axis=1).view(np.int64)), n


class PointTestParams(C.Structure):
    _fields_ = [('abserr', C.c_double), ('nearf', C.c_double), ('ddslack', C.c_double),
                ('abskip', C.c_int), ('abcheck', C.c_int), ('dropunres', C.c_int), ('alldd', C.c_int),
                ('fma', C.c_int), ('split', C.c_int)]


class Level(C.Structure):
    """sqb_level_t (sqb_rt.h), every field: no fold, no predictor"""
    _fields_ = [('g', C.c_void_p), ('cells', C.c_void_p), ('ncell', C.c_long), ('next', C.c_void_p),
                ('next_cap', C.c_long), ('st', C.c_int), ('last', C.c_int), ('pw', C.c_double), ('thr', C.c_double),
                ('t', PointTestParams), ('max_children', C.c_long), ('sym', C.c_void_p), ('vt', C.c_void_p),
                ('vput', C.c_int), ('predict', C.c_double), ('esok', C.c_int), ('X', C.c_void_p), ('Wt', C.c_void_p),
                ('K', C.c_int)]


class Acc(C.Structure):
    """sqb_acc_t (sqb_rt.h), every field"""
    _fields_ = [('S', C.c_double * 2), ('A', C.c_double * 2), ('drop', C.c_double * 2), ('b1', C.c_double * 2),
                ('b2', C.c_double * 2), ('u', C.c_double * 2), ('ne', C.c_ulonglong), ('keep', C.c_ulonglong),
                ('nq', C.c_ulonglong), ('unres', C.c_ulonglong), ('skipped', C.c_ulonglong), ('overflow', C.c_ulonglong),
                ('pskip', C.c_ulonglong)]


ABSERR, NEARF, DDSLACK = 1e-15, 1e-3, 1.0


def level(route, graph, k, flags, K, h, last, thr, alldd=0):
    """one batch by the general kernels, by the axis form's, or in the caller's memory; the cells 4 bytes past an
    8-byte boundary"""
    import torch
    L, (n, d) = library(), k.shape
    pts = np.zeros((n, 12), dtype=np.int8)
    pts[:, :d], pts[:, 11] = k, flags
    dev = torch.from_numpy(np.concatenate([np.zeros(4, np.int8), pts.reshape(-1)])).cuda()
    nxt = torch.zeros((n << d, 12), dtype=torch.int8, device='cuda')
    torch.cuda.synchronize()
    at, to = dev.data_ptr() + 4, None if last else nxt.data_ptr()
    if route == 'noalloc':
        s, c = (C.c_double*12)(), (C.c_longlong*6)()
        rc = L.sqb_level_noalloc(graph.encode(), h, K, at, n, 1, int(last), 1.0, thr, ABSERR, NEARF, DDSLACK, 1, 0, 1, to, n << d, s, c,
                                 torch.cuda.current_stream().cuda_stream)
        s, c = np.array(s), list(c)
    else:
        L.sqb_find_graph.restype = C.c_void_p
        L.sqb_dev_axis.argtypes = [C.c_void_p, C.c_int]
        g = L.sqb_find_graph(graph.encode())
        X = (C.c_double*(2*K + 1))(*[math.exp(i*h) for i in range(-K, K + 1)])
        W = (C.c_double*(2*K + 1))(*[x*h for x in X])
        assert L.sqb_dev_init(0) == 0 and L.sqb_dev_tables(X, W, K) == 0
        assert route == 'general' or L.sqb_dev_axis(g, 1) == 0
        lv = Level(g=g, cells=at, ncell=n, next=to, next_cap=n << d, st=1, last=int(last), pw=1.0, thr=thr,
                   t=PointTestParams(ABSERR, NEARF, DDSLACK, 1, 0, 1, alldd, 1, 0), max_children=0)
        acc, nn, ms = Acc(), C.c_long(), C.c_double()
        rc = L.sqb_dev_level(C.byref(lv), C.byref(acc), C.byref(nn), C.byref(ms))
        s = np.array([x for f in ('S', 'A', 'drop', 'b1', 'b2', 'u') for x in getattr(acc, f)])
        c = [acc.ne, acc.keep, acc.nq, acc.unres, acc.skipped, acc.overflow]
    assert rc == 0, L.sqb_error()
    torch.cuda.synchronize()
    return s, c, nxt[:0 if last else c[1]].cpu().numpy()


@pytest.mark.parametrize('last', [False, True])
@pytest.mark.parametrize('graph', ['syn_d5', 'syn_d8', 'syn_d11'])
def test_level_batch_equals_the_general_kernels(graph, last):
    d, K, h = int(graph[5:]), 32, 1.0
    g = np.random.default_rng(d)
    # the last: tiles summed by the FP64 pass, their fallback points added by a warp per tile
    for n in (1, 2, 37, 1 << 18 - d, (1 << 18 - d) + 1, (1 << 20 - d) - 3, ((13 << 20) >> d) + 3):
        k = nodes(d, K, n, 2, n)
        flags = (g.random(n) < 0.5) + 2*g.integers(0, 3, n)
        for alldd in (0, 1) if n < 1000 else (0,):
            s, c, nxt = level('general', graph, k, flags, K, h, last, 1e-9, alldd)
            assert c[0] > 0 and (n < 1000 or c[2] > 0)
            for route in ('axis', 'noalloc') if n << d <= 1 << 18 and not alldd else ('axis',):
                s1, c1, nxt1 = level(route, graph, k, flags, K, h, last, 1e-9, alldd)
                assert c1 == c and np.array_equal(nxt1, nxt), (n, route, alldd)
                # equal values; a thread's plain sums of |v| and of the dropped weight have 64 additions or fewer
                assert np.all(np.abs((s1 - s)[0::2] + (s1 - s)[1::2]) <= 64*EPS*s[2]), (n, route, alldd)


@pytest.mark.parametrize('graph', ['syn_d5', 'syn_d8', 'syn_d11'])
def test_level_batch_beyond_the_window_of_shared_reciprocals(graph):
    # |z| to 300: table entries to 2^700, quotients and products of variables beyond 2^+-450, to zero and infinity
    d, K, h, n = int(graph[5:]), 120, 2.5, 300
    g = np.random.default_rng(d)
    k = np.where(g.random((n, d)) < 0.4, K*g.choice([-1, 1], (n, d)), nodes(d, K, n, 2, d))
    k[::3] = 2*g.integers(-K//2, K//2 + 1, k[::3].shape)
    flags = g.random(n) < 0.5
    for last in (False, True):
        s, c, nxt = level('general', graph, k, flags, K, h, last, 1e-30)
        s1, c1, nxt1 = level('axis', graph, k, flags, K, h, last, 1e-30)
        assert c1 == c and np.array_equal(nxt1, nxt) and np.all(np.isfinite(s))
        assert np.all(np.abs((s1 - s)[0::2] + (s1 - s)[1::2]) <= 64*EPS*s[2])


def same(a, b):
    return all(x == y or (x != x and y != y) for x, y in zip(np.ravel(a), np.ravel(b)))


@pytest.mark.parametrize('graph,kw', [('syn_d5', {}), ('syn_d5', {'fma': 0}), ('syn_d8', {})])
def test_group_and_batch_are_each_integral_alone(graph, kw):
    jobs = [(graph, h, 2*math.ceil(30/h - 1e-9) + 1, 1e-9) for h in (1.6, 1.3, 1.1, 1.0)]
    alone = [sq.hsum(*j, **kw) for j in jobs]
    group = sq.hsum_group(jobs, **kw)
    batch = sq.hsum_batch([j + (-1, 1.0) for j in jobs], workers=3, **kw)[0]
    for j, a, b, c in zip(jobs, alone, group, batch):
        for f in FIELDS:
            assert same(a[f], b[f]) and same(a[f], c[f]), (j, f, a[f], b[f], c[f])


@pytest.mark.parametrize('ab', [0, 1])
@pytest.mark.parametrize('prec', [0, 1, 2])
def test_pointwise_values_do_not_depend_on_the_staging(prec, ab):
    # 40 bytes a point in, 32 (prec 1) or 16 out: one piece each way, several, and the sizes about each edge
    sf = np.exp(np.random.default_rng(5).uniform(-12, 12, size=(60001, 5)))
    want = [np.concatenate(x) for x in zip(*[sq.eval_points('syn_d5', sf[i:i + 1000], prec, ab) for i in range(0, len(sf), 1000)])]
    for n in (1, 13107, 13108, 16384, 16385, 26214, 26215, 32768, 32769, 60001):
        for got, w in zip(sq.eval_points('syn_d5', sf[:n], prec, ab), want):
            assert np.array_equal(got.view(np.int64), w[:n].view(np.int64)), n


@pytest.mark.parametrize('graph,h,eps,top,N', [('syn_d5', 0.5, 1e-9, 1, (105, 113)), ('syn_d8', 1.0, 1e-7, 3, (65, 97))])
def test_dilation_by_bitmap_and_by_sort(graph, h, eps, top, N):
    # 53^5 and 57^5 nodes, 9^8 and 13^8, about 2^29; at the smaller grid's edge the integrand is 1e-11 and 1e-9 of its peak
    a, b = (sq.hsum(graph, h, n, eps, top=top) for n in N)
    for f in FIELDS:
        assert f == 'trunc' or same(a[f], b[f]), (f, a[f], b[f])

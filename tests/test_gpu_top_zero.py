"""A sum whose top level is the lattice itself (top = 0, GPU) against a replay of its grow on the host: the pruning
column is |sum f w| over the points that a frontier leaves out (driver/sumkey.h:225-245), and not over those that only
the final threshold removes, whose weight goes to the dropped |f w| alone (driver/sumkey.h:399-401).  Runs whose
frontiers stand at the sizes where the grow changes its route: 4096 points are the most that one cluster takes, in
chains that a larger frontier ends."""
import math

import numpy as np
import pytest

from sincfeyn_b200 import sq

pytestmark = pytest.mark.gpu


def replay(graph, h, N, eps):
    """(the frontiers' sizes, the running sum of |f w|, all values, the frontiers' dropped ones, kept ones below the final
    threshold), f w as the FP64 kernel rounds it"""
    D, K = int(graph[5:]), (N - 1)//2
    K += K % 2                                    # driver/lattice.c:16
    X = np.array([math.exp(k*h) for k in range(-K, K + 1)])
    P = (2*K + 1)**np.arange(D - 1, -1, -1)
    step = np.repeat(np.eye(D, dtype=np.int64), 2, axis=0)*np.tile([-1, 1], D)[:, None]
    front, seen, a = np.zeros((1, D), dtype=np.int64), np.zeros(1, dtype=np.int64), 0.0
    sizes, every, out, kept = [], [], [], []
    while len(front):
        f, _ = sq.eval_points(graph, X[front + K], 0, 1)
        w = np.ones(len(front))
        for d in range(D):
            w = w*(X*h)[front[:, d] + K]
        v = np.where(np.isfinite(f*w), f*w, 0.0)
        a = np.add.accumulate(np.concatenate([[a], np.abs(v)]))[-1]
        keep = np.abs(v) >= eps*1e-3*a
        sizes.append(len(v))
        every.append(v)
        out.append(v[~keep])
        kept.append(np.abs(v[keep]))
        c = (front[keep][:, None, :] + step[None]).reshape(-1, D)      # (kept point, axis, sign)
        c = c[(np.abs(c) <= K).all(1)]
        key, first = np.unique(c @ P, return_index=True)
        first = np.sort(first[~np.isin(key, seen)])
        front, seen = c[first], np.union1d(seen, key)
    kept = np.concatenate(kept)
    return sizes, a, np.concatenate(every), np.concatenate(out), kept[kept < eps*1e-3*a]


@pytest.mark.parametrize('graph,h,N,eps', [('syn_d5', 1.5, 41, 1e-6), ('syn_d5', 1.5, 41, 1e-2), ('syn_d5', 2.0, 31, 1e-4)])
def test_prune_is_the_frontiers_signed_sum(graph, h, N, eps):
    sizes, _, _, out, late = replay(graph, h, N, eps)
    assert len(out) and (len(late) or eps != 1e-6)
    r = sq.hsum(graph, h, N, eps, 0, fma=0, abserr0=1e300)
    assert r['nev'] == sum(sizes)
    # a double-double sum, rounded once: an ulp of the exact one each way
    want = abs(math.fsum(out))
    assert abs(r['prune'] - want) <= 2*np.spacing(want), (r['prune'], want, len(late), late.sum())


@pytest.mark.parametrize('h,N,eps,size', [(1.706, 37, 1.935e-6, 4095), (1.765, 35, 1.08e-6, 4096), (1.76, 37, 1.133e-6, 4097)])
def test_frontiers_at_the_size_of_one_cluster(h, N, eps, size):
    sizes, a, every, _, _ = replay('syn_d5', h, N, eps)
    assert size in sizes and max(sizes) > 4097
    r = sq.hsum('syn_d5', h, N, eps, 0, fma=0, abserr0=1e300)
    assert r['nev'] == sum(sizes) and r['ref'] == a
    want = math.fsum(every)
    assert abs(r['S'][0] - want) <= 2*np.spacing(want)

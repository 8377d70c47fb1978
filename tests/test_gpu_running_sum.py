"""The grow's running sum (GPU): the parallel replay of a + |v0| w + |v1| w + ..., every addition rounded, against
the sequential sum on the host (numpy's accumulate), bit for bit, by both of its routes: at the edges of their
chunks and tiles, over binade changes, ties to even, zeros, tiny, huge and infinite values."""
import ctypes as C

import numpy as np
import pytest

from sincfeyn_b200 import sq

pytestmark = pytest.mark.gpu


def device_sum(v, a, pw, tiles):
    import torch
    L = sq.lib()
    L.sqb_running_sum.argtypes = [C.c_void_p, C.c_long, C.c_double, C.c_double, C.c_int, C.c_void_p, C.c_void_p]
    d = torch.from_numpy(np.ascontiguousarray(v)).cuda()
    torch.cuda.synchronize()
    out = C.c_double()
    assert L.sqb_running_sum(d.data_ptr(), len(v), a, pw, tiles, None, C.byref(out)) == 0
    return out.value


def values(kind, n):
    g = np.random.default_rng(n)
    if kind == 'support':          # a frontier's values: many decades, both signs
        return np.exp(g.uniform(-60, 3, n))*g.choice([-1.0, 1.0], n)
    if kind == 'growing':          # a binade change every few elements, then every few thousand
        return 2.0**(np.arange(n) % 40 - 20)*(1 + g.integers(0, 1 << 52, n)*2.0**-52)
    if kind == 'ties':             # multiples of 2^-54 and 2^-53 about a = 1: half units, to even either way
        return g.integers(0, 8, n)*2.0**-54
    if kind == 'zeros':
        return np.where(g.random(n) < 0.999, 0.0, g.random(n))
    if kind == 'tiny':
        return g.integers(0, 3, n)*5e-324
    if kind == 'huge':             # one that ends all binades at the middle
        v = g.random(n)
        v[n//2] = 1e301
        return v
    v = g.random(n)                # 'infinite'
    v[n//3] = np.inf
    return v


@pytest.mark.parametrize('tiles', [0, 1])
@pytest.mark.parametrize('kind', ['support', 'growing', 'ties', 'zeros', 'tiny', 'huge', 'infinite'])
def test_running_sum_is_the_sequential_one(kind, tiles):
    for n in (1, 31, 2048, 2049, 4096, 4097, 10000, 300001) if kind != 'growing' else (1, 100, 5000):
        for a, pw in ((0.0, 1.0), (1.0, 1.0), (0.7, 32.0), (1 - 2.0**-53, 1.0)):
            if kind == 'tiny' and a == 0:
                n = min(n, 300)
            v = values(kind, n)
            want = np.add.accumulate(np.concatenate([[a], np.abs(v)*pw]))[-1]
            got = device_sum(v, a, pw, tiles)
            assert got == want, (kind, n, a, pw, got, want)

"""The evaluator's work as its users call it, as a list of cases that can be timed and checked one by one.

Every case runs through a public entry point: sq.hsum, sq.hsum_batch and sq.hsum_group (the hierarchical
Sinc sum of one integral, of a batch on worker streams, of one graph at several h in shared level launches),
sq.eval_points (pointwise values), sqb_level_noalloc (one refinement-level batch in a caller's own memory),
and the plug-in ABI in its two forms, gpu_setup / gpu_submit_cells / gpu_wait on host cells and
sqb_plugin_launch on device buffers.  The integrands are the repository's own synthetic ones (syn_d5, syn_d8,
syn_d11), which every build of the library holds; h, N and eps are those of the benchmark, the tests and the
reference's published runs (h = 0.7 .. 2, eps = 1e-8 .. 1e-12, N = 2 ceil(30/h) + 1 unless a case says
otherwise).  A sum has no array inputs: its inputs are its parameters, and the seed moves h by up to 0.2 %, as
a scan over h does.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

from sincfeyn_b200 import sq

SEEDS = {5: 1, 8: 2, 11: 3}                       # the integrands' parameter seeds
REF = {5: 155.25, 8: 3339.0, 11: 4.3e5}           # size of the sum, which scales a level's thresholds
EPS1 = 1e-9                                       # the integrands' epsilon


def _d(case):
    return int(case['graph'].split('_d')[1])


def _n(h, reach=30.0):
    return 2*math.ceil(reach/h - 1e-9) + 1


def _hsum(name, graph, h, eps, form='contracted', N=None):
    return dict(name=name, kind='hsum', graph=graph, h=h, N=N or _n(h), eps=eps, form=form)


def listed():
    return [
        # the smallest whole call: one coarse two-loop-sized integral, as a first look at a new h is run
        # (h = 1.5, eps = 1e-10 is the reference's published scan); launches and waits decide
        _hsum('sum d5 h1.5', 'syn_d5', 1.5, 1e-10),
        # an ordinary small integral in the parity form, whose point set is checked against the reference
        _hsum('sum d5 h1.0 as written', 'syn_d5', 1.0, 1e-12, 'as written'),
        # the error reference of the precision table: every point in double-double, two refinement levels
        _hsum('sum d5 h0.7 all dd', 'syn_d5', 0.7, 1e-12, 'all dd'),
        # three-loop-sized integrals at the benchmark's settings: a slowly decaying one whose coarse grid
        # keeps 4e6 cells, so that the top level counts, and one whose two refinement levels do all the work
        _hsum('sum d8 h1.0', 'syn_d8', 1.0, 1e-12),
        _hsum('sum d8 h0.7', 'syn_d8', 0.7, 1e-12),
        # four-loop-sized integrals (dimension 11): a coarse exploratory run, and the largest case
        _hsum('sum d11 h2.0', 'syn_d11', 2.0, 1e-10),
        _hsum('sum d11 h1.5', 'syn_d11', 1.5, 1e-10),
        # a mixed batch: two graphs at the benchmark's four h on four worker streams
        dict(name='batch d5 d8', kind='batch', graphs='syn_d5 syn_d8', hs='1.0 0.9 0.8 0.7', eps=1e-10, workers=4),
        # one graph's h ladder as a group with shared level launches
        dict(name='group d5', kind='group', graph='syn_d5', hs='1.0 0.9 0.8 0.7', eps=1e-12),
        # one refinement-level batch in a program that owns its device memory: 1000 cells, 256,000 children
        dict(name='level d8 1000 cells', kind='level', graph='syn_d8', h=1.0, K=32, ncell=1000, last=False),
        # the reference driver on this library: one of its batches, cells in and f w, |f| w back in host memory
        dict(name='submit d5', kind='submit', graph='syn_d5', h=0.7, K=44, ncell=32768),
        # a pointwise table in double-double (a check of an integrand at given points)
        dict(name='points d11 dd', kind='points', graph='syn_d11', n=20001, prec=1),
    ]


def draw(rng):
    """One more case: the kinds by how often each is called, sizes over the listed cases' whole range."""
    log = lambda a, b: math.exp(rng.uniform(math.log(a), math.log(b)))   # noqa: E731
    kind = rng.choice(['hsum', 'hsum', 'hsum', 'hsum', 'batch', 'group', 'level', 'submit', 'launch', 'points'])
    d = rng.choice([5, 8, 11])
    graph = 'syn_d%d' % d
    if kind == 'hsum':
        lo, hi, e = {5: (0.6, 2.0, -12), 8: (0.7, 2.0, -12), 11: (1.4, 2.2, -9)}[d]
        h = round(log(lo, hi), 4)
        form = rng.choice(['contracted', 'contracted', 'as written', 'all dd'] if d == 5 else ['contracted', 'contracted', 'as written'])
        return dict(kind=kind, graph=graph, h=h, N=_n(h, rng.uniform(26, 36)), eps=float('%.3g' % 10**rng.uniform(e, -8)), form=form)
    if kind in ('batch', 'group'):
        hs = ' '.join('%.3f' % x for x in sorted({round(log(0.75, 1.6), 3) for _ in range(rng.randint(2, 6))}))
        eps = float('%.3g' % 10**rng.uniform(-11, -8))
        if kind == 'batch':
            return dict(kind=kind, graphs='syn_d5 syn_d8', hs=hs, eps=eps, workers=rng.choice([2, 3, 4]))
        return dict(kind=kind, graph=rng.choice(['syn_d5', 'syn_d8']), hs=hs, eps=eps)
    h = round(log(0.7, 2.0), 3)
    K = math.ceil(30/h/4)*4
    if kind == 'level':
        return dict(kind=kind, graph=graph, h=h, K=K, ncell=int(log(3, (1 << 18) >> d)), last=rng.random() < 0.5)
    if kind == 'submit':
        return dict(kind=kind, graph=graph, h=h, K=K, ncell=max(1, int(log(1 << 8, 1 << 20)) >> d))
    if kind == 'launch':
        return dict(kind=kind, graph=graph, h=h, K=K, ncell=max(1, int(log(1 << 8, 1 << 22)) >> d), contracted=rng.random() < 0.7)
    return dict(kind='points', graph=graph, n=int(log(17, 100000)), prec=rng.choice([0, 1, 2]))


# ------------------------------------------- inputs ----------------------------------------------------
def _near(h, rng):
    return h*(1 + 0.002*rng.uniform(-1, 1))


def _jobs(case, rng):
    graphs = case['graphs'].split() if case['kind'] == 'batch' else [case['graph']]
    return [(g, _near(float(h), rng), _n(float(h)), case['eps'], -1, float(h)**-_d({'graph': g})) for g in graphs for h in case['hs'].split()]


def _cells(d, K, h, n, seed):
    """n cells of a refinement level as the run keeps them: distinct nodes of the step-2 grid around the
    integrand's support, in lexicographic order, the far ones marked as needing no |.| sums, with their tiers."""
    g = np.random.default_rng(seed)
    got = np.zeros((0, d), dtype=np.int64)
    scale = 6.0/h/d**0.5
    while len(got) < n:
        k = 2*np.rint(g.laplace(0, scale, size=(2*n + 64, d))/2).astype(np.int64)
        got = np.unique(np.concatenate([got, np.clip(k, -(K//2)*2, (K//2)*2)]), axis=0)
        scale *= 1.2
    k = got[np.sort(g.permutation(len(got))[:n])]
    r = np.abs(k).sum(1)*h
    return k, (r > np.median(r)), np.minimum(2, (4*r.max() - 4*r)//max(1e-9, r.max())).astype(np.int64)


FORMS = {'contracted': {}, 'as written': dict(fma=0), 'all dd': dict(alldd=1)}
COLUMNS = ('Ah', 'ref', 'prune', 'trunc', 'unres', 'es1', 'es2')
COUNTS = ('nev', 'nq', 'kept_top', 'abskipped', 'unresdrop')


def _library():
    L = sq.lib()
    p = C.c_void_p
    L.sqb_level_noalloc.argtypes = [C.c_char_p, C.c_double, C.c_int, p, C.c_long, C.c_int, C.c_int] + [C.c_double]*5 + \
        [C.c_int]*3 + [p, C.c_long, p, p, p]
    L.sqb_plugin_launch.argtypes = [C.c_char_p, C.c_int, p, C.c_long, p, p, p, C.c_int, C.c_double, p, p, C.c_int, C.c_int]
    L.gpu_setup.argtypes = [C.c_char_p, C.c_int, p, C.c_int, C.c_double]
    L.gpu_submit_cells.argtypes = [C.c_int, C.c_long, p, C.c_int, p, C.c_int]
    L.gpu_wait.argtypes = [C.c_int, C.POINTER(C.POINTER(C.c_double)), C.POINTER(C.POINTER(C.c_double))]
    return L


def prepare(case, seed):
    kind, rng = case['kind'], random.Random(seed)
    s = dict(case)
    if kind == 'hsum':
        s['h'] = _near(case['h'], rng)
        return s
    if kind in ('batch', 'group'):
        s['jobs'] = _jobs(case, rng)
        return s
    d = _d(case)
    if kind == 'points':
        s['sf'] = np.exp(np.random.default_rng(seed).uniform(-12, 12, size=(case['n'], d)))
        return s
    s['lib'] = _library()
    k, skip, tier = _cells(d, case['K'], case['h'], case['ncell'], seed)
    table = np.exp(np.arange(-case['K'], case['K'] + 1)*case['h'])
    n = case['ncell'] << d
    if kind == 'level':
        pts = np.zeros((len(k), 12), dtype=np.int8)
        pts[:, :d] = k
        pts[:, 11] = skip + 2*tier
        s['cells'] = torch.from_numpy(pts).cuda()
        s['next'] = torch.zeros((n, 12), dtype=torch.int8, device='cuda')
    elif kind == 'submit':
        s['cells'], s['skip'], s['table'] = k.astype(np.int32), skip.astype(np.uint8), table
    else:
        s['cells'] = torch.from_numpy(k.astype(np.int16)).cuda()
        s['skip'] = torch.from_numpy(skip.astype(np.uint8)).cuda()
        s['table'] = torch.from_numpy(table).cuda()
        s['f'], s['ab'] = (torch.zeros(n, dtype=torch.float64, device='cuda') for _ in range(2))
    if kind != 'level':
        torch.cuda.synchronize()
    return s


# --------------------------------------------- one pass ------------------------------------------------
def _sums(r):
    out = {'S_h': r['S'][0], 'S_2h': r['S'][1], 'S_4h': r['S'][2]}
    out.update({k: r[k] for k in COLUMNS})
    out['counts'] = [r[k] for k in COUNTS]
    return out


def run(s):
    kind = s['kind']
    if kind == 'hsum':
        return _sums(sq.hsum(s['graph'], s['h'], s['N'], s['eps'], **FORMS[s['form']]))
    if kind == 'batch':
        return _table([_sums(r) for r in sq.hsum_batch(s['jobs'], workers=s['workers'])[0]])
    if kind == 'group':
        return _table([_sums(r) for r in sq.hsum_group([j[:5] for j in s['jobs']])])
    if kind == 'points':
        f, ab = sq.eval_points(s['graph'], s['sf'], s['prec'], 1)
        if s['prec'] != 1:
            return {'f': f, 'ab': ab}
        return {'f': f[:, 0], 'f_low': f[:, 1], 'ab': ab[:, 0], 'ab_low': ab[:, 1]}
    L, d, g = s['lib'], _d(s), s['graph'].encode()
    n = s['ncell'] << d
    if kind == 'level':
        ref = REF[d]
        sums, counts = (C.c_double*12)(), (C.c_longlong*6)()
        rc = L.sqb_level_noalloc(g, s['h'], s['K'], s['cells'].data_ptr(), s['ncell'], 1, int(s['last']), 1.0, 1e-14*ref, 1e-15*ref,
                                 1e-3, 1.0, 1, 0, 1, None if s['last'] else s['next'].data_ptr(), n, sums, counts,
                                 torch.cuda.current_stream().cuda_stream)
        if rc:
            raise sq.SqbError(L.sqb_error().decode())
        x = np.array(sums)
        out = {k: float(x[2*i] + x[2*i + 1]) for i, k in enumerate(('S', 'A', 'drop', 'es1', 'es2', 'u'))}
        out['counts'] = list(counts)
        if not s['last']:
            out['next'] = s['next']
        return out
    if kind == 'submit':
        if L.gpu_setup(g, d, s['table'].ctypes.data, s['K'], s['h']) != 1:
            raise sq.SqbError('no kernel for ' + s['graph'])
        f, ab = C.POINTER(C.c_double)(), C.POINTER(C.c_double)()
        L.gpu_submit_cells(0, s['ncell'], s['cells'].ctypes.data, d, s['skip'].ctypes.data, 1)
        L.gpu_wait(0, C.byref(f), C.byref(ab))
        return {'f': np.ctypeslib.as_array(f, shape=(n,)), 'ab': np.ctypeslib.as_array(ab, shape=(n,))}
    rc = L.sqb_plugin_launch(g, 2 if s['contracted'] else 0, torch.cuda.current_stream().cuda_stream, n, s['cells'].data_ptr(), s['skip'].data_ptr(),
                             s['table'].data_ptr(), s['K'], s['h'], s['f'].data_ptr(), s['ab'].data_ptr(), 1, 1)
    if rc:
        raise sq.SqbError(L.sqb_error().decode())
    return {'f': s['f'], 'ab': s['ab']}


def _table(rows):
    """Several sums as one column each."""
    out = {k: np.array([r[k] for r in rows]) for k in rows[0] if k != 'counts'}
    out['counts'] = np.array([r['counts'] for r in rows], dtype=np.int64)
    return out


# ------------------------------------- what a pass cannot do without -----------------------------------
def _point_flops(d):
    """+ - * / of the integrand (sq.flops) and its 3 d + 1 exponentials and logarithms, one each"""
    return sq.flops('syn_d%d' % d, 0) + 3*d + 1


def work(case):
    """A sum's floor is its evaluated points' arithmetic (the point set is the result of the run itself); its
    inputs and outputs are a few numbers.  The other calls read their cells or points once and write every
    value once."""
    kind = case['kind']
    if kind == 'hsum':
        r = sq.hsum(case['graph'], case['h'], case['N'], case['eps'], **FORMS[case['form']])
        return {'bytes': 16.0*case['N'] + 8*16, 'flops': float(r['nev'])*_point_flops(_d(case))}
    if kind in ('batch', 'group'):
        jobs = _jobs(case, random.Random(0))
        rows = sq.hsum_batch(jobs)[0]
        return {'bytes': sum(16.0*j[2] + 8*16 for j in jobs), 'flops': float(sum(r['nev']*_point_flops(_d({'graph': j[0]})) for j, r in zip(jobs, rows)))}
    d = _d(case)
    if kind == 'points':
        return {'bytes': case['n']*(8.0*d + (32 if case['prec'] == 1 else 16)), 'flops': float(case['n'])*_point_flops(d)}
    n = case['ncell'] << d
    per_cell, per_child = {'level': (12, 0), 'submit': (4*d + 1, 16), 'launch': (2*d + 1, 16)}[kind]
    return {'bytes': float(case['ncell']*per_cell + n*per_child), 'flops': float(n)*_point_flops(d)}


# ---------------------------------------- the values in 64 bits ----------------------------------------
def _params(d):
    """a_i in [0.5, 2], b_i in [-1, 1] from splitmix64"""
    m, s, u = (1 << 64) - 1, SEEDS[d], []
    for _ in range(2*d):
        s = (s + 0x9E3779B97F4A7C15) & m
        z = s
        z = ((z ^ (z >> 30))*0xBF58476D1CE4E5B9) & m
        z = ((z ^ (z >> 27))*0x94D049BB133111EB) & m
        u.append(((z ^ (z >> 31)) >> 11)*2.0**-53)
    return 0.5 + 1.5*np.array(u[:d]), -1 + 2*np.array(u[d:])


def _values(z):
    """f prod s and |f| prod s at z (n x d), the cancelling difference taken by expm1"""
    a, b = _params(z.shape[1])
    p = np.prod(1/np.cosh(a*z + b), axis=1)
    x = np.exp(-np.abs(z)).sum(1)
    return p*np.expm1(x*EPS1)/EPS1, p*(np.exp(x*EPS1) + 1)/EPS1


def _box(d, h, K, step):
    """The sum over the whole lattice |k| <= K, k a multiple of step, which the pruned sum approximates: a
    product over the axes, its difference from the eps = 0 product taken by expm1."""
    a, b = _params(d)
    z = np.arange(-(K//step)*step, K + 1, step)*h
    total, dif = 1.0, 0.0
    for i in range(d):
        g = step*h/np.cosh(a[i]*z + b[i])
        total *= g.sum()
        dif += math.log1p((g*np.expm1(EPS1*np.exp(-np.abs(z)))).sum()/g.sum())
    return total*math.expm1(dif)/EPS1


def _exact_sum(graph, h, N, eps):
    d, top = _d({'graph': graph}), sq.default_top(h)
    m = 2 << top
    K = ((N - 1)//2 + m - 1)//m*m
    out = {'S_h': _box(d, h, K, 1), 'S_2h': _box(d, h, K, 2), 'S_4h': _box(d, h, K, 4) if top > 1 else None}
    out.update({k: None for k in COLUMNS})
    out['counts'] = None
    return out


def exact(case, seed):
    kind, rng = case['kind'], random.Random(seed)
    if kind == 'hsum':
        return _exact_sum(case['graph'], _near(case['h'], rng), case['N'], case['eps'])
    if kind in ('batch', 'group'):
        rows = [_exact_sum(*j[:4]) for j in _jobs(case, rng)]
        return {k: np.array([r[k] for r in rows]) if all(r[k] is not None for r in rows) else None for k in rows[0]}
    s = prepare(case, seed)
    d = _d(case)
    if kind == 'points':
        z = np.log(s['sf'])
        f, ab = (v/np.prod(s['sf'], axis=1) for v in _values(z))
        return {'f': f, 'ab': ab} if case['prec'] != 1 else {'f': f, 'f_low': None, 'ab': ab, 'ab_low': None}
    k, _, tier = _cells(d, case['K'], case['h'], case['ncell'], seed)
    bits = (np.arange(1 << d)[:, None] >> np.arange(d)) & 1
    f, ab = np.zeros(len(k) << d), np.zeros(len(k) << d)
    for c0 in range(0, len(k), 1024):
        kk = (k[c0:c0 + 1024, None, :] - bits[None]).reshape(-1, d)
        v, w = _values(kk*case['h'])
        inside = (kk >= -case['K']).all(1)*case['h']**d
        f[c0 << d:(c0 << d) + len(v)], ab[c0 << d:(c0 << d) + len(v)] = v*inside, w*inside
    if kind != 'level':
        return {'f': f, 'ab': ab}
    small, t = np.abs(f) < 1e-14*REF[d], np.repeat(tier, 1 << d)
    out = {'S': f.sum(), 'A': np.abs(f).sum(), 'drop': None if case['last'] else np.abs(f[small]).sum(),
           'es1': f[t >= 1].sum() if case['last'] else None, 'es2': f[t >= 2].sum() if case['last'] else None, 'u': None, 'counts': None}
    if not case['last']:
        out['next'] = None
    return out

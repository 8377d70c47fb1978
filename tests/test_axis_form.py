"""The axis form of an integrand (kgen.axis_plan, class template KA) against the point function it is derived
from, on the CPU: the scan over table columns gives f and the |.| sum bit for bit, in double and in
double-double, at lattice nodes over the whole box (its corners, where factors underflow, among them); the
division by a tabulated divisor (sq_divu) gives the rounded quotient over normal and extreme operands; and
kgen leaves alone what is not such a scan."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from sincfeyn_b200.codegen import kgen

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, 'sincfeyn_b200', 'csrc')
SYNTH = os.path.join(ROOT, 'sincfeyn_b200', 'synth')
NAMES = ['syn_d5', 'syn_d8', 'syn_d11']

SRC = r'''
#include <math.h>
#include "sqdd.cuh"
#define SQ_AXIS_FORM
#define SQ_TABLE static const
#define SQ_FUNC
#define SQ_FUNC_K
#define SQ_CHUNK
#define SQ_CHUNK_DD
#define RABS(x) sq_rabs(x)
#define SQ_EXP(x) sq_exp(x)
#define SQ_LOG(x) sq_log(x)
#define SQG_NS(n) sqg_##n
static void put(double x, double *o){ o[0] = x; o[1] = 0; }
static void put(const sqdd &x, double *o){ o[0] = x.hi; o[1] = x.lo; }
template<class K, class A, class R, int D> static void both(const K &fn, long n, const double *s, double *o){
    for(long i = 0; i < n; i++){
        R sf[D], a1, a2;
        typename A::st S; A::init(S);
        for(int d = 0; d < D; d++){
            sf[d] = R(s[i*D + d]);
            R u[A::NU]; double r[A::NR];
            A::axis(d, sf[d], u);
            for(int q = 0; q < A::NR; q++) r[q] = sqdd_rcp(u[A::rc(q)]);
            A::step(S, sf[d], u, r);
        }
        put(fn(sf, &a1), o + 8*i); put(a1, o + 8*i + 2); put(A::fin(S, &a2), o + 8*i + 4); put(a2, o + 8*i + 6);
    }
}
#define SQ_GRAPH_AXIS(NAME, V, L, D, W, NP, FIX) \
extern "C" void ax_##NAME(long n, const double *s, int dd, double *o){ \
    if(dd) both<decltype(&sqg_##NAME::K<sqdd, 1>::f_##NAME), sqg_##NAME::KA<sqdd, 1>, sqdd, D>(&sqg_##NAME::K<sqdd, 1>::f_##NAME, n, s, o); \
    else both<decltype(&sqg_##NAME::K<double, 1>::f_##NAME), sqg_##NAME::KA<double, 1>, double, D>(&sqg_##NAME::K<double, 1>::f_##NAME, n, s, o); }
extern "C" void divu(long n, const double *a, const double *b, double *o){
    for(long i = 0; i < n; i++) o[i] = sq_divu(a[i], b[i], sqdd_rcp(b[i])); }
extern "C" void divc(long n, const double *a, const double *b, double *o, int *bad){
    for(long i = 0; i < n; i++){
        unsigned f = 0;
        const double r = sq_rcpc<0>(b[i], &f);
        o[i] = sq_divc<0>(a[i], b[i], r, &f); bad[i] = sqdd_bad(f);
    } }
'''


@pytest.fixture(scope='module')
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp('axis')
    cc = d / 'axis.cc'
    text = SRC
    for n in NAMES:
        _, cuh = kgen.emit(os.path.join(SYNTH, n + '.c'))
        assert 'struct KA' in cuh, n
        (d / (n + '.cuh')).write_text(cuh)
        text += '#include "%s.cuh"\n' % n
    cc.write_text(text)
    so = d / 'axis.so'
    subprocess.run(['g++', '-O1', '-ffp-contract=off', '-std=c++17', '-shared', '-fPIC', '-I' + CSRC, '-o', str(so), str(cc)], check=True)
    return C.CDLL(str(so))


@pytest.mark.parametrize('dd', [0, 1])
@pytest.mark.parametrize('name', NAMES)
def test_scan_equals_the_point_function(lib, name, dd):
    D = int(name.split('_d')[1])
    rng = np.random.default_rng(D)
    for h, K in ((1.0, 30), (0.7, 44), (2.0, 16), (0.55, 127)):
        k = rng.integers(-K, K + 1, size=(400 if dd else 4000, D))
        k[:4] = [[K]*D, [-K]*D, [0]*D, [K, -K]*(D//2) + [K]*(D % 2)]
        s = np.ascontiguousarray(np.exp(k*h))
        o = np.empty((len(k), 8))
        getattr(lib, 'ax_' + name)(C.c_long(len(k)), s.ctypes.data_as(C.c_void_p), dd, o.ctypes.data_as(C.c_void_p))
        assert np.array_equal(o[:, :4], o[:, 4:], equal_nan=True), (h, K)


def test_division_by_a_table_column_rounds_correctly(lib):
    rng = np.random.default_rng(3)
    n = 200000
    mant = lambda: (1 + rng.integers(0, 1 << 52, n)*2.0**-52)          # noqa: E731
    edge = np.array([1.0, 1 + 2.0**-52, 2 - 2.0**-52, 2 - 2.0**-51, 1.5])
    for ea, eb in ((0, 0), (480, -190), (-499, 3), (499, 199), (499, 0), (501, 0), (-1000, 30), (0, -1060), (1000, 1000), (0, 401), (899, 399), (-899, -399)):
        a, b = mant(), mant()
        a[:25], b[:25] = np.repeat(edge, 5), np.tile(edge, 5)
        with np.errstate(all='ignore'):
            a, b = a*2.0**ea*rng.choice([-1, 1], n), np.ldexp(b, eb)
            want = a/b
        o = np.empty(n)
        lib.divu(C.c_long(n), *(x.ctypes.data_as(C.c_void_p) for x in (a, b, o)))
        assert np.array_equal(o, want), (ea, eb)
    a, b = (x.ravel() for x in np.meshgrid([0.0, -0.0, np.inf, -np.inf, np.nan, 1.0, 5e-324], [0.0, np.inf, np.nan, 2.0, 5e-324]))
    a, b, o = np.ascontiguousarray(a), np.ascontiguousarray(b), np.empty(len(a))
    lib.divu(C.c_long(len(a)), *(x.ctypes.data_as(C.c_void_p) for x in (a, b, o)))
    with np.errstate(all='ignore'):
        assert np.array_equal(o, a/b, equal_nan=True)


@pytest.mark.parametrize('change', [
    ('x=x+SQ_EXP(-RABS(z));', 'x=x+SQ_EXP(-RABS(z))*sf[0];'),       # a coordinate of another axis
    ('js=js*sf[i];', 'js=js*sf[i]; p=p+y;'),                       # an unknown name
    ('for(int i=0;i<5;i++)', 'for(int i=0;i<4;i++)'),              # not every axis
    ('const REAL ex=', 'x=x+sf[0];\n  const REAL ex='),            # the tail reads a coordinate
])
def test_other_functions_keep_their_form(tmp_path, change):
    with open(os.path.join(SYNTH, 'syn_d5.c')) as f:
        text = f.read()
    i = text.index('#define REAL QREAL')
    assert change[0] in text[i:]
    src = tmp_path / 'syn_d5.c'
    src.write_text(text[:i] + text[i:].replace(*change))
    assert kgen.axis_plan(kgen.KernelSource(str(src))) is None
    assert 'KA' not in kgen.emit(str(src))[1]


def test_an_added_product_keeps_its_factors_apart(tmp_path):
    """x + e*z: the contracted build fuses it in f_, and so it must in the scan"""
    with open(os.path.join(SYNTH, 'syn_d5.c')) as f:
        text = f.read().replace('x=x+SQ_EXP(-RABS(z));', 'x=x+e*SQ_EXP(z);')
    src = tmp_path / 'syn_d5.c'
    src.write_text(text)
    plan = kgen.axis_plan(kgen.KernelSource(str(src)))
    assert 'S.x=S.x+u[1]*u[2];' in plan and 'u[1]=e;' in plan and 'u[2]=SQ_EXP(z);' in plan


def test_put_off_tests_of_a_division(lib):
    # either the rounded quotient or flagged, and flagged only outside 2^+-450
    rng = np.random.default_rng(3)
    n = 200000
    a, b = (rng.choice([-1, 1], n)*(1 + rng.integers(0, 1 << 52, n)*2.0**-52)*2.0**rng.integers(-1000, 1000, n) for _ in range(2))
    b[n//2:] = b[n//2:]/2.0**(2*np.frexp(b[n//2:])[1]//3)
    a[:7], b[:7] = [0, 1, np.inf, np.nan, 1, 1, 0], [1, 0, 1, 1, np.inf, np.nan, 0]
    o, bad = np.empty(n), np.empty(n, dtype=np.intc)
    lib.divc(C.c_long(n), a.ctypes.data_as(C.c_void_p), b.ctypes.data_as(C.c_void_p), o.ctypes.data_as(C.c_void_p), bad.ctypes.data_as(C.c_void_p))
    with np.errstate(all='ignore'):
        q = a/b
        inside = (np.abs(q) >= 2.0**-449) & (np.abs(q) < 2.0**449) & (np.abs(b) >= 2.0**-450) & (np.abs(b) < 2.0**450)
    assert not np.any(bad[inside]) and np.all(bad[:7] != 0)
    good = bad == 0
    assert good.sum() > n//10 and np.array_equal(o[good], q[good])

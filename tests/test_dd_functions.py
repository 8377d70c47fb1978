"""The double-double exp and log of the device code (sqdd.cuh) on the host, against 60-digit decimal values: over the
whole range of exp, at the edges of its reduction (multiples of ln2/256, where the table entry changes) and at extreme
arguments.  exp keeps one rounding of its low part (2^-107) and products a few 2^-112 below it: within 2^-106.  log
adds a product of two numbers near 1: within 2^-104 max(1, |log a|)."""
import ctypes as C
import os
import subprocess
from decimal import Decimal, getcontext

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'sincfeyn_b200', 'csrc')
SRC = r'''
#include "sqdd.cuh"
extern "C" void ddexp(long n, const double *x, double *o){
    for(long i = 0; i < n; i++){ sqdd r = sqdd_exp(sqdd(x[2*i], x[2*i+1])); o[2*i] = r.hi; o[2*i+1] = r.lo; } }
extern "C" void ddlog(long n, const double *x, double *o){
    for(long i = 0; i < n; i++){ sqdd r = sqdd_log(sqdd(x[2*i], x[2*i+1])); o[2*i] = r.hi; o[2*i+1] = r.lo; } }
'''


@pytest.fixture(scope='module')
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp('dd')
    (d / 'dd.cc').write_text(SRC)
    subprocess.run(['g++', '-O1', '-ffp-contract=off', '-shared', '-fPIC', '-I' + CSRC, '-o', str(d / 'dd.so'), str(d / 'dd.cc')], check=True)
    return C.CDLL(str(d / 'dd.so'))


def call(fn, pairs):
    x = np.ascontiguousarray(pairs, dtype=np.float64)
    o = np.empty_like(x)
    fn(C.c_long(len(x)), x.ctypes.data_as(C.c_void_p), o.ctypes.data_as(C.c_void_p))
    return o


def exact(p):
    return Decimal(float(p[0])) + Decimal(float(p[1]))


def split(v):
    return float(v), float(v - Decimal(float(v)))


def arguments():
    g = np.random.default_rng(11)
    hi = np.concatenate([g.uniform(-w, w, 500) for w in (1e-9, 0.01, 1, 35, 660)] +
                        [np.array([0.0, 1e-300, -1e-300, 660.0, -660.0]),
                         (np.arange(-300, 300) + 0.5)*np.log(2)/128*(1 + g.choice([-1, 1], 600)*1e-15)])
    return np.stack([hi, hi*g.uniform(-1, 1, len(hi))*2.0**-54], 1)


def test_exp(lib):
    getcontext().prec = 60
    for p, o in zip(arguments(), call(lib.ddexp, arguments())):
        t = exact(p).exp()
        assert abs(exact(o) - t) <= Decimal(2)**-106*t, p


def test_log(lib):
    getcontext().prec = 60
    x = np.array([split(exact(p).exp()) for p in arguments()])
    for p, o in zip(x, call(lib.ddlog, x)):
        t = exact(p).ln()
        assert abs(exact(o) - t) <= Decimal(2)**-104*max(Decimal(1), abs(t)), p


def test_extreme_arguments(lib):
    e = call(lib.ddexp, [(710, 0), (np.inf, 0), (-746, 0), (-np.inf, 0), (np.nan, 0), (709, 0), (-744, 0)])[:, 0]
    assert list(e[:4]) == [np.inf, np.inf, 0, 0] and np.isnan(e[4])
    assert abs(e[5]/8.218407461554972e307 - 1) < 1e-15 and e[6] == 1e-323
    log = call(lib.ddlog, [(0, 0), (-1, 0), (np.nan, 0)])[:, 0]
    assert log[0] == -np.inf and np.isnan(log[1]) and np.isnan(log[2])

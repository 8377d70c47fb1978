"""Integrands whose text has what the axis form's class could trip over (CPU): every one compiles, and where kgen writes the
class its scan gives the point function's values bit for bit.  A unary minus after a minus stays two signs; an
accumulator, a constant or a value of the tail may have the name of anything that the class declares."""
import ctypes as C
import os
import re
import subprocess

import numpy as np
import pytest

from sincfeyn_b200.codegen import kgen

import test_axis_form as form

RENAMED = ['S', 'u', 'r', 'si', 'st', 'KA', 'CK', 'NU', 'NR', 'rc', 'axis', 'init', 'step', 'fin', 'sq_bad', 'r_js', 'S0', 'c']
CASES = [('minus', [('x=x+SQ_EXP(-RABS(z));', 'x=x- -SQ_EXP(-RABS(z));')], True),
         ('minus of an accumulator', [('x=x+SQ_EXP(-RABS(z));', 'x=SQ_EXP(-RABS(z))- -x;')], True),
         ('minus in a column', [('x=x+SQ_EXP(-RABS(z));', 'x=x+SQ_EXP(z- -z);')], True),
         ('minus in the tail', [('return (ex-1)', 'return (ex- -1)')], True)]
CASES += [('accumulator ' + n, [(r'\bjs\b', n)], None) for n in RENAMED if n != 'r_js']
CASES += [('constant ' + n, [(r'\be\b', n)], None) for n in RENAMED]
CASES += [('tail ' + n, [(r'\bex\b', n)], None) for n in RENAMED]


@pytest.mark.parametrize('name,changes,form_wanted', CASES, ids=[c[0] for c in CASES])
def test_text_compiles_and_agrees(tmp_path, name, changes, form_wanted):
    with open(os.path.join(form.SYNTH, 'syn_d5.c')) as f:
        head, body = f.read().split('#define REAL double', 1)
    for a, b in changes:
        new = re.sub(a, b, body) if a.startswith('\\b') else body.replace(a, b)
        assert new != body
        body = new
    src = tmp_path / 'syn_d5.c'
    src.write_text(head + '#define REAL double' + body)
    _, cuh = kgen.emit(str(src))
    has = 'struct KA' in cuh
    assert has or not form_wanted
    (tmp_path / 'syn_d5.cuh').write_text(cuh)
    text = form.SRC if has else form.SRC[:form.SRC.index('#define SQ_GRAPH_AXIS')] + \
        '#define SQ_GRAPH(NAME, V, L, D, W, NP, FIX) extern "C" double value(const double *s){ double ab; return sqg_##NAME::K<double, 1>::f_##NAME(s, &ab); }\n'
    (tmp_path / 'a.cc').write_text(text + '#include "syn_d5.cuh"\n')
    so = tmp_path / 'a.so'
    r = subprocess.run(['g++', '-O0', '-ffp-contract=off', '-std=c++17', '-shared', '-fPIC', '-I' + form.CSRC, '-o', str(so), str(tmp_path / 'a.cc')],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[:2000]
    if not has:
        return
    L = C.CDLL(str(so))
    k = np.random.default_rng(1).integers(-30, 31, size=(300, 5))
    s, o = np.ascontiguousarray(np.exp(k*0.7)), np.empty((300, 8))
    for dd in (0, 1):
        L.ax_syn_d5(C.c_long(300), s.ctypes.data_as(C.c_void_p), dd, o.ctypes.data_as(C.c_void_p))
        assert np.array_equal(o[:, :4], o[:, 4:], equal_nan=True)

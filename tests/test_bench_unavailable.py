"""bench.py where the library holds the synthetic integrands alone, or the reference's CPU build is absent (CPU): each arm
says so in one JSON line and ends with status 0."""
import json
import os
import subprocess
import sys

import pytest

import refpy
from sincfeyn_b200 import sq


def lines(root, *args):
    r = subprocess.run([sys.executable, os.path.join(root, 'bench.py')] + list(args), cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return [json.loads(x) for x in r.stdout.splitlines()]


@pytest.mark.skipif(any(not g['name'].startswith('syn_') for g in sq.graphs()), reason='the library holds graphs')
@pytest.mark.parametrize('workload', ['all3', 'mixed', 'vp4', 'single', 'points'])
def test_our_arm_without_the_graphs(root, workload):
    out = lines(root, '--gpus', '1', '--steps', '1', '--workload', workload)
    assert len(out) == 1 and out[0]['impl'] == 'ours' and out[0]['value'] is None and 'kernels' in out[0]['unavailable']


@pytest.mark.skipif(refpy.available(), reason='the reference is built')
def test_reference_arm_without_the_reference(root):
    out = lines(root, '--impl', 'reference', '--gpus', '1', '--steps', '2', '--warmup', '1')
    assert len(out) == 1 and out[0]['impl'] == 'reference' and 'not built' in out[0]['unavailable']

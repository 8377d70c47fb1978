"""sq.preload (GPU) loads every kernel that a graph's integrals run: for an integrand with an axis form the three general
ones, the level kernel of the contracted build, and of each build the level kernel's four forms, three kernels for other
launches and the one that fills the tables."""
import json
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r'''
import json
from sincfeyn_b200 import sq
L = sq.lib()
assert L.sqb_dev_init(0) == 0
print(json.dumps([sq.preload('syn_d5'), sq.preload('syn_d8'), sq.preload('no_such_graph')]))
'''


def test_preload_loads_the_axis_form(root):
    r = subprocess.run([sys.executable, '-c', CHILD], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert json.loads(r.stdout) == [3 + 1 + 2*8, 3 + 1 + 2*8, 0]

"""The reference's per-graph launcher GG_<graph> (GPU), which returns nothing: a launch that the device refuses (lattice
tables beyond a CTA's shared memory) prints and exits with status 3, as the rest of the plain form; an error that an
earlier call left behind does not count against a good one."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r'''
import ctypes as C, sys, torch
import numpy as np
from sincfeyn_b200 import sq
p = C.c_void_p
class Desc(C.Structure):
    _fields_ = [('name', C.c_char_p), ('D', C.c_int),
                ('launch', C.CFUNCTYPE(None, p, C.c_long, p, p, p, C.c_int, C.c_double, p, p, C.c_int, C.c_int))]
L, K = sq.lib(), int(sys.argv[1])
L.sqb_l2_flush.argtypes = [C.c_size_t]
g = Desc.in_dll(L, 'GG_syn_d5')
k = torch.zeros((8, 5), dtype=torch.int16, device='cuda')
X = torch.from_numpy(np.exp(0.001*np.arange(-K, K + 1))).cuda()
out = torch.full((2, 8), -7.0, dtype=torch.float64, device='cuda')
torch.cuda.synchronize()
assert L.sqb_l2_flush(1 << 50) != 0            # an allocation refused, its error left in the library's runtime
g.launch(None, 8, k.data_ptr(), None, X.data_ptr(), K, 0.5, out[0].data_ptr(), out[1].data_ptr(), 0, 0)
torch.cuda.synchronize()
f, ab = sq.eval_points('syn_d5', np.ones((8, 5)), 0, 1)
assert np.array_equal(out.cpu().numpy(), np.stack([f, ab])*0.5**5), out
print('launched')
'''


@pytest.mark.parametrize('K,code', [(40, 0), (2000, 3)])
def test_a_refused_launch_is_reported(root, K, code):
    r = subprocess.run([sys.executable, '-c', CHILD, str(K)], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == code, r.stderr
    assert ('launched' in r.stdout) == (code == 0) and ('CUDA error' in r.stderr) == (code == 3)

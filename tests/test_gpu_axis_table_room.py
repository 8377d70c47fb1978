"""The plug-in's launches on wide lattices (GPU): the axis table that a CTA fills in shared memory either side of the K at
which it no longer fits beside the lattice tables and the kernel's own shared memory (syn_d11: 85, syn_d8: 115; syn_d5's
fits at every K).  Every |k| <= 127 is accepted, and the values are those of launches below the table's size, bit for
bit."""
import numpy as np
import pytest

from test_gpu_axis_paths import launch, nodes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('form', [0, 2])
@pytest.mark.parametrize('graph,K', [('syn_d11', 85), ('syn_d11', 86), ('syn_d11', 87), ('syn_d11', 88), ('syn_d11', 127),
                                     ('syn_d8', 115), ('syn_d8', 116), ('syn_d8', 117), ('syn_d8', 118), ('syn_d5', 127)])
def test_raw_launch_on_a_wide_lattice(graph, K, form):
    d, h, n = int(graph[5:]), 0.5, 1 << 17
    k = nodes(d, K, n, 1, K)
    skip = np.random.default_rng(K).random(n) < 0.3
    whole = launch(graph, form, k, skip, K, h, 0, d, 1)
    parts = [launch(graph, form, k[i:i + n//2], skip[i:i + n//2], K, h, 0, d, 1) for i in (0, n//2)]
    assert np.array_equal(whole.view(np.int64), np.concatenate(parts, axis=1).view(np.int64))

"""Test configuration: the `gpu` marker (tests that need a CUDA device, run on a B200), the paths, and the tests that need
graphs which the built library may not hold."""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
sys.path.insert(0, os.path.join(ROOT, 'oracle'))


def pytest_configure(config):
    config.addinivalue_line('markers', 'gpu: needs a CUDA device (sm_100a); run with -m gpu on a B200')


# Tests of the reference's graphs, by the class of the graphs that they run (a file, or some of its tests).  A library that
# was built without the reference's kernels holds the synthetic integrands alone: there they skip.  The other files of
# graphs skip by themselves.
NEEDS = {
    'test_abi.py': {'test_registry_and_plugin_descriptors': 'g2_', 'test_selectors_match_the_reference_groups': 'g2_'},
    'test_build_policy.py': {'test_occupancy_record_follows_the_policy': 'g3_'},
    'test_gpu_all3.py': 'g3_',
    'test_gpu_batch.py': {'test_batch_equals_one_at_a_time': 'g2_', 'test_batch_order_by_cost_and_tuner': 'g2_'},
    'test_gpu_ckpt.py': 'g2_',
    'test_gpu_fold.py': 'g3_',
    'test_gpu_group.py': 'g2_',
    'test_gpu_hsum.py': 'g2_',
    'test_gpu_pi6.py': 'w4_p6',
    'test_gpu_precision.py': 'g3_',
    'test_gpu_predict.py': 'g2_',
    'test_gpu_scale.py': 'g2_',
    'test_gpu_split.py': 'g3_',
    'test_gpu_ties.py': 'v3_',
    'test_gpu_vp4_sets.py': 'v4_',
    'test_zz_no_alloc.py': 'g3_',
}


def pytest_collection_modifyitems(config, items):
    from sincfeyn_b200 import sq
    try:
        names = [g['name'] for g in sq.graphs()]
    except (sq.SqbError, OSError):
        return                       # no library, or none that loads: the tests say so themselves
    for item in items:
        need = NEEDS.get(os.path.basename(str(item.fspath)))
        if isinstance(need, dict):
            need = need.get(getattr(item, 'originalname', item.name))
        if need and not any(n.startswith(need) for n in names):
            item.add_marker(pytest.mark.skip(reason='the library holds no %s graph (built without the reference\'s kernels)' % need))


@pytest.fixture(scope='session')
def root():
    return ROOT

"""Which sources the build compiles without the reference's kernel tree: the synthetic integrands where no
library is built or the built one holds nothing else, and nothing (the library is kept) where it holds other
graphs."""
import json

import pytest

from sincfeyn_b200 import build


@pytest.mark.parametrize('built, want', [(None, 3), (['syn_d5', 'syn_d8', 'syn_d11'], 3), (['g2_00', 'syn_d5'], 0)])
def test_sources_without_a_kernel_tree(tmp_path, monkeypatch, built, want):
    monkeypatch.setattr(build, 'LIBSO', str(tmp_path / 'lib.so'))
    monkeypatch.setattr(build, 'FLOPS', str(tmp_path / 'flops.json'))
    if built:
        (tmp_path / 'lib.so').write_text('')
        (tmp_path / 'flops.json').write_text(json.dumps({n: {} for n in built}))
    for kdir in (None, str(tmp_path)):
        assert len(build.kernel_sources(kdir, 'g2 g3')) == want

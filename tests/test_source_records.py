"""The source files whose hashes a run's record and checkpoints carry: with every listed file of csrc/ also the
headers of csrc/ that it includes, so that no change of the library's arithmetic goes unrecorded."""
import importlib
import re

import pytest

from conftest import PKG_DIR, PKG_NAME, load_package


@pytest.mark.parametrize('module,name', [('ghost', 'MAC_CylinderFlow'), ('cutcell', 'CutCellFlow'), ('staircase', 'StaircaseFlow'),
                                         ('staircase', 'LegacyGhostFlow')])
def test_records_cover_included_headers(module, name):
    load_package()
    files = set(getattr(importlib.import_module(f'{PKG_NAME}.{module}'), name)._source_hashes(None))
    for f in sorted(x for x in files if x.startswith('csrc/')):
        for header in re.findall(r'^#include "([\w.]+)"', (PKG_DIR / f).read_text(), re.M):
            assert f'csrc/{header}' in files, (f, header)

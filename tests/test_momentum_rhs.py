"""The FP64 momentum right-hand side of inner faces (csrc/momentum.cuh) keeps a constant field to the bit and
rounds only its increment and their sum (momentum_check.cu, built for the host with nvcc)."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_constant_fields_stay(tmp_path):
    nvcc = shutil.which('nvcc') or ('/usr/local/cuda/bin/nvcc' if Path('/usr/local/cuda/bin/nvcc').exists() else None)
    if nvcc is None:
        pytest.skip('nvcc not available')
    exe = tmp_path / 'momentum_check'
    subprocess.run([nvcc, '-std=c++17', '-I', str(ROOT / 'cfd-cylinder-flow-ghost-cell_gb300' / 'csrc'), '-o', str(exe),
                    str(ROOT / 'tests' / 'momentum_check.cu')], check=True, capture_output=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr

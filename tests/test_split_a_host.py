"""The split of the tensor-core A operands without FP64 instructions
(fpconv::split_a) gives the pieces of the FP64 arithmetic: host build,
random entries and the neighbourhoods of every rounding's midpoints."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


def test_split_a_matches_fp64(tmp_path):
    nvcc = shutil.which('nvcc') or '/usr/local/cuda/bin/nvcc'
    if not os.path.exists(nvcc):
        pytest.skip('nvcc not available')
    exe = tmp_path / 'split_a_check'
    subprocess.run([nvcc, '-O2', '-std=c++17', '-I', os.path.join(ROOT, 'lime_gb300', 'csrc'),
                    os.path.join(ROOT, 'tests', 'native', 'split_a_check.cu'), '-o', str(exe)],
                   check=True, capture_output=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith('ok'), out.stdout[-2000:]

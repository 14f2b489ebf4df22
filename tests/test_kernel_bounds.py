"""Addresses of a stencil kernel, walked on the CPU: the kernel's own source is
compiled for the host (tests/host_kernels) and every load and store that it
makes outside its staged planes must stay inside its arrays.  An access past
an array does not show in the outputs when it only feeds sums that are
dropped, as the potential of a halo plane does."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which('g++') is None, reason='needs g++')
def test_cell_staged_star(tmp_path):
    exe = str(tmp_path / 'cells')
    src = os.path.join(HERE, 'host_kernels')
    subprocess.run(['g++', '-std=c++17', '-O1', '-w', '-I', src, '-I',
                    os.path.dirname(HERE), os.path.join(src, 'cells.cpp'),
                    '-o', exe], check=True)
    run = subprocess.run([exe], stdout=subprocess.PIPE)
    assert (run.returncode, run.stdout) == (0, b'in bounds\n')

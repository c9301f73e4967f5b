"""Float64 quotients by Float32, Float16 and integer differences run on the integer
pipes (meshing.jl_gb300/csrc/mesh_quot.h) and must equal the IEEE quotient bit for
bit.  narrow_division.cpp compiles that header for the host, with reciprocal seeds
off by up to two ulps, and compares random and edge operands with a / b; the GPU
parity tests then compare the kernels' vertices with the oracle's.
"""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_quotients_equal_the_ieee_division(tmp_path):
    cc = shutil.which('g++')
    if cc is None:
        pytest.skip('no C++ compiler')
    exe = str(tmp_path / 'narrow_division')
    subprocess.run([cc, '-O2', '-std=c++17', '-ffp-contract=off', '-I',
                    os.path.join(HERE, '..', 'meshing.jl_gb300', 'csrc'), '-o', exe,
                    os.path.join(HERE, 'narrow_division.cpp')], check=True)
    out = subprocess.run([exe, '4000000'], check=True, capture_output=True, text=True)
    bad, taken = (int(x) for x in out.stdout.split())
    assert taken > 10_000_000
    assert bad == 0

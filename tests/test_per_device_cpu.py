"""Settings that belong to a device are made on every device that needs them
(``csrc/per_device.cuh``), compiled here as plain C++."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), 'lentil_gb300', 'csrc')

PROGRAM = r'''
#include "per_device.cuh"
#include <cstdio>
int main() {
  static lgb::OncePerDevice once;
  int calls[3] = {0, 0, 0}, fail = 1;
  auto on = [&](int dev, int slot) { return once.run(dev, 0, [&] { ++calls[slot]; return slot == 1 ? fail : 0; }); };
  const int a = on(0, 0), b = on(0, 0);            // device 0: once
  const int c = on(1, 1);                          // device 1 fails ...
  fail = 0;
  const int d = on(1, 1), e = on(1, 1);            // ... is tried again, then known
  const int f = on(1000, 2), g = on(1000, 2);      // beyond the table: each time
  std::printf("%d %d %d %d %d %d %d | %d %d %d\n", a, b, c, d, e, f, g, calls[0], calls[1], calls[2]);
}
'''


def test_once_on_each_device(tmp_path):
    cxx = shutil.which('g++') or shutil.which('c++')
    if cxx is None:
        pytest.skip('no C++ compiler')
    src, exe = tmp_path / 'once.cpp', tmp_path / 'once'
    src.write_text(PROGRAM)
    subprocess.run([cxx, '-std=c++17', '-I', CSRC, str(src), '-o', str(exe), '-pthread'], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out.strip() == '0 0 1 0 0 0 0 | 1 2 2'


def test_kernel_attributes_are_set_per_device():
    # a kernel's attributes are set by the helper above or on every launch, never
    # under a flag of the whole process
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as fh:
            text = fh.read()
        if 'cudaFuncSetAttribute' in text or 'allow_shared_memory' in text:
            assert 'call_once' not in text, name

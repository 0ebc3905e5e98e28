"""What a launcher does once, it does once on every device: shared-memory opt-ins belong to the device that is current."""
import glob
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r'''
#include "common/host.h"
static int device = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return device < 0 ? cudaErrorNoDevice : cudaSuccess; }
int main() {
  static lt::OncePerDevice once;
  int done = 0;
  auto launch = [&](int d) { device = d; if (once.pending()) { ++done; once.finish(); } };
  for (int d : {0, 0, 1, 0, 1, 63, 63, 2}) launch(d);
  if (done != 4) return 1;
  launch(-1);          // no device, or more of them than are kept apart: due every time
  launch(-1);
  launch(64);
  launch(64);
  return done == 8 ? 0 : 2;
}
'''


def test_once_per_device(tmp_path):
    src, exe = str(tmp_path / "once.cpp"), str(tmp_path / "once")
    with open(src, "w") as f:
        f.write(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "csrc", "kernels"), "-I", "/usr/local/cuda/include", src, "-o", exe], check=True)
    assert subprocess.run([exe]).returncode == 0


def test_launchers_opt_in_on_every_device():
    for path in glob.glob(os.path.join(ROOT, "csrc", "**", "*.cu"), recursive=True):
        text = open(path).read()
        for at in re.finditer(r"cudaFuncSetAttribute\(", text):
            assert "static bool" not in text[max(0, at.start() - 900):at.start()], (path, text[at.start() - 200:at.start()])

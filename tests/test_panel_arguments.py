"""Host checks of the Householder panel's launcher (qr.cu), in a small program that needs no GPU."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "zolo-svd_b200", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
# a panel past every register form, its rows in no buffer of V: refused before anything is launched
MAIN = r"""
#include <cstdio>
#include "kernels.h"
namespace zolo { int num_sms() { return 148; } }
int main() {
  double* p = reinterpret_cast<double*>(4096);  // never touched on the host
  const int m = 16 * 512 + 1;
  const cudaError_t e = zolo::qr_panel(m, 32, p, m, 0, p, 32, p, 1024, nullptr, 0, 0, 1, nullptr);
  std::printf("%d\n", static_cast<int>(e));
  return e == cudaErrorInvalidValue ? 0 : 1;
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
def test_large_panel_needs_v(tmp_path):
    (tmp_path / "main.cu").write_text(MAIN)
    exe = str(tmp_path / "t")
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", f"-I{CSRC}", "-o", exe,
                    str(tmp_path / "main.cu"), os.path.join(CSRC, "qr.cu")], check=True)
    env = dict(os.environ, CUDA_VISIBLE_DEVICES="")  # the launcher alone, on a GPU box too
    r = subprocess.run([exe], capture_output=True, text=True, env=env)
    assert r.returncode == 0, f"cudaError {r.stdout.strip()}"

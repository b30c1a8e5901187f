"""The stage-by-stage kernels take one instance: a table of instances is refused before any
launch (checked on the host, without a GPU)."""

import subprocess

from fesom_jax_b200 import build

SOURCE = r"""
#include <cstdio>
#include "fct_host.h"
extern "C" const char* fct_last_error(void);
int main() {
  fct::LaunchDims d{};
  d.ntr = 1;
  d.fused = false;
  d.copy_dry = d.any_wi = false;
  fct::Inst single{};
  const fct::Inst* table = reinterpret_cast<const fct::Inst*>(uintptr_t(256));   // never read
  const int st = fct::launch_forward(single, table, 1, d, nullptr);
  std::printf("%d %s\n", st, fct_last_error());
  return 0;
}
"""


def test_stage_kernels_refuse_a_table(tmp_path):
    src, exe = tmp_path / "t.cu", tmp_path / "t"
    src.write_text(SOURCE)
    lib = build.build()
    subprocess.run([build.nvcc(), "-std=c++17", "-I", str(build.CSRC), "-I",
                    str(build.PKG.parent / "include"), str(src), str(lib), "-Xlinker",
                    f"-rpath={lib.parent}", "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True,
                         env={"CUDA_VISIBLE_DEVICES": ""}).stdout
    status, message = out.split(maxsplit=1)
    assert int(status) == -1 and "one instance" in message

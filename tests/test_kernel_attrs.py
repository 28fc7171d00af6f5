"""Launch attributes and occupancies are kept per context, since they belong to
the context's device: a second device's context sets and asks for its own. Run on
the CPU against a stand-in for cudaFuncSetAttribute that counts per device."""
import re
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "lfric_core_b200" / "csrc"

PROGRAM = r"""
#include "lfx_kernel_attrs.h"
#include <cassert>
#include <cstdio>
static int device = 0, calls[2], limit[2], fail = 0;
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute a, int v) {
  if (fail) return cudaErrorInvalidValue;
  assert(a == cudaFuncAttributeMaxDynamicSharedMemorySize);
  calls[device]++;
  limit[device] = v;
  return cudaSuccess;
}
int main() {
  lfx::KernelAttrs ctx[2];
  const void *f = &device, *g = &fail;
  for (device = 0; device < 2; ++device) {
    for (int k = 0; k < 3; ++k) assert(ctx[device].allow_smem(f, 100000) == cudaSuccess);
    assert(calls[device] == 1 && limit[device] == 100000);
    assert(ctx[device].allow_smem(f, 50000) == cudaSuccess && calls[device] == 1);
    assert(ctx[device].allow_smem(f, 200000) == cudaSuccess && limit[device] == 200000);
    fail = 1;  // a refused limit is asked for again
    assert(ctx[device].allow_smem(g, 60000) != cudaSuccess);
    fail = 0;
    assert(ctx[device].allow_smem(g, 60000) == cudaSuccess && calls[device] == 3);
    int asked = 0;
    for (int k = 0; k < 3; ++k) assert(ctx[device].once(f, [&] { ++asked; return device; }) == device);
    assert(asked == 1);
  }
  std::puts("ok");
}
"""


def test_each_context_has_its_own(tmp_path):
    src, exe = tmp_path / "attrs.cpp", tmp_path / "attrs"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", "-I/usr/local/cuda/include", str(src), "-o",
                    str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout == "ok\n"


def test_no_launch_state_in_the_process():
    for f in [*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]:
        assert not re.search(r"^ +static (bool|int) ", f.read_text(), re.M), f.name

"""A result that is read after its number: no data race by the thread
sanitizer's rules (a plain or volatile look at the number, tried beside it, is
one: on a host that reorders loads the result could be an older one)."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "lfric_core_b200" / "csrc"

PROGRAM = r"""
#include "lfx_host_number.h"
#include <cstdio>
#include <thread>
static double result;
static unsigned number;
int main() {
  std::thread writer([] {
    result = 3.5;
    __atomic_store_n(&number, 1u, __ATOMIC_RELEASE);
  });
  while (LOOK(&number) != 1u) {
  }
  std::printf("%g\n", result);
  writer.join();
}
"""


@pytest.mark.parametrize("look,race", [("lfx::host_number", False),
                                       ("*(const volatile unsigned*)", True)])
def test_result_follows_its_number(tmp_path, look, race):
    src, exe = tmp_path / "number.cpp", tmp_path / "number"
    src.write_text(PROGRAM)
    r = subprocess.run(["g++", "-std=c++17", "-g", "-O1", "-fsanitize=thread", f"-DLOOK={look}",
                        f"-I{CSRC}", str(src), "-o", str(exe), "-lpthread"], capture_output=True)
    if r.returncode:
        pytest.skip("no thread sanitizer")
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    if "FATAL: ThreadSanitizer" in r.stderr:  # it cannot map its shadow memory here
        pytest.skip("the thread sanitizer does not start")
    assert r.stdout == "3.5\n"
    assert ("data race" in r.stderr) == race


def test_the_host_waits_so():
    wait = (CSRC / "lfx_ctx.cu").read_text().split("int host_wait(")[1].split("\n}\n")[0]
    assert "host_number(" in wait and "volatile" not in wait

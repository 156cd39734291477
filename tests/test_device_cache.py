"""Whether idle device blocks serve a list of requests (csrc/dbuf.h, `dcache::holds`): the rule
by which a handle may leave out the look at the free memory.  Host code alone, compiled
with nvcc; the blocks are made-up addresses that no one touches."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "sdpx.jl_b200", "csrc")

PROGRAM = r"""
#include "dbuf.h"
#include <cstdio>
using namespace sdpx;
static int bad = 0;
static void check(bool got, bool want, const char* what) {
  if (got != want) std::printf("%s: %d\n", what, (int)got), ++bad;
}
static void idle(size_t bytes, int dev, size_t address) {
  dcache::cache().idle.insert({bytes, {dev, reinterpret_cast<void*>(address)}});
}
int main() {
  const size_t M = 1 << 20;
  check(dcache::holds(0, {M}), false, "nothing idle");
  check(dcache::holds(0, {}), true, "nothing asked");
  idle(8 * M, 0, 0x1000);
  check(dcache::holds(0, {8 * M}), true, "the same size");
  check(dcache::holds(0, {8 * M + 1}), false, "too small by a byte");
  check(dcache::holds(0, {6 * M}), true, "within a quarter and 1 MB");
  check(dcache::holds(0, {5 * M}), false, "much too large");
  check(dcache::holds(1, {8 * M}), false, "another device's");
  check(dcache::holds(0, {8 * M, 8 * M}), false, "one block for two");
  idle(8 * M, 1, 0x2000);
  check(dcache::holds(0, {8 * M, 8 * M}), false, "two, one on another device");
  idle(8 * M, 0, 0x3000);
  check(dcache::holds(0, {8 * M, 8 * M}), true, "two for two");
  check(dcache::holds(0, {8 * M, 7 * M, 7 * M}), false, "two for three");
  dcache::cache().idle.clear();
  return bad;
}
"""


def test_requests_against_idle_blocks(tmp_path):
    sys.path.insert(0, os.path.join(ROOT, "sdpx.jl_b200"))
    from build import nvcc
    try:
        compiler = nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    src, exe = tmp_path / "cache.cu", tmp_path / "cache"
    src.write_text(PROGRAM)
    subprocess.run([compiler, "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I", CSRC, "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout

"""The rule that sends a channel move to the kernels with 32-bit group counters, at its limits (compiled for the host):
a counter that is one step past the last group must not have wrapped round, or its loop would never end."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "vortexlab_b200", "csrc")

PROGRAM = r"""
#include "vl_groups.hpp"
#include <cstdio>
#include <initializer_list>
int main() {
  const long long groups[] = {1, 0x7ffffffeLL, 0x7fffffffLL, 0x80000000LL, 0xffffffffLL - vl::kMoveThreads, 0xfffffffeLL, 0xffffffffLL};
  for (long long g : groups)
    for (int v : {4, 8}) {
      const bool in = vl::move_grouped(0, 16, g * v, 8, 16, 8, v);
      const bool ends = g + vl::kMoveThreads <= 0xffffffffLL;   // the last counter value fits 32 bits
      std::printf("%d %d\n", (int)in, (int)ends);
      if (in && !ends) return 1;
      if (in != (g <= 0x7fffffffLL)) return 2;
    }
  if (vl::move_grouped(8, 16, 64, 8, 16, 8, 4) || vl::move_grouped(0, 16, 64, 6, 16, 8, 4) || vl::move_grouped(0, 0, 64, 8, 18, 8, 4) ||
      vl::move_grouped(0, 0, 64, 8, 16, 2, 4)) return 3;
  return 0;
}
"""


def test_limits(tmp_path):
    src = tmp_path / "groups.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "groups")
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_the_kernels_use_the_rule():
    with open(os.path.join(CSRC, "vl_nn.cu")) as f:
        t = f.read()
    for name in ("up2", "up2_bwd", "copy_channels", "slice_channels"):
        body = t[t.index(f"int vl_nn_{name}("):]
        assert body.index("if (grouped(") < body.index(f"k_{name}_v<<<")
    assert "return vl::move_grouped(" in t

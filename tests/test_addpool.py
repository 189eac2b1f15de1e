"""The host threads that add forces and copy states as their pieces land (csrc/pmb_addpool.h): results,
and a failed wait.  The waits are the test's own; no device is needed."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "protomol3_b200", "csrc")
CODE = r"""
#include <cstdio>
#include "pmb_addpool.h"
static int ok(const void *, int) { return 0; }
static int third_fails(const void *e, int c) { return c < 2 ? 0 : *static_cast<const int *>(e); }
int main() {
  const int n = 1003, chunk = 251, pieces = 4;
  const int code = 77;
  for (int threads = 1; threads <= 4; threads++) {
    pmb::AddPool pool;
    pool.start(threads, [](int) {}, 0);
    for (int round = 0; round < 3; round++) {
      std::vector<double> src(n), dst(n, 1.0);
      for (int i = 0; i < n; i++) src[i] = i;
      if (pool.run(dst.data(), src.data(), n, chunk, pieces, ok, nullptr)) return 1;
      for (int i = 0; i < n; i++) if (dst[i] != 1.0 + i) return 2;
      if (pool.run(dst.data(), src.data(), n, chunk, pieces, ok, nullptr, true)) return 3;
      for (int i = 0; i < n; i++) if (dst[i] != i) return 4;
      std::vector<double> kept(n, -1.0);
      if (pool.run(kept.data(), src.data(), n, chunk, pieces, third_fails, &code, true) != code) return 5;
      for (int i = 0; i < n; i++) if (kept[i] != (i < 2 * chunk ? i : -1.0)) return 6;
    }
  }
  std::puts("ok");
  return 0;
}
"""


def test_pieces_and_failed_waits(tmp_path):
    (tmp_path / "t.cpp").write_text(CODE)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-pthread", "-I", CSRC, "-o", str(tmp_path / "t"), str(tmp_path / "t.cpp")])
    out = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout == "ok\n", out

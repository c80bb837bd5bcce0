"""ulps_of (kernels.cuh), the whole ulps of a sum that a term rounds to, on the host:
against long double over terms from far above the sum's binade to far below it, of
both signs, subnormal ones among them, with every undefined operation an error."""
import os
import subprocess

from brawl_gb300 import build as B

SOURCE = r"""
#include "kernels.cuh"
#include <cmath>
#include <cstdio>
#include <cstring>
int main() {
  unsigned long long s = 88172645463325252ull;
  auto word = [&]() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; };
  const unsigned long long signed_fraction = 0x800fffffffffffffull;
  long settled = 0;
  for (long i = 0; i < 1000000; ++i) {
    const int ex = 61 + (int)(word() % 1900), below = (int)(word() % 90) - 20;
    const int tx = ex - below < 0 ? 0 : ex - below > 2047 ? 2047 : ex - below;
    const long long e = (long long)((word() & signed_fraction) | (unsigned long long)ex << 52);
    const long long t = (long long)((word() & signed_fraction) | (unsigned long long)tx << 52);
    bool ok = true;
    const long long k = (long long)brawl::ulps_of(t, e, ok);
    if (!ok) continue;
    ++settled;
    double td, ed;
    std::memcpy(&td, &t, 8);
    std::memcpy(&ed, &e, 8);
    // in ulps of e, in the direction in which e's bits grow
    long double q = std::ldexp((long double)td, 1075 - ex);
    if (ed < 0) q = -q;
    if ((long double)k != std::nearbyint(q)) {
      std::printf("term %a, sum %a: %lld\n", td, ed, k);
      return 1;
    }
  }
  std::printf("%ld settled\n", settled);
  return settled > 500000 ? 0 : 2;
}
"""


def test_ulps_of_a_term(tmp_path):
    src, exe = tmp_path / "ulps.cu", tmp_path / "ulps"
    src.write_text(SOURCE)
    subprocess.run([B.nvcc(), *B.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", B.CSRC, "-Xcompiler",
                    "-fsanitize=undefined,-fno-sanitize-recover=undefined", "-o", str(exe), str(src), "-lubsan"],
                   check=True, env=dict(os.environ))
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr

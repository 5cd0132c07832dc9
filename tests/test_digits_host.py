"""dg::digits7 (csrc/mh_digits.cuh), the digits of the FP64 tensor-core products, compiled for the host
with signed overflow trapped: over the whole range |X| < 2^55, its ends above all."""
import os
import random
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "marinehydro.jl_gb300", "csrc")

MAIN = """
#include <cstdio>
%s
int main() {
  long long X;
  while (std::scanf("%%lld", &X) == 1) {
    int d[kDigits7];
    digits7(X, d);
    for (int p = 0; p < kDigits7; ++p) std::printf("%%d ", d[p]);
    std::printf("\\n");
  }
}
"""


def test_digits7_over_its_range(tmp_path):
    with open(os.path.join(CSRC, "mh_digits.cuh")) as f:
        body = re.search(r"constexpr int kDigits7 = 7;.*?\n}\n", f.read(), re.S).group(0)
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(MAIN % body.replace("__device__ __forceinline__", "static"))
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=signed-integer-overflow",
                    "-fsanitize-undefined-trap-on-error", str(src), "-o", str(exe)], check=True)
    rng = random.Random(5)
    top = 2 ** 55
    xs = [0, 1, -1, top - 1, 1 - top]
    for bits in range(55):
        xs += [s * (top - 2 ** bits) + e for s in (1, -1) for e in (-1, 0, 1)]
        xs += [s * 2 ** bits + e for s in (1, -1) for e in (-1, 0, 1)]
    xs += [rng.randrange(1 - top, top) for _ in range(2000)]
    xs = [x for x in xs if abs(x) < top]
    out = subprocess.run([str(exe)], input="\n".join(map(str, xs)), check=True, capture_output=True, text=True).stdout
    for x, line in zip(xs, out.splitlines(), strict=True):
        d = [int(v) for v in line.split()]
        assert all(-128 <= v <= 128 for v in d) and sum(v * 256 ** (6 - p) for p, v in enumerate(d)) == x, (x, d)

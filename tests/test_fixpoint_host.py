"""fx::to_q (csrc/mh_fixpoint.cuh) over its whole range, compiled for the host with signed overflow
trapped: the exact term's tables take it to x 2^64 = -2^63, which has no positive counterpart."""
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "marinehydro.jl_gb300", "csrc")

MAIN = """
#include <cstdio>
#include <cstdlib>
#include <cstring>
static long long __double_as_longlong(double x) { long long b; std::memcpy(&b, &x, 8); return b; }
%s
int main(int argc, char** argv) {
  for (int i = 1; i + 1 < argc; i += 2) std::printf("%%lld\\n", to_q(std::strtod(argv[i], nullptr), std::atoi(argv[i + 1])));
}
"""


def test_to_q_over_its_range(tmp_path):
    with open(os.path.join(CSRC, "mh_fixpoint.cuh")) as f:
        body = re.search(r"__device__ __forceinline__ long long to_q\(.*?\n}\n", f.read(), re.S).group(0)
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(MAIN % body.replace("__device__ __forceinline__", "static"))
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=signed-integer-overflow",
                    "-fsanitize-undefined-trap-on-error", str(src), "-o", str(exe)], check=True)
    cases = [(-0.5, 64), (0.5 - 2.0 ** -54, 64), (-0.5 + 2.0 ** -54, 64), (-0.5, 63), (7.999, 60), (-1.0, 62),
             (0.0, 64), (-0.0, 64), (1e-320, 64), (2.0 ** -64, 64), (-(2.0 ** -65), 64), (0.3, 60), (-0.3, 60)]
    args = [s for x, q in cases for s in (repr(x), str(q))]
    got = [int(v) for v in subprocess.run([str(exe), *args], check=True, capture_output=True, text=True).stdout.split()]

    def trunc(x, s):
        num, den = abs(x).as_integer_ratio()
        return (-1 if x < 0 else 1) * (num * 2 ** s // den)

    # subnormal numbers count as 0
    assert got == [0 if abs(x) < 2.0 ** -1022 else trunc(x, s) for x, s in cases]

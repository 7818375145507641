"""Launch limits of kernels are raised on every device that launches them.

A kernel's shared-memory limit (and its leave to run in clusters of 16) is an
attribute of the kernel on one device.  func_limits.hpp is compiled here against
stand-ins for the two runtime calls it makes, with contexts on two devices in
turn; and no kernel of the Lanczos or tensor-core files raises a limit elsewhere.
"""
import re
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "nssdmrg_gb300" / "csrc"

PROGRAM = r"""
#include "func_limits.hpp"
#include <cstdio>
static int current = 0;
extern "C" cudaError_t cudaGetDevice(int *d) { *d = current; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) {
    std::printf("set %d %ld %d %d\n", current, (long)f, (int)a, v);
    return v > 300000 ? cudaErrorInvalidValue : cudaSuccess;
}
int main() {
    long fn, bytes;
    while (std::scanf("%d %ld %ld", &current, &fn, &bytes) == 3)
        std::printf("rc %d\n", (int)nss::allow_smem((const void *)fn, (size_t)bytes));
}
"""


def test_each_device_gets_the_limit(tmp_path):
    (tmp_path / "p.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", "-I/usr/local/cuda/include", "-o", str(tmp_path / "p"),
                    str(tmp_path / "p.cpp")], check=True)
    a, b = 16, 32                                        # two kernels
    asked = [(0, a, 40000), (0, a, 172032), (1, a, 172032), (0, a, 172032), (1, b, 100000), (0, a, 100000),
             (1, a, 200000), (0, a, 172032), (1, a, 400000), (1, a, 400000)]
    out = subprocess.run([str(tmp_path / "p")], input="".join("%d %d %d\n" % x for x in asked), text=True,
                         capture_output=True, check=True).stdout.split("\n")
    rc = [int(x.split()[1]) for x in out if x.startswith("rc")]
    got = [tuple(map(int, x.split()[1:])) for x in out if x.startswith("set")]
    assert rc[:8] == [0] * 8 and rc[8] != 0 and rc[9] != 0
    assert [(d, f, v) for d, f, _, v in got] == [(0, a, 172032), (1, a, 172032), (1, b, 100000), (1, a, 200000),
                                                 (1, a, 400000), (1, a, 400000)]
    assert len({x[2] for x in got}) == 1


def test_limits_are_raised_there_alone():
    for name in ("k_lanczos.cu", "k_sector_mma.cu", "k_sector_split.cu"):
        assert "cudaFuncSetAttribute" not in (CSRC / name).read_text(), name
    # elsewhere it is set before each launch; nothing remembers that for the process
    for f in CSRC.glob("*.c*"):
        src = f.read_text()
        for m in re.finditer(r"cudaFuncSetAttribute", src):
            assert not re.search(r"static std::atomic<bool>|static bool", src[max(0, m.start() - 300):m.start()]), f.name

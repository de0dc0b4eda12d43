"""Index arithmetic of the kernels at the ends of its range (csrc/lp_index.h, compiled for the host)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

WALK = """
    // every block of 128 entries: the entries it takes, those it looks at one round ahead and the
    // number of rounds, near the end of the walk
    const long long n = atoll(argv[1]), blocks = atoll(argv[2]), width = 128, stride = blocks * width;
    const long long skip = n / stride > 3 ? n / stride - 3 : 0;
    for (int b = 0; b < blocks; b += blocks > 1 ? (int)blocks - 1 : 1) {
        ListWalk w(b, (int)blocks, (int)width, (int)n);
        for (long long r = 0; r < skip; ++r) w.next();
        long long at = b * width + skip * stride;
        for (int rounds = 0; rounds < 6; ++rounds, at += stride, w.next()) {
            if (w.more() != (at < n)) return puts("more"), 0;
            if (!w.more()) break;
            for (int ahead = 0; ahead < 2; ++ahead)
                for (int i : {0, 1, 126, 127}) {
                    const long long e = at + ahead * stride + i;
                    if (w.entry(ahead, i) != (e < n ? e : -1)) return puts("entry"), 0;
                }
        }
        if (w.more()) return puts("end"), 0;
    }
    return puts("ok"), 0;
"""

BARRIER = """
    // barriers k ... of a run: arrivals before, at and up to one barrier after
    const uint32_t k0 = (uint32_t)atoll(argv[1]), blocks = (uint32_t)atoll(argv[2]);
    unsigned long long total = (unsigned long long)k0 * blocks;
    for (uint32_t k = k0; k != k0 + 3; ++k, total += blocks)
        for (uint32_t missing = 0; missing <= blocks; ++missing) {
            if (barrier_waits((uint32_t)(total - missing), k, blocks) != (missing > 0)) return puts("waits"), 0;
            if (barrier_waits((uint32_t)(total + missing), k, blocks)) return puts("closed"), 0;
        }
    return puts("ok"), 0;
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("index")

    def build(name, body):
        src, exe = d / (name + ".cpp"), d / name
        src.write_text('#include <cstdio>\n#include <cstdlib>\n#include <initializer_list>\n#include "lp_index.h"\n'
                       "using namespace galp;\nint main(int argc, char **argv)\n{" + body + "}\n")
        if not exe.exists():
            subprocess.run([cxx, "-O1", "-std=c++17", "-fwrapv", "-I", os.path.join(ROOT, "galp_gb300", "csrc"),
                            str(src), "-o", str(exe)], check=True)

        def run(*args):
            return subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True,
                                  timeout=60).stdout.split()
        return run
    return build


@pytest.mark.parametrize("n", [1, 127, 128, 129, 155647, 155648, 155649, 2**31 - 155649, 2**31 - 155648,
                               2**31 - 129, 2**31 - 2, 2**31 - 1])
@pytest.mark.parametrize("blocks", [1, 152 * 8, 2048])
def test_list_walk(program, n, blocks):
    assert program("walk", WALK)(n, blocks) == ["ok"]


@pytest.mark.parametrize("blocks", [1, 16, 152, 256])
@pytest.mark.parametrize("k", [1, 2, 1000, 2**31 // 152, 2**32 // 152, 2**32 // 152 - 2, 2**32 // 256 - 1,
                               2**32 // 16 - 1, 2**32 // 16, 2**32 - 2])
def test_barrier_count_wraps(program, k, blocks):
    # a run without early exit has two barriers an iteration and as many iterations as asked for
    assert program("barrier", BARRIER)(k, blocks) == ["ok"]

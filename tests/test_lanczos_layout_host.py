"""The places of a Lanczos run's small device buffers, without a GPU: csrc/lanczos_layout.h compiled as plain
C++.  Complex numbers are read 16 bytes at a time, so they lie on 16-byte boundaries, and the partial sums
of every number of basis vectors fit in front of them."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "exactdiagonalization.jl_gb300", "csrc")


def run_cpp(tmp_path, body):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text('#include "lanczos_layout.h"\n#include <cmath>\n#include <cstdio>\n#include <vector>\n'
                   "using namespace edgpu;\nint main() {\n" + body + "\n}\n")
    subprocess.run([cxx, "-O1", "-std=c++17", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()


def test_places(tmp_path):
    out = run_cpp(tmp_path, """
        long bad = 0, checked = 0;
        for (int sms : {1, 7, 132, 148, 152, 160}) {
            for (int m = 1; m <= 12000; m += m < 200 ? 1 : 7) {
                const LanczosSmall o = lanczos_small(m, sms);
                ++checked;
                if (o.scratch % 2 || o.h % 2) ++bad;
                if (o.hmax < o.h + 2 * (size_t)(m + 1) || o.tickets < o.hmax + o.n_groups || o.total < o.tickets + (o.n_groups + 1) / 2) ++bad;
                for (int64_t n : {1ll, 255ll, 100000ll, 1ll << 32})
                    for (int k = 1; k <= m + 1; k += 1 + k / 8) {
                        const size_t g = lz_groups(k), rb = lz_row_blocks(n, (int)g, sms);
                        if (g > o.n_groups || o.scratch + 2 * g * rb * LZ_G + rb > o.h) ++bad;
                    }
                if (o.scratch + 2 * (size_t)LZ_MAX_BLOCKS > o.h || o.scratch + 2 * (size_t)RED_BLOCKS > o.h) ++bad;
            }
        }
        std::printf("%ld %ld", bad, checked);
    """)
    assert out[0] == "0" and int(out[1]) > 10000, out

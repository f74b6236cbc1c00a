"""The places of a Lanczos run's small device buffers and the rule for the precision of its correction, without
a GPU: csrc/lanczos_layout.h compiled as plain C++.  Complex numbers are read 16 bytes at a time, so they lie on 16-byte boundaries, and the partial sums
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


def test_single_precision_rule(tmp_path):
    """Where the rule just allows it, the correction's sum in single precision (the kernel's order: chains over
    chunks of LZ_CHUNK vectors, vectors cut and coefficients rounded to 24 bits) is within 2^-54 of the
    vector's norm of the sum in long double.  Equal vectors add up most."""
    out = run_cpp(tmp_path, """
        std::srand(1);
        auto rnd = [] { return (double)std::rand() / RAND_MAX + 1e-10 * std::rand() / RAND_MAX; };
        auto cut = [](double v) { int e; const double m = std::frexp(v, &e); return (float)std::ldexp(std::trunc(std::ldexp(m, 24)), e - 24); };
        long bad = 0, allowed = 0;
        for (int K : {1, 2, 8, 50, 95, 100, 200, 255, 256, 257, 300, 511, 512, 513, 2000})
            for (int kind = 0; kind < 4; ++kind) {
                const int N = 64;
                // the largest hmax the rule allows beside |w1| = 1, by bisection of the exponent and mantissa
                double lo = 0x1p-200, hi = 1.0;
                for (int it = 0; it < 200; ++it) {
                    const double mid = std::sqrt(lo * hi);
                    (lz_single_precision(K, mid, 1.0) ? lo : hi) = mid;
                }
                const double H = lo;
                allowed += lz_single_precision(K, H, 1.0);
                std::vector<double> vx(N), vy(N);
                auto fresh = [&] {
                    double n2 = 0.0;
                    for (int i = 0; i < N; ++i) {
                        vx[i] = kind & 1 ? rnd() - 0.5 : rnd() + 0.1;
                        vy[i] = kind & 1 ? rnd() - 0.5 : -rnd() - 0.1;
                        n2 += vx[i] * vx[i] + vy[i] * vy[i];
                    }
                    for (int i = 0; i < N; ++i) vx[i] /= std::sqrt(n2), vy[i] /= std::sqrt(n2);
                };
                fresh();
                const int e = std::ilogb(H);
                std::vector<float> cx(N, 0.f), cy(N, 0.f);
                std::vector<double> sx(N, 0.0), sy(N, 0.0);
                std::vector<long double> tx(N, 0.0L), ty(N, 0.0L);
                for (int k = 0; k < K; ++k) {
                    if (kind & 2) fresh();
                    const double hx = H * (0.5 + 0.5 * rnd()), hy = H * (0.5 + 0.5 * rnd());
                    const float fx = (float)std::ldexp(hx, -e), fy = (float)std::ldexp(hy, -e);
                    for (int i = 0; i < N; ++i) {
                        const float ux = cut(vx[i]), uy = cut(vy[i]);
                        cx[i] = std::fmaf(fx, ux, cx[i]);
                        cx[i] = std::fmaf(-fy, uy, cx[i]);
                        cy[i] = std::fmaf(fx, uy, cy[i]);
                        cy[i] = std::fmaf(fy, ux, cy[i]);
                        tx[i] += (long double)hx * vx[i] - (long double)hy * vy[i];
                        ty[i] += (long double)hx * vy[i] + (long double)hy * vx[i];
                        if ((k + 1) % LZ_CHUNK == 0 || k + 1 == K) {
                            sx[i] += std::ldexp((double)cx[i], e), sy[i] += std::ldexp((double)cy[i], e);
                            cx[i] = cy[i] = 0.f;
                        }
                    }
                }
                long double err = 0.0L;
                for (int i = 0; i < N; ++i) err += (sx[i] - tx[i]) * (sx[i] - tx[i]) + (sy[i] - ty[i]) * (sy[i] - ty[i]);
                if (!(std::sqrt((double)err) <= 0x1p-54)) ++bad;
            }
        bad += lz_single_precision(5, NAN, 1.0) + lz_single_precision(5, INFINITY, 1.0) + lz_single_precision(5, 0.0, 1.0) +
               lz_single_precision(5, 1e-300, 1.0) + lz_single_precision(5, 1e-20, NAN);
        std::printf("%ld %ld", bad, allowed);
    """)
    assert out == ["0", "60"], out

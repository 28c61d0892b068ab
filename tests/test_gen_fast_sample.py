"""The device generator's sampler (gen.h, fast_sample) against its definition,
Zipf::sample, draw by draw: table sizes from 1 to 2^27, every skew the
generator takes, draws over the whole range and close to its upper end, where
the result is near a whole number; and its polynomial against long double,
whose error has to stay inside the bound that its cell carries.  CPU only."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHECK = r"""
#include <cmath>
#include <cstdio>
#include <initializer_list>
#include "gen.h"
using namespace ltpg::gen;
int main() {
    static FixTables tab;
    static PolyCell cells[POLY_CELLS];
    fix_tables_fill(tab);
    for (uint64_t n : {1ull, 2ull, 3ull, 20ull, 1000ull, 100000ull, 3000000ull, 134217728ull})
        for (double theta : {0.0, 1e-9, 0.3, 0.6, 0.9, 0.99, 0.9999, 0.9999999}) {
            Zipf z;
            z.n = n;
            z.theta = theta;
            if (theta != 0.0) {  // zeta(n): summed to 100,000, the rest by its integral (any value serves here)
                double sum = 0;
                const uint64_t m = n < 100000 ? n : 100000;
                for (uint64_t i = 1; i <= m; ++i) sum += 1.0 / std::pow((double)i, theta);
                sum += (std::pow((double)n, 1 - theta) - std::pow((double)m, 1 - theta)) / (1 - theta);
                z.zetan = sum;
                z.alpha = 1.0 / (1.0 - theta);
                z.eta = (1.0 - std::pow(2.0 / (double)n, 1.0 - theta)) / (1.0 - (1.0 + std::pow(0.5, theta)) / sum);
                z.half_pow = std::pow(0.5, theta);
            }
            const FastZipf f = fast_zipf(z, cells);
            long bad = 0;
            double part = 0;
            Rng r(n + (uint64_t)(theta * 1e6));
            for (int i = 0; i < 60000; ++i) {
                uint64_t draw = r.next();
                if (i % 3 == 0) draw = ~0ull - (draw >> (16 + i % 44));
                const double u = (double)(draw >> 11) * 0x1.0p-53, uz = u * z.zetan;
                uint64_t want;
                if (theta == 0.0) want = mulhi64(draw, n);
                else if (uz < 1.0) want = 0;
                else if (uz < 1.0 + z.half_pow) want = n > 1 ? 1 : 0;
                else {
                    want = fix_pow_floor(tab, z.eta * u - z.eta + 1.0, z.alpha, n);
                    if (want >= n) want = n - 1;
                }
                bad += fast_sample(f, cells, tab, draw) != want;
                if (!f.fast || (draw >> 11) < f.t2) continue;
                uint32_t le;
                const uint64_t val = poly_rank(cells, f.sh, draw >> 11, le);
                if (le == POLY_NEVER) continue;
                const long double b = 1.0L - (long double)z.eta * (1.0L - (long double)u);
                const long double ref = (long double)n * powl(b, (long double)z.alpha) * (long double)(1ull << 36);
                part = std::fmax(part, (double)(fabsl((long double)val - ref) / (long double)(1ull << le)));
            }
            std::printf("%llu %g %ld %g\n", (unsigned long long)n, theta, bad, part);
        }
}
"""


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    d = tmp_path_factory.mktemp("fast")
    src, exe = d / "check.cpp", d / "check"
    src.write_text(CHECK)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "ltpg_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    return [ln.split() for ln in out.splitlines()]


def test_same_ranks(lines):
    assert len(lines) == 64
    assert all(int(ln[2]) == 0 for ln in lines), [ln for ln in lines if int(ln[2])]


def test_cells_bound_their_error(lines):
    # half of a cell's bound is for the definition's own rounding
    assert all(float(ln[3]) < 0.5 for ln in lines), lines


"""The search tables of sampled spectra (csrc/spec_lut.h), compiled for the host: for every table they give
the index of the plain search, at its entries, beside them, between them and beyond both ends."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <limits>
#include <random>
#include "spec_lut.h"
using namespace liar_gpu;
static long checked = 0, bad = 0, tables = 0;
static void check(std::vector<float> a, bool table) {
    std::vector<uint32_t> luts(7);  // (tables are appended)
    const SearchLut t = add_lut(luts, a.data(), a.size());
    if ((t.scale != 0.0f) != table) ++bad;
    tables += t.scale != 0.0f;
    const float inf = INFINITY;
    std::vector<float> x{-inf, inf, NAN, 0.0f, -1.0f, 1e30f, -1e30f};
    for (float v : a) {
        x.push_back(v);
        x.push_back(std::nextafter(v, -inf));
        x.push_back(std::nextafter(v, inf));
    }
    std::mt19937 g(1);
    std::uniform_real_distribution<double> u(-0.05, 1.05);
    for (int i = 0; i < 20000; ++i) x.push_back((float)(a.front() + u(g) * ((double)a.back() - a.front())));
    for (int c = 0; c <= kLutCells; ++c) {  // the cells' edges
        const float e = (float)(a.front() + (double)c * ((double)a.back() - a.front()) / kLutCells);
        x.push_back(e);
        x.push_back(std::nextafter(e, -inf));
        x.push_back(std::nextafter(e, inf));
    }
    for (float v : x) {
        ++checked;
        bad += lut_upper_bound(luts.data(), t, a.data(), (int)a.size(), v) != upper_bound_in(a.data(), 0, (int)a.size(), v);
    }
}
int main() {
    std::mt19937 g(2);
    std::uniform_real_distribution<float> u(0.0f, 1.0f);
    check({300e-9f, 900e-9f}, true);
    check({380e-9f, 550e-9f, 720e-9f}, true);
    check({0.0f, 0.0f, 0.25f, 0.25f, 1.0f, 1.0f}, true);   // a cdf with flat ends
    check({5.0f, 5.0f, 5.0f}, false);                       // no range
    check({2.0f, 1.0f}, false);
    check({1.0f, std::numeric_limits<float>::quiet_NaN(), 3.0f}, false);
    check({-3e38f, 3e38f}, false);                          // the range overflows
    check({1.0f, std::nextafter(1.0f, 2.0f)}, true);
    check({0.0f, 1e-42f}, false);                           // its reciprocal does
    for (int n : {3, 17, 95, 300, 471, 4001, 65535, 70000}) {
        std::vector<float> even, uneven, cdf, cluster;
        double s = 0.0;
        for (int i = 0; i < n; ++i) {
            even.push_back((float)(360e-9 + 470e-9 * i / (n - 1)));
            uneven.push_back(u(g));
            cluster.push_back(i == 0 ? 0.0f : i == n - 1 ? 2.0f : 1.0f + 1e-6f * u(g));
            s += std::exp(-30.0 * (i / (double)n - 0.5) * (i / (double)n - 0.5));
            cdf.push_back((float)s);
        }
        std::sort(uneven.begin(), uneven.end());
        std::sort(cluster.begin(), cluster.end());
        for (float& v : cdf) v /= (float)s;
        for (const auto& a : {even, uneven, cdf, cluster}) check(a, n <= 65535);
    }
    std::printf("%ld tables, %ld searches, %ld bad\n", tables, checked, bad);
    return bad != 0;
}
"""


def test_search_tables_give_the_plain_search(tmp_path):
    (tmp_path / "lut.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "liar_b200" / "csrc"),
                    str(tmp_path / "lut.cpp"), "-o", str(tmp_path / "lut")], check=True)
    r = subprocess.run([str(tmp_path / "lut")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr

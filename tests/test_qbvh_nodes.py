"""The tree's quantised child boxes (csrc/qbvh.h, csrc/qbvh_build.cpp), checked on the host: every
primitive's box lies inside the decoded box of each node slot above it, empty slots are inverted, and
every primitive is reached once."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>
#include "qbvh.h"
using namespace liar_gpu;
static QBVHHost q;
static std::vector<int> seen;
static std::vector<float> V, S;
static std::vector<uint32_t> T;
static long bad = 0, empty = 0, slots = 0;
struct Range { double lo[3], hi[3]; };
static Range prim(int i) {
    Range r;
    const int nt = (int)(T.size() / 3);
    for (int a = 0; a < 3; ++a) {
        if (i >= nt) {
            const float* s = &S[4 * (i - nt)];
            r.lo[a] = (double)s[a] - s[3];
            r.hi[a] = (double)s[a] + s[3];
        } else {
            const float x = V[3 * T[3 * i] + a], y = V[3 * T[3 * i + 1] + a], z = V[3 * T[3 * i + 2] + a];
            r.lo[a] = std::fmin(x, std::fmin(y, z));
            r.hi[a] = std::fmax(x, std::fmax(y, z));
        }
    }
    return r;
}
static Range walk(int node) {
    const QNode& n = q.nodes[node];
    Range all;
    for (int a = 0; a < 3; ++a) all.lo[a] = INFINITY, all.hi[a] = -INFINITY;
    for (int c = 0; c < 4; ++c) {
        const uint32_t w = (uint32_t)n.child[c];
        Range r;
        ++slots;
        if (w & 0x80000000u) {
            const uint32_t count = (w >> 27) & 15u, first = w & 0x07ffffffu;
            if (count == 0) {
                ++empty;
                for (int a = 0; a < 3; ++a)
                    if (((n.lo[a] >> (8 * c)) & 255u) != 255u || ((n.hi[a] >> (8 * c)) & 255u) != 0u) ++bad;
                continue;
            }
            for (int a = 0; a < 3; ++a) r.lo[a] = INFINITY, r.hi[a] = -INFINITY;
            for (uint32_t k = first; k < first + count; ++k) {
                int i;
                std::memcpy(&i, &q.tris[k].v0.w, 4);
                ++seen[i];
                const Range p = prim(i);
                for (int a = 0; a < 3; ++a) r.lo[a] = std::fmin(r.lo[a], p.lo[a]), r.hi[a] = std::fmax(r.hi[a], p.hi[a]);
            }
        } else {
            r = walk((int)w);
        }
        for (int a = 0; a < 3; ++a) {
            const uint32_t lq = (n.lo[a] >> (8 * c)) & 255u, hq = (n.hi[a] >> (8 * c)) & 255u;
            uint32_t lb = 0x40000000u | (lq << 16), hb = 0x40000000u | (hq << 16);
            float lv, hv;
            std::memcpy(&lv, &lb, 4);
            std::memcpy(&hv, &hb, 4);
            if (lv != plane_value(lq) || hv != plane_value(hq)) ++bad;
            if (n.scl[a] > 0.0f) {
                if (!((double)n.org[a] + (double)lv * n.scl[a] < r.lo[a])) ++bad;
                if (!((double)n.org[a] + (double)hv * n.scl[a] > r.hi[a])) ++bad;
            } else if (lq != 0 || hq != 255) {
                ++bad;
            }
            all.lo[a] = std::fmin(all.lo[a], r.lo[a]);
            all.hi[a] = std::fmax(all.hi[a], r.hi[a]);
        }
    }
    return all;
}
int main(int argc, char** argv) {
    const int nt = std::atoi(argv[1]), ns = std::atoi(argv[2]), leaf = std::atoi(argv[3]);
    const double offset = std::atof(argv[4]), size = std::atof(argv[5]), flat = std::atof(argv[6]);
    std::mt19937 rng(7);
    std::uniform_real_distribution<double> u(-1, 1);
    for (int i = 0; i < nt; ++i) {
        double c[3] = {u(rng), u(rng), u(rng) * flat};
        for (int k = 0; k < 3; ++k)
            for (int a = 0; a < 3; ++a) V.push_back((float)(offset + size * (c[a] + 0.05 * u(rng) * (a == 2 ? flat : 1.0))));
        for (int k = 0; k < 3; ++k) T.push_back(3 * i + k);
    }
    for (int i = 0; i < ns; ++i) {
        for (int a = 0; a < 3; ++a) S.push_back((float)(offset + size * u(rng)));
        S.push_back((float)(size * (0.01 + 0.1 * std::fabs(u(rng)))));
    }
    BuildOptions o;
    o.max_leaf_size = leaf;
    char msg[256] = {0};
    const int rc = build_qbvh(V.data(), V.size() / 3, T.data(), nt, S.empty() ? nullptr : S.data(), ns, o, q, msg, sizeof(msg));
    if (rc) { std::printf("build failed: %s\n", msg); return 2; }
    seen.assign(nt + ns, 0);
    walk(0);
    for (int s : seen) bad += s != 1;
    std::printf("%ld slots, %ld empty, %ld bad\n", slots, empty, bad);
    free_qbvh(q);
    return bad ? 1 : 0;
}
"""


@pytest.fixture(scope="module")
def walker(tmp_path_factory):
    d = tmp_path_factory.mktemp("qbvh")
    (d / "walk.cpp").write_text(PROGRAM)
    csrc = ROOT / "liar_b200" / "csrc"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(csrc), "-I", str(ROOT / "include"),
                    str(d / "walk.cpp"), str(csrc / "qbvh_build.cpp"), "-o", str(d / "walk"), "-lpthread"], check=True)
    return d / "walk"


@pytest.mark.parametrize("args", [
    (1, 0, 4, 0, 1, 1), (2, 0, 1, 0, 1, 1), (5, 1, 4, 0, 1, 1), (3000, 40, 1, 0, 1, 1), (3000, 0, 4, 0, 1, 1),
    (3000, 0, 8, 1000, 1, 1),          # far from the origin: planes of few distinct floats
    (500, 0, 4, 0, 1, 0),              # flat on z
    (500, 0, 4, 0, 1e-30, 1), (500, 0, 4, 0, 1e30, 1),
    (500, 0, 4, 0, 3.2e38, 1),         # the grid would pass the float range
    (0, 200, 4, -5, 2, 1),
], ids=str)
def test_child_boxes_hold_their_primitives(walker, args):
    r = subprocess.run([str(walker), *map(str, args)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr

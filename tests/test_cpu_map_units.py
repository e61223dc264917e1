"""Every row of a constraint map belongs to exactly one work unit, without a GPU.

A small C++ driver compiles csrc/map_units.h with g++, deals the rows of A and
A^T to buckets and units as the table builder and the launchers do, and walks
the units as the kernels' CTAs do, for the launched maps (each in the form that
it asks for) and for the persistent CG, whose kernel applies both maps in one
form.  Layouts where only one of the two asks for the deep form are among
them."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DRIVER = r"""
#include <cstdio>
#include <map>
#include <vector>
#include "map_units.h"
using namespace v2g;

struct Map {
    int nb = 0, width[kMaxBuckets] = {};
    int64_t nslots[kMaxBuckets] = {};
    int nlong = 0, nmid = 0, packed = 0;
    std::vector<int64_t> longs;
};

static Map read_map() {
    int64_t head[2];
    if (std::fread(head, 8, 2, stdin) != 2) throw 1;
    std::vector<int32_t> len(head[0]);
    if (std::fread(len.data(), 4, len.size(), stdin) != len.size()) throw 1;
    Map M;
    M.packed = (int)head[1];
    int64_t count[kMaxBuckets] = {};
    std::map<int64_t, int> same;
    for (int32_t l : len) {
        const int b = row_bucket(head[0], l);
        if (b < kMaxBuckets) count[b]++;
        else M.longs.push_back(l), same[l]++;
    }
    for (int b = 0; b < kMaxBuckets; b++)
        if (count[b]) M.width[M.nb] = kBucketWidths[b], M.nslots[M.nb++] = count[b];
    M.nlong = (int)M.longs.size();
    for (int64_t l : M.longs) M.nmid += row_is_mid(l, same[l]);
    return M;
}

// Rows not taken exactly once by a grid of G CTAs of `threads` in the kernel's form.
static long faults(const Map& M, const Blocks& bl, int B, int threads, int G, bool deep) {
    const int64_t rpp = threads / lanes_of(B);
    const int warps = threads / 32;
    std::vector<std::vector<char>> seen(M.nb);
    for (int i = 0; i < M.nb; i++) seen[i].assign(M.nslots[i], 0);
    std::vector<int> slow(M.nlong, 0);
    for (int blk = 0; blk < G; blk++) {
        int u = blk;
        for (; u < bl.mid; u += G) slow[M.nmid + u]++;
        for (; u < bl.start[0]; u += G) {
            const int k = (u - bl.mid) / bl.midchunks, chunk = (u - bl.mid) % bl.midchunks;
            for (int w = 0; w < warps; w++)
                if (k * warps + w < M.nmid && chunk == 0) slow[k * warps + w]++;
        }
        for (int i = 0; i < M.nb; i++) {
            const int t0 = first_tile(bl, i, blk, G);
            if (t0 < 0) break;
            if (t0 >= bl.start[i + 1] - bl.start[i]) continue;
            const int R = unit_passes(deep, M.width[i]);
            for (int64_t at = (int64_t)t0 * rpp * R; at < M.nslots[i]; at += (int64_t)G * rpp * R)
                for (int64_t p = at; p < at + rpp * R && p < M.nslots[i]; p++) seen[i][p]++;
        }
    }
    long bad = 0;
    for (auto& s : seen)
        for (char c : s) bad += c != 1;
    for (int c : slow) bad += c != 1;
    return bad;
}

int main(int argc, char**) {
    const Map A = read_map(), AT = read_map();
    if (argc > 1) return loop_applies(A, AT) ? 0 : 2;
    for (int B = 1; B <= 40; B++) {
        const int t = map_threads(B);
        for (const Map* M : {&A, &AT}) {
            const bool deep = wants_deep(*M, B, t, 148 * 4);
            const Blocks bl = map_blocks(*M, B, t, deep);
            const int G = std::min(bl.start[kMaxBuckets], 148 * 4);
            std::printf("map %d %ld\n", B, faults(*M, bl, B, t, G, deep));
        }
        if (B > 8) continue;
        for (int sms : {148, 132, 7}) {
            const LoopUnits u = loop_units(A, AT, B, 512, 4 * sms);
            const int G = std::min(sms, std::max(u.A.start[kMaxBuckets], u.AT.start[kMaxBuckets]));
            std::printf("loop %d %ld\n", B, faults(A, u.A, B, 512, G, u.deep) + faults(AT, u.AT, B, 512, G, u.deep));
            if (sms == 148)
                std::printf("mixed %d %d\n", B,
                            wants_deep(A, B, 512, 4 * sms) != wants_deep(AT, B, 512, 4 * sms) ? 1 : 0);
        }
    }
}
"""

# (n, POSITIVITY, CONSTRAIN_SPIN, instance counts where only one map asks for the deep form)
LAYOUTS = [(4, "DQG", True, ()), (7, "DQGT2", True, ()), (10, "DQG", True, ()), (13, "DQG", True, ()),
           (14, "DG", True, (1, 2)), (12, "DQ", True, (7, 8)), (13, "DQ", True, (5, 6)), (15, "D", True, (5,)),
           (10, "DQG", False, (7, 8)), (14, "DQG", False, (1, 2))]


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    d = tmp_path_factory.mktemp("units")
    (d / "units.cpp").write_text(DRIVER)
    exe = str(d / "units")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "v2rdm_casscf_b200", "csrc"),
                    str(d / "units.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("n,positivity,spin,mixed", LAYOUTS)
def test_every_row_has_one_unit(v2g, driver, n, positivity, spin, mixed):
    s = v2g.V2RDMSolver([n], n // 2, n // 2, options=dict(POSITIVITY=positivity, CONSTRAIN_SPIN=spin))
    rowptr, col, val = s.A_csr()
    lens = [np.diff(rowptr), np.bincount(col, minlength=s.dimx)]
    assert len(np.unique(val)) <= 16  # so both tables are packed
    data = b"".join(np.array([len(k), 1], dtype=np.int64).tobytes() + k.astype(np.int32).tobytes() for k in lens)
    out = subprocess.run([driver], input=data, check=True, capture_output=True).stdout.decode()
    rows = [r.split() for r in out.splitlines()]
    assert {int(b) for kind, b, v in rows if kind == "mixed" and int(v)} >= set(mixed)
    assert [r for r in rows if r[0] != "mixed" and int(r[2])] == []


@pytest.mark.parametrize("packed", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_one_kernel_for_both_maps_needs_one_packing(driver, packed):
    data = b"".join(np.array([3, p], dtype=np.int64).tobytes() + np.array([1, 2, 3], dtype=np.int32).tobytes()
                    for p in packed)
    assert (subprocess.run([driver, "applies"], input=data).returncode == 0) == (packed[0] == packed[1])

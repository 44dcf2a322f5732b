"""CPU tests of the list scan's plan (csrc/list_plan.h): what a pass allocates
over the whole range of rows, queries and candidates, and that its sample and
chunks are what the kernels take."""
import itertools
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "similaritysearch.jl_gb300", "csrc")
BUDGET = 1 << 30
FIELDS = ["ok", "splits", "cap", "groups", "per_tile", "keys", "samples", "chunk", "alone", "query_bytes"]

DRIVER = r"""
#include "list_plan.h"
#include <cstdio>
int main() {
    long long n, m, wide, splits, pairs;
    int kk, streamed, locality;
    while (std::scanf("%lld %lld %d %lld %d %lld %lld %d", &n, &m, &kk, &wide, &streamed, &splits, &pairs, &locality) == 8) {
        ssg::ListCall c;
        c.n = n; c.m = m; c.kk = kk; c.wide = wide; c.streamed = streamed; c.splits = splits; c.pairs = pairs;
        ssg::ListPlan p;
        const bool ok = locality ? ssg::list_plan_locality(c, &p) : ssg::list_plan(c, &p);
        std::printf("%d %d %d %d %d %d %lld %lld %lld %lld\n", int(ok), p.splits, p.cap, p.groups, p.per_tile, p.keys,
                    (long long)p.samples, (long long)p.chunk,
                    (long long)ssg::wave_splits((m + 255) / 256, pairs, (n + wide - 1) / wide), (long long)ssg::list_query_bytes(p));
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not found")
    d = tmp_path_factory.mktemp("plan")
    src = d / "plan.cpp"
    src.write_text(DRIVER)
    exe = d / "plan"
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True)

    def run(calls):
        text = "\n".join(" ".join(str(int(v)) for v in c) for c in calls) + "\n"
        out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout
        return [dict(zip(FIELDS, map(int, line.split()))) for line in out.splitlines()]

    return run


def pass_bytes(p):
    """Lists (8 bytes an entry), minima, bounds and counts of a chunk, as the scan addresses them."""
    segs = 2 * p["splits"]
    return p["chunk"] * (segs * p["cap"] * 8 + p["groups"] * 4 + 4 + segs * 4)


N = [2048, 5000, 30_011, 100_000, 1_000_003, 2_000_000, 10_000_000, 100_000_000, 1_000_000_000, 2**32 - 2]
M = [1, 64, 256, 257, 1000, 10_000, 100_000, 1_000_000]
KK = [1, 3, 10, 64, 65, 160, 161, 480]


def test_pass_stays_within_its_budget(plans):
    calls = [(n, m, kk, wide, st, 0, 76, 0) for n, m, kk, (wide, st) in itertools.product(
        N, M, KK, [(256, 0), (256, 1), (240, 0)])]
    calls += [(n, n, kk, 256, 0, 0, 76, 0) for n in N for kk in KK]  # allknn in id order
    taken = 0
    for c, p in zip(calls, plans(calls)):
        n, m, kk, wide = c[:4]
        if not p["ok"]:
            assert n // wide // 4 * 64 < 4 * kk or n // wide < 8
            continue
        taken += 1
        assert pass_bytes(p) == p["chunk"] * p["query_bytes"] <= BUDGET
        assert p["chunk"] % 256 == 0 and 256 <= p["chunk"] <= -(-m // 256) * 256
        # the bound: enough minima, from whole tiles
        assert p["groups"] == p["samples"] * p["per_tile"] >= 4 * kk
        assert p["per_tile"] in (2, 8, 64)
        assert 4 * p["samples"] <= n // wide
        # the lists: kk stay after a compaction, beside a tile's columns and a buffer
        assert 1 <= p["splits"] <= -(-n // wide)
        assert p["cap"] % 32 == 0 and p["cap"] <= 1024 and p["cap"] - 128 - 12 >= kk
        # one pass wherever it fits, split as for all queries
        if p["chunk"] >= m:
            assert p["splits"] == p["alone"]
    assert taken > 500


def test_small_chunks_fill_the_device(plans):
    """A chunk bounded by the minima is split until its CTA pairs fill the 76."""
    calls = [(n, m, kk, 256, 0, 0, 76, 0) for n in (10_000_000, 30_000_000, 100_000_000, 1_000_000_000)
             for m in (20_000, 100_000, 1_000_000) for kk in (10, 100)]
    for p in plans(calls):
        pairs = p["chunk"] // 256 * p["splits"]
        waves = -(-pairs // 76)
        assert pairs / (76 * waves) > 0.85


def test_locality_pass_stays_within_its_budget(plans):
    calls = [(n, n, kk, 256, 0, 0, 76, 1) for n in N if n >= 65_536 for kk in KK]
    for c, p in zip(calls, plans(calls)):
        if p["ok"]:
            assert pass_bytes(p) <= BUDGET
            assert p["groups"] >= 4 * c[2]


@pytest.mark.parametrize("locality", [0, 1])
def test_splits_asked_for_yield_to_the_budget(plans, locality):
    calls = [(n, n if locality else m, kk, 256, 0, splits, 76, locality) for n in (100_000, 2_000_000, 1_000_000_000)
             for m in (1, 300) for kk in (10, 200) for splits in (1, 3, 17, 300, 5000, 65_535)]
    for c, p in zip(calls, plans(calls)):
        if not p["ok"]:
            continue
        assert pass_bytes(p) <= BUDGET
        assert 1 <= p["splits"] <= c[5]
        if not locality and c[5] <= 300 and c[0] < 1_000_000_000:
            assert p["splits"] == min(c[5], -(-c[0] // 256))


SAMPLE_DRIVER = r"""
#include "list_plan.h"
#include <cstdio>
#include <vector>
// Every sampled place is a row of its own, of a whole tile; prints the largest
// run of rows without a sampled one among the tiles sampled from, and their number.
int main() {
    long long n, samples;
    int tile_rows;
    while (std::scanf("%lld %d %lld", &n, &tile_rows, &samples) == 3) {
        const int atoms = tile_rows / 8;
        const ssg::SampleRows s = ssg::sample_rows(n, tile_rows, samples);
        std::vector<bool> seen(static_cast<size_t>(n));
        bool ok = true;
        for (long long v = 0; v < 2 * samples; ++v) {
            int64_t tile;
            int line;
            ssg::sample_unit(s, atoms, v, &tile, &line);
            ok = ok && tile >= 0 && tile < s.q && line >= 0 && line < atoms;
            for (int c = 0; ok && c < tile_rows; ++c) {
                const int64_t row = ssg::sample_row(s, tile_rows, tile, line, c);
                ok = row >= 0 && row < n / tile_rows * tile_rows && !seen[size_t(row)];
                if (ok) seen[size_t(row)] = true;
            }
        }
        const long long reach = s.q * atoms * tile_rows;
        long long gap = 0, run = 0;
        for (long long i = 0; i < reach; ++i) {
            run = seen[size_t(i)] ? 0 : run + 1;
            gap = run > gap ? run : gap;
        }
        std::printf("%d %lld %lld\n", int(ok), gap, reach);
    }
    return 0;
}
"""


def test_sample_is_distinct_rows_from_everywhere(plans, tmp_path):
    src = tmp_path / "sample.cpp"
    src.write_text(SAMPLE_DRIVER)
    exe = tmp_path / "sample"
    subprocess.run([shutil.which("g++"), "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    sizes = [2048, 2100, 3839, 4095, 4096, 5000, 24_600, 30_011, 100_000, 777_777]
    calls = [(n, m, kk, wide, st, 0, 76, 0) for n in sizes for m in (1, 1000) for kk in (1, 10, 100)
             for wide, st in ((256, 0), (256, 1), (240, 0))]
    text, asked = "", []
    for c, p in zip(calls, plans(calls)):
        if p["ok"]:
            asked.append((c[0], c[3] // 2, p["samples"]))
            text += "%d %d %d\n" % asked[-1]
    out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout.split("\n")
    for (n, tile_rows, samples), line in zip(asked, out):
        ok, gap, reach = map(int, line.split())
        assert ok == 1
        assert reach > n - tile_rows * (tile_rows // 8) - tile_rows  # less than a span of tiles is left out
        assert gap <= 2 * (reach // (2 * samples * 8 * (tile_rows // 8))) * 8 + 16  # evenly spread


VISIT_DRIVER = r"""
#include "list_plan.h"
#include <cstdio>
#include <vector>
// The wide tiles' first units, from any tile on: every one of them once; prints
// their stride and the shortest way between any two of four visited in a row.
int main() {
    long long samples;
    while (std::scanf("%lld", &samples) == 1) {
        const ssg::SampleRows s = ssg::sample_rows(256 * 4 * samples, 128, samples);
        std::vector<int> at(static_cast<size_t>(samples));
        std::vector<bool> seen(static_cast<size_t>(samples));
        bool ok = true;
        int v = ssg::sample_first(s, 0);
        for (long long w = 0; ok && w < samples; ++w, v = ssg::sample_next(s, v)) {
            ok = v >= 0 && v < samples && !seen[size_t(v)] && v == ssg::sample_first(s, w);
            if (ok) seen[size_t(v)] = true;
            at[size_t(w)] = v;
        }
        long long least = samples;
        for (long long w = 0; w < samples; ++w)
            for (long long x = w + 1; x < w + 4 && x < samples; ++x) {
                const long long d = at[size_t(w)] > at[size_t(x)] ? at[size_t(w)] - at[size_t(x)] : at[size_t(x)] - at[size_t(w)];
                least = d < least ? d : least;
            }
        std::printf("%d %d %lld\n", int(ok), s.stride, least);
    }
    return 0;
}
"""


def test_sample_visits_every_unit_once_and_far_apart(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not found")
    src = tmp_path / "visit.cpp"
    src.write_text(VISIT_DRIVER)
    exe = tmp_path / "visit"
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    sizes = list(range(1, 400)) + [651, 1389, 7812, 65_537, 262_144]
    out = subprocess.run([str(exe)], input="\n".join(map(str, sizes)), capture_output=True, text=True, check=True).stdout
    for s, line in zip(sizes, out.splitlines()):
        ok, stride, least = map(int, line.split())
        assert ok == 1
        # three golden sections g = 0.618 come to 1.854: four in a row are 0.146
        # of the sample apart at least, less three times the way to a coprime stride
        off = stride - 0.618034 * s
        assert 0 <= off + 1 < 12
        assert least >= min(s, 0.1458 * s - 3 * abs(off))


def test_large_groups_have_the_tiles_to_keep_places_apart(plans):
    calls = [(n, m, kk, wide, 0, splits, 76, 0) for n in N for m in M for kk in (1, 10, 100) for wide in (240, 256)
             for splits in (0, 1, 5)]
    seen = set()
    for c, p in zip(calls, plans(calls)):
        if p["ok"]:
            seen.add(p["per_tile"])
            assert p["per_tile"] != 2 or p["samples"] >= 4 * p["splits"]
    assert {2, 8} <= seen

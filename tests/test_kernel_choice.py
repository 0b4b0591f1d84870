"""What the library chooses when the caller fixes nothing, asked on the CPU: a small C++ program linked against the library calls the rules.  The
numbers are those of a B200 (148 SMs, clusters of 2 to 8 CTAs that fit at once)."""
import math
import os
import random
import subprocess

import pytest

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include "kernels.h"
namespace t0 { int w4a16_umma_form(uint32_t sms, uint32_t M, uint32_t N, uint32_t K, uint32_t count, uint32_t cluster_split, uint32_t cluster_rounds, uint32_t* ctas); }     // w4a16_umma_cut.cu
using namespace t0;
int main() {
    static const uint32_t clusters[kMaxClusterParts + 1] = {0, 148, 74, 40, 33, 24, 20, 14, 15};
    char what[16];
    while (scanf("%15s", what) == 1) {
        unsigned m, n, k, nn, bf16;
        if (!strcmp(what, "w4a16")) {
            unsigned count, split, rounds, ctas;
            if (scanf("%u %u %u %u %u %u", &m, &n, &k, &count, &split, &rounds) != 6) return 1;
            const int form = w4a16_umma_form(148, m, n, k, count, split, rounds, &ctas);
            printf("%d %u\n", form, ctas);
            continue;
        }
        if (scanf("%u %u %u %u %u", &m, &n, &k, &nn, &bf16) != 5) return 1;
        t0_gemm_config c;
        bool forced;
        cached_config(m, k, n, &c, &forced);
        const uint32_t split = c.split_k > 1 && k % c.split_k == 0 ? c.split_k : 1;
        const GemmChoice g = choose_gemm(m, n, k, nn != 0, bf16 != 0, split, 148, clusters);
        printf("%u %u %d %d %u\n", g.tile_n, g.parts, (int)g.pair, (int)g.halves, split);
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def ask(t0, tmp_path_factory):
    root, lib = os.path.dirname(os.path.dirname(t0.HEADER_PATH)), os.path.dirname(t0.LIB_PATH)
    where = tmp_path_factory.mktemp("choice")
    (where / "ask.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(root, "rust-gpu_b200", "csrc"), "-I", "/usr/local/cuda/include", str(where / "ask.cpp"), "-o", str(where / "ask"),
                    os.path.join(lib, "libt0b200.so"), f"-Wl,-rpath,{lib}"], check=True)

    def run(lines):
        env = {k: v for k, v in os.environ.items() if k != "T0_FORCE_CFG"}
        out = subprocess.run([str(where / "ask")], input="\n".join(" ".join(map(str, line)) for line in lines), capture_output=True, text=True, check=True, env=env).stdout
        return [tuple(map(int, line.split())) for line in out.splitlines()]

    return run


def gemm_choices(ask, shapes):
    """(tile_n, parts, pair, halves) and the k blocks of the longest accumulation, per (m, n, k, nn, bf16)."""
    out = []
    for (m, n, k, nn, bf16), (tile_n, parts, pair, halves, split) in zip(shapes, ask([("gemm",) + s for s in shapes])):
        blocks = -(-(-(-k // 64)) // parts) if parts else -(-(k // split) // 64)
        out.append(((tile_n, parts, bool(pair), bool(halves)), (blocks + 1) // 2 if halves else blocks))
    return out


# k blocks of the longest accumulation that the library has given these shapes since its sums were cut; the tensor cores' error grows with it
LONGEST = [((1352, 248, 1672, 0, 0), 5), ((56, 7952, 1984, 0, 0), 8), ((1016, 272, 1456, 0, 0), 4), ((2168, 168, 560, 0, 0), 5), ((112, 144, 952, 1, 0), 2),
           ((64, 3136, 1536, 0, 1), 3), ((3289, 115, 1936, 0, 0), 4), ((24, 64, 624, 1, 0), 1), ((696, 56, 944, 1, 0), 2), ((392, 32, 872, 0, 1), 2), ((136, 64, 784, 1, 1), 2),
           ((384, 768, 1464, 0, 1), 4), ((400, 520, 1432, 0, 1), 4), ((192, 384, 880, 0, 1), 3), ((1448, 384, 1024, 0, 0), 8), ((80, 2120, 1216, 1, 0), 5),
           ((106, 3492, 1185, 0, 1), 10), ((7976, 40, 576, 0, 0), 5), ((2605, 509, 1320, 0, 1), 21), ((448, 3456, 5176, 0, 0), 41), ((2048, 1024, 4096, 0, 0), 32),
           ((128, 4096, 4096, 0, 0), 8), ((4096, 4096, 4096, 0, 0), 64)]


def test_sums_are_no_longer_than_they_have_been(ask):
    for ((m, n, k, nn, bf16), longest), (choice, blocks) in zip(LONGEST, gemm_choices(ask, [s for s, _ in LONGEST])):
        assert blocks <= longest, (m, n, k, nn, bf16, choice, blocks, longest)


CLUSTERS, WHOLE, CUT = 0, 1, 2


def w4a16_split(n, k, count):
    """The tiles and 64-deep chunks of `count` problems (0: one that is not given as a list), and for such a one into how many parts clusters would cut its K and
    in how many rounds they run."""
    tiles, chunks = -(-n // 256) * (count or 1), k // 64
    split = 0 if count else min(max(1, min(4, 148 // tiles)), chunks)
    at_once = {0: tiles, 1: tiles, 2: 74, 3: 48, 4: 33}[split]                                                # clusters of `split` CTAs that fit at once
    return tiles, chunks, split, -(-tiles // at_once)


def w4a16_longest(form, ctas, tiles, chunks, split):
    """The chunks of the longest accumulation."""
    if form != CUT:
        return -(-chunks // max(split, 1))
    ends = sorted({c * tiles * chunks // ctas for c in range(ctas + 1)} | {t * chunks for t in range(tiles)})      # of the CTAs' ranges, and of the tiles
    return max(b - a for a, b in zip(ends, ends[1:]))


def w4a16_forms(ask, problems):
    """How each (m, n, k, count) is shared out, and the 64-deep chunks of the longest accumulation."""
    splits = [w4a16_split(n, k, count) for _, n, k, count in problems]
    answers = ask([("w4a16", m, n, k, count or 1, split, rounds) for (m, n, k, count), (_, _, split, rounds) in zip(problems, splits)])
    return [(form, w4a16_longest(form, ctas, tiles, chunks, split)) for (form, ctas), (tiles, chunks, split, _) in zip(answers, splits)]


def w4a16_form(ask, m, n, k, count):
    return w4a16_forms(ask, [(m, n, k, count)])[0]


# lists whose tiles have been cut, and single problems, with the chunks of the longest accumulation the library has given them
W4A16_LONGEST = [((113, 4456, 1920, 3), 11), ((125, 9800, 2944, 2), 25), ((114, 4680, 1664, 2), 7), ((128, 1632, 2240, 8), 14), ((121, 5144, 3008, 4), 27),
                 ((58, 592, 960, 0), 4), ((50, 4840, 576, 0), 3), ((36, 304, 576, 0), 3), ((20, 3200, 768, 0), 3), ((50, 7736, 832, 0), 4), ((128, 256, 64, 0), 1),
                 ((17, 1024, 256, 0), 1), ((52, 8968, 576, 0), 3), ((128, 11008, 4096, 0), 22), ((20, 14336, 2048, 0), 16), ((100, 28672, 1024, 0), 16),
                 ((70, 2320, 1280, 3), 5), ((84, 4352, 1280, 2), 5), ((77, 6024, 1408, 2), 8), ((42, 3488, 1024, 2), 4), ((28, 8224, 1408, 2), 11),
                 ((17, 2408, 832, 4), 5), ((39, 9776, 1152, 1), 6), ((25, 22296, 2368, 0), 22), ((120, 19352, 2944, 0), 24)]


def test_w4a16_sums_are_no_longer_than_they_have_been(ask):
    for (m, n, k, count), longest in W4A16_LONGEST:
        form, chunks = w4a16_form(ask, m, n, k, count)
        assert chunks <= longest, (m, n, k, count, form, chunks)


def w4a16_bound(m, n, k, count):
    """The longest accumulation by the rule whose lengths the library keeps: the times of the kernels as they were before two warps issued, with the grid of cut tiles."""
    tiles, chunks, split, rounds = w4a16_split(n, k, count)
    total = tiles * chunks
    ctas = min(max(1, total // 4), 148)
    if tiles * 2 <= 148:
        parts = max(1, min(4, 148 // tiles, chunks // 4))
        if parts == 4 or parts * 8 > chunks or tiles * parts * 5 >= 148 * 4:
            ctas = tiles * parts
    other = CLUSTERS if split > 1 else WHOLE
    if other == CLUSTERS and -(-total // ctas) > -(-chunks // split):
        ctas = tiles * split
    form = other
    if tiles % ctas:
        waves, chunk = -(-tiles // 148), 0.42 + 0.0008 * m
        whole = rounds * (-(-chunks // split) * 0.495 + 8.2) + 2.0 if other == CLUSTERS else waves * chunks * chunk + 4.2
        if total / ctas * chunk + 6.2 + 0.055 * m + (2.0 if ctas >= 148 else 0.0) <= 0.97 * whole or \
                (split == 0 and total / ctas * 0.67 + 14.4 <= 0.97 * (waves * chunks * 0.63 + 4.0)):
            form = CUT
    return w4a16_longest(form, ctas, tiles, chunks, split)


def test_w4a16_sums_are_no_longer_over_the_range(ask):
    rng = random.Random(11)
    def size(low, high, step):
        return max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))) / step) * step)
    problems = [(rng.randint(17, 128), size(256, 32768, 8), size(128, 8192, 64), rng.choice([0, 0, 1, 2, 2, 3, 4, 8, 16])) for _ in range(20000)]
    longer = [(p, got, w4a16_bound(*p)) for p, got in zip(problems, w4a16_forms(ask, problems)) if got[1] > w4a16_bound(*p)]
    assert not longer, (len(longer), longer[:5])


def test_w4a16_uneven_parts_of_many_rows_leave_clusters_alone(ask):
    # measured slower cut than as clusters (56, 53, 38, 58 tiles on 148 CTAs); even parts, few rows, or more of K: cut
    for m, n, k in [(93, 14112, 1536), (81, 13416, 1536), (66, 9720, 1664), (85, 14784, 1152)]:
        assert w4a16_form(ask, m, n, k, 0)[0] == CLUSTERS, (m, n, k)
    for m, n, k in [(92, 3232, 6272), (49, 14112, 1536), (96, 15312, 2816), (121, 12128, 7424)]:
        assert w4a16_form(ask, m, n, k, 0)[0] == CUT, (m, n, k)


def test_w4a16_clusters_in_two_rounds_are_weighed_as_such(ask):
    # 33 clusters of four CTAs fit at once: 33 tiles take one round, 34 take two and are cut in their place
    assert w4a16_form(ask, 128, 33 * 256, 4096, 0)[0] == CLUSTERS
    for tiles in (34, 37):
        assert w4a16_form(ask, 128, tiles * 256, 4096, 0)[0] == CUT


# The shapes by which the GPU tests mean to reach a kernel: a refit that moved one would leave the kernel untested.
PAIR_128_HALVES = [(2048, 1024, 4096, 0, 0), (2048, 1024, 4096, 1, 0), (1664, 1056, 3248, 0, 0), (1664, 1056, 3248, 1, 0), (280, 3339, 2036, 0, 1), (280, 3339, 2040, 1, 1),
                   (263, 3318, 2218, 0, 1), (263, 3320, 2218, 1, 0), (768, 2048, 4096, 1, 1), (645, 7493, 4864, 0, 0)]


def test_shapes_of_the_gpu_tests_reach_pair_tiles_128_wide(ask):
    for shape, (choice, _) in zip(PAIR_128_HALVES, gemm_choices(ask, PAIR_128_HALVES)):
        assert choice == (128, 1, True, True), (shape, choice)
    tiles = -(-645 // 256) * -(-7493 // 128)                                     # more than the 74 pairs, and the last wave at most half full
    assert tiles > 74 and 0 < 2 * (tiles % 74) <= 74


@pytest.mark.parametrize("form,problems", [
    (CUT, [(20, 14344, 2048, 0), (33, 2312, 1024, 3), (17, 200, 128, 0), (20, 1030, 256, 0), (64, 8960, 256, 0), (40, 9000, 576, 0), (39, 3264, 768, 0), (128, 9300, 1024, 0),
           (33, 255, 512, 0), (20, 2560, 2048, 0), (40, 2560, 4096, 2)]),
    (CLUSTERS, [(128, 2560, 2048, 0), (128, 1030, 1024, 0), (100, 1001, 1024, 0), (128, 7, 1024, 0), (128, 11008, 4096, 0)]),
    (WHOLE, [(16, 38144, 64, 0), (17, 1030, 64, 0)])])
def test_shapes_of_the_gpu_tests_reach_every_w4a16_form(ask, form, problems):
    for m, n, k, count in problems:
        assert w4a16_form(ask, m, n, k, count)[0] == form, (m, n, k, count)

"""What the library chooses when the caller fixes nothing, asked on the CPU: a small C++ program linked against the library calls the rules.  The
numbers are those of a B200 (148 SMs, clusters of 2 to 8 CTAs that fit at once)."""
import os
import subprocess

import pytest

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include "kernels.h"
using namespace t0;
int main() {
    static const uint32_t clusters[kMaxClusterParts + 1] = {0, 148, 74, 40, 33, 24, 20, 14, 15};
    char what[16];
    while (scanf("%15s", what) == 1) {
        unsigned m, n, k, nn, bf16;
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

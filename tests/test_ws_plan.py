"""CPU test of the weight-stationary matmul's choice of token tiles and K slices: the same as a search over every number
of token tiles, in a number of steps that does not grow with the rows."""
import os
import random
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MAIN = r"""
#include <cstdio>
#include "ws_plan.h"
int main() {
  long long m, rt; int u, f, c[4];
  while (std::scanf("%lld %lld %d %d %d %d %d %d", &m, &rt, &u, &f, c, c + 1, c + 2, c + 3) == 8) {
    const b200::WsSplit s = b200::choose_ws_split(m, rt, u, f, c);
    std::printf("%d %d %d %d\n", s.nb, s.ksplit, s.tried, (int)b200::prefill_kernel_is_ahead(m, 128 * rt, 256LL * u, s, rt, c[0]));
  }
}
"""


def exhaustive(m, row_tiles, units, forced, clusters):
    """Every number of token tiles in turn, times 1, 2, 4 and 8 slices; the first of equal costs."""
    best = None
    mt0 = -(-m // 192)
    for mt in range(mt0, (1 if m <= 128 else mt0 + mt0 // 2 + 3) + 1):
        nb = -(-(-(-m // mt)) // 16) * 16
        tiles = row_tiles * -(-m // nb)
        for i, c in enumerate((1, 2, 4, 8)):
            if c > units or (forced and not (c <= forced and (c * 2 > forced or c * 2 > units or c == 8))):
                continue
            rounds = -(-tiles // clusters[i])
            span = max(520 + nb if nb <= 128 else 760 + nb, tiles * c // rounds * (nb * 512 + 18432) // 14000)
            tile = -(-units // c) * span
            drain = 300 + 12 * nb if c == 1 else 800 + 50 * nb
            room = m <= 128 and c >= 4 and 2 * tiles <= clusters[i] + (2 if c == 8 else 0)
            if room:
                start = 1600 - 8 * nb if c == 8 and tiles > 4 else 0
            else:
                start = (0, 500, 1000, 3500)[i]
                if m <= 128 and rounds == 1 and 2 * tiles > clusters[i]:
                    crowd = (0, 500, 2400, 0)[i] * (2 * tiles - clusters[i]) // clusters[i]
                    start = max(start, crowd) if c == 4 else start + crowd
            tail = drain if c == 1 else 900 + 38 * nb if room else 600 + 35 * nb
            cost = start + tile + (rounds - 1) * max(tile, drain) + tail
            if m > 128 and c > 1:
                cost += cost * 15 // 1000
            if best is None or cost < best[0]:
                best = (cost, nb, c)
    return best[1:]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("ws_plan")
    (d / "main.cc").write_text(MAIN)
    exe = str(d / "plan")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", os.path.join(ROOT, "relax_b200", "csrc"), str(d / "main.cc"),
                    "-o", exe], check=True)
    return lambda cases: [tuple(map(int, line.split())) for line in subprocess.run(
        [exe], input="\n".join(" ".join(map(str, (m, rt, u, f, *c))) for m, rt, u, f, c in cases), capture_output=True, text=True,
        check=True).stdout.splitlines()]


def test_choice_equals_the_exhaustive_search(program):
    rng = random.Random(7)
    cases = [(m, rt, 16, 0, (148, 74, 36, 16)) for m in list(range(1, 700)) + [2047, 2048, 5000, 100000] for rt in (1, 32, 172)]
    cases += [(int(2 ** rng.uniform(0, 15)), rng.randint(1, 300), rng.randint(1, 64), rng.choice((0, 0, 1, 2, 4, 8)),
               rng.choice(((148, 74, 36, 16), (132, 66, 33, 16), (8, 4, 2, 1)))) for _ in range(3000)]
    for case, got in zip(cases, program(cases)):
        assert got[:2] == exhaustive(*case), case


def test_the_search_does_not_grow_with_the_rows(program):
    for m in (2048, 65536, 1_000_000, 0x7fffffff // 64):
        (nb, ksplit, tried, _), = program([(m, 86, 16, 0, (148, 74, 36, 16))])
        assert tried <= 48 and nb in range(16, 193, 16) and ksplit in (1, 2, 4, 8)


def test_long_prompts_that_one_wave_of_the_prefill_kernel_holds(program):
    # as measured: ahead on the left, not on the right
    for ahead, shapes in ((1, [(2048, 4096, 11008), (4096, 2048, 8192), (2048, 4096, 8192), (8192, 1024, 11008)]),
                          (0, [(1024, 8192, 8192), (2048, 4096, 4096), (4096, 2048, 4096), (777, 3584, 8192), (2048, 11008, 8192),
                               (512, 8192, 8192), (128, 8192, 8192), (4096, 4096, 8192)])):
        got = program([(m, n // 128, k // 256, 0, (148, 74, 36, 16)) for m, n, k in shapes])
        assert [g[3] for g in got] == [ahead] * len(shapes), list(zip(shapes, got))


def test_slices_where_clusters_crowd_the_gpu(program):
    # as measured: the best number of slices (four, two or one were taken for them: 5-30 % slower)
    for best, shapes in ((2, [(8, 4096, 2080), (16, 4096, 2080), (16, 4096, 2560)]),
                         (1, [(64, 8192, 2080), (96, 8192, 2560), (96, 6144, 2560), (777, 12288, 7168), (777, 12288, 8192)]),
                         (4, [(9, 10240, 5120), (33, 10240, 7168), (16, 2560, 4096), (64, 2560, 2560), (16, 4096, 11008), (16, 4096, 5120), (24, 1024, 4096), (16, 2048, 11008)]),
                         (8, [(16, 512, 8192)])):
        for clusters in ((148, 74, 36, 16), (148, 74, 33, 15)):                     # (two GPUs of one kind)
            got = program([(m, -(-n // 128), -(-k // 256), 0, clusters) for m, n, k in shapes])
            assert [g[1] for g in got] == [best] * len(shapes), (clusters, list(zip(shapes, got)))


def test_choice_on_a_gpu_with_fewer_clusters_equals_the_exhaustive_search(program):
    rng = random.Random(8)
    cases = [(int(2 ** rng.uniform(0, 15)), rng.randint(1, 300), rng.randint(1, 64), rng.choice((0, 0, 1, 2, 4, 8)), (148, 74, 33, 15)) for _ in range(1000)]
    for case, got in zip(cases, program(cases)):
        assert got[:2] == exhaustive(*case), case

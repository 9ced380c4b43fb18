"""How a Floyd-Warshall batch is shared out between teams of CTAs (host code)."""
import os
import random
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pagani-toolkit_b200", "csrc")
MAIN = """#include "fw_plan.h"
#include <cstdio>
int main(int argc, char** argv)
{
    std::vector<int> nb;
    for (int x; scanf("%d", &x) == 1;) nb.push_back(x);
    const FwPlan p = fw_batch_plan(nb.data(), (int)nb.size(), 148, 64);
    printf("%d", p.teams);
    for (int q : p.bundle0) printf(" %d", q);
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", str(d / "main.cpp"), "-o", str(d / "plan")], check=True)

    def run(sizes):
        nb = sorted((max(1, (n + 63) // 64) for n in sizes), reverse=True)
        out = subprocess.run([str(d / "plan")], input=" ".join(map(str, nb)), capture_output=True, text=True, check=True)
        t, *b = map(int, out.stdout.split())
        return nb, t, b
    return run


def _sizes(count, lo, hi):
    rng = random.Random(count + hi)
    return [rng.randint(lo, hi) for _ in range(count)]


@pytest.mark.parametrize("sizes", [[1], [2500], _sizes(2, 90, 1024), _sizes(8, 90, 260), _sizes(16, 90, 520),
                                   _sizes(32, 90, 1024), _sizes(64, 90, 1024), _sizes(64, 90, 130), [1024] + [120] * 20,
                                   [1500] + [120] * 60, [700] + [120] * 300, [512] * 40])
def test_small_and_uneven_batches_are_swept_in_step(plan, sizes):
    """A team of their own left most of the GPU idle: up to six times slower."""
    nb, teams, cuts = plan(sizes)
    assert teams == 1 and cuts == [0, len(nb)]


@pytest.mark.parametrize("sizes", [_sizes(512, 90, 1024), _sizes(2000, 65, 128), [64] * 20000, [1024] * 370])
def test_large_batches_are_shared_evenly(plan, sizes):
    nb, teams, cuts = plan(sizes)
    assert teams == 37
    assert cuts[0] == 0 and cuts[-1] == len(nb) and all(a < b for a, b in zip(cuts, cuts[1:]))
    busy = [0] * teams
    for a, b in zip(cuts, cuts[1:]):
        assert b == a + 1 or sum((64 * x) ** 2 * 4 for x in nb[a:b]) <= 1 << 20
        busy[busy.index(min(busy))] += sum(x ** 3 for x in nb[a:b])
    assert max(busy) <= 1.25 * sum(busy) / teams

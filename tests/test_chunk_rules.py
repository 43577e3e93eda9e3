"""The rules for the planes per block of the sweeps (host arithmetic): within the grid for every size, and for the cp.async
sweep the lengths that were fastest (within 3 %) where a rule for other tiles and another residency had cost 10 %."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "sphericalstokes_gb300" / "csrc"
MAIN = """
#include <cstdio>
#include "sph_chunk.h"
int main() {
    int n1, n2, n3;
    while (std::scanf("%d %d %d", &n1, &n2, &n3) == 3) {
        const long long a = (long long)((n1 + 31) / 32) * ((n2 + 13) / 14), b = (long long)((n1 + 31) / 32) * ((n2 + 7) / 8);
        std::printf("%d %d %d\\n", sph::grid_chunk(a, n3, 152), sph::fallback_chunk(b, n3, 152), sph::chunk_rule({{a, n3}, {a, n3}}, 152));
    }
}
"""
FASTEST = {(47, 31, 39): (2,), (63, 63, 63): (4, 7), (23, 40, 200): (4, 7), (28, 29, 158): (3, 5)}


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("chunk")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", "-o", str(d / "rules"), str(d / "main.cpp")], check=True)

    def run(sizes):
        out = subprocess.run([str(d / "rules")], input="\n".join("%d %d %d" % n for n in sizes), capture_output=True, text=True, check=True)
        return [tuple(map(int, line.split())) for line in out.stdout.splitlines()]
    return run


def test_picks_are_within_the_grid(rules):
    sizes = [(a, b, c) for a in (5, 32, 33, 511, 2000) for b in (5, 14, 15, 255) for c in (5, 6, 23, 24, 25, 101, 4000)]
    for n, picks in zip(sizes, rules(sizes), strict=True):
        assert all(1 <= k <= 24 for k in picks) and max(picks[:2]) <= n[2], (n, picks)


def test_cp_async_sweep_takes_a_fast_length(rules):
    for (n, fast), picks in zip(FASTEST.items(), rules(FASTEST), strict=True):
        assert picks[1] in fast, (n, picks)

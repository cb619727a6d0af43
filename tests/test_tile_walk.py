"""The persistent column stage's walk over its tiles, the device code compiled for the CPU: CTAs in any order of
progress, one of them alone among them, take every tile exactly once, from the counter and from ranges."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gmtsar-gpu_gb300", "csrc")
MAIN = r"""
#include <stdio.h>
#include <stdlib.h>
#include <vector>
#include "tile_walk.cuh"
// one CTA's state as the kernel keeps it: the walk and the counter's last value it took
struct Cta { xcg::TileWalk w; int grab; bool in, done; };
int main(int argc, char **argv) {
    const int ntiles = atoi(argv[1]), K = atoi(argv[2]), ctas = atoi(argv[3]), seed = atoi(argv[4]), ranges = atoi(argv[5]);
    int counter = 0, left = ctas;
    std::vector<int> seen(ntiles, 0);
    std::vector<Cta> c(ctas);
    for (Cta &x : c) { x.in = x.done = false; x.grab = ntiles; x.w.ntiles = ntiles; x.w.K = K; }
    srand(seed);
    while (left > 0) {
        // seed 0: one CTA runs as far as it can before the next starts
        int i = 0;
        if (seed == 0) while (c[i].done) i++;
        else do i = rand() % ctas; while (c[i].done);
        Cta &x = c[i];
        if (!x.in) {
            x.in = true;
            if (ranges) {
                x.w.t = (int)((long long)ntiles * i / ctas);
                x.w.end = (int)((long long)ntiles * (i + 1) / ctas);
            } else {
                x.grab = counter;
                counter += K;
                x.w.enter(x.grab);
            }
            if (x.w.t >= x.w.end) { x.done = true; left--; }
            continue;
        }
        if (!ranges && x.w.last()) { x.grab = counter; counter += K; }
        const int tn = x.w.next(x.grab);
        if (x.w.t < 0 || x.w.t >= ntiles) return 2;
        if (++seen[x.w.t] > 1) { printf("tile %d again\n", x.w.t); return 1; }
        if (tn < 0) { x.done = true; left--; } else x.w.go(tn);
    }
    for (int t = 0; t < ntiles; t++) if (seen[t] != 1) { printf("tile %d: %d times\n", t, seen[t]); return 1; }
}
"""


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    d = tmp_path_factory.mktemp("walk")
    (d / "m.cpp").write_text(MAIN)
    subprocess.run(["g++", "-O2", "-I" + CSRC, str(d / "m.cpp"), "-o", str(d / "m")], check=True)
    return str(d / "m")


@pytest.mark.parametrize("ntiles,K,ctas", [(1, 1, 1), (7, 1, 3), (320, 1, 760), (320, 2, 160), (321, 4, 1), (64, 16, 5), (1000, 3, 304)])
def test_every_tile_once(walk, ntiles, K, ctas):
    for seed in range(6):
        for ranges in (0, 1):
            r = subprocess.run([walk] + [str(v) for v in (ntiles, K, ctas, seed, ranges)], capture_output=True, text=True)
            assert r.returncode == 0, (seed, ranges, r.stdout)

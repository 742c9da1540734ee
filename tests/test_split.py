"""The split of an exact k-NN pass over the GPU (``csrc/split.cuh``), compiled for the host, against trying
every number of CTAs a query tile."""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "hnsw_engine_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include "split.cuh"

static Split every(int qt, int tiles, int sms) {
    const int most = std::min(tiles, std::max(1, (8 * sms + qt - 1) / qt));
    Split g{tiles, 1};
    int64_t best = INT64_MAX;
    for (int s = 1; s <= most; s++) {
        const int tps = (tiles + s - 1) / s, splits = (tiles + tps - 1) / tps;
        const int64_t waves = (int64_t(qt) * splits + sms - 1) / sms, cost = waves * (tps + FIXED_TILES);
        if (cost < best) {
            best = cost;
            g = Split{tps, splits};
        }
    }
    return g;
}

int main() {
    int bad = 0;
    for (int sms : {1, 20, 132, 148, 160})
        for (int qt = 1; qt <= 300; qt += qt < 160 ? 1 : 13)
            for (int64_t t = 1; t <= 8388608; t += t < 700 ? 1 + t / 97 : t / 5) {
                const Split a = split_tiles(qt, int(t), sms), b = every(qt, int(t), sms);
                if (a.tps != b.tps || a.splits != b.splits) {
                    if (bad++ < 5)
                        std::printf("qt %d tiles %d sms %d: %d x %d, not %d x %d\n", qt, int(t), sms, a.splits, a.tps,
                                    b.splits, b.tps);
                }
                if (int64_t(a.tps) * a.splits < t || int64_t(a.tps) * (a.splits - 1) >= t) return 2;
            }
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host compiler")
def test_split_is_the_best_of_all(tmp_path: Path) -> None:
    src, exe = tmp_path / "split_test.cpp", tmp_path / "split_test"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and run.stdout == "", run.stdout

"""The cut of a tensor-core LWE key switch (csrc/lwe_mma_plan.h) over the contractions that a context accepts, on the
CPU: every split has steps, none more than the 258 that keep 32-bit sums exact, and the grid is one CUDA takes."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
SMS, STEP, MOST = 148, 128, 258


@pytest.fixture(scope="module")
def plan():
    out_dir = ROOT / "tests" / "_build"  # git-ignored build folder
    out_dir.mkdir(exist_ok=True)
    exe = out_dir / "lwe_mma_plan_driver"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT / 'fhetoothpaste_b200' / 'csrc'}",
                    str(ROOT / "tests" / "cpp" / "lwe_mma_plan_driver.cpp"), "-o", str(exe)], check=True)

    def run(rows):
        res = subprocess.run([str(exe)], input="\n".join(" ".join(map(str, r)) for r in rows) + "\n",
                             capture_output=True, text=True, check=True)
        return [tuple(map(int, line.split())) for line in res.stdout.splitlines()]
    return run


# 64 splits of 258 steps end at 16512 steps; a context accepts up to 2^30 bytes of K
STEPS = [1, 2, 3, 64, 257, 258, 259, 516, 517, 8192, 16511, 16512, 16513, 16770, 16771, 40000, 1 << 17, (1 << 23)]


def test_every_contraction_has_a_plan(plan):
    cases = [(planes, steps * STEP, width, batch, SMS) for steps in STEPS for planes in (1, 2)
             for width in (2, 32, 631) for batch in (1, 129, 20000)]
    for (planes, kpad, width, batch, _), (rows, rows_pad, splits, plane_bytes, part_bytes, fits) in zip(cases, plan(cases)):
        steps = kpad // STEP
        assert fits and 1 <= splits <= steps and splits <= 65535
        share = -(-steps // splits)
        assert share <= MOST and (splits - 1) * share < steps
        assert 1 <= rows <= batch and rows_pad == -(-rows // 128) * 128
        assert plane_bytes == planes * rows_pad * kpad and (plane_bytes <= 1 << 28 or rows_pad == 128)
        assert part_bytes == splits * rows * width * 8


def test_what_does_not_fit(plan):
    assert [p[5] for p in plan([(1, 128, 65535 * 32, 1, SMS), (1, 128, 65535 * 32 + 1, 1, SMS), (3, 128, 2, 1, SMS)])] == [1, 0, 0]


def test_largest_share(plan):
    """Tiles that fill the SMs leave K whole up to 258 steps (what the GPU test of the largest sums relies on)."""
    for planes in (1, 2):
        (rows, rows_pad, splits, *_), = plan([(planes, MOST * STEP, 37 * 32, 4 * 128, SMS)])
        assert splits == 1 and rows == 4 * 128

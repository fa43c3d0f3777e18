"""Which form a forward projection takes (csrc/tk_fp_plan.h), on the host: the row lanes where a CTA's shared memory
holds enough slices, the slice lanes where short chunks would make the row lanes the slower form (measured: up to three
times slower) or few projections leave its warps idle, the row lanes again where the volume does not fill the GPU."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# (W, N, X, Z, D / W, scale, cells of the slice lanes' box, whether two of their CTAs fit an SM), the row lanes expected
# to run; measured ms of row lanes and slice lanes beside them
CASES = [
    ((784, 60, 512, 512, 5.2, 1.5, 3328, 1), True),               # 12.7, 16.3
    ((784, 60, 512, 512, 4.0, 1.5, 3808, 1), False),              # 36.1, 17.1
    ((707, 60, 512, 512, 3.0, 1.35, 4140, 1), False),             # 35.6, 17.4
    ((630, 60, 512, 512, 2.0, 1.2, 5304, 1), False),              # 55.0, 20.5
    ((1040, 60, 512, 512, 8.0, 2.0, 4680, 1), False),             # 37.3, 20.0
    ((400, 120, 256, 256, 4.0, 1.5, 3808, 1), False),             # 9.3, 4.7
    ((323, 120, 256, 256, 4.0, 1.2, 2688, 1), True),              # 2.8, 4.4
    ((272, 1, 256, 256, 4.0, 1.0, 1880, 1), False),               # 0.165, 0.093
    ((272, 9, 256, 256, 4.0, 1.0, 1880, 1), True),                # 0.342, 0.374
    ((208, 200, 128, 128, 4.0, 1.5, 3752, 1), False),             # 2.28, 1.45
    ((144, 200, 128, 128, 3.0, 1.0, 2244, 1), True),              # 1.03, 1.32
    ((112, 200, 64, 64, 4.0, 1.5, 3696, 1), True),                # 0.34, 1.14
    ((64, 200, 64, 64, 3.0, 0.7, 1120, 1), True),                 # 0.14, 1.02
    ((80, 1, 64, 64, 4.0, 1.0, 1840, 1), False),                  # 0.021, 0.014
    ((80, 5, 64, 64, 4.0, 1.0, 1840, 1), True),                   # 0.025, 0.035
]


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fp") / "fp_plan_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "tomokvas_gb300", "csrc"), "-I",
                    os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "cpp", "fp_plan_check.cpp"), "-o", exe],
                   check=True)

    def run(W, N, X, Z, ratio, scale, cells=2000, two=1):
        line = f"{W} {W} {N} {X} {X} {Z} {ratio * W} {scale} {cells} {two}\n"
        return tuple(int(v) for v in subprocess.run([exe], input=line, capture_output=True, text=True).stdout.split())

    return run


@pytest.mark.parametrize("case,rows", CASES)
def test_faster_form_is_taken(plan, case, rows):
    K, TZ, zchunks, faster = plan(*case)
    assert K > 0 and TZ * zchunks >= case[3]
    assert bool(faster) == rows


def test_more_chunks_than_a_grid_has(plan):
    """1200000 slices in chunks of at most twelve would be 100000 blocks in a grid's y: left to the slice lanes."""
    assert plan(64, 8, 4, 120000, 2e5, 2.3)[:2] == (2, 12)
    assert plan(64, 8, 4, 1200000, 2e5, 2.3)[0] == 0

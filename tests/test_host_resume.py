"""The two pieces a point runs in when its sweep takes two launches (transient,
then averaging phase), compiled for the host, against the point run whole: the
same bits of status, steps and spectrum for every model, precision, integrator
and way to end, in either piece."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SCENARIOS = ["plain", "align", "mgs", "own_times", "max_steps", "hmin", "escape", "nonfinite"]


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path_factory.mktemp("resume") / "resume_driver")
    subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I" + os.path.join(os.path.dirname(HERE), "include"), "-o", exe,
                    os.path.join(HERE, "host", "resume_driver.cu")], check=True, capture_output=True)
    out = subprocess.run([exe, "60"], check=True, capture_output=True, text=True).stdout
    return [(f[:4], [int(v) for v in f[4:]]) for f in map(str.split, out.splitlines())]


@pytest.mark.parametrize("scenario", SCENARIOS)
def test_two_pieces_are_the_whole(lines, scenario):
    rows = [r for r in lines if r[0][3] == scenario]
    assert len(rows) == 5 * 2 * 2
    for name, (points, *counts, ended, differ) in rows:
        assert differ == 0 and points == 60 and sum(counts) == points, name
    total = [sum(r[1][1 + s] for r in rows) for s in range(5)]
    ended = sum(r[1][6] for r in rows)
    want = {"max_steps": 3, "hmin": 2, "escape": 4, "nonfinite": 1}.get(scenario)
    if want is None:
        assert total[0] == 1200 and ended == 0
    else:  # some end so, in the transient and (a non-finite point apart) after it
        assert total[want] > ended // 2 > 0
        assert scenario == "nonfinite" or total[want] > ended

"""The fixed-step sweep's choice between its launch forms, on runs measured in
both (a B200's 148 SMs): never more than 6.5 % slower than the better form."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))

# phases: t_skip, t_skip_clp, calc_time, add_skip at a step of 0.01
PHASES = {"skip": (3.0, 0.05, 0.05, 5.0), "tan": (0.02, 0.2, 3.0, 5.0), "gs": (0.02, 2.0, 1.0, 1.0),
          "rare": (0.02, 0.02, 3.0, 100.0), "half": (1.6, 0.1, 1.5, 5.0),
          "quart": (0.8, 0.1, 2.3, 10.0)}
# model, method, k, points per SM, phases, us with a thread per point, us with a group
MEASURED = [
    ("lorenz", "fd", 3, 87, "skip", 113, 260),
    ("lorenz", "fd", 3, 1, "skip", 112, 102),
    ("lorenz", "fd", 3, 52, "tan", 538, 278),
    ("lorenz", "fd", 3, 87, "half", 320, 325),
    ("lorenz", "fd", 1, 66, "skip", 106, 188),
    ("lorenz", "fd", 1, 1, "tan", 256, 188),
    ("lorenz", "fd", 1, 87, "tan", 262, 269),
    ("lorenz", "var", 1, 87, "tan", 257, 308),
    ("lorenz", "var", 2, 52, "skip", 108, 188),
    ("lorenz", "var", 2, 52, "tan", 432, 312),
    ("lorenz", "var", 3, 87, "gs", 777, 573),
    ("lorenz", "qr", 3, 87, "tan", 820, 619),
    ("lorenz", "qr", 3, 75, "skip", 111, 260),
    ("chua", "fd", 1, 1, "skip", 122, 148),
    ("chua", "var", 1, 31, "half", 178, 193),
    ("chua", "var", 3, 87, "tan", 573, 424),
    ("chua", "qr", 3, 52, "skip", 142, 208),
    ("chua", "fd", 3, 15, "tan", 601, 231),
    ("hyper_rossler", "fd", 4, 87, "skip", 157, 615),
    ("hyper_rossler", "fd", 4, 1, "skip", 154, 124),
    ("hyper_rossler", "fd", 4, 15, "tan", 890, 239),
    ("hyper_rossler", "var", 4, 52, "half", 530, 536),
    ("hyper_rossler", "qr", 4, 34, "skip", 142, 322),
    ("hyper_rossler", "qr", 4, 31, "tan", 1461, 597),
    ("shimizu", "fd", 1, 87, "rare", 183, 217),
    ("shimizu", "var", 3, 34, "quart", 401, 253),
    ("rossler", "qr", 3, 66, "half", 429, 418),
]
METHODS = {"fd": 0, "var": 1, "qr": 2}


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path_factory.mktemp("rule") / "compat_rule_driver")
    subprocess.run([gxx, "-std=c++17", "-O1", "-o", exe,
                    os.path.join(HERE, "host", "compat_rule_driver.cpp")], check=True)

    def run(questions):
        text = "".join(" ".join(repr(v) for v in q) + "\n" for q in questions)
        out = subprocess.run([exe], input=text, check=True, capture_output=True, text=True).stdout
        return [int(v) for v in out.split()]
    return run


def test_choice_on_measured_runs(ask):
    groups = ask([(METHODS[m], k, int(model == "chua"), 148 * n, 148, 0.01, *PHASES[ph])
                  for model, m, k, n, ph, _, _ in MEASURED])
    assert len(groups) == len(MEASURED)
    for g, row in zip(groups, MEASURED):
        thread, group = row[-2:]
        assert (group if g else thread) <= 1.065 * min(thread, group), row


@pytest.mark.parametrize("method", [0, 1, 2])
def test_range_and_odd_arguments(ask, method):
    """Above 88 points per SM always threads; phases of no or negative length,
    and a renormalisation period that is never reached, are no steps."""
    tan = PHASES["tan"]
    assert ask([(method, 3, 0, P, 148, 0.01, *tan) for P in (1, 148 * 20, 148 * 88 + 1)]) == [1, 1, 0]
    assert ask([(method, 3, 0, 148, 148, 0.01, *ph) for ph in
                ((-1.0, -1.0, 1.0, 5.0), (0.0, 0.0, 1.0, 2.5), (0.0, 0.0, 1.0, float("inf")),
                 (0.0, 0.0, 1.0, 0.0), (0.0, 0.0, 1.0, float("nan")))]) == [1] * 5

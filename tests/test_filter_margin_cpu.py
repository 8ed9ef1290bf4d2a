"""The narrow phase's filter settles items by a bound on how far its Bernstein
coefficients can be from the reference formulation's.  Both are run operation
for operation on the host, with the filter's own weights, over random pairs of
several kinds of coefficients: the difference stays below the bound at every
order."""

import pathlib
import subprocess

import pytest

HERE = pathlib.Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = tmp_path_factory.mktemp("filter") / "harness"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-x", "c++",
                    f"-I{HERE.parent / 'mizuba_b200' / 'csrc'}", str(HERE / "filter_margin_harness.cpp"), "-o", str(exe)],
                   check=True)
    return exe


@pytest.mark.parametrize("order", range(2, 33))
def test_difference_within_the_margin(harness, order):
    r = subprocess.run([str(harness), str(order), "400", str(order)], check=True, capture_output=True, text=True)
    worst = {int(k): float(v) for k, v in (line.split() for line in r.stdout.splitlines())}
    assert len(worst) == 5
    for kind, v in worst.items():
        assert 0.0 < v < 1.0, (kind, v)

"""The delay kernel's tiles and lists on the CPU: every sum as the kernel forms it equals the
direct one (tests/delay_plan_check.cpp), in one order whatever the batch."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("plan") / "check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-mfma", "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "delay_plan_check.cpp")], check=True)

    def run(*args):
        p = subprocess.run([exe] + [str(x) for x in args], capture_output=True, text=True)
        assert p.returncode == 0, (args, p.stdout)
        w = p.stdout.split()
        return dict(zip(w[::2], w[1::2]))
    return run


# precision, nodes, density, shortest and longest delay, noise terms
SHAPES = [("double", 1, 1.0, 1, 1, 2), ("double", 2, 0.9, 32, 33, 2), ("float", 31, 0.5, 33, 63, 2), ("double", 33, 0.5, 1, 300, 1),
          ("float", 100, 0.3, 10, 300, 2), ("double", 100, 0.9, 40, 64, 2), ("float", 97, 0.9, 2, 400, 2),
          ("double", 601, 0.1, 20, 300, 2), ("float", 701, 0.04, 20, 300, 2), ("float", 1000, 0.1, 31, 200, 1),
          ("float", 1024, 0.02, 32, 1000, 2), ("double", 64, 0.0, 5, 50, 2)]


@pytest.mark.parametrize("precision,nodes,density,lo,hi,noise", SHAPES)
def test_lists_give_the_direct_sums_in_any_batch(check, precision, nodes, density, lo, hi, noise):
    plans = [check(precision, nodes, sims, 148, density, lo, hi, 1, noise) for sims in (1, 300, 2000)]
    assert all(p["plan"] == "1" for p in plans), plans
    assert len({p["sum"] for p in plans}) == 1, plans


@pytest.mark.parametrize("precision", ["float", "double"])
def test_only_near_heavy_tables_are_left_out(check, precision):
    """Delays of 60-400 steps and 2 to 20 times as fast, five simulations of each: the fast
    tables' simulations are left to the per-step kernel, the others stay."""
    p = check(precision, 60, 100, 148, 0.4, 60, 400, 20, 2)
    assert p["plan"] == "1" and 0 < int(p["rest"]) < 100
    assert check(precision, 60, 400, 148, 0.4, 60, 400, 20, 2)["plan"] == "0"   # most of a large batch
    q = check(precision, 60, 5, 148, 0.4, 60, 400, 1, 2)   # the slowest alone
    assert q["rest"] == "0"


def test_one_slow_table_does_not_decide_for_the_others(check):
    """Delays to 12,000 steps leave no tile of four sources, half of them do."""
    p = check("double", 30, 10, 148, 0.5, 100, 12000, 2, 2)
    assert (p["plan"], p["rest"]) == ("1", "5")


def test_two_passes_are_planned(check):
    assert check("float", 701, 3, 148, 0.04, 25, 300, 1, 2)["passes"] == "2"
    assert check("float", 1000, 3, 148, 0.1, 25, 300, 1, 2)["passes"] == "2"
    assert check("double", 701, 3, 148, 0.04, 25, 300, 1, 2)["passes"] == "1"

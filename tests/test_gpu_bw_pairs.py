"""The Balloon-Windkessel step of several items at once (bw_step64_n): which form an item
takes is its own affair, and a step that leaves a table centre's series takes the general
power.  Jansen-Rit drives the inflow f to 1 + 0.41 (y1 - y2); an SC weight of 1e4 and more
takes f to thousands and the volume nu out of the power table."""
import numpy as np
import pytest

import cases
from cubnm_b200 import core
from oracle import oracle

pytestmark = pytest.mark.gpu

NODES = 40


def _args(N, G, precision="fp64", nodes=NODES, ms=600):
    a = list(cases.synthetic_args("JR", N=N, nodes=nodes, duration_s=4, seed=3, density=0.6, G=G, bold_remove_s=0,
                                  do_fcd=False, precision=precision))
    a[7] = dict(a[7], do_fc="0", noise_time_steps="200")
    a[16], a[17], a[18] = ms, 100, 100
    return a


@pytest.mark.parametrize("precision,nodes,N,kernel", [("fp64", NODES, 1203, "k_tile64"), ("fp32", NODES, 1200, "k_integrate_mma"),
                                                      ("fp32", 120, 2500, "k_integrate_tc")])
def test_a_simulation_does_not_depend_on_its_neighbours(precision, nodes, N, kernel):
    calm = np.linspace(0.3, 0.9, N)
    mixed = np.where(np.arange(N) % 2 == 0, calm, 3e4)
    bold = []
    for G in (calm, mixed):
        bold.append(core.run_simulations(*_args(N, G, precision, nodes, ms=2000))["sim_bold"])
        assert core.last_kernel() == kernel
    assert np.abs(bold[1][1] - bold[0][1]).max() > 0.1        # the odd ones are elsewhere
    np.testing.assert_array_equal(bold[1][::2], bold[0][::2])


@pytest.mark.parametrize("N", [6, 1203])
def test_large_inflow_matches_oracle(N):
    """f in the thousands: the volume moves by more than its centre's series reaches in one step.
    FP64 at the bound of the other parity tests."""
    G = np.resize(np.array([0.5, 300.0, 2e3, 1e4, 3e4, 6e4]), N)
    got = core.run_simulations(*_args(N, G, ms=400))
    ref = oracle.run_simulations(*_args(6, G[:6], ms=400))
    assert ref["sim_bold"].max() > 0.1 and np.isfinite(ref["sim_bold"]).all()
    np.testing.assert_allclose(got["sim_bold"][-6 - N % 6:][:6], ref["sim_bold"], rtol=1e-8, atol=1e-12)

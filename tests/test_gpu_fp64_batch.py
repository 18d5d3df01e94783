"""An FP64 simulation without delays gives the same bits in any batch: k_one64 (few
simulations, one per CTA) and k_tile64 (tiles of eight) form the coupling sum in one order.
Node counts at and around the 8-source tiles and the compiled extents of both kernels."""
import numpy as np
import pytest

import cases
from cubnm_b200 import core

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", ["rWW", "WC", "JR", "rWWEx"])
@pytest.mark.parametrize("nodes", [2, 7, 8, 31, 33, 64, 65, 88, 96, 97, 104, 105, 121, 128])
def test_one_simulation_equals_the_same_in_a_large_batch(model, nodes):
    N = 1203
    a = list(cases.synthetic_args(model, N=N, nodes=nodes, duration_s=4, seed=nodes, density=0.6,
                                  G=np.linspace(0.2, 1.5, N), bold_remove_s=0, do_fcd=False))
    a[7] = dict(a[7], do_fc="0", noise_time_steps="150")
    a[16], a[17], a[18] = 300, 100, 100
    a[1] = np.stack([cases.synthetic_sc(nodes, 0.6, s).reshape(-1) for s in (1, 2)])
    a[2] = (np.arange(N) % 2).astype(np.intc)
    whole = core.run_simulations(*a)
    assert core.last_kernel() == "k_tile64"
    pick = np.r_[0:3, 600:602, N - 3:N]
    b = list(a)
    b[2], b[6], b[14] = a[2][pick], a[6][pick], pick.size
    b[4] = np.ascontiguousarray(a[4][:, pick])
    b[5] = np.ascontiguousarray(a[5].reshape(-1, N, nodes)[:, pick].reshape(a[5].shape[0], -1))
    alone = core.run_simulations(*b)
    assert core.last_kernel() == "k_one64"
    np.testing.assert_array_equal(alone["sim_bold"], whole["sim_bold"][pick])
    np.testing.assert_array_equal(alone["_sim_states"], whole["_sim_states"][:, pick])

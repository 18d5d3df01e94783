"""The Balloon-Windkessel step away from rest: strong activity drives the inflow f and the
volume nu through several centres of the power table (and past them where the general
form takes over).  FP64 against the oracle at the bound of the other parity tests (the
powers are within a few ulp of pow(), and the model is a stable relaxation)."""
import numpy as np
import pytest

import cases
from cubnm_b200 import core
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("delay", [False, True])
@pytest.mark.parametrize("N", [6, 700])
def test_strong_activity_matches_oracle(N, delay):
    nodes = 20
    # w_p to 30 drives S_E to saturation (f to about 1.4); TR / bw_dt as in the other tests
    a = list(cases.synthetic_args("rWW", N=N, nodes=nodes, duration_s=9, seed=2, density=0.6,
                                  G=np.linspace(0.1, 30.0, N), w_p=np.linspace(0.0, 30.0, N),
                                  J_N=np.linspace(0.05, 2.0, N), bold_remove_s=0, do_fcd=False))
    a[7] = dict(a[7], noise_time_steps="500")
    a[17] = a[18] = 500
    if delay:
        a[3] = np.ascontiguousarray(cases.synthetic_lengths(nodes, 2).ravel())
        a[6] = np.full(N, 6.0)
        a[11] = True
    got = core.run_simulations(*[x.copy() if isinstance(x, np.ndarray) else x for x in a])
    pick = np.arange(N) if N < 10 else np.r_[0:3, N // 2:N // 2 + 3, N - 3:N]
    b = list(a)
    b[2], b[6], b[14] = a[2][pick], a[6][pick], pick.size
    b[4] = np.ascontiguousarray(a[4][:, pick])
    b[5] = np.ascontiguousarray(a[5].reshape(4, N, nodes)[:, pick].reshape(4, -1))
    ref = oracle.run_simulations(*b)
    assert ref["sim_bold"].max() > 0.05          # the haemodynamic state has left rest
    np.testing.assert_allclose(got["sim_bold"][pick], ref["sim_bold"], rtol=1e-8, atol=1e-12)

"""The delay kernel: the same bits in any batch, and the forms that other tests do not reach.

The coupling sums run over the sources in ascending order whatever the tiles are (which
depend on the number of simulations, on the longest delay and on the fullest SC of the
batch).  FP64 against the oracle at the bound of the other parity tests (1e-8 relative,
1e-12 absolute); FP32 against FP64 at the bounds the FP32 delay tests have."""
import numpy as np
import pytest

import cases
from cubnm_b200 import core
from oracle import oracle

pytestmark = pytest.mark.gpu


def _args(model, nodes, N, dist, velocity, ms, density, precision="fp64"):
    a = list(cases.synthetic_args(model, N=N, nodes=nodes, duration_s=4, seed=nodes, density=density,
                                  G=np.linspace(0.2, 1.2, N), bold_remove_s=0, do_fcd=False, precision=precision))
    a[7] = dict(a[7], do_fc="0", noise_time_steps="300")
    a[3] = np.ascontiguousarray(dist.ravel())
    a[6] = np.broadcast_to(np.asarray(velocity, dtype=float), (N,)).copy()
    a[11] = True
    a[16], a[17], a[18] = ms, 100, 100
    return a


def _uniform(nodes, lo, hi, seed=0):
    """Symmetric lengths for delays of lo to hi steps at 6 m/s and 0.1 ms (0.6 mm a step)."""
    d = np.random.default_rng(seed).uniform(0.6 * lo, 0.6 * hi, (nodes, nodes))
    return np.tril(d, -1) + np.tril(d, -1).T


def _copy(args):
    return [x.copy() if isinstance(x, np.ndarray) else x for x in args]


def _subset(a, pick):
    b, N, n = _copy(a), a[14], a[15]
    b[2], b[6], b[14] = a[2][pick], a[6][pick], pick.size
    b[4] = np.ascontiguousarray(a[4][:, pick])
    b[5] = np.ascontiguousarray(a[5].reshape(-1, N, n)[:, pick].reshape(a[5].shape[0], -1))
    return b


@pytest.mark.parametrize("model,precision,nodes", [("rWW", "fp64", 100), ("JR", "fp64", 45), ("rWWEx", "fp64", 200),
                                                   ("rWW", "fp32", 100), ("WC", "fp32", 230)])
def test_one_simulation_equals_the_same_in_a_large_batch(model, precision, nodes):
    N = 600
    v = np.where(np.arange(N) % 3 == 0, 6.0, np.linspace(2.0, 7.0, N))   # slower ones lengthen every window
    a = _args(model, nodes, N, _uniform(nodes, 12, 250), v, 250, 0.5, precision)
    whole = core.run_simulations(*_copy(a))
    assert core.last_kernel() == "k_integrate_delay"
    pick = np.array([0, 3, 300])
    alone = core.run_simulations(*_subset(a, pick))
    assert core.last_kernel() == "k_integrate_delay"
    np.testing.assert_array_equal(alone["sim_bold"], whole["sim_bold"][pick])
    np.testing.assert_array_equal(alone["_sim_states"], whole["_sim_states"][:, pick])


@pytest.mark.parametrize("model,nodes,lo,hi,density", [("rWW", 97, 1, 400, 0.9), ("WC", 130, 2, 500, 0.9),
                                                       ("rWW", 601, 20, 300, 0.1)])
def test_fp64_matches_oracle(model, nodes, lo, hi, density):
    """Near pairs in several warps (a barrier every step), and more than 512 nodes."""
    a = _args(model, nodes, 2, _uniform(nodes, lo, hi), 6.0, 201, density)
    got = core.run_simulations(*_copy(a))
    assert core.last_kernel() == "k_integrate_delay"
    ref = oracle.run_simulations(*_copy(a))
    vols = 2 * nodes   # 200 of the 201 ms
    np.testing.assert_allclose(got["sim_bold"][:, :vols], ref["sim_bold"][:, :vols], rtol=1e-8, atol=1e-12)
    np.testing.assert_allclose(got["_sim_states"], ref["_sim_states"], rtol=1e-8, atol=1e-12)


@pytest.mark.parametrize("nodes,density,ms", [(701, 0.04, 331), (1000, 0.1, 200)])
def test_two_passes_over_the_targets(nodes, density, ms):
    dist = _uniform(nodes, 25, 300)
    o64 = core.run_simulations(*_args("rWW", nodes, 2, dist, 6.0, ms, density))
    o32 = core.run_simulations(*_args("rWW", nodes, 2, dist, 6.0, ms, density, "fp32"))
    assert core.last_kernel() == "k_integrate_delay/2"
    np.testing.assert_allclose(o32["_sim_states"], o64["_sim_states"], rtol=1e-4, atol=1e-5)
    assert np.abs(o32["sim_bold"] - o64["sim_bold"]).max() < 1e-4


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("fic", [0, 2])
def test_mixed_velocities_run_on_two_kernels_at_once(precision, fic):
    """Simulations whose delays are mostly below a block of 32 steps run on the per-step
    kernel, beside the others: each gives what it gives alone."""
    nodes, N = 60, 40
    a = _args("rWW", nodes, N, _uniform(nodes, 60, 300), np.linspace(4.0, 60.0, N), 1200 if fic else 300, 0.5, precision)
    a[7] = dict(a[7], do_fic=str(int(fic > 0)), max_fic_trials="3" if fic == 2 else "0", I_SAMPLING_START="0",
                I_SAMPLING_END="1000")
    b = _copy(a)
    whole = core.run_simulations(*b)
    assert core.last_kernel() == "k_integrate_delay+k_integrate_sim"
    assert not fic or whole["_global_ints"].max() > 0   # trials of the numerical FIC
    kernels = set()
    for i in (0, 5, 20, 39):
        c = _subset(a, np.array([i]))
        alone = core.run_simulations(*c)
        kernels.add(core.last_kernel())
        np.testing.assert_array_equal(alone["sim_bold"], whole["sim_bold"][[i]])
        np.testing.assert_array_equal(alone["_sim_states"], whole["_sim_states"][:, [i]])
        np.testing.assert_array_equal(alone["_global_ints"], whole["_global_ints"][:, [i]])
        np.testing.assert_array_equal(c[5], b[5].reshape(-1, N, nodes)[:, i])   # wIE as written back
    assert kernels == {"k_integrate_delay", "k_integrate_sim"}
    if precision == "fp64":
        pick = np.array([0, 39])
        ref = oracle.run_simulations(*_subset(a, pick))
        np.testing.assert_allclose(whole["sim_bold"][pick], ref["sim_bold"], rtol=1e-8, atol=1e-12)

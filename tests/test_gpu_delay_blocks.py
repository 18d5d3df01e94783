"""The delay kernel (blocks of 32 steps) where its index arithmetic can go wrong.

FP64 against the oracle at the bound of the other parity tests (1e-8 relative,
1e-12 absolute: the kernel sums far pairs before near ones, a reordering of a
double sum).  Cases: fewer nodes than a warp, one more than a warp or a block,
rows of one and several warps, delays below, at and above a block and a
power-of-two ring, run lengths that are no multiple of a block, networks with
and without near pairs, several (SC, velocity) pairs, and more simulations than
resident CTAs.
"""
import numpy as np
import pytest

import cases
from cubnm_b200 import core
from oracle import oracle

pytestmark = pytest.mark.gpu

KEYS = ("sim_bold", "sim_fc_trils", "_sim_states")


def _args(model, nodes, N, dist, velocity, ms, density=0.5, precision="fp64", dt=0.1):
    a = list(cases.synthetic_args(model, N=N, nodes=nodes, duration_s=4, seed=nodes, density=density,
                                  G=np.linspace(0.2, 1.2, N), bold_remove_s=0, do_fcd=False, precision=precision))
    a[7] = dict(a[7], noise_time_steps="300")
    a[3] = np.ascontiguousarray(dist.ravel())
    a[6] = np.broadcast_to(np.asarray(velocity, dtype=float), (N,)).copy()
    a[11] = True
    a[16], a[17], a[18], a[20] = ms, 100, 100, dt
    return a


def _copy(args):
    return [x.copy() if isinstance(x, np.ndarray) else x for x in args]


def _uniform(nodes, lo, hi, seed=0):
    d = np.random.default_rng(seed).uniform(lo, hi, (nodes, nodes))
    d = np.tril(d, -1) + np.tril(d, -1).T
    return d


# (model, nodes, sims, shortest and longest delay in steps, duration in ms)
SHAPES = [("rWW", 2, 3, 32, 33, 700), ("rWW", 31, 2, 33, 63, 333), ("rWW", 33, 2, 40, 64, 301),
          ("WC", 65, 2, 32, 65, 407), ("rWW", 97, 3, 3, 140, 501), ("rWWEx", 40, 2, 1, 300, 512),
          ("JR", 48, 2, 20, 129, 300), ("rWW", 130, 2, 31, 513, 203)]


@pytest.mark.parametrize("model,nodes,N,lo,hi,ms", SHAPES)
def test_fp64_matches_oracle(model, nodes, N, lo, hi, ms):
    dist = _uniform(nodes, lo * 0.6, hi * 0.6, nodes)   # 6 m/s at dt 0.1 ms: 0.6 mm a step
    density = 0.5 if lo >= 32 else 0.9
    a = _args(model, nodes, N, dist, 6.0, ms, density=max(density, 0.5))
    got, ref = core.run_simulations(*_copy(a)), oracle.run_simulations(*_copy(a))
    # the truncated iteration count (0.7 s / 1 ms = 699) can leave the last volume
    # unwritten on both sides, and with it the FC undefined
    written, vols = int((ms / 1000.0) / 0.001) // 100, ms // 100
    np.testing.assert_allclose(got["sim_bold"][:, :written * nodes], ref["sim_bold"][:, :written * nodes], rtol=1e-8,
                               atol=1e-12)
    for k in KEYS[1:] if written == vols else KEYS[2:]:
        np.testing.assert_allclose(got[k], ref[k], rtol=1e-8, atol=1e-12, err_msg=k)


def test_fp32_follows_fp64():
    dist = _uniform(160, 2.0, 150.0)
    a = _args("rWW", 160, 5, dist, 6.0, 2000)
    o64 = core.run_simulations(*_copy(a))
    o32 = core.run_simulations(*_copy(_args("rWW", 160, 5, dist, 6.0, 2000, precision="fp32")))
    # FP32 states: rounding of 6e-8 a step on states of order 0.1
    np.testing.assert_allclose(o32["_sim_states"], o64["_sim_states"], rtol=1e-4, atol=1e-5)
    assert np.abs(o32["sim_bold"] - o64["sim_bold"]).max() < 1e-4


def test_pairs_and_more_simulations_than_ctas():
    """Two SCs x two velocities; 6,001 two-node-warp simulations against the same ones alone."""
    nodes, N = 20, 6001
    dist = _uniform(nodes, 10.0, 60.0)
    a = _args("rWW", nodes, N, dist, np.where(np.arange(N) % 3 == 0, 4.0, 7.0), 200)
    a[1] = np.stack([cases.synthetic_sc(nodes, 0.5, s).reshape(-1) for s in (1, 2)])
    a[2] = (np.arange(N) % 2).astype(np.intc)
    whole = core.run_simulations(*_copy(a))
    pick = np.r_[0:6, 3000:3006, N - 6:N]
    b = _copy(a)
    b[2], b[6], b[14] = a[2][pick], a[6][pick], pick.size
    b[4] = np.ascontiguousarray(a[4][:, pick])
    b[5] = np.ascontiguousarray(a[5].reshape(4, N, nodes)[:, pick].reshape(4, -1))
    ref = oracle.run_simulations(*_copy(b))
    for k in ("sim_bold", "sim_fc_trils"):
        np.testing.assert_allclose(whole[k][pick], ref[k], rtol=1e-8, atol=1e-12, err_msg=k)


def test_two_passes_over_the_targets():
    """Above 512 nodes in FP32 with few entries per tile the sums are formed for half the
    targets at a time (an odd node count, near pairs, 331 ms = no whole number of blocks)."""
    nodes = 701
    dist = _uniform(nodes, 6.0, 190.0)
    a = _args("rWW", nodes, 3, dist, 6.0, 331, density=0.08)
    o64 = core.run_simulations(*_copy(a))
    o32 = core.run_simulations(*_copy(_args("rWW", nodes, 3, dist, 6.0, 331, density=0.08, precision="fp32")))
    np.testing.assert_allclose(o32["_sim_states"], o64["_sim_states"], rtol=1e-4, atol=1e-5)
    assert np.abs(o32["sim_bold"] - o64["sim_bold"]).max() < 1e-4

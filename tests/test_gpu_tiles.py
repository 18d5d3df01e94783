"""The register-resident tile kernels (no delays) where their index arithmetic can go wrong.

FP64 (up to 128 nodes: one simulation per CTA, or tiles of eight above four
simulations per SM) against the oracle at the bound of the other parity tests
(1e-8 relative, 1e-12 absolute: the sums are formed in another order).  FP32 tiles
(up to 224 nodes) against the FP64 run: rounding of 6e-8 a step on states of order
0.1, held to the bounds the FP32 kernels have against each other.  Node counts at
and around the 8- and 16-node tiles and the compiled extents, batches that leave
empty columns, several SCs, more noise repeats than one, steps per millisecond
other than ten.
"""
import numpy as np
import pytest

import cases
from cubnm_b200 import core
from oracle import oracle

pytestmark = pytest.mark.gpu


def _args(model, nodes, N, precision="fp64", ms=400, dt=0.1, seed=0):
    a = list(cases.synthetic_args(model, N=N, nodes=nodes, duration_s=4, seed=seed + nodes, density=0.6,
                                  G=np.linspace(0.2, 1.2, N), bold_remove_s=0, do_fcd=False, precision=precision))
    a[7] = dict(a[7], noise_time_steps="150")
    a[16], a[17], a[18], a[20] = ms, 100, 100, dt
    if nodes < 2:
        a[7]["do_fc"] = "0"
        a[1] = np.zeros((1, 1))   # synthetic_sc divides by its mean row sum, 0 for one node
    return a


def _copy(args):
    return [x.copy() if isinstance(x, np.ndarray) else x for x in args]


def _subset(a, pick):
    b, N, n = _copy(a), a[14], a[15]
    b[2], b[6], b[14] = a[2][pick], a[6][pick], pick.size
    b[4] = np.ascontiguousarray(a[4][:, pick])
    b[5] = np.ascontiguousarray(a[5].reshape(-1, N, n)[:, pick].reshape(a[5].shape[0], -1))
    return b


@pytest.mark.parametrize("model,nodes", [("rWW", 1), ("rWW", 8), ("WC", 9), ("rWW", 33), ("JR", 64), ("rWWEx", 65),
                                         ("rWW", 100), ("WC", 105), ("JR", 113), ("rWW", 128)])
@pytest.mark.parametrize("N", [3, 1203])
def test_fp64_matches_oracle(model, nodes, N):
    a = _args(model, nodes, N)
    if nodes > 1:
        a[1] = np.stack([cases.synthetic_sc(nodes, 0.6, s).reshape(-1) for s in (1, 2)])
        a[2] = (np.arange(N) % 2).astype(np.intc)
    got = core.run_simulations(*_copy(a))
    pick = np.arange(N) if N < 10 else np.r_[0:5, 600:603, N - 5:N]
    ref = oracle.run_simulations(*_subset(a, pick))
    np.testing.assert_allclose(got["sim_bold"][pick], ref["sim_bold"], rtol=1e-8, atol=1e-12)
    np.testing.assert_allclose(got["_sim_states"][:, pick], ref["_sim_states"], rtol=1e-8, atol=1e-12)


@pytest.mark.parametrize("model,nodes", [("rWW", 1), ("rWW", 16), ("WC", 17), ("JR", 48), ("rWW", 81), ("rWWEx", 97),
                                         ("rWW", 112), ("WC", 129), ("rWW", 161), ("JR", 177), ("rWW", 200),
                                         ("rWWEx", 224)])
def test_fp32_follows_fp64(model, nodes):
    N = 21
    a = _args(model, nodes, N)
    if nodes > 1:
        a[1] = np.stack([cases.synthetic_sc(nodes, 0.6, s).reshape(-1) for s in (1, 2)])
        a[2] = (np.arange(N) % 2).astype(np.intc)
    o64 = core.run_simulations(*_copy(a))
    a[7] = dict(a[7], precision="fp32")
    o32 = core.run_simulations(*_copy(a))
    assert core.last_integrator() == "tc1"
    for v in range(o64["_sim_states"].shape[0]):
        scale = max(1.0, float(np.abs(o64["_sim_states"][v]).max()))
        assert np.abs(o32["_sim_states"][v] - o64["_sim_states"][v]).max() < 1e-4 * scale, v
    assert np.abs(o32["sim_bold"] - o64["sim_bold"]).max() < 1e-4


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("dt", [1.0, 0.5, 0.04])
def test_steps_per_millisecond(precision, dt):
    """1, 2 and 25 (chunks of ten, ten and five) integration steps per Balloon-Windkessel step."""
    for N in (3, 1203) if precision == "fp64" else (9,):
        a = _args("rWW", 40, N, precision=precision, ms=300, dt=dt)
        pick = np.r_[0:3] if N < 10 else np.r_[0:3, N - 3:N]
        got = core.run_simulations(*_copy(a))
        b = _subset(a, pick)
        b[7] = dict(b[7], precision="fp64")
        ref = oracle.run_simulations(*b)
        tol = dict(rtol=1e-8, atol=1e-12) if precision == "fp64" else dict(rtol=1e-3, atol=1e-4)
        np.testing.assert_allclose(got["sim_bold"][pick], ref["sim_bold"], **tol)


@pytest.mark.parametrize("model,nodes", [("rWW", 113), ("rWW", 128), ("WC", 128), ("JR", 120), ("rWWEx", 127)])
def test_fp32_wide_tiles_match_narrow_ones(model, nodes):
    """More than 16 simulations per SM of 113-128 nodes take the 32-wide tcgen05 tiles; the
    same simulations alone the eight-wide ones.  Both form the coupling from 16-bit halves with FP32 sums."""
    N = 2500
    a = _args(model, nodes, N, precision="fp32", ms=300)
    a[1] = np.stack([cases.synthetic_sc(nodes, 0.6, s).reshape(-1) for s in (1, 2)])
    a[2] = (np.arange(N) % 2).astype(np.intc)
    wide = core.run_simulations(*_copy(a))
    assert core.last_integrator() == "tc1"
    pick = np.r_[0:5, 1200:1203, N - 5:N]
    narrow = core.run_simulations(*_subset(a, pick))
    assert np.abs(wide["sim_bold"][pick] - narrow["sim_bold"]).max() < 1e-5
    for v in range(wide["_sim_states"].shape[0]):
        scale = max(1.0, float(np.abs(narrow["_sim_states"][v]).max()))
        assert np.abs(wide["_sim_states"][v][pick] - narrow["_sim_states"][v]).max() < 1e-4 * scale, v


@pytest.mark.parametrize("model,nodes", [("rWW", 33), ("WC", 97), ("JR", 200)])
@pytest.mark.parametrize("exponent", [-60, 40])
def test_fp32_weights_scale_exactly(model, nodes, exponent):
    """The tiles scale each row of the SC into the range of their 16-bit halves.  A power of
    two moved from G to the SC changes no bit: every product and sum scales with it."""
    a = _args(model, nodes, 9, precision="fp32", ms=300)
    ref = core.run_simulations(*_copy(a))
    assert core.last_integrator() == "tc1"
    b = _copy(a)
    b[1] = b[1] * 2.0 ** exponent
    b[4] = b[4] * 2.0 ** -exponent
    got = core.run_simulations(*b)
    np.testing.assert_array_equal(got["sim_bold"], ref["sim_bold"])


@pytest.mark.parametrize("nodes,rounded", [(100, False), (129, True), (224, True), (225, True)])
def test_fp32_fic_returns_wie_as_integrated(nodes, rounded):
    """Above 128 nodes an FP32 run returns the wIE of the analytical FIC in FP32, whichever
    kernel it takes; the solver itself is FP64 in both precisions."""
    N = 5
    a = list(cases.synthetic_args("rWW", N=N, nodes=nodes, duration_s=1, seed=nodes, density=0.3,
                                  G=np.linspace(0.2, 1.2, N), bold_remove_s=0, do_fcd=False, do_fic=1,
                                  precision="fp64"))
    a[16], a[17], a[18] = 200, 100, 100
    wie = []
    for precision in ("fp64", "fp32"):
        b = _copy(a)
        b[7] = dict(a[7], precision=precision)
        core.run_simulations(*b)
        wie.append(b[5][2].copy())
    np.testing.assert_array_equal(wie[1], wie[0].astype(np.float32).astype(np.float64) if rounded else wie[0])

"""Which kernel integrates a run, by its sizes (core.last_kernel)."""
import numpy as np
import pytest

import cases
from cubnm_b200 import core

pytestmark = pytest.mark.gpu


def _run(model, nodes, N, precision, velocity=0.0, density=0.3, scs=1, ms=100, **config):
    a = list(cases.synthetic_args(model, N=N, nodes=nodes, duration_s=1, seed=nodes, density=density,
                                  G=np.linspace(0.2, 1.2, N), bold_remove_s=0, do_fcd=False, precision=precision))
    a[7] = dict(a[7], do_fc="0", noise_time_steps="100", **config)
    a[16], a[17], a[18] = ms, 100, 100
    if scs > 1:
        a[1] = np.stack([cases.synthetic_sc(nodes, density, s).reshape(-1) for s in range(scs)])
        a[2] = (np.arange(N) % scs).astype(np.intc)
    if velocity:
        a[3] = np.ascontiguousarray(cases.synthetic_lengths(nodes, nodes).ravel())
        a[6] = np.full(N, velocity)
        a[11] = True
    core.run_simulations(*a)
    return core.last_kernel()


@pytest.mark.parametrize("model,nodes,N,precision,kernel", [
    ("rWW", 68, 5, "fp64", "k_one64"), ("rWW", 128, 1200, "fp64", "k_tile64"), ("rWW", 129, 5, "fp64", "k_integrate_sim"),
    ("Kuramoto", 40, 5, "fp64", "k_integrate_sim"), ("rWW", 100, 5000, "fp32", "k_integrate_mma"),
    ("WC", 128, 100, "fp32", "k_integrate_mma"), ("WC", 128, 2500, "fp32", "k_integrate_tc"),
    ("JR", 200, 9, "fp32", "k_integrate_mma"), ("rWW", 225, 9, "fp32", "k_integrate_sim")])
def test_without_delays(model, nodes, N, precision, kernel):
    assert _run(model, nodes, N, precision) == kernel


@pytest.mark.parametrize("nodes,N,scs,kernel", [
    (100, 148, 1, "k_one64"), (100, 450, 1, "k_tile64"), (100, 592, 1, "k_tile64"), (68, 450, 1, "k_tile64"),
    (100, 600, 75, "k_tile64"), (100, 600, 600, "k_one64"), (32, 1184, 1, "k_tile64"), (32, 1000, 1000, "k_one64")])
def test_fp64_form_by_waves(nodes, N, scs, kernel):
    """Tiles of eight where they finish first on 148 SMs: not for few simulations, nor where
    each has an SC of its own and a tile one live column."""
    assert _run("rWW", nodes, N, "fp64", scs=scs) == kernel


@pytest.mark.parametrize("model,nodes,precision,density,kernel", [
    ("rWW", 100, "fp64", 0.2, "k_integrate_delay"), ("WC", 400, "fp32", 0.2, "k_integrate_delay"),
    ("rWW", 1000, "fp32", 0.1, "k_integrate_delay/2"), ("rWW", 600, "fp64", 0.2, "k_integrate_delay"),
    ("rWW", 900, "fp64", 0.1, "k_integrate_sim"), ("Kuramoto", 60, "fp64", 0.2, "k_integrate_sim")])
def test_with_delays(model, nodes, precision, density, kernel):
    assert _run(model, nodes, 3, precision, velocity=6.0, density=density) == kernel


@pytest.mark.parametrize("nodes,N,scs,density,kernel", [
    (200, 300, 1, 0.1, "k_integrate_mma"), (200, 300, 300, 0.1, "k_integrate_sim"),
    (200, 148, 148, 0.8, "k_integrate_mma"), (128, 300, 300, 0.1, "k_integrate_mma")])
def test_fp32_tiles_by_their_filling(nodes, N, scs, density, kernel):
    """Above 128 nodes a sparse SC for every simulation leaves the tiles in a run that is long enough for
    packing the sparse tables on the host not to count."""
    assert _run("rWW", nodes, N, "fp32", scs=scs, density=density, ms=3000) == kernel


def test_forced_kernels(monkeypatch):
    monkeypatch.setenv("CBNM_FP32_KERNEL", "simt")
    assert _run("rWW", 100, 20, "fp32") == "k_integrate_sim"
    monkeypatch.setenv("CBNM_FP32_KERNEL", "lanes")
    assert _run("rWW", 150, 20, "fp32", velocity=6.0) == "k_integrate_lanes"
    monkeypatch.delenv("CBNM_FP32_KERNEL")
    monkeypatch.setenv("CBNM_FP32_TC", "pp")
    assert _run("rWW", 100, 100, "fp32") == "k_integrate_pp"


@pytest.mark.parametrize("value,fp64,delayed", [("auto", "k_one64", "k_integrate_delay"),
                                                ("sparse", "k_integrate_sim", "k_integrate_sim"),
                                                ("dense", "k_integrate_sim", "k_integrate_sim")])
def test_coupling_form(value, fp64, delayed, monkeypatch):
    """CBNM_COUPLING asks for the per-step kernels by naming a coupling form, not by being set."""
    monkeypatch.setenv("CBNM_COUPLING", value)
    assert _run("rWW", 60, 5, "fp64") == fp64
    assert _run("rWW", 60, 5, "fp64", velocity=6.0) == delayed

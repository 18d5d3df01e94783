"""The adjoint kernels around their compiled extents (48, 112, 160, 208 nodes in registers,
above that one thread per node): BOLD against an ordinary FP32 run and an FP64 run, and the
gradient of a weighted sum of BOLD along a random direction of all parameters against FP64
central differences (relative 1e-3, the bound of the other gradient tests)."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


def _run(sc, p, dur, tr, precision):
    from cubnm_b200 import core
    G, reg = p[0], p[1:]
    N, nodes = reg[0].shape
    cfg = cases.model_config("rWW", 0, window_size=4, window_step=2, bold_remove_s=0, do_fc=False, do_fcd=False)
    cfg["precision"] = precision
    out = core.run_simulations(
        "rWW", np.ascontiguousarray(sc.reshape(1, -1)), np.zeros(N, np.intc), np.zeros(nodes * nodes), G[None, :].copy(),
        np.ascontiguousarray(np.vstack([x.reshape(1, -1) for x in reg])), np.zeros(N), cfg, True, False, False, False, False,
        False, N, nodes, dur * 1000, tr, tr, 0, 0.1, 1.0)
    return out["sim_bold"].reshape(N, -1, nodes)


@pytest.mark.parametrize("nodes", [2, 48, 49, 112, 113, 160, 161, 208, 209])
def test_bold_and_gradient(nodes):
    import torch
    from cubnm_b200 import core
    from cubnm_b200.grad import RWWProblem
    N, dur, tr = 3, 2, 100
    rng = np.random.default_rng(nodes)
    sc = cases.synthetic_sc(nodes, 0.9 if nodes < 10 else 0.4, 3)
    p = [rng.uniform(0.5, 2.0, N), rng.uniform(0.8, 1.4, (N, nodes)), rng.uniform(0.1, 0.3, (N, nodes)),
         rng.uniform(0.8, 1.2, (N, nodes)), np.full((N, nodes), 0.01)]
    prob = RWWProblem(sc, nodes, dur, bold_tr=tr, segment_steps=1000)
    t = [torch.tensor(x, dtype=torch.float64, device="cuda:0", requires_grad=True) for x in p]
    bold = prob.bold(*t)
    wgt = rng.normal(size=tuple(bold.shape))
    (bold * torch.tensor(wgt, device="cuda:0")).sum().backward()
    got = bold.detach().cpu().numpy()

    ref = _run(sc, p, dur, tr, "fp64")
    ordinary = _run(sc, p, dur, tr, "fp32")
    assert core.last_kernel() == "k_integrate_mma"
    # FP32 states: rounding of 6e-8 a step on a relaxing system, both routes
    for x in (got, ordinary):
        assert np.linalg.norm(x - ref) < 1e-6 * np.linalg.norm(ref)

    v = [rng.normal(size=x.shape) * s for x, s in zip(p, (1.0, 0.3, 0.1, 0.3, 0.003))]
    h = 1e-4
    up, down = ([x + s * h * d for x, d in zip(p, v)] for s in (1, -1))
    fd = ((_run(sc, up, dur, tr, "fp64") - _run(sc, down, dur, tr, "fp64")) * wgt).sum(axis=(1, 2)) / (2 * h)
    adj = sum((x.grad.cpu().numpy().reshape(N, -1) * d.reshape(N, -1)).sum(axis=1) for x, d in zip(t, v))
    assert np.abs(fd - adj).max() <= 1e-3 * np.abs(fd).max() + 1e-8, (fd, adj)

"""The KS distance of the fit kernel at the target lengths where its split over
warps and CTAs changes, with ties among the targets and with simulated values,
against the oracle (GPU)."""
import numpy as np
import pytest

import bnm_cuda_b200 as B


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 31, 1023, 4095, 4096, 5001, 70000])
def test_ks_matches_oracle(port, m):
    rng = np.random.default_rng(m)
    N, frames, n = 12, 60, 3
    z = rng.standard_normal((n, frames + 4, N))
    bold = sum(z[:, k:k + frames] for k in range(5)).astype(np.float32).astype(np.float64)
    cfg = B.Config(nodes=N, max_sims=n, time_steps=1000 * (frames - 1), bold_tr=1000, bold_remove_s=0, window_size=8,
                   window_step=1, exc_interhem=False)
    emp_fc = rng.uniform(-0.2, 0.8, cfg.sizes()["n_pairs"])
    emp = rng.uniform(-0.3, 0.9, m)
    emp[: m // 3] = np.round(emp[: m // 3], 1)  # ties
    with B.Plan(cfg, np.zeros((N, N)), emp_fc, rng.permutation(emp)) as p:
        fcd = p.check_fit_bold(bold)["fcd"]
        # values of the first series among the targets
        k = min(m, 200)
        emp[:k] = fcd[0][:k]
    with B.Plan(cfg, np.zeros((N, N)), emp_fc, rng.permutation(emp)) as p:
        r = p.check_fit_bold(bold)
    for i in range(n):
        # of the device's own FCD: counts over lengths, exact up to the last ulp
        assert r["fcd_ks"][i] == pytest.approx(port.port_ks(np.sort(emp), r["fcd"][i]), abs=1e-12)


@pytest.mark.gpu
@pytest.mark.parametrize("m", [600, 70000])
def test_graph_launch_counts_the_same(m):
    rng = np.random.default_rng(m)
    N, n = 12, 4
    cfg = B.Config(nodes=N, max_sims=n, time_steps=4000, bold_tr=100, bold_remove_s=1, window_size=8, window_step=1,
                   exc_interhem=False, i_sampling_start=100, i_sampling_end=600)
    G, w = rng.uniform(0.5, 3, n), rng.uniform(0.1, 0.7, (n, N))
    with B.Plan(cfg, rng.random((N, N)) * 0.05, rng.uniform(-0.2, 0.8, cfg.sizes()["n_pairs"]),
                rng.uniform(-0.2, 0.9, m)) as p:
        first = p.run(G, w, w, outputs=())
        second = p.run(G, w, w, outputs=())
        assert p.graph_launched()
    for k in ("cost", "fcd_ks"):
        np.testing.assert_array_equal(first[k], second[k])

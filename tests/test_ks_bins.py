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

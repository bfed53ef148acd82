"""Integrator shapes of a group that leaves SMs idle and of one that does not:
the results are those of the plans alone (GPU)."""
import numpy as np
import pytest

import bnm_cuda_b200 as B
from bnm_cuda_b200 import synth


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3, 70, 90])
def test_group_results_do_not_depend_on_the_shape_rule(n):
    nodes = (24, 68)
    plans, alone, params = [], [], []
    rng = np.random.default_rng(n)
    for N in nodes:
        cfg = B.Config(nodes=N, max_sims=n, time_steps=3000, bold_tr=100, bold_remove_s=1, window_size=8,
                       i_sampling_start=200, i_sampling_end=900)
        s = cfg.sizes()
        args = (cfg, synth.make_sc(N, 0.3, N), rng.uniform(-0.2, 0.8, s["n_pairs"]), rng.uniform(-0.2, 0.9, 60))
        plans.append(B.Plan(*args))
        alone.append(B.Plan(*args))
        params.append(synth.uniform_params(n, N, n))
    with B.Group(plans) as g:
        first, second = g.run(params), g.run(params)
    if 2 * n <= 148:  # every particle has an SM of its own
        assert all(p.integrator()["slots"] == 1 for p in plans)
    for p, q, a, b in zip(alone, params, first, second):
        r = p.run(*q, outputs=("w_ie",))
        for k in ("cost", "fic_penalty", "fcd_ks", "w_ie", "fic_ntrials"):
            np.testing.assert_array_equal(r[k], a[k], err_msg=k)
            np.testing.assert_array_equal(r[k], b[k], err_msg=k)
    for p in plans + alone:
        p.close()

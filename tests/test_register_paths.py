"""The register integrator's kernel for one particle per CTA against the one
for two (BNM_B200_SLOTS), bit for bit, where its layout and its control flow
change: warps per CTA, buffer strides, odd node counts, FIC decisions at the
ends of a run, frames every millisecond, more particles than the GPU holds,
placement (GPU)."""
import numpy as np
import pytest

import bnm_cuda_b200 as B
from bnm_cuda_b200 import synth

# nodes, particles, model ms, TR, FIC window start, end, max trials, fixed wIE
CASES = [(2, 3, 700, 50, 100, 400, 10, False), (31, 5, 900, 100, 100, 500, 3, False),
         (32, 2, 900, 100, 100, 901, 2, False), (33, 40, 600, 100, 1, 1, 4, False),
         (64, 700, 300, 50, 50, 150, 2, False), (65, 9, 999, 111, 900, 1500, 10, False),
         (96, 310, 300, 50, 50, 150, 2, False), (97, 6, 600, 100, 100, 300, 2, False),
         (128, 5, 500, 100, 100, 300, 0, False), (50, 4, 400, 1, 10, 300, 2, False),
         (84, 4, 1000, 200, 100, 500, 10, True), (40, 3, 800, 100, 700, 100, 2, False)]


def _run(monkeypatch, slots, case, calls):
    N, n, T, TR, start, end, trials, fixed = case
    monkeypatch.setenv("BNM_B200_SLOTS", str(slots))
    rng = np.random.default_rng(N)
    cfg = B.Config(nodes=N, max_sims=n, time_steps=T, bold_tr=TR, bold_remove_s=0, window_size=2, window_step=2,
                   exc_interhem=False, i_sampling_start=start, i_sampling_end=end, max_fic_trials=trials,
                   do_fic=not fixed, no_fcd=N < 3, noise_seed=N)
    sc = synth.make_sc(N, 0.5, N) * (1 + 0.3 * rng.random((N, N)))  # not symmetric
    s = cfg.sizes()
    with B.Plan(cfg, sc, rng.uniform(-0.2, 0.8, s["n_pairs"]), rng.uniform(-0.2, 0.9, 30)) as p:
        G, wEE, wEI = synth.uniform_params(n, N, N)
        wIE = rng.uniform(0.8, 1.5, (n, N)) if fixed else None
        out = [p.run(G, wEE * (1 + 0.1 * rng.random(wEE.shape)), wEI, wIE, outputs=("bold", "ext_means", "w_ie"))
               for _ in range(calls)]
        assert p.integrator()["slots"] == slots
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES)
def test_one_and_two_particles_per_cta_agree(monkeypatch, case):
    # the second call of the first plan is a graph launch, with placement from the first call's restarts
    one, two = _run(monkeypatch, 1, case, 2), _run(monkeypatch, 2, case, 2)
    for a, b in zip(one, two):
        for k in ("bold", "ext_means", "w_ie", "fic_ntrials", "fic_failed"):
            np.testing.assert_array_equal(a[k], b[k], err_msg=k)

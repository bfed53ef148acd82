"""The reference-order FP64 kernel on the largest node counts, where a CTA has
more threads than its registers at their natural number allow (GPU)."""
import numpy as np
import pytest

import bnm_cuda_b200 as B
from bnm_cuda_b200 import synth


def _case(N, n, T, TR):
    rng = np.random.default_rng(N)
    cfg = B.Config(nodes=N, max_sims=n, time_steps=T, bold_tr=TR, bold_remove_s=0, window_size=2, window_step=1,
                   exc_interhem=False, do_fic=False, calculate_fic_penalty=False, precision=B.PREC_F64,
                   noise_mode=B.NOISE_HOST)
    s = cfg.sizes()
    sc = synth.make_sc(N, 0.4, N) * (1 + 0.3 * rng.random((N, N)))  # not symmetric
    G, wEE, wEI = synth.uniform_params(n, N, N)
    wIE = rng.uniform(0.8, 1.5, (n, N))
    targets = rng.uniform(-0.2, 0.8, s["n_pairs"]), rng.uniform(-0.2, 0.9, 50)
    return cfg, s, sc, targets, (G, wEE * (1 + 0.1 * rng.random(wEE.shape)), wEI, wIE)


@pytest.mark.gpu
@pytest.mark.parametrize("N", [640, 641, 1024])
def test_fp64_large_node_counts_match_oracle(port, N):
    T, TR = 60, 10
    cfg, s, sc, targets, (G, wEE, wEI, wIE) = _case(N, 1, T, TR)
    noise = port.port_noise(410, s["noise_len"])
    with B.Plan(cfg, sc, *targets, host_noise=noise) as p:
        r = p.run(G, wEE, wEI, wIE, outputs=("bold",))
    o = port.port_integrate(sc, G[0], wEE[0], wEI[0], wIE[0], time_steps=T, bold_tr=TR, n_vols_remove=0, noise=noise,
                            adjust_fic=False)
    # the operations and their order are the oracle's; exp and pow differ in the last ulp
    np.testing.assert_allclose(r["bold"][0], o["bold"], rtol=1e-9, atol=1e-12)

"""The reference-order FP64 kernel at the node counts where its layout changes
(padded columns, SC in or out of shared memory, one or two threads a node),
against the oracle's integration of the same noise (GPU)."""
import numpy as np
import pytest

import bnm_cuda_b200 as B
from bnm_cuda_b200 import synth


@pytest.mark.gpu
@pytest.mark.parametrize("N", [3, 31, 33, 102, 164, 165, 256, 257])
def test_fp64_layouts_match_oracle(port, N):
    rng = np.random.default_rng(N)
    T, TR = (1200, 100) if N < 200 else (300, 20)
    cfg = B.Config(nodes=N, max_sims=2, time_steps=T, bold_tr=TR, bold_remove_s=0, window_size=4, window_step=1,
                   exc_interhem=False, do_fic=False, calculate_fic_penalty=False, precision=B.PREC_F64,
                   noise_mode=B.NOISE_HOST)
    s = cfg.sizes()
    sc = synth.make_sc(N, 0.4, N) * (1 + 0.3 * rng.random((N, N)))  # not symmetric
    noise = port.port_noise(410, s["noise_len"])
    G, wEE, wEI = synth.uniform_params(2, N, N)
    wEE = wEE * (1 + 0.1 * rng.random(wEE.shape))
    wIE = rng.uniform(0.8, 1.5, (2, N))
    with B.Plan(cfg, sc, rng.uniform(-0.2, 0.8, s["n_pairs"]), rng.uniform(-0.2, 0.9, 50), host_noise=noise) as p:
        r = p.run(G, wEE, wEI, wIE, outputs=("bold", "ext_means"))
    for i in range(2):
        o = port.port_integrate(sc, G[i], wEE[i], wEI[i], wIE[i], time_steps=T, bold_tr=TR, n_vols_remove=0,
                                noise=noise, adjust_fic=False)
        # the operations and their order are the oracle's; exp and pow differ in the last ulp
        np.testing.assert_allclose(r["bold"][i], o["bold"], rtol=1e-9, atol=1e-12)

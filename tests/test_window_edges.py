"""FC and FCD of given BOLD against the oracle where the window kernel's tiles,
ring and frame chunks end: node counts around the 16-node tiles, hemispheres,
window steps beyond the window, windows longer than the ring, few frames (GPU)."""
import numpy as np
import pytest

import bnm_cuda_b200 as B

CASES = [  # nodes, frames, window size, step, exclude inter-hemispheric pairs
    (3, 9, 2, 1, False), (16, 40, 10, 2, False), (17, 41, 4, 7, False), (34, 90, 20, 3, True), (66, 64, 8, 1, True),
    (130, 33, 6, 1, False), (40, 500, 400, 11, True), (258, 24, 4, 1, False)]


@pytest.mark.gpu
@pytest.mark.parametrize("N,frames,size,step,exc", CASES)
def test_window_edges_match_oracle(port, N, frames, size, step, exc):
    rng = np.random.default_rng(N + frames)
    n = 2
    z = rng.standard_normal((n, frames + 4, N))
    bold = sum(z[:, k:k + frames] for k in range(5)) + rng.standard_normal((n, frames, 1)) * rng.standard_normal((n, 1, N))
    bold = bold.astype(np.float32).astype(np.float64)  # what the FP32 path holds
    cfg = B.Config(nodes=N, max_sims=n, time_steps=1000 * (frames - 1), bold_tr=1000, bold_remove_s=0,
                   window_size=size, window_step=step, exc_interhem=exc, gram=B.GRAM_F32)
    s = cfg.sizes()
    with B.Plan(cfg, np.zeros((N, N)), rng.uniform(-0.2, 0.8, s["n_pairs"]), rng.uniform(-0.2, 0.9, 40)) as p:
        r = p.check_fit_bold(bold)
    for i in range(n):
        # co-moments in FP64, rounded once to FP32
        np.testing.assert_allclose(r["fc"][i], port.port_fc_tril(bold[i], exc), rtol=2e-7, atol=1e-7)
        np.testing.assert_allclose(r["fcd"][i], port.port_fcd_tril(bold[i], step, size, exc), atol=1e-4)

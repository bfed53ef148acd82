"""FCD of the FP32 path where its output tiles and K chunks end, with both tile
sizes (few and many simulations), against the oracle (GPU)."""
import numpy as np
import pytest

import bnm_cuda_b200 as B


@pytest.mark.gpu
@pytest.mark.parametrize("N,frames,n", [(4, 40, 2), (9, 72, 1), (9, 73, 3), (12, 105, 400), (24, 137, 110)])
def test_fcd_tiles_match_oracle(port, N, frames, n):
    rng = np.random.default_rng(frames)
    z = rng.standard_normal((n, frames + 4, N))
    bold = sum(z[:, k:k + frames] for k in range(5)).astype(np.float32).astype(np.float64)
    cfg = B.Config(nodes=N, max_sims=n, time_steps=1000 * (frames - 1), bold_tr=1000, bold_remove_s=0, window_size=8,
                   window_step=1, exc_interhem=False, gram=B.GRAM_F32)
    with B.Plan(cfg, np.zeros((N, N)), rng.uniform(-0.2, 0.8, cfg.sizes()["n_pairs"]), rng.uniform(-0.2, 0.9, 40)) as p:
        r = p.check_fit_bold(bold)
    for i in sorted({0, n // 2, n - 1}):
        # FP32 rows and sums of at most 276 products of unit vectors' entries: a few hundred ulps of 1
        np.testing.assert_allclose(r["fcd"][i], port.port_fcd_tril(bold[i], 1, 8, False), atol=3e-5)

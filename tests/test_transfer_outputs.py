"""Host arrays that cross in several pieces and through several threads, against
the oracle, which shares none of that path: FCD of more than one, two and nine
pieces, the last one ragged; series longer than a piece (GPU)."""
import numpy as np
import pytest

import bnm_cuda_b200 as B

# nodes, frames, series, window step; values of the FCD: 1.4, 2.7 and 9.6 pieces of 131,072; BOLD rows of 143,000 values
CASES = [(8, 610, 1, 1), (8, 610, 2, 1), (8, 610, 7, 1), (130, 1100, 2, 40), (130, 1100, 5, 40)]


@pytest.mark.gpu
@pytest.mark.parametrize("N,frames,n,step", CASES)
def test_pieces_match_oracle(port, N, frames, n, step):
    rng = np.random.default_rng(N + n)
    z = rng.standard_normal((n, frames + 4, N))
    bold = sum(z[:, k:k + frames] for k in range(5)).astype(np.float32).astype(np.float64)
    cfg = B.Config(nodes=N, max_sims=n, time_steps=1000 * (frames + 9), bold_tr=1000, bold_remove_s=10, window_size=8,
                   window_step=step, exc_interhem=False)
    s = cfg.sizes()
    with B.Plan(cfg, np.zeros((N, N)), rng.uniform(-0.2, 0.8, s["n_pairs"]), rng.uniform(-0.2, 0.9, 500)) as p:
        for _ in range(2):  # the second call finds the slots in use
            r = p.check_fit_bold(bold)
            for i in range(n):
                # split-BF16 Grams of unit vectors: 2^-16 relative per factor
                np.testing.assert_allclose(r["fc"][i], port.port_fc_tril(bold[i], False), atol=1e-4)
                np.testing.assert_allclose(r["fcd"][i], port.port_fcd_tril(bold[i], step, 8, False), atol=1e-4)

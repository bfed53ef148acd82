"""The caller's double arrays cross to and from the device in FP32 through
pieces converted by several threads: batches on both sides of the piece and
thread limits give what each series gives alone, through one pageable copy
where it is small (GPU)."""
import numpy as np
import pytest

import bnm_cuda_b200 as B


@pytest.mark.gpu
@pytest.mark.parametrize("N,frames,n", [(40, 400, 5), (40, 400, 19), (130, 505, 5), (130, 1100, 2), (6, 30, 2000)])
def test_batches_equal_single_series(N, frames, n):
    rng = np.random.default_rng(N + n)
    z = rng.standard_normal((n, frames + 3, N))
    bold = sum(z[:, k:k + frames] for k in range(4))
    cfg = B.Config(nodes=N, max_sims=n, time_steps=1000 * (frames + 9), bold_tr=1000, bold_remove_s=10, window_size=20,
                   window_step=4, exc_interhem=False)
    s = cfg.sizes()
    efc, efcd = rng.uniform(-0.2, 0.8, s["n_pairs"]), rng.uniform(-0.2, 0.9, 500)
    with B.Plan(cfg, np.zeros((N, N)), efc, efcd) as p:
        r = p.check_fit_bold(bold)
        r2 = p.check_fit_bold(bold[::-1])  # the page-locked slots again
        for i in sorted({0, 1, n // 2, n - 1}):
            one = p.check_fit_bold(bold[i:i + 1])
            for k in ("cost", "fc_corr", "fcd_ks", "fc", "fcd"):
                np.testing.assert_array_equal(r[k][i], one[k][0], err_msg=k)
                np.testing.assert_array_equal(r2[k][n - 1 - i], one[k][0], err_msg=k)

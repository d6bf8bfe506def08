"""The mixed site density matrix of positive tensors at sizes whose FP32 contractions
take the large and the small tiles with remainders, odd K and split K.

FP32 products of length K carry an error of at most K u times the sum of magnitudes;
with the entries positive that is relative, and the largest chain here (six
contractions of K <= 2241) gives 6 * 2241 * 6e-8 = 8e-4.  The rounding errors are
random, not aligned (6 * 47 * 6e-8 = 2e-5), and a tile row lost would be 1 in 2400,
so the bar is 1e-4 against the FP64 path.
"""

import numpy as np
import pytest
import torch

import acetn_gb300 as gb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,chi", [(4, 150), (4, 139), (3, 249)])
def test_mixed_site_rdm_wide(D, chi):
    rng = np.random.default_rng(D * chi)

    def positive(*shape):
        return torch.from_numpy(rng.uniform(0.5, 1.5, shape) / shape[0]).to("cuda")

    st = gb.random_state(D, 4, 1, nx=1, ny=1, device="cuda")
    s = st.site_list[0]
    st[s] = {"A": positive(D, D, D, D, 2), "C": [positive(chi, chi) for _ in range(4)],
             "E": [positive(chi, chi, D, D) for _ in range(4)]}
    exact = gb.RDM(st, "fp64")[s].cpu().numpy()
    mixed = gb.RDM(st, "mixed")[s].cpu().numpy()
    assert np.abs(mixed / exact - 1.0).max() < 1e-4

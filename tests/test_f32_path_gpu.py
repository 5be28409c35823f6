"""The 32-bit path's product: every kernel a batch may go to gives a row the same bits."""
from __future__ import annotations

import pytest
import torch

from test_kernels_gpu import DEV, K, randn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(130, 257), (130, 260), (33, 16), (16, 5), (513, 129), (3072, 128)])
def test_product_rows_have_the_same_bits_in_every_kernel(n, k):
    """1 to 16 rows take the kernel of decode steps, more take tiles of 32, 64 or 128 rows; edges of all of them.
    The error of a sum of k products, each addition rounded: below k/2 units of 2^-24 of the terms' magnitudes."""
    x, w = randn(700, k, dtype=torch.float32, seed=1), randn(n, k, dtype=torch.float32, seed=2)
    bias = randn(n, dtype=torch.float32, seed=3)
    full = K().linear(x, w, bias)
    bound = (x.double().abs() @ w.double().abs().T + bias.double().abs()) * ((k + 2) * 2.0 ** -24)
    assert ((full.double() - (x.double() @ w.double().T + bias.double())).abs() <= bound).all()
    for rows in (1, 7, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129, 300):
        assert torch.equal(K().linear(x[:rows].contiguous(), w, bias), full[:rows]), rows
    wide = torch.zeros(20, k + 3, dtype=torch.float32, device=DEV)          # rows that start off 16-byte boundaries
    wide[:, 3:] = x[:20]
    assert torch.equal(K().linear(wide[:, 3:], w, bias), full[:20])

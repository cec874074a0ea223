"""The library's own launch shape changes with the batch size: one shot below the change, at it, and well below
it, every result equal to an explicit shape's (results do not depend on the shape, so equality is exact)."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from pelagos_b200 import RelayBPDecoder, codes

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
KW = dict(algo="relay", pre_iter=12, num_sets=3, set_max_iter=6, gamma0=0.65, gamma_dist_interval=(-0.24, 0.66),
          stop_nconv=2, seed=5, device=[0])
# code, shape whose resident blocks the change is counted in, shots per resident block, another explicit shape
RULES = [
    (codes.bb_code_capacity_72, (32, 1, 1, 2), 4, (96, 1)),
    (lambda: codes.bb_phenomenological_144(12), (448, 1, 1, 2), 16, (704, 1)),
]


@pytest.mark.parametrize("make,counted,per_block,other", RULES)
def test_default_shape_changes_with_the_batch(make, counted, per_block, other):
    H = make()
    p = np.full(H.shape[1], 0.01)
    ref = RelayBPDecoder(H, p, **KW)
    ref.configure_launch(*counted)
    n = per_block * ref.launch_info()["blocks"]
    ref.configure_launch(*other)
    rng = np.random.default_rng(11)
    err = (rng.random((n, H.shape[1])) < 0.012).astype(np.uint8)
    syn = torch.from_numpy((err @ H.T % 2).astype(np.uint8)).to(DEV)
    want = ref.decode(syn, return_last_posterior=True)
    dec = RelayBPDecoder(H, p, **KW)
    for B in (3, n - 1, n):
        got = dec.decode(syn[:B].contiguous(), return_last_posterior=True)
        for k in ("errors", "weights", "valid_mask", "iterations", "found_count", "last_posterior"):
            assert torch.equal(got[k], want[k][:B]), (k, B)

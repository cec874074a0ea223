"""Result arrays and queue order of a batch against torch, around the compacting block's rounds of 4,096."""

from __future__ import annotations

import pytest
import torch

from pelagos_b200.decoder import finish_results, queue_order

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.mark.parametrize("share", [0.0, 0.01, 0.5, 1.0])
@pytest.mark.parametrize("B", [0, 1, 3, 31, 1024, 4095, 4096, 4097, 65537])
def test_results_and_order(B, share):
    g = torch.Generator(device=DEV).manual_seed(B + 1)
    buf = torch.randint(1, 6, (B + 1,), generator=g, device=DEV, dtype=torch.int32)
    buf[torch.rand(B + 1, generator=g, device=DEV) < share] = 0
    wfix = torch.randint(-(1 << 62), 1 << 62, (B,), generator=g, device=DEV, dtype=torch.int64)
    for found in (buf[:B], buf[1:]):  # aligned to 16 bytes or not
        w = torch.where(found > 0, wfix, torch.iinfo(torch.int64).max)
        exact = torch.where(found > 0, w.to(torch.float64) * 2.0 ** -32, float("inf"))
        for dtype in (torch.float32, torch.float64):
            weights, valid, unconverged = finish_results(found, w, 3, dtype)
            assert weights.dtype == dtype and torch.equal(weights, exact.to(dtype))
            assert valid.dtype == torch.bool and torch.equal(valid, found >= 3)
            assert unconverged.dtype == torch.int32
            assert torch.equal(unconverged.long(), torch.nonzero(found < 3).flatten())
        count = torch.full((1,), -1, dtype=torch.int32, device=DEV)
        order = queue_order(found, count)
        assert torch.equal(order.long(), torch.argsort((found > 0).to(torch.uint8), stable=True))
        assert int(count) == int((found <= 0).sum())


# rounds of 16,384 shots from 8,192 on, a cluster of 8 blocks from 32,768 on: around the changes, parts of one round
# and of several, blocks without a part, and a partial last round
@pytest.mark.parametrize("share", [0.0, 0.01, 1.0])
@pytest.mark.parametrize("B", [8191, 8192, 16384, 16385, 32767, 32768, 32769, 131071, 131072, 131073, 262147, 600001])
def test_results_and_order_in_a_cluster(B, share):
    test_results_and_order(B, share)

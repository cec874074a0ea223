"""GF(2) products at the edges of their tiles: partial words of shots and columns, few and many rows,
every alignment of rows and buffers, the longest rows."""

from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp
import torch

from pelagos_b200.adapter import _DeviceCSR

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 4, 1])
@pytest.mark.parametrize("B,N,R", [(1, 33, 5), (31, 64, 64), (33, 100, 70), (1185, 2592, 936), (20000, 48, 63),
                                   (40, 49152, 3), (70, 16, 128), (5, 1, 1)])
def test_matches_integer_product(B, N, R, offset):
    rng = np.random.default_rng(B + N)
    A = sp.random(R, N, density=min(1.0, 8 / N), format="csr", random_state=1, dtype=np.float64)
    A.data[:] = 1
    buf = torch.from_numpy(rng.integers(0, 256, size=B * N + 16, dtype=np.uint8)).cuda()  # only low bits count
    x = buf[offset:offset + B * N].view(B, N)
    got = _DeviceCSR(A, x.device).apply(x).cpu().numpy()
    want = (A.astype(np.int64) @ (x.cpu().numpy().T.astype(np.int64) & 1)).T % 2
    np.testing.assert_array_equal(got, want)

"""GF(2) products at the edges of their tiles: partial words of shots and columns, few and many rows,
every alignment of rows and buffers, the longest rows."""

from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp
import torch

from pelagos_b200.adapter import _DeviceCSR
from pelagos_b200.montecarlo import MonteCarlo

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


# rows staged as whole 16-byte pieces: the shortest and longest, a half word at the end, one shot, and past the limit
@pytest.mark.parametrize("B,N,R", [(1, 32, 5), (33, 48, 70), (1300, 2608, 12), (40, 12288, 70), (40, 12304, 70)])
def test_staged_rows_match_integer_product(B, N, R):
    test_matches_integer_product(B, N, R, 0)
    test_failure_counts_match_the_general_products(B, N, R, 0)


@pytest.mark.parametrize("offset", [0, 4, 1])
@pytest.mark.parametrize("B,N,R", [(1, 33, 5), (31, 64, 64), (33, 100, 70), (1185, 2592, 12), (20000, 48, 63),
                                   (40, 49152, 3), (70, 16, 300), (5, 1, 1)])
def test_failure_counts_match_the_general_products(B, N, R, offset):
    rng = np.random.default_rng(B + N)
    O = sp.random(R, N, density=min(1.0, 3 / N), format="csr", random_state=2, dtype=np.float64)
    O.data[:] = 1
    O[0, N - 1] = 1
    mc = MonteCarlo(sp.csr_matrix(np.ones((1, N))), np.full(N, 0.1), O)
    buf = torch.from_numpy(rng.integers(0, 256, size=2 * B * N + 32, dtype=np.uint8)).cuda()  # only low bits count
    e = buf[offset:offset + B * N].view(B, N)
    est = buf[B * N + 16 + offset:2 * B * N + 16 + offset].view(B, N)
    est[: B // 2] = e[: B // 2]  # half of the shots do not flip
    if B > 2:
        est[1, N - 1] ^= 1  # one whose only difference is the last column
    found = torch.from_numpy(rng.integers(0, 3, size=B).astype(np.int32)).cuda()
    iters = torch.from_numpy(rng.integers(0, 6081, size=B).astype(np.int32)).cuda()
    got = mc.failures(e, {"errors": est, "found_count": found, "iterations": iters}).cpu().numpy()
    A = O.astype(np.int64)
    d = (e.cpu().numpy() ^ est.cpu().numpy()).astype(np.int64) & 1
    flip = ((A @ d.T) % 2).any(axis=0)
    unsolved = found.cpu().numpy() <= 0
    want = [(flip | unsolved).sum(), unsolved.sum(), (flip & ~unsolved).sum(), iters.cpu().numpy().astype(np.int64).sum()]
    np.testing.assert_array_equal(got, want)
    # int64 counts take the general products
    other = mc.failures(e, {"errors": est, "found_count": found.long(), "iterations": iters.long()})
    np.testing.assert_array_equal(other.cpu().numpy(), want)


# rows read by column: tiles of 9, 17 and 32 shots with a partial last one, odd and 4-byte rows, a warp and a
# thread per matrix row, one and four bytes per store
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("B,N,R", [(5323, 101, 70), (5323, 100, 63), (10001, 37, 5), (19003, 36, 68), (1900, 20001, 65)])
def test_rows_read_by_column(B, N, R, offset):
    test_matches_integer_product(B, N, R, offset)
    test_failure_counts_match_the_general_products(B, N, R, offset)

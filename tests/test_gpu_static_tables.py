"""rbp_decode_static builds its graph tables on the host in pieces: graphs whose checks are far from equal (empty,
single-edge and very wide rows), and tables longer than one piece, against rbp_decode."""

from __future__ import annotations

import numpy as np
import pytest
import torch
from scipy.sparse import csr_matrix

from pelagos_b200 import RelayBPDecoder, codes
from test_zz_no_alloc import DEV, _assert_identical, _decoder_entry, _static_decode

pytestmark = pytest.mark.gpu


def _uneven(wide_first: bool):
    rng = np.random.default_rng(4)
    H = np.zeros((60, 300), np.uint8)
    H[0, rng.choice(300, 250, replace=False)] = 1
    for v in range(300):
        H[rng.integers(20, 60), v] = 1  # checks 1..19 are empty
    H[59, :] = 0
    H[59, 7] = 1
    return csr_matrix(H if wide_first else H[::-1].copy())


def _degree_five():
    """2,500 variables of up to five edges: two blocks of the tables."""
    rng = np.random.default_rng(8)
    H = np.zeros((1300, 2500), np.uint8)
    H[rng.permutation(np.arange(12500) % 1300), np.arange(12500) % 2500] = 1
    return csr_matrix(H)


@pytest.mark.parametrize("make", [lambda: _uneven(True), lambda: _uneven(False), _degree_five,
                                  lambda: codes.regular_ldpc(C=2000, V=4000, seed=3)])
def test_tables_of_uneven_and_large_graphs(make):
    H = make()
    dec = RelayBPDecoder(H, np.full(H.shape[1], 0.02), algo="relay", pre_iter=20, num_sets=3, set_max_iter=10,
                         gamma0=0.65, gamma_dist_interval=(-0.24, 0.66), stop_nconv=2, seed=5)
    rng = np.random.default_rng(6)
    err = (rng.random((200, H.shape[1])) < 0.02).astype(np.int64)
    syn = torch.from_numpy(((H.astype(np.int64) @ err.T) % 2).T.astype(np.uint8).copy()).to(DEV)
    _assert_identical(_static_decode(dec, syn), _decoder_entry(dec, syn))

"""Launch shapes: what a shape that asks for two resident blocks per SM gets, and the library's own choice."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from pelagos_b200 import RelayBPDecoder, codes

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
KW = dict(algo="relay", pre_iter=12, num_sets=3, set_max_iter=6, gamma0=0.65, gamma_dist_interval=(-0.24, 0.66),
          stop_nconv=2, seed=5, device=[0])


def _decoder(H, dtype):
    return RelayBPDecoder(H, np.full(H.shape[1], 0.01), data_type=dtype, **KW)


def _sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


# two blocks of the 2,000 x 4,000 code fit an SM with 16-bit messages, without the optional kept sums
@pytest.mark.parametrize("dtype,per_sm", [("float16", 2), ("bfloat16", 2), ("float32", 1)])
def test_two_blocks_per_sm_come_before_the_kept_sums(dtype, per_sm):
    H = codes.regular_ldpc(C=2000, V=4000, seed=3)
    dec = _decoder(H, dtype)
    rng = np.random.default_rng(3)
    err = (rng.random((40, 4000)) < 0.02).astype(np.uint8)
    syn = torch.from_numpy((err @ H.T % 2).astype(np.uint8)).to(DEV)
    want = dec.decode(syn, return_last_posterior=True)
    dec.configure_launch(256, 1, 1, 2)
    assert dec.launch_info()["blocks"] == per_sm * _sms()
    got = dec.decode(syn, return_last_posterior=True)  # results do not depend on the shape
    for k in ("errors", "weights", "valid_mask", "iterations", "found_count", "last_posterior"):
        assert torch.equal(got[k], want[k]), k


# the message types of one code on either side of the batch size where the library's shape changes: 16 shots per
# resident block of the second one
@pytest.mark.parametrize("make,dtype,small,bulk", [
    (lambda: codes.bb_phenomenological_144(12), "float32", (864, 1, 1), (448, 1, 2)),
    (lambda: codes.bb_phenomenological_144(12), "bfloat16", (864, 1, 1), (448, 1, 2)),
    (lambda: codes.regular_ldpc(C=2000, V=4000, seed=3), "float16", (512, 1, 1), (256, 1, 2)),
    (lambda: codes.regular_ldpc(C=2000, V=4000, seed=3), "float32", (512, 1, 1), None),
])
def test_reported_shape_is_that_of_the_batch(make, dtype, small, bulk):
    dec = _decoder(make(), dtype)
    n = 16 * 2 * _sms()
    keys = ("group_threads", "groups_per_block", "blocks_per_sm")
    for shots, want in ((None, small), (n - 1, small), (n, bulk or small)):
        info = dec.launch_info(shots)
        assert tuple(info[k] for k in keys) == want, shots
        assert tuple(info["pre"][k] for k in keys) == want, shots
    dec.configure_launch(512, 1)  # an explicit shape holds for every batch
    assert dec.launch_info(n) == dec.launch_info(1) == dec.launch_info()

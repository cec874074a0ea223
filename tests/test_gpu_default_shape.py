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


# large batches of codes of at most 2,048 variables: shots per resident group from which their shape runs, and
# (threads, groups per block, blocks per SM) below and from there
@pytest.mark.parametrize("make,dtype,per_group,small,bulk", [
    (codes.bb_code_capacity_144, "float32", 224, (160, 1, 2), (64, 1, 2)),
    (lambda: codes.bb_phenomenological_144(2), "float16", 224, (448, 1, 2), (128, 1, 2)),
    (lambda: codes.bb_phenomenological_144(3), "bfloat16", 224, (352, 1, 2), (192, 1, 2)),
    (lambda: codes.bb_phenomenological_144(8), "float32", 224, (448, 1, 2), (288, 1, 2)),
    (codes.bb_code_capacity_72, "float64", 8, (96, 1, 2), (64, 1, 2)),
    (lambda: codes.bb_phenomenological_144(2), "float64", 256, (448, 1, 2), (224, 1, 2)),
    (lambda: codes.bb_phenomenological_144(3), "float64", 512, (352, 1, 2), (192, 4, 1)),
    (lambda: codes.bb_phenomenological_144(8), "float64", 512, (576, 1, 1), (224, 2, 1)),
])
def test_large_batches_of_small_codes(make, dtype, per_group, small, bulk):
    H = make()
    dec = _decoder(H, dtype)
    keys = ("group_threads", "groups_per_block", "blocks_per_sm")
    n = 1 << 30
    info = dec.launch_info(n)
    assert tuple(info[k] for k in keys) == bulk
    n = per_group * info["blocks"] * info["groups_per_block"]
    assert tuple(dec.launch_info(n - 1)[k] for k in keys) == small
    assert tuple(dec.launch_info(n)[k] for k in keys) == bulk
    # the batch at the change, every result equal to another shape's (results do not depend on the shape)
    gen = torch.Generator(device=DEV).manual_seed(n)
    A = torch.from_numpy(H.toarray().T.astype(np.float32)).to(DEV)
    syn = torch.empty(n, H.shape[0], dtype=torch.uint8, device=DEV)
    for i in range(0, n, 65536):
        e = torch.rand(min(65536, n - i), H.shape[1], generator=gen, device=DEV) < 0.012
        syn[i:i + 65536] = torch.remainder(e.float() @ A, 2).to(torch.uint8)
    got = dec.decode(syn)
    dec.configure_launch(*small[:2], 1, small[2])
    want = dec.decode(syn)
    for k in ("errors", "weights", "valid_mask", "iterations", "found_count"):
        assert torch.equal(got[k], want[k]), k


@pytest.mark.parametrize("V,threads", [(2200, 384), (3000, 512)])
def test_float64_codes_above_2048_variables(V, threads):
    info = _decoder(codes.regular_ldpc(C=V // 2, V=V, seed=3), "float64").launch_info()
    assert (info["group_threads"], info["groups_per_block"], info["blocks_per_sm"]) == (threads, 1, 1)

"""Check rows, variable updates and the convergence test of the decode loop where they can go wrong:
rows with padding and single edges, absent edges, rows that fill 8 or 16 slots, more than 1,024 checks
(32 words of the convergence test), masked rows, offsets, per-shot priors with NaN, infinities and -0.
Every output equals the CPU oracle's."""

from __future__ import annotations

import numpy as np
import pytest
import torch
from scipy.sparse import csr_matrix

from oracle import oracle as O
from pelagos_b200 import RelayBPDecoder

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
SHAPES = [None, (0, -1), (64, 2), (0, 1), (0, 1, 2), (0, 1, 1, 2)]  # the library's choice, groups in a block, ...
BASE = dict(pre_iter=24, num_sets=4, set_max_iter=15, gamma0=0.65, gamma_dist_interval=(-0.24, 0.66), stop_nconv=3,
            algo="relay", seed=5)
VARIANTS = {
    "base": {},
    "alpha": dict(normalized_min_sum_alpha=0.8),
    # 1 - 2^((t + 1) / 0.7): magnitudes that need the masked rows
    "wild_alpha": dict(normalized_min_sum_alpha=0.0, alpha_iteration_scaling_factor=-0.7),
    "beta": dict(offset_min_sum_beta=0.3),
    "fma_lp_last_leg": dict(mix_rounding="fma_lp", unconverged_correction="last_leg"),
}


def _graph(C, V, dc, dv, seed):
    """Every row between 1 and dc edges, one of them exactly dc; columns between 0 and dv edges."""
    rng = np.random.default_rng(seed)
    H = np.zeros((C, V), np.uint8)
    H[0, rng.choice(V, dc, replace=False)] = 1
    for v in rng.permutation(V):
        free = np.nonzero((H.sum(1) < dc) & (H[:, v] == 0))[0]
        n = min(int(rng.integers(0, dv + 1)) - int(H[:, v].sum()), free.size)
        if n > 0:
            H[rng.choice(free, n, replace=False), v] = 1
    H[C - 1] = 0
    H[C - 1, int(np.argmin(H.sum(0)))] = 1  # a check with one edge
    return csr_matrix(H)


def _syndromes(H, p, B, seed):
    rng = np.random.default_rng(seed)
    e = (rng.random((B, H.shape[1])) < p).astype(np.int64)
    s = ((H @ e.T) % 2).T.astype(np.uint8)
    s[::3] = rng.integers(0, 2, size=s[::3].shape)  # shots that never converge
    return np.ascontiguousarray(s)


def _compare(dec, out, ref):
    for k in ("errors", "found_count", "iterations", "weight_fixed"):
        np.testing.assert_array_equal(out[k].cpu().numpy(), ref[k], err_msg=k)
    np.testing.assert_array_equal(out["last_posterior"].cpu().numpy().astype(np.float64), ref["last_posterior"])


def _oracle(dec, syn, mix, **kw):
    return O.decode(O.reference_graph(dec.H_csr), syn, dec.log_prior_ratios, pre_iter=dec.pre_iter,
                    num_sets=dec.num_sets, set_max_iter=dec.set_max_iter, stop_nconv=dec.stop_nconv,
                    gamma0=dec.gamma0, gamma_legs=dec._leg_table(0), algo=dec.algo,
                    last_leg=dec.unconverged_correction == "last_leg", alpha=dec.normalized_min_sum_alpha,
                    alpha_scaling=dec.alpha_iteration_scaling_factor, beta=dec.offset_min_sum_beta,
                    data_type=dec.dtype_str, mix=mix, **kw)


@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16", "float64"])
@pytest.mark.parametrize("size", [(40, 90, 8, 3), (33, 70, 16, 8), (1100, 1500, 8, 3), (24, 60, 20, 5)])
def test_irregular_graphs_match_oracle(size, dtype):
    H = _graph(*size, seed=size[0])
    syn = _syndromes(H, 0.03, 48, seed=3)
    shapes = [s for s in SHAPES if s != (64, 2) or size[1] <= 1024]  # 64 threads own at most 1,024 variables
    for shape in shapes if size[2] <= 16 else shapes[:2]:
        for name, kw in VARIANTS.items():
            dec = RelayBPDecoder(H, np.full(size[1], 0.03), data_type=dtype, launch=shape, **{**BASE, **kw})
            out = dec.decode(torch.from_numpy(syn).to(DEV), return_last_posterior=True)
            _compare(dec, out, _oracle(dec, syn, kw.get("mix_rounding", "separate")))


@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16", "float64"])
def test_special_priors_match_oracle(dtype):
    H = _graph(40, 90, 8, 3, seed=2)
    syn = _syndromes(H, 0.03, 32, seed=4)
    rng = np.random.default_rng(1)
    pl = (3.5 + rng.normal(0, 1, (32, 90))).astype(np.float32)
    for i, x in enumerate((np.nan, np.inf, -np.inf, -0.0, 0.0, 1e30, 3e38, -3e38, 1e-42)):
        pl[i, rng.integers(0, 90, 4)] = x
    for shape in SHAPES:
        dec = RelayBPDecoder(H, np.full(90, 0.03), data_type=dtype, launch=shape, **BASE)
        out = dec.decode(torch.from_numpy(syn).to(DEV), prior_llr=torch.from_numpy(pl).to(DEV),
                         return_last_posterior=True)
        _compare(dec, out, _oracle(dec, syn, "separate", llr_per_shot=pl))


@pytest.mark.parametrize("dtype", ["float32", "bfloat16", "float64"])
@pytest.mark.parametrize("size", [(40, 90, 8, 3), (33, 70, 16, 8), (24, 60, 20, 5)])
def test_legs_with_per_shot_priors_match_oracle(size, dtype):
    """Many short legs: the first pass from the shot's messages, later ones from its kept sums, converging or not."""
    H = _graph(*size, seed=size[0])
    syn = _syndromes(H, 0.04, 40, seed=6)
    syn[:4] = np.random.default_rng(8).integers(0, 2, (4, size[0]))  # shots whose legs do not converge
    pl = (3.0 + np.random.default_rng(9).normal(0, 1, (40, size[1]))).astype(np.float32)
    for shape in SHAPES if size[2] <= 16 else SHAPES[:2]:
        dec = RelayBPDecoder(H, np.full(size[1], 0.03), data_type=dtype, launch=shape,
                             **{**BASE, "num_sets": 9, "set_max_iter": 4, "stop_nconv": 6})
        out = dec.decode(torch.from_numpy(syn).to(DEV), prior_llr=torch.from_numpy(pl).to(DEV),
                         return_last_posterior=True)
        _compare(dec, out, _oracle(dec, syn, "separate", llr_per_shot=pl))

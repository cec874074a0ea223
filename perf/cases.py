"""Performance cases: the work users have this decoder do, through its public entry points.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges.  ``prepare`` makes what a
user's program holds before the call (decoder, network, syndromes on the GPU), ``run`` is one pass and
returns everything the call returns, but for the list of unconverged shots: its length is the batch's
own, and the shots are those with ``valid_mask`` unset.  The codes, schedules and noise rates are those of the
benchmark, the tests and the experiments of this repository.

Kinds of cases:

* ``decode``   RelayBPDecoder.decode: one shot to 65,536, the four codes (and the phenomenological
               matrices of fewer rounds), every message type, relay and plain min-sum, per-shot priors;
* ``learned``  LearnedRelayBPDecoder.decode, the network for every shot or for the unsolved ones;
* ``mixed``    MixedDecoder.decode, four codes in one launch;
* ``train``    ProposalNet.train_step: forward, backward and AdamW of the proposal network;
* ``judge``    the Monte-Carlo loop's syndromes (H e) and failure counts (O e against O e_hat).
"""

from __future__ import annotations

import math
from functools import lru_cache

import numpy as np
import torch

from pelagos_b200 import RelayBPDecoder, autotune, codes

DEVICE = "cuda:0"

# The benchmark's schedule.
RELAY = dict(pre_iter=80, num_sets=100, set_max_iter=60, gamma0=0.65, gamma_dist_interval=(-0.24, 0.66),
             stop_nconv=5, seed=1234)
# Iterations a shot needs on average under that schedule, for the work estimate (measured: the
# phenomenological code at p = 0.003; the learned decode's are lower).
ITERATIONS = {"bb72_cc": 14.0, "bb144_cc": 14.0, "phen": 15.0, "ldpc2000": 20.0}
LEARNED_ITERATIONS = 10.0
NOISE = {"bb72_cc": (0.03, 0.05), "bb144_cc": (0.03,), "phen": (0.002, 0.003, 0.004), "ldpc2000": (0.02,)}
MSG_BYTES = {"float32": 4, "float64": 8, "float16": 2, "bfloat16": 2}


def listed() -> list:
    return [
        # a real-time service: one syndrome as it arrives, latency is all
        dict(name="one_shot", kind="decode", code="phen", rounds=12, p=0.003, shots=1),
        # a small test batch of the smallest code: launches and host work
        dict(name="bb72_small_batch", kind="decode", code="bb72_cc", p=0.05, shots=100),
        # code-capacity Monte Carlo, an ordinary batch of a small code
        dict(name="bb144_cc_batch", kind="decode", code="bb144_cc", p=0.03, shots=20001),
        # a classical LDPC matrix, normalized min-sum, large graph
        dict(name="ldpc2000_alpha", kind="decode", code="ldpc2000", p=0.02, shots=6000, alpha=0.8,
             correction="last_leg"),
        # soft information: every shot with its own prior LLRs, posterior returned, few rounds (ragged sizes)
        dict(name="phen5_soft_priors", kind="decode", code="phen", rounds=5, p=0.003, shots=2047, priors=True),
        # 16-bit messages, bit-packed corrections
        dict(name="phen_bf16_packed", kind="decode", code="phen", rounds=12, p=0.003, shots=12289,
             data_type="bfloat16", packed=True),
        # throughput Monte Carlo of the benchmark code: the seeded decoder with the committed launch shapes
        dict(name="phen_plain", kind="decode", code="phen", rounds=12, p=0.003, shots=65536, committed=True,
             graph=True),
        # the benchmark itself: the learned decode, network for the unsolved shots
        dict(name="phen_learned_gated", kind="learned", p=0.003, shots=65536, gate=True, committed=True),
        # the learned decode as its constructor defaults have it: network for every shot
        dict(name="phen_learned_all", kind="learned", p=0.003, shots=16384, gate=False, committed=True),
        # a service decoding four codes at once
        dict(name="mixed_four_codes", kind="mixed", shots=16384),
        # training the proposal network: one step of the default batch
        dict(name="train_step", kind="train", p=0.003, shots=1024),
        # the Monte-Carlo loop around the decode: syndromes of the drawn errors, failures of the estimates
        dict(name="syndromes_failures", kind="judge", p=0.003, shots=65536),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(("decode", "decode", "decode", "decode", "learned", "mixed", "train", "judge"))
    if kind == "decode":
        code = rng.choice(("bb72_cc", "bb144_cc", "phen", "phen", "phen", "ldpc2000"))
        c = dict(kind=kind, code=code, p=rng.choice(NOISE[code]))
        if code == "phen":
            c["rounds"] = rng.choice((1, 2, 3, 5, 8, 12, 12, 12))
        # the larger p is, the more iterations a shot takes
        # one shot at a time is a real-time service's call; the small matrices come in batches
        least = 1 if c.get("rounds", 0) >= 8 else 16
        c["shots"] = _log_int(rng, least, 8192 if code == "ldpc2000" else (32768 if c["p"] > 0.003 else 65536))
        # float64 messages of the 2000 x 4000 matrix exceed a block's shared memory
        c["data_type"] = rng.choice(("float32", "float32", "float32", "float16", "bfloat16") if code == "ldpc2000" else
                                    ("float32", "float32", "float32", "float16", "bfloat16", "float64"))
        if c["data_type"] == "float64":
            c["shots"] = min(c["shots"], 8192)
        if rng.random() < 0.2:
            c["alpha"] = rng.choice((0.8, 0.875))
        elif rng.random() < 0.1:
            c["beta"] = 0.25
        if rng.random() < 0.2:
            c["packed"] = True
        if rng.random() < 0.2:
            c["correction"] = "last_leg"
        if rng.random() < 0.2:
            c["algo"] = "plain"
        if rng.random() < 0.15:
            c["priors"] = True
            c["shots"] = min(c["shots"], 16384)
        elif rng.random() < 0.4:
            c["graph"] = True
        if rng.random() < 0.5:
            c["committed"] = True
        return c
    if kind == "learned":
        return dict(kind=kind, p=rng.choice(NOISE["phen"]), shots=_log_int(rng, 64, 32768),
                    gate=rng.random() < 0.5, committed=rng.random() < 0.7)
    if kind == "mixed":
        return dict(kind=kind, shots=_log_int(rng, 16, 16384))
    if kind == "train":
        return dict(kind=kind, p=rng.choice(NOISE["phen"]), shots=_log_int(rng, 16, 2048))
    return dict(kind=kind, p=rng.choice(NOISE["phen"]), shots=_log_int(rng, 16, 65536))


# ---------------------------------------------------------------------------- matrices and inputs


@lru_cache(maxsize=None)
def _matrix(code: str, rounds: int):
    if code == "bb72_cc":
        return codes.bb_code_capacity_72()
    if code == "bb144_cc":
        return codes.bb_code_capacity_144()
    if code == "phen":
        return codes.bb_phenomenological_144(rounds)
    if code == "ldpc2000":
        return codes.regular_ldpc(C=2000, V=4000, seed=3)
    raise ValueError(code)


@lru_cache(maxsize=None)
def _observables():
    from pelagos_b200.montecarlo import observables_for

    return observables_for(codes.workload("bb144_phen", p=0.003))


@lru_cache(maxsize=None)
def _dense_t(code: str, rounds: int) -> torch.Tensor:
    return torch.from_numpy(_matrix(code, rounds).toarray().T.astype(np.float32)).to(DEVICE)


def _errors(code: str, rounds: int, p: float, shots: int, seed: int) -> torch.Tensor:
    """Seeded i.i.d. Bernoulli(p) errors on every column, [shots, V] uint8."""
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    V = _matrix(code, rounds).shape[1]
    return (torch.rand(shots, V, generator=gen, device=DEVICE) < p).to(torch.uint8)


def _syndromes(code: str, rounds: int, e: torch.Tensor) -> torch.Tensor:
    """s = H e mod 2 by a dense product (0/1 inputs, row sums below 2^11: exact in any mode)."""
    return torch.remainder(e.float() @ _dense_t(code, rounds), 2).to(torch.uint8)


def _posteriors(e: torch.Tensor, p: float, seed: int) -> torch.Tensor:
    """Posterior LLRs as they are after the pre-iterations: magnitudes of some prior LLRs, negative
    where an error is decided; a few variables decided wrongly."""
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed + 1)
    shape = tuple(e.shape)
    mag = math.log((1 - p) / p) * torch.exp(1.2 + 0.7 * torch.randn(shape, generator=gen, device=DEVICE))
    wrong = torch.rand(shape, generator=gen, device=DEVICE) < torch.where(e > 0, 0.03, 0.0003)
    return torch.where((e > 0) != wrong, -mag, mag)


def _decoder(case: dict, code: str, rounds: int, p: float) -> RelayBPDecoder:
    H = _matrix(code, rounds)
    dec = RelayBPDecoder(
        H, np.full(H.shape[1], p), algo=case.get("algo", "relay"), data_type=case.get("data_type", "float32"),
        normalized_min_sum_alpha=case.get("alpha"), offset_min_sum_beta=case.get("beta"),
        bitpack_output=bool(case.get("packed", False)), unconverged_correction=case.get("correction", "first_leg"),
        cuda_graph=bool(case.get("graph", False)), device=[0], **RELAY)
    if case.get("committed"):
        autotune.apply_default_shapes(dec)
    return dec


MIXED = (("bb72_cc", 0, 0.03), ("bb144_cc", 0, 0.03), ("phen", 12, 0.003), ("ldpc2000", 0, 0.02))


# ---------------------------------------------------------------------------- prepare and run


def prepare(case: dict, seed: int) -> dict:
    kind, shots = case["kind"], case["shots"]
    if kind == "decode":
        code, rounds, p = case["code"], case.get("rounds", 0), case["p"]
        e = _errors(code, rounds, p, shots, seed)
        st = {"kind": kind, "dec": _decoder(case, code, rounds, p), "syn": _syndromes(code, rounds, e), "opts": {}}
        if case.get("priors"):
            # soft readout: each shot's LLRs scattered around the prior's, smaller where it did flip
            gen = torch.Generator(device=DEVICE)
            gen.manual_seed(seed + 1)
            llr = math.log((1 - p) / p)
            noise = torch.randn(shots, e.shape[1], generator=gen, device=DEVICE)
            st["opts"] = {"prior_llr": torch.where(e > 0, 0.3 * llr, llr) + noise, "return_last_posterior": True}
        return st
    if kind == "learned":
        from pelagos_b200.proposal import LearnedRelayBPDecoder, ProposalNet, default_weights_path, load_params

        dec = _decoder(case, "phen", 12, case["p"])
        net = ProposalNet(dec, load_params(default_weights_path())[0])
        e = _errors("phen", 12, case["p"], shots, seed)
        return {"kind": kind, "dec": LearnedRelayBPDecoder(dec, net, learned_legs=4, gate=case["gate"]),
                "syn": _syndromes("phen", 12, e), "opts": {}}
    if kind == "mixed":
        from pelagos_b200.mixed import MixedDecoder

        decs, syns = [], []
        for i, (code, rounds, p) in enumerate(MIXED):
            decs.append(_decoder({}, code, rounds, p))
            # the larger codes get the smaller share, odd sizes among them
            n = max(1, shots if i < 2 else shots // 2 + 1)
            syns.append(_syndromes(code, rounds, _errors(code, rounds, p, n, seed + i)))
        return {"kind": kind, "dec": MixedDecoder(decs, graph=True), "syn": syns}
    if kind == "train":
        from pelagos_b200.proposal import ProposalNet, TrainConfig

        syn, post, target = _tuples(case, seed)
        net = ProposalNet(_decoder({}, "phen", 12, case["p"]), _network())
        return {"kind": kind, "net": net, "cfg": TrainConfig(w_neg=W_NEG), "syn": syn, "post": post, "target": target,
                "loss": torch.zeros(1, device=DEVICE), "grads": torch.zeros(net.n_params, device=DEVICE)}
    if kind == "judge":
        from pelagos_b200.montecarlo import MonteCarlo

        H = _matrix("phen", 12)
        mc = MonteCarlo(H, np.full(H.shape[1], case["p"]), _observables(), device=DEVICE, seed=seed)
        e, out = _judged(case, seed)
        return {"kind": kind, "mc": mc, "e": e, "out": out}
    raise ValueError(kind)


W_NEG = 20.0  # loss weight of the wrongly decided variables
NETWORK = [("E", (64, 6))] + [(n + layer, s) for layer in "12" for n, s in
                              (("W", (16, 64)), ("G", (4, 16)), ("U", (64, 16)), ("b", (64,)))] + \
          [("O", (64,)), ("Oz", (4,)), ("ob", (1,))]


def _network() -> np.ndarray:
    """Flat parameters of a fresh network."""
    rng = np.random.default_rng(0)
    scale = {"E": 6 ** -0.5, "W": 0.125, "U": 0.125, "b": 0.05, "O": 0.0125, "Oz": 1.0, "ob": 1.0}
    return np.concatenate([0.25 + rng.normal(0, 0.05, shape).reshape(-1) if name[0] == "G" else
                           rng.normal(0, scale[name.rstrip("12")], shape).reshape(-1)
                           for name, shape in NETWORK]).astype(np.float32)


def _tuples(case: dict, seed: int):
    """Training tuples: syndromes, posteriors after the pre-iterations, target [decision == error]."""
    e = _errors("phen", 12, case["p"], case["shots"], seed)
    post = _posteriors(e, case["p"], seed)
    return _syndromes("phen", 12, e), post, ((post <= 0).to(torch.uint8) == e).to(torch.uint8)


def _judged(case: dict, seed: int):
    """Errors and a decode's result on them: most estimates equal the error, some shots differ in a few
    bits, a few did not converge."""
    e = _errors("phen", 12, case["p"], case["shots"], seed)
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed + 1)
    bad = torch.rand(case["shots"], 1, generator=gen, device=DEVICE) < 0.01
    est = e ^ ((torch.rand(e.shape, generator=gen, device=DEVICE) < 0.002) & bad).to(torch.uint8)
    found = torch.where(torch.rand(case["shots"], generator=gen, device=DEVICE) < 0.001, 0, 5).to(torch.int32)
    iters = torch.randint(5, 40, (case["shots"],), generator=gen, device=DEVICE, dtype=torch.int32)
    return e, {"errors": est, "found_count": found, "iterations": iters}


def run(state: dict):
    kind = state["kind"]
    if kind in ("decode", "learned"):
        return _fixed(state["dec"].decode(state["syn"], **state["opts"]))
    if kind == "mixed":
        return [_fixed(o) for o in state["dec"].decode(state["syn"])]
    if kind == "train":
        cfg = state["cfg"]
        state["net"].train_step(state["syn"], state["post"], state["target"], cfg, cfg.lr, loss_out=state["loss"],
                                grads_out=state["grads"])
        return {"loss": state["loss"], "grads": state["grads"]}
    mc = state["mc"]
    return {"syndromes": mc.H.apply(state["e"]), "counts": mc.failures(state["e"], state["out"])}


def _fixed(out: dict) -> dict:
    return {k: v for k, v in out.items() if k != "unconverged_indices"}


# ---------------------------------------------------------------------------- work and exact values


def _decode_work(code: str, rounds: int, shots: int, msg: int, iters: float, priors: bool = False,
                 packed: bool = False) -> dict:
    H = _matrix(code, rounds)
    (C, V), E = H.shape, H.nnz
    per_shot = C + (4 * ((V + 31) // 32) if packed else V) + 4 + 1 + 4 + 4 + 8
    if priors:
        per_shot += 8 * V
    # a check pass compares, selects and signs each message, a variable pass adds it in and takes it out
    return {"bytes": shots * per_shot, "flops": shots * iters * (8 * E + 6 * V)}


NET_FLOPS_PER_CHECK = 2 * (6 * 64 + 2 * (64 * 16 + 16 * 64) + 64)  # the network's dense layers


def work(case: dict) -> dict:
    kind, shots = case["kind"], case["shots"]
    if kind == "decode":
        return _decode_work(case["code"], case.get("rounds", 0), shots, MSG_BYTES[case.get("data_type", "float32")],
                            ITERATIONS[case["code"]], bool(case.get("priors")), bool(case.get("packed")))
    if kind == "mixed":
        parts = [_decode_work(code, rounds, max(1, shots if i < 2 else shots // 2 + 1), 4, ITERATIONS[code])
                 for i, (code, rounds, _) in enumerate(MIXED)]
        return {k: sum(w[k] for w in parts) for k in ("bytes", "flops")}
    H = _matrix("phen", 12)
    (C, V), E = H.shape, H.nnz
    net = C * NET_FLOPS_PER_CHECK + 2 * 2 * 16 * 2 * E  # dense layers, two rounds of sums both ways
    if kind == "learned":
        w = _decode_work("phen", 12, shots, 4, LEARNED_ITERATIONS)
        return {"bytes": w["bytes"], "flops": w["flops"] + (0 if case["gate"] else shots * net)}
    if kind == "train":
        return {"bytes": shots * (C + 4 * V + V) + 4 * 4805 * 8, "flops": 3 * shots * net}
    # H e, O e and O e_hat: each set bit's columns; both error arrays read once, the syndromes written
    return {"bytes": shots * (2 * V + C + 8), "flops": shots * (E + 2 * int(_observables().sum()))}


def exact(case: dict, seed: int):
    if case["kind"] == "judge":
        return _exact_judge(case, seed)
    if case["kind"] == "train":
        return _exact_train(case, seed)
    # A decode's outputs are decisions, counts and sums of chosen priors: the value of an iteration that
    # is chaotic in its rounding, with no 64-bit counterpart.
    return None


def _exact_judge(case: dict, seed: int) -> dict:
    e, out = _judged(case, seed)
    H = torch.from_numpy(_matrix("phen", 12).toarray().astype(np.float64)).to(DEVICE)
    O = torch.from_numpy(_observables().astype(np.float64)).to(DEVICE)
    syn = torch.remainder(e.double() @ H.T, 2).to(torch.uint8)
    diff = (e ^ out["errors"]).double()
    flip = (torch.remainder(diff @ O.T, 2) > 0).any(dim=1)
    unconv = out["found_count"] <= 0
    counts = torch.stack([(flip | unconv).sum(), unconv.sum(), (flip & ~unconv).sum(),
                          out["iterations"].to(torch.int64).sum()])
    return {"syndromes": syn, "counts": counts}


def _round_bf16(x: torch.Tensor) -> torch.Tensor:
    """The network's bf16 rounding; its derivative is taken as 1."""
    return x + (x.to(torch.float32).to(torch.bfloat16).to(x.dtype) - x).detach()


def _exact_train(case: dict, seed: int) -> dict:
    """Loss and gradients of the first step in 64 bits: the network as pelagos_b200.proposal describes it
    (node width 64, message width 16, four edge types, bf16 weights and messages)."""
    syn, post, target = _tuples(case, seed)
    Hm = _matrix("phen", 12).tocsr()
    C, V = Hm.shape
    A = torch.from_numpy(Hm.toarray().astype(np.float64)).to(DEVICE)  # [C, V]
    dc, dv = A.sum(1), A.sum(0)
    theta = torch.from_numpy(_network()).to(DEVICE)
    w = theta.to(torch.bfloat16).double().requires_grad_(True)
    P, o = {}, 0
    for name, shape in NETWORK:
        n = int(np.prod(shape))
        P[name] = w[o:o + n].view(shape)
        o += n
    llr = float(np.float32(math.log((1 - case["p"]) / case["p"])))
    shots = case["shots"]
    chk, var = (torch.from_numpy(x.astype(np.int64)).to(DEVICE) for x in Hm.nonzero())
    loss_sum, grad = 0.0, torch.zeros_like(theta, dtype=torch.float64)
    for b0 in range(0, shots, 64):
        s, pc, y = (x[b0:b0 + 64].double() for x in (syn, post.clamp(-1e4, 1e4), target))
        hard = (pc <= 0).double()
        z = torch.stack([torch.tanh(pc / 16), hard, (s @ A) / dv, torch.full_like(pc, math.tanh(llr / 16))], -1)
        ty = (2 * hard + (pc.abs() < 8).double()).long()
        zc = torch.einsum("cv,bvf->bcf", A, z) / dc[:, None]
        x = torch.cat([s[..., None], _round_bf16(zc), torch.ones_like(s)[..., None]], -1)
        q = x @ P["E"].T
        for layer in "12":
            g = torch.relu(q)
            m = _round_bf16(_round_bf16(g) @ P["W" + layer].T)
            n = _round_bf16(torch.einsum("cv,bcd->bvd", A, m))
            gate = P["G" + layer][ty]                                          # [b, V, 16]
            edge = gate[:, var] * (n[:, var] - m[:, chk])
            a = torch.zeros_like(m).index_add(1, chk, edge)
            q = g + _round_bf16(a) @ P["U" + layer].T + P["b" + layer]
        oc = _round_bf16(torch.relu(q)) @ P["O"]
        r = (oc @ A) / dv + z @ P["Oz"] + P["ob"]
        weight = torch.where(y > 0, 1.0, W_NEG)
        loss = (weight * (torch.nn.functional.softplus(r) - y * r)).sum() / (shots * V)
        grad += torch.autograd.grad(loss, w)[0]
        loss_sum += float(loss)
    return {"loss": torch.tensor([loss_sum], dtype=torch.float64, device=DEVICE), "grads": grad}

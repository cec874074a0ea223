"""RelayBPDecoder: drop-in host interface over the sm_100a Relay-BP-S kernel.

Mirrors the reference class ``RelayBPDecoder`` (src/pelagos/decoder.py:247-3891):
same constructor arguments, the same argument validation and error types, and
``decode(syndromes, ...)`` returning a dict with the same keys.  All decoding
runs in one persistent CUDA kernel per call (pelagos_b200/csrc/relaybp.cu)
reached through the C ABI of include/relaybp.h; there is no CPU path.

Differences from the reference, by design:

* message precision: ``data_type`` "float16" / "bfloat16" store messages in
  16 bits while posteriors, memory and sums stay float32 (the reference keeps
  everything in float16 for "float16");
* solution weights are exact (64-bit fixed point, 2^-32 units), so the
  lowest-weight selection does not depend on a summation order;
* results are fresh tensors (the reference returns views of per-batch-size
  cached buffers that the next decode overwrites);
* ``scheduling="layered"`` is not provided;
* ``fast_max_unconverged_pct`` decodes leg-synchronously (one launch per leg,
  each resuming the shots' saved state), since its early exit is a batch-level
  decision; every other call runs all legs in one launch.
"""

from __future__ import annotations

from typing import Dict, List, Optional, Sequence, Tuple, Union

import ctypes as ct
from contextlib import nullcontext

import numpy as np
import torch
from scipy.sparse import csr_matrix

from . import _native as nat
from .graph import TannerGraph
from .utils import (
    GAMMA_DRAW_MODES,
    alpha_schedule,
    compute_log_prior_ratios,
    sample_gamma_per_variable,
    sample_gamma_uniform,
    validate_csr_matrix,
    validate_error_priors,
)

#: Values accepted by ``unconverged_correction`` (decoder.py:222-223).
UNCONVERGED_CORRECTIONS = ("first_leg", "last_leg")

_DTYPE_ALIASES = {
    "float": "float32",
    "half": "float16",
    "double": "float64",
    "fp16": "float16",
    "fp32": "float32",
    "fp64": "float64",
    "bf16": "bfloat16",
}
_MSG_TYPES = {
    "float32": nat.RBP_MSG_F32,
    "float16": nat.RBP_MSG_F16,
    "bfloat16": nat.RBP_MSG_BF16,
    "float64": nat.RBP_MSG_F64,
}
_MIX_MODES = {"separate": nat.RBP_MIX_SEPARATE, "fma_gp": nat.RBP_MIX_FMA_GP, "fma_lp": nat.RBP_MIX_FMA_LP}


def _ptr(t: Optional[torch.Tensor]):
    return ct.c_void_p(t.data_ptr()) if t is not None else ct.c_void_p(0)


#: Batches at least this large decode with the unconverged shots queued first (hard_shots_first).
HARD_FIRST_MIN_BATCH = 1024

_HERE = nullcontext()


def on_device(device: Union[int, torch.device]):
    """Context in which ``device`` is the current one: native entries without a handle launch on the current
    device.  Nothing to enter where it is already (asking takes 0.25 us, torch.cuda.device 1.5)."""
    index = device if isinstance(device, int) else device.index
    return _HERE if torch.cuda.current_device() == index else torch.cuda.device(device)


def finish_results(found: torch.Tensor, wfix: torch.Tensor, stop_nconv: int, weights_dtype=torch.float32):
    """(weights, valid mask, unconverged indices) of a decode's device counts and exact weights, on their
    device and its current stream; reading the number of unconverged shots synchronises the host."""
    B, dev = int(found.shape[0]), found.device
    weights = torch.empty(B, dtype=weights_dtype, device=dev)
    valid = torch.empty(B, dtype=torch.bool, device=dev)
    unconverged = torch.empty(B + 1, dtype=torch.int32, device=dev)  # their number comes after the capacity
    f64 = 1 if weights_dtype == torch.float64 else 0
    u = unconverged.data_ptr()
    with on_device(dev):
        nat.check(nat.lib().rbp_results(found.data_ptr(), wfix.data_ptr(), B, int(stop_nconv), weights.data_ptr(), f64,
                                        valid.data_ptr(), u, u + 4 * B, torch.cuda.current_stream(dev).cuda_stream),
                  "rbp_results")
    return weights, valid, unconverged[:int(unconverged[B])]


def queue_order(found: torch.Tensor, count: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Shot order with the shots that have no solution first (their number in ``count``), on the
    device of ``found`` and its current stream."""
    dev = found.device
    order = torch.empty(found.shape[0], dtype=torch.int32, device=dev)
    with on_device(dev):
        nat.check(nat.lib().rbp_queue_order(found.data_ptr(), int(found.shape[0]), order.data_ptr(),
                                            count.data_ptr() if count is not None else None,
                                            torch.cuda.current_stream(dev).cuda_stream), "rbp_queue_order")
    return order


class _NativeDecoder:
    """Owns one device's rbp_graph + rbp_decoder handles."""

    def __init__(self, graph: TannerGraph, device: int, params: nat.RbpParams, llr: np.ndarray,
                 gamma_legs: np.ndarray, alpha: np.ndarray):
        L = nat.lib()
        self.device = device
        self._graph = ct.c_void_p()
        self._dec = ct.c_void_p()
        nat.check(L.rbp_graph_create(graph.C, graph.V, graph.E, nat.i32_ptr(graph.chk_ptr),
                                     nat.i32_ptr(graph.edge_var), nat.i32_ptr(graph.var_ptr),
                                     nat.i32_ptr(graph.var_edges), device, ct.byref(self._graph)),
                  "rbp_graph_create")
        llr = np.ascontiguousarray(llr, dtype=np.float32)
        gamma_legs = np.ascontiguousarray(gamma_legs, dtype=np.float32)
        alpha = np.ascontiguousarray(alpha, dtype=np.float32)
        rc = L.rbp_decoder_create(self._graph, ct.byref(params), nat.f32_ptr(llr),
                                  nat.f32_ptr(gamma_legs) if gamma_legs.size else None,
                                  nat.f32_ptr(alpha), int(alpha.size), ct.byref(self._dec))
        if rc != nat.RBP_OK:
            L.rbp_graph_destroy(self._graph)
            self._graph = ct.c_void_p()
        nat.check(rc, "rbp_decoder_create")

    def set_llr(self, llr: np.ndarray):
        llr = np.ascontiguousarray(llr, dtype=np.float32)
        nat.check(nat.lib().rbp_decoder_set_llr(self._dec, nat.f32_ptr(llr)), "rbp_decoder_set_llr")

    def configure(self, group_threads: int, groups_per_block: int, shots_per_group: int = 0,
                  blocks_per_sm: int = 0, kind: int = nat.RBP_LAUNCH_ALL):
        nat.check(nat.lib().rbp_decoder_configure_kind(self._dec, int(kind), int(group_threads),
                                                       int(groups_per_block), int(shots_per_group),
                                                       int(blocks_per_sm)), "rbp_decoder_configure")

    def query(self, shots: Optional[int] = None) -> dict:
        L = nat.lib()
        gs, bs = ct.c_int64(), ct.c_int64()

        def shape(kind):
            v = {k: ct.c_int32() for k in ("group_threads", "groups_per_block", "shots_per_group", "blocks_per_sm",
                                           "blocks")}
            refs = [ct.byref(x) for x in v.values()]
            if shots is None:
                nat.check(L.rbp_decoder_query_kind(self._dec, kind, *refs), "rbp_decoder_query")
            else:
                sizes = (ct.byref(gs), ct.byref(bs)) if kind == nat.RBP_LAUNCH_LEGS else (None, None)
                nat.check(L.rbp_decoder_query_batch(self._dec, kind, int(shots), *sizes, *refs), "rbp_decoder_query")
            return {k: x.value for k, x in v.items()}

        legs = shape(nat.RBP_LAUNCH_LEGS)
        if shots is None:
            nat.check(L.rbp_decoder_query(self._dec, ct.byref(gs), ct.byref(bs), None, None, None, None),
                      "rbp_decoder_query")
        return {"group_smem": gs.value, "block_smem": bs.value, **legs, "pre": shape(nat.RBP_LAUNCH_PRE)}

    def decode(self, B: int, batch: nat.RbpBatch, outs: nat.RbpOutputs, stream: int):
        nat.check(nat.lib().rbp_decode(self._dec, int(B), ct.byref(batch), ct.byref(outs),
                                       ct.c_void_p(stream)), "rbp_decode")

    def close(self):
        if getattr(self, "_dec", None):
            nat.lib().rbp_decoder_destroy(self._dec)
            self._dec = ct.c_void_p()
        if getattr(self, "_graph", None):
            nat.lib().rbp_graph_destroy(self._graph)
            self._graph = ct.c_void_p()

    def __del__(self):  # pragma: no cover - interpreter shutdown order
        try:
            self.close()
        except Exception:
            pass


class RelayBPDecoder:
    """Relay-BP-S decoder on one (or, as independent replicas, several) B200 GPUs.

    Constructor arguments and their validation follow decoder.py:271-784.
    Extra keyword arguments of this implementation:

    * ``mix_rounding``: rounding of the memory mix (1-g)*llr + g*posterior:
      "separate" (default; one rounding per operation), "fma_gp" or "fma_lp";
    * ``launch``: optional (group_threads, groups_per_block[, shots_per_group[, blocks_per_sm]])
      kernel shape of every launch (by default the library chooses by the code's size and each
      batch's); blocks_per_sm 2 selects the kernel compiled for two resident blocks per SM, and
      shots_per_group 2 (one group per block, under two shots' limits) changes nothing else.
      ``configure_launch(..., kind="pre")`` gives the pre-iteration launches their own shape.
    * ``hard_shots_first`` (default True): a relay decode of at least 1024 shots
      runs as two launches, the pre-iterations and then the relay legs resumed
      from each shot's saved state, with the shots the pre-iterations left
      unconverged queued first.  Those few shots run up to
      pre_iter + num_sets * set_max_iter iterations; started first, they finish
      alongside the bulk instead of after it.  Results are identical.
    * ``parity_first`` (0, 1 or 2): accepted and without effect; the kernel tests
      every iteration's convergence before the next min-sum pass.
    * ``cuda_graph`` (default False): a one-GPU decode of at least 1024 shots
      with no per-call options replays a CUDA graph of its launches, captured
      on the first call of each batch size (and again after a launch-shape
      change); the syndromes are copied into the graph's input and the
      results cloned out of its buffers, so each call costs one graph launch
      on the host instead of a dozen kernel and library calls.  Results are
      identical.
    """

    def __init__(
        self,
        H_csr: csr_matrix,
        error_priors: np.ndarray,
        pre_iter: int = 80,
        num_sets: int = 100,
        set_max_iter: int = 60,
        gamma0: float = 0.65,
        gamma_dist_interval: Tuple[float, float] = (-0.24, 0.66),
        stop_nconv: int = 5,
        normalized_min_sum_alpha: Optional[float] = None,
        offset_min_sum_beta: Optional[float] = None,
        data_type: str = "float32",
        device: Union[str, List[int], int] = [0],  # noqa: B006 - reference default
        seed: int = 1234,
        gamma_draw: str = "broadcast",
        bitpack_output: bool = False,
        algo: Optional[str] = None,
        perf: Optional[str] = None,
        alpha_iteration_scaling_factor: Optional[float] = 1.0,
        explicit_gammas: Optional[np.ndarray] = None,
        gamma_dist_interval_by_error: Optional[np.ndarray] = None,
        fast_max_unconverged_pct: Optional[float] = None,
        scheduling: str = "flood-fill",
        layered_k_iters: int = 0,
        layered_block_policy: str = "contiguous",
        layered_num_blocks: Optional[int] = None,
        layered_target_edges_per_block: Optional[int] = None,
        layered_block_seed: int = 42,
        unconverged_correction: str = "first_leg",
        *,
        mix_rounding: str = "separate",
        launch: Optional[Tuple[int, int]] = None,
        hard_shots_first: bool = True,
        parity_first: int = 2,
        cuda_graph: bool = False,
    ):
        if unconverged_correction not in UNCONVERGED_CORRECTIONS:
            raise ValueError(
                f"unconverged_correction must be one of {UNCONVERGED_CORRECTIONS} "
                f"(got {unconverged_correction!r})")
        self.unconverged_correction = unconverged_correction
        validate_csr_matrix(H_csr)
        error_priors = validate_error_priors(error_priors)
        if normalized_min_sum_alpha is not None and offset_min_sum_beta is not None:
            raise ValueError("Cannot specify both normalized_min_sum_alpha and offset_min_sum_beta")
        if normalized_min_sum_alpha is not None and not (0 <= normalized_min_sum_alpha <= 1):
            raise ValueError("normalized_min_sum_alpha must be in [0, 1]")
        if offset_min_sum_beta is not None and offset_min_sum_beta < 0:
            raise ValueError("offset_min_sum_beta must be >= 0")
        self.H_csr = H_csr
        self.check_permutation = None
        self.error_priors = error_priors
        self.pre_iter = int(pre_iter)
        self.num_sets = int(num_sets)
        self.set_max_iter = int(set_max_iter)
        self.gamma0 = gamma0
        self.gamma_dist_interval = gamma_dist_interval
        self.stop_nconv = int(stop_nconv)
        if fast_max_unconverged_pct is not None:
            if not (0.0 <= fast_max_unconverged_pct <= 1.0):
                raise ValueError(
                    f"fast_max_unconverged_pct must be between 0.0 and 1.0, got {fast_max_unconverged_pct}")
        self.fast_max_unconverged_pct = fast_max_unconverged_pct
        self.normalized_min_sum_alpha = normalized_min_sum_alpha
        self.offset_min_sum_beta = offset_min_sum_beta

        data_type = _DTYPE_ALIASES.get(data_type, data_type)
        if data_type not in _MSG_TYPES:
            raise ValueError(
                f"data_type must be 'float16', 'bfloat16', 'float32', or 'float64', got {data_type}")
        self.dtype_str = data_type
        self.dtype = {"float16": torch.float16, "bfloat16": torch.bfloat16, "float32": torch.float32,
                      "float64": torch.float64}[data_type]
        self._acc_dtype = torch.float64 if data_type == "float64" else torch.float32
        self.device_ids = self._parse_device_spec(device)
        self.num_gpus = len(self.device_ids)
        if not torch.cuda.is_available():
            raise RuntimeError("GPU not available (install a GPU-enabled PyTorch build: CUDA or ROCm)")
        self.device_type = "cuda"
        self._device_strs = {g: f"cuda:{g}" for g in self.device_ids}
        self.seed = int(seed)
        if gamma_draw not in GAMMA_DRAW_MODES:
            raise ValueError(f"gamma_draw must be one of {GAMMA_DRAW_MODES}; got {gamma_draw!r}")
        self.gamma_draw = gamma_draw
        self.bitpack_output = bool(bitpack_output)
        if algo not in ("relay", "plain"):
            raise ValueError(f"Unknown algo '{algo}'. Use 'relay' or 'plain'.")
        self.algo = algo
        perf_norm = (perf or "throughput").strip().lower()
        perf_aliases = {"default": "default", "row": "default", "rowwise": "default",
                        "throughput": "throughput", "btile": "throughput"}
        if perf_norm not in perf_aliases:
            raise ValueError(f"Unknown perf '{perf_norm}'. Use 'default'/'throughput'.")
        self.perf = perf_aliases[perf_norm]
        self.alpha_iteration_scaling_factor = float(alpha_iteration_scaling_factor or 1.0)
        scheduling_norm = (scheduling or "flood-fill").strip().lower()
        if scheduling_norm not in ("flood-fill", "layered"):
            raise ValueError(f"Unknown scheduling '{scheduling_norm}'. Use 'flood-fill' or 'layered'.")
        if scheduling_norm == "layered" and self.perf != "throughput":
            raise ValueError("scheduling='layered' requires perf='throughput'")
        if scheduling_norm == "layered":
            raise NotImplementedError("scheduling='layered' is not provided; use 'flood-fill'")
        self.scheduling = scheduling_norm
        if mix_rounding not in _MIX_MODES:
            raise ValueError(f"mix_rounding must be one of {tuple(_MIX_MODES)}")
        self.mix_rounding = mix_rounding

        V = int(H_csr.shape[1])
        self._explicit_gammas = None
        if explicit_gammas is not None:
            eg = np.asarray(explicit_gammas, dtype=np.float32)
            if eg.ndim != 2 or eg.shape[1] != V:
                raise ValueError(f"explicit_gammas must have shape (K, V={V})")
            self._explicit_gammas = eg
        self._gamma_by_error = None
        if gamma_dist_interval_by_error is not None:
            gd = np.asarray(gamma_dist_interval_by_error, dtype=np.float32)
            if gd.ndim != 2 or gd.shape[0] != V or gd.shape[1] != 2:
                raise ValueError(
                    f"gamma_dist_interval_by_error must have shape (V={V}, 2), got {tuple(gd.shape)}")
            if np.any(gd[:, 0] > gd[:, 1]):
                raise ValueError("gamma_dist_interval_by_error: lower bounds must be <= upper bounds")
            self._gamma_by_error = gd

        self.graph = TannerGraph(H_csr)
        self.C, self.V, self.E = self.graph.C, self.graph.V, self.graph.E
        self.log_prior_ratios = compute_log_prior_ratios(error_priors)          # [V] f32
        self.wj = np.where(np.isfinite(self.log_prior_ratios), self.log_prior_ratios, 0).astype(np.float32)
        # The reference seeds the global torch RNG here (decoder.py:774).
        torch.manual_seed(seed)

        self._launch = tuple(launch) if launch is not None else None
        self._pre_launch = None  # shape of the pre-iteration launches when it differs from _launch
        self.cuda_graph = bool(cuda_graph)
        self._cuda_graphs: Dict[int, tuple] = {}  # batch size -> (key, graph, static input, buffers)
        self.hard_shots_first = bool(hard_shots_first)
        if parity_first not in (0, 1, 2):
            raise ValueError("parity_first must be 0, 1 or 2")
        self.parity_first = int(parity_first)
        self._native: Dict[int, _NativeDecoder] = {}
        self._legs_broadcast: Dict[int, torch.Tensor] = {}
        self._alpha_len = max(self.pre_iter, self.set_max_iter, 1)
        for g in self.device_ids:
            self._native[g] = self._make_native(g, self._alpha_len)

    # ------------------------------------------------------------------ construction helpers

    def _parse_device_spec(self, device) -> List[int]:
        """decoder.py:1403-1452."""
        if isinstance(device, int):
            if device < 1:
                raise ValueError(f"Number of GPUs must be >= 1, got {device}")
            available = torch.cuda.device_count()
            if device > available:
                raise ValueError(f"Requested {device} GPUs but only {available} available")
            return list(range(device))
        if isinstance(device, list):
            if not device:
                raise ValueError("Device list cannot be empty")
            available = torch.cuda.device_count()
            for gpu_id in device:
                if not isinstance(gpu_id, int):
                    raise ValueError(f"Device IDs must be integers, got {type(gpu_id)}")
                if gpu_id < 0 or gpu_id >= available:
                    raise ValueError(f"Device ID {gpu_id} out of range [0, {available - 1}]")
            return list(device)
        if isinstance(device, str):
            if device.strip().lower() in ("auto", "cuda", "rocm"):
                return [0]
            raise ValueError(f"Unsupported device string '{device}'. Use List[int], int, or 'auto'/'cuda'.")
        raise ValueError(f"Invalid device type: {type(device)}. Expected List[int], int, or str.")

    def _leg_table(self, gpu_id: int) -> np.ndarray:
        """[num_sets, V] memory strengths of the relay legs with broadcast draws (decoder.py:3684-3700)."""
        R, V = self.num_sets, self.V
        if R == 0:
            return np.zeros((0, V), np.float32)
        if self._explicit_gammas is not None:
            K = self._explicit_gammas.shape[0]
            return np.stack([self._explicit_gammas[(leg + 1) % K] for leg in range(R)]).astype(np.float32)
        dev = self._device_strs[gpu_id]
        rows = []
        if self._gamma_by_error is not None:
            iv = torch.from_numpy(self._gamma_by_error).to(dev)
            for leg in range(R):
                rows.append(sample_gamma_per_variable(1, V, iv, dev, self.seed + leg))
        else:
            lo, hi = self.gamma_dist_interval
            for leg in range(R):
                rows.append(sample_gamma_uniform(1, V, lo, hi, dev, self.seed + leg))
        return torch.cat(rows, 0).float().cpu().numpy()

    def _per_row_legs(self, B: int, gpu_id: int, row0: int) -> torch.Tensor:
        """[B, num_sets, V] per-shot leg strengths for gamma_draw='per_row' (rows row0..row0+B of each draw)."""
        dev = self._device_strs[gpu_id]
        total = row0 + B
        out = torch.empty(B, self.num_sets, self.V, dtype=torch.float32, device=dev)
        for leg in range(self.num_sets):
            if self._gamma_by_error is not None:
                iv = torch.from_numpy(self._gamma_by_error).to(dev)
                g = sample_gamma_per_variable(total, self.V, iv, dev, self.seed + leg)
            else:
                lo, hi = self.gamma_dist_interval
                g = sample_gamma_uniform(total, self.V, lo, hi, dev, self.seed + leg)
            out[:, leg, :] = g[row0:total].float()
        return out

    def _params(self) -> nat.RbpParams:
        use_alpha, _ = alpha_schedule(self.normalized_min_sum_alpha, self.alpha_iteration_scaling_factor, 1)
        return nat.RbpParams(
            pre_iter=self.pre_iter, num_sets=self.num_sets, set_max_iter=self.set_max_iter,
            stop_nconv=self.stop_nconv, msg_type=_MSG_TYPES[self.dtype_str],
            last_leg=1 if self.unconverged_correction == "last_leg" else 0,
            use_alpha=1 if use_alpha else 0,
            use_beta=1 if self.offset_min_sum_beta is not None else 0,
            beta=float(self.offset_min_sum_beta or 0.0), mix_mode=_MIX_MODES[self.mix_rounding])

    def _make_native(self, gpu_id: int, alpha_len: int) -> _NativeDecoder:
        _, alpha = alpha_schedule(self.normalized_min_sum_alpha, self.alpha_iteration_scaling_factor, alpha_len)
        with torch.cuda.device(gpu_id):
            nd = _NativeDecoder(self.graph, gpu_id, self._params(), self.log_prior_ratios,
                                self._leg_table(gpu_id), alpha)
            if self._launch is not None:
                nd.configure(*self._launch)
            if self._pre_launch is not None:
                nd.configure(*self._pre_launch, kind=nat.RBP_LAUNCH_PRE)
        return nd

    # ------------------------------------------------------------------ public helpers

    def configure_launch(self, group_threads: int, groups_per_block: int, shots_per_group: int = 0,
                         blocks_per_sm: int = 0, kind: str = "all") -> None:
        """Set the kernel shape (threads per shot group, groups per thread block, shots a group
        decodes at once, resident blocks per SM the kernel is compiled for; 0 picks the default)
        of every launch (``kind="all"``), of the launches that run only the pre-iterations
        (``"pre"``: the first launch of a two-launch decode), or of the others (``"legs"``)."""
        if kind not in ("all", "pre", "legs"):
            raise ValueError("kind must be 'all', 'pre' or 'legs'")
        shape = (int(group_threads), int(groups_per_block), int(shots_per_group), int(blocks_per_sm))
        code = {"all": nat.RBP_LAUNCH_ALL, "pre": nat.RBP_LAUNCH_PRE, "legs": nat.RBP_LAUNCH_LEGS}[kind]
        for nd in self._native.values():
            nd.configure(*shape, kind=code)
        if kind == "all":
            self._launch, self._pre_launch = shape, None
        elif kind == "pre":
            self._pre_launch = shape
        else:
            if self._pre_launch is None:  # the pre-iteration launches keep their current shape
                self._pre_launch = self._launch if self._launch is not None else (0, 0, 0, 0)
            self._launch = shape

    def launch_info(self, shots: Optional[int] = None) -> dict:
        """The configured launch shape (the pre-iteration launches' under ``"pre"``).  Where the library chooses,
        it depends on the batch: ``shots`` gives that of a launch of so many shots, without it the shape of
        small batches."""
        return self._native[self.device_ids[0]].query(shots)

    def override_llr_columns(self, cols, value):
        """Overwrite prior LLRs (and selection weights) of some columns; returns a restore callable.

        decoder.py:786-834.  Values bypass the prior clipping, so negative LLRs are allowed.
        """
        cols = np.asarray(cols, dtype=np.int64)
        saved_llr = self.log_prior_ratios[cols].copy()
        saved_wj = self.wj[cols].copy()
        self.log_prior_ratios[cols] = np.asarray(value, dtype=np.float32)
        self.wj[cols] = np.asarray(value, dtype=np.float32)
        self._push_llr()

        def _restore():
            self.log_prior_ratios[cols] = saved_llr
            self.wj[cols] = saved_wj
            self._push_llr()

        return _restore

    def _push_llr(self):
        for nd in self._native.values():
            nd.set_llr(self.log_prior_ratios)

    def get_stats(self) -> Dict:
        return {
            "graph": self.graph.get_stats(),
            "parameters": {
                "pre_iter": self.pre_iter, "num_sets": self.num_sets, "set_max_iter": self.set_max_iter,
                "gamma0": self.gamma0, "gamma_dist_interval": self.gamma_dist_interval,
                "stop_nconv": self.stop_nconv, "dtype": self.dtype_str, "device": self.device_ids,
                "algo": self.algo, "perf": self.perf,
            },
        }

    # ------------------------------------------------------------------ decode

    def decode(
        self,
        syndromes: torch.Tensor,
        *,
        init_posterior: Optional[torch.Tensor] = None,
        init_gamma: Optional[torch.Tensor] = None,
        skip_relay_legs: bool = False,
        pre_iter_override: Optional[int] = None,
        return_last_posterior: bool = False,
        prior_llr: Optional[torch.Tensor] = None,
        leg_gammas: Optional[torch.Tensor] = None,
    ) -> Dict[str, torch.Tensor]:
        """Decode [B, C] uint8 syndromes; see decoder.py:2317-2361 for the keyword arguments.

        ``leg_gammas`` ([B, L, V], this implementation only) gives each shot its own
        memory strengths for relay legs 0..L-1; later legs use the seeded table.
        """
        if not isinstance(syndromes, torch.Tensor):
            syndromes = torch.as_tensor(np.asarray(syndromes))
        if syndromes.ndim != 2:
            raise ValueError(f"Expected a [B, {self.C}] syndrome tensor, got shape {tuple(syndromes.shape)}")
        B = int(syndromes.shape[0])
        if syndromes.shape[1] != self.C:
            raise ValueError(f"Expected {self.C} syndrome bits, got {syndromes.shape[1]}")
        advanced = (init_posterior is not None or init_gamma is not None or skip_relay_legs
                    or pre_iter_override is not None or return_last_posterior or prior_llr is not None)
        if advanced:
            if self.perf != "throughput":
                raise ValueError(
                    "init_posterior / init_gamma / skip_relay_legs / pre_iter_override / "
                    f"return_last_posterior are only supported in throughput perf mode (got perf={self.perf!r}).")
            if self.num_gpus > 1:
                raise ValueError(
                    "init_posterior / init_gamma / skip_relay_legs / pre_iter_override / "
                    "return_last_posterior / prior_llr require single-GPU decode "
                    f"(self.num_gpus={self.num_gpus}).")
            for name, t in (("init_posterior", init_posterior), ("init_gamma", init_gamma),
                            ("prior_llr", prior_llr)):
                if t is not None and tuple(t.shape) != (B, self.V):
                    raise ValueError(f"{name} shape {tuple(t.shape)} != ({B}, {self.V})")
        if leg_gammas is not None and (leg_gammas.ndim != 3 or leg_gammas.shape[0] != B
                                       or leg_gammas.shape[2] != self.V):
            raise ValueError(f"leg_gammas must have shape ({B}, L, {self.V})")
        pre = self.pre_iter if pre_iter_override is None else int(pre_iter_override)
        if pre < 0:
            raise ValueError("pre_iter_override must be >= 0")
        if pre > self._alpha_len and self.normalized_min_sum_alpha is not None:
            self._alpha_len = pre
            for g in self.device_ids:
                self._native[g].close()
                self._native[g] = self._make_native(g, self._alpha_len)

        if self.num_gpus == 1:
            if self.fast_max_unconverged_pct is not None and not skip_relay_legs:
                return self._decode_leg_synchronous(syndromes, pre, init_posterior, init_gamma,
                                                    return_last_posterior, prior_llr, leg_gammas)
            if (self.hard_shots_first and not skip_relay_legs and self.num_sets > 0 and pre > 0
                    and B >= HARD_FIRST_MIN_BATCH):
                if self.cuda_graph and not advanced and leg_gammas is None:
                    return self._decode_graphed(syndromes, pre)
                return self._decode_hard_first(self.device_ids[0], syndromes, pre, init_posterior, init_gamma,
                                               return_last_posterior, prior_llr, leg_gammas)
            return self._decode_on(self.device_ids[0], syndromes, 0, pre, init_posterior, init_gamma,
                                   skip_relay_legs, return_last_posterior, prior_llr, leg_gammas)
        # Replicas: every shard's kernels are enqueued on its own device before any result is
        # read back (the reads synchronise the host), so the devices decode concurrently, as the
        # reference's one host thread per GPU does (decoder.py:2475-2543).
        splits = self._split_batch(B, self.num_gpus)
        raws = []
        for gpu_id, (s0, s1) in zip(self.device_ids, splits):
            lg = leg_gammas[s0:s1] if leg_gammas is not None else None
            if self.hard_shots_first and self.num_sets > 0 and pre > 0 and s1 - s0 >= HARD_FIRST_MIN_BATCH:
                raws.append(self._launch_hard_first(gpu_id, syndromes[s0:s1], pre, None, None, False, None, lg))
            else:
                raws.append(self._launch_on(gpu_id, syndromes[s0:s1], s0, pre, None, None, False, False, None, lg))
        parts = [self._finish(r) for r in raws]
        return self._gather(parts, splits)

    @staticmethod
    def _split_batch(B: int, num_gpus: int) -> List[Tuple[int, int]]:
        """Contiguous, near-equal shards; the first B % n get one extra shot (decoder.py:2451-2473)."""
        base, rem = divmod(B, num_gpus)
        out, start = [], 0
        for i in range(num_gpus):
            end = start + base + (1 if i < rem else 0)
            out.append((start, end))
            start = end
        return out

    def _gather(self, parts: Sequence[dict], splits) -> Dict[str, torch.Tensor]:
        target = self._device_strs[self.device_ids[0]]
        out = {}
        for k in ("errors", "weights", "valid_mask", "iterations", "found_count"):
            out[k] = torch.cat([p[k].to(target) for p in parts], 0)
        unc = [p["unconverged_indices"].to(target) + s0 for p, (s0, _) in zip(parts, splits)]
        out["unconverged_indices"] = torch.cat(unc, 0).to(torch.int32)
        return out

    def state_bytes(self, gpu_id: Optional[int] = None) -> int:
        """Bytes of one shot's saved decode state (resumable decoding)."""
        b = ct.c_int64()
        gid = self.device_ids[0] if gpu_id is None else gpu_id
        nat.check(nat.lib().rbp_state_bytes(self._native[gid]._dec, ct.byref(b)), "rbp_state_bytes")
        return int(b.value)

    def new_state(self, B: int) -> torch.Tensor:
        """Device buffer for B shots' saved decode state."""
        return torch.empty(B, self.state_bytes(), dtype=torch.uint8, device=self._device_strs[self.device_ids[0]])

    def decode_phases(self, syndromes: torch.Tensor, *, resume: Optional[torch.Tensor] = None,
                      suspend: Optional[torch.Tensor] = None, legs_begin: int = 0, legs_end: int = 0,
                      skip_relay_legs: bool = False, leg_gammas: Optional[torch.Tensor] = None,
                      leg_gammas_legs: Optional[int] = None,
                      return_last_posterior: bool = False) -> Dict[str, torch.Tensor]:
        """Run part of a decode: from the pre-iterations (or, with `resume`, from relay leg
        `legs_begin` of the saved state) up to relay leg `legs_end` (0: all), saving the state in
        `suspend`.  Outputs reflect the shots' state after the last phase run.  `leg_gammas`
        ([B, R, V]) gives each shot its own strengths for the first `leg_gammas_legs` legs (default
        R); leg l uses row min(l, R - 1)."""
        if self.num_gpus != 1:
            raise ValueError("resumable decoding runs on one GPU")
        if resume is not None and not 0 <= legs_begin <= self.num_sets:
            raise ValueError("legs_begin out of range")
        return self._decode_on(self.device_ids[0], syndromes, 0, self.pre_iter, None, None, skip_relay_legs,
                               return_last_posterior, None, leg_gammas, resume, suspend, legs_begin, legs_end,
                               leg_gammas_legs)

    def _decode_leg_synchronous(self, syndromes, pre, init_posterior, init_gamma, return_last_posterior,
                                prior_llr, leg_gammas):
        """decode() with fast_max_unconverged_pct: the pre-iterations, then one relay leg per launch,
        checking after each phase, as the reference does (decoder.py:3619-3662, 3812-3831), whether
        every shot is done or the unconverged fraction fell below the threshold."""
        gid = self.device_ids[0]
        B = int(syndromes.shape[0])
        state = self.new_state(B)
        out = self._decode_on(gid, syndromes, 0, pre, init_posterior, init_gamma, True,
                              return_last_posterior, prior_llr, leg_gammas, None, state, 0, 0)
        thr = self.fast_max_unconverged_pct
        for leg in range(-1, self.num_sets):
            if leg >= 0:
                out = self._decode_on(gid, syndromes, 0, pre, None, None, False, return_last_posterior,
                                      prior_llr, leg_gammas, state, state, leg, leg + 1)
            unconv = float((out["found_count"] < self.stop_nconv).float().mean()) if B else 0.0
            if unconv == 0.0:
                break
            if unconv < thr and unconv < 1.0:
                break
        return out

    def _state_buffer(self, gpu_id: int, B: int) -> torch.Tensor:
        """Per-device saved-state buffer of the two-launch decode, kept for the next call of the same
        or a smaller batch (a fresh 11 KB-per-shot allocation per call stalls the allocator)."""
        cache = self.__dict__.setdefault("_state_cache", {})
        buf = cache.get(gpu_id)
        if buf is None or buf.shape[0] < B:
            cache[gpu_id] = None
            buf = torch.empty(B, self.state_bytes(gpu_id), dtype=torch.uint8, device=self._device_strs[gpu_id])
            cache[gpu_id] = buf
        return buf[:B]

    def _decode_hard_first(self, gpu_id, syndromes, pre, init_posterior, init_gamma, return_last_posterior,
                           prior_llr, leg_gammas) -> Dict[str, torch.Tensor]:
        """Pre-iterations, then the relay legs with the unconverged shots queued first."""
        return self._finish(self._launch_hard_first(gpu_id, syndromes, pre, init_posterior, init_gamma,
                                                    return_last_posterior, prior_llr, leg_gammas))

    def _decode_graphed(self, syndromes: torch.Tensor, pre: int) -> Dict[str, torch.Tensor]:
        """_decode_hard_first as one CUDA-graph replay (``cuda_graph``): the graph of a batch size
        is captured from the two launches and the device ops between them after an eager warm-up
        call; a call copies the syndromes (host or device) into the graph's input buffer, replays
        it and clones the results out of the graph's buffers."""
        gid = self.device_ids[0]
        B = int(syndromes.shape[0])
        key = (pre, self._launch, self._pre_launch)
        entry = self._cuda_graphs.get(B)
        if entry is None or entry[0] != key:
            self._cuda_graphs = {}  # one batch size at a time; a graph holds its buffers
            with torch.cuda.device(gid):
                static = torch.empty(B, self.C, dtype=torch.uint8, device=self._device_strs[gid])
                static.copy_(syndromes)
                self._launch_hard_first(gid, static, pre, None, None, False, None, None)  # state buffer, attributes
                torch.cuda.synchronize(gid)
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g):
                    raw = self._launch_hard_first(gid, static, pre, None, None, False, None, None)
            entry = (key, g, static, raw)
            self._cuda_graphs[B] = entry
        _, g, static, raw = entry
        with torch.cuda.device(gid):
            static.copy_(syndromes, non_blocking=True)
            g.replay()
            out = {k: v.clone() if isinstance(v, torch.Tensor) else v for k, v in raw.items()}
            return self._finish(out)

    def _launch_hard_first(self, gpu_id, syndromes, pre, init_posterior, init_gamma, return_last_posterior,
                           prior_llr, leg_gammas) -> dict:
        """_decode_hard_first's two launches, enqueued without a host synchronisation."""
        B = int(syndromes.shape[0])
        dev = self._device_strs[gpu_id]
        with on_device(gpu_id):
            syn = syndromes.to(device=dev, dtype=torch.uint8).contiguous()
            state = self._state_buffer(gpu_id, B)
            first = self._decode_on(gpu_id, syn, 0, pre, init_posterior, init_gamma, True, False, prior_llr,
                                    leg_gammas, None, state, 0, 0, light=True)
            order = queue_order(first["found_count"])  # the unconverged ones, then the converged, both in order
            return self._launch_on(gpu_id, syn, 0, pre, None, None, False, return_last_posterior, prior_llr,
                                   leg_gammas, state, None, 0, 0, order=order)

    def _decode_on(self, gpu_id, syndromes, row0, pre, init_posterior, init_gamma, skip_relay_legs,
                   return_last_posterior, prior_llr, leg_gammas, resume=None, suspend=None, legs_begin=0,
                   legs_end=0, leg_gammas_legs=None, order=None, light=False) -> Dict[str, torch.Tensor]:
        """One launch and its result dict.  ``order`` sets the queue order; ``light`` returns only
        found_count and iterations (no error rows, no host synchronisation)."""
        raw = self._launch_on(gpu_id, syndromes, row0, pre, init_posterior, init_gamma, skip_relay_legs,
                              return_last_posterior, prior_llr, leg_gammas, resume, suspend, legs_begin, legs_end,
                              leg_gammas_legs, order, light)
        if light:
            return {"found_count": raw["found"], "iterations": raw["iters"]}
        return self._finish(raw)

    def _launch_on(self, gpu_id, syndromes, row0, pre, init_posterior, init_gamma, skip_relay_legs,
                   return_last_posterior, prior_llr, leg_gammas, resume=None, suspend=None, legs_begin=0,
                   legs_end=0, leg_gammas_legs=None, order=None, light=False) -> dict:
        """Enqueue one decode launch on the device's current stream and return its output buffers
        (no host synchronisation)."""
        B = int(syndromes.shape[0])
        dev = self._device_strs[gpu_id]
        with on_device(gpu_id):
            syn = syndromes.to(device=dev, dtype=torch.uint8).contiguous()
            f32 = dict(device=dev, dtype=torch.float32)
            ip = init_posterior.to(**f32).contiguous() if init_posterior is not None else None
            ig = None
            gamma0 = 0.0
            if self.algo == "relay":
                if init_gamma is not None:
                    ig = init_gamma.to(**f32).contiguous()
                else:
                    gamma0 = float(np.float32(self.gamma0))
            pl = prior_llr.to(**f32).contiguous() if prior_llr is not None else None
            shot_legs, n_shot_legs, shot_rows = None, 0, 0
            if self.gamma_draw == "per_row" and self._explicit_gammas is None and self.num_sets > 0:
                # each device draws rows 0..B_i-1, as the reference's per-GPU loop does
                shot_legs = self._per_row_legs(B, gpu_id, 0)
                n_shot_legs = self.num_sets
            if leg_gammas is not None:
                lg = leg_gammas.to(**f32).contiguous()
                R = int(lg.shape[1])
                L = min(R if leg_gammas_legs is None else int(leg_gammas_legs), self.num_sets)
                if shot_legs is not None:
                    for leg in range(L):
                        shot_legs[:, leg] = lg[:, min(leg, R - 1)]
                else:
                    shot_legs, n_shot_legs, shot_rows = lg, L, R
            W = (self.V + 31) // 32
            found = torch.empty(B, dtype=torch.int32, device=dev)
            iters = torch.empty(B, dtype=torch.int32, device=dev)
            wfix = torch.empty(B, dtype=torch.int64, device=dev)
            errors = packed = None
            if light:
                pass
            elif self.bitpack_output:
                packed = torch.empty(B, W, dtype=torch.int32, device=dev)
            else:
                errors = torch.empty(B, self.V, dtype=torch.uint8, device=dev)
            last_post = torch.empty(B, self.V, dtype=self._acc_dtype, device=dev) if return_last_posterior else None
            batch = nat.RbpBatch(syndromes=_ptr(syn), llr_per_shot=_ptr(pl), gamma_pre=_ptr(ig),
                                 gamma0=gamma0, init_posterior=_ptr(ip), gamma_legs_shot=_ptr(shot_legs),
                                 n_shot_legs=n_shot_legs, pre_iter=pre,
                                 skip_relay_legs=1 if skip_relay_legs else 0,
                                 resume_state=_ptr(resume), suspend_state=_ptr(suspend),
                                 legs_begin=int(legs_begin), legs_end=int(legs_end), shot_leg_rows=shot_rows,
                                 shot_order=_ptr(order), parity_first=self.parity_first)
            outs = nat.RbpOutputs(errors=_ptr(errors), errors_packed=_ptr(packed), weights=None,
                                  weight_fixed=_ptr(wfix), found_count=_ptr(found), iterations=_ptr(iters),
                                  last_posterior=_ptr(last_post))
            stream = torch.cuda.current_stream(gpu_id).cuda_stream
            self._native[gpu_id].decode(B, batch, outs, stream)
            # Inputs freed after this call stay safe: the caching allocator reuses their memory
            # only for work ordered after this stream's kernel.
            return {"gpu_id": gpu_id, "found": found, "iters": iters, "wfix": wfix, "errors": errors,
                    "packed": packed, "last_post": last_post}

    def _finish(self, raw: dict) -> Dict[str, torch.Tensor]:
        """The result dict of a launch's buffers (the unconverged-index list synchronises the host)."""
        found, iters, wfix = raw["found"], raw["iters"], raw["wfix"]
        wdt = torch.float64 if self.dtype_str == "float64" else torch.float32
        weights, valid, unconverged = finish_results(found, wfix, self.stop_nconv, wdt)
        result = {
            "errors": raw["packed"] if self.bitpack_output else raw["errors"],
            "weights": weights,
            "valid_mask": valid,
            "iterations": iters,
            "found_count": found,
            "unconverged_indices": unconverged,
            "weight_fixed": wfix,
        }
        if raw["last_post"] is not None:
            result["last_posterior"] = raw["last_post"]
        return result

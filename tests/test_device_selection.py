"""Native calls that take only device pointers launch on the calling thread's current device, so their
callers select the tensors' device first.  Checked on the CPU: a stand-in library records the device that is
selected at each call, for a decoder whose device is not the current one."""

from __future__ import annotations

import ctypes as ct
from types import SimpleNamespace

import numpy as np
import pytest
import scipy.sparse as sp
import torch

from pelagos_b200 import _native as nat
from pelagos_b200.adapter import _DeviceCSR
from pelagos_b200.decoder import finish_results, queue_order
from pelagos_b200.proposal import LearnedRelayBPDecoder

DEV = torch.device("cpu")  # the tensors' device; the current one is another
C, V = 3, 5


@pytest.fixture
def calls(monkeypatch):
    """(entry, device selected) of every native call."""
    log, selected = [], ["another device"]

    class Select:
        def __init__(self, device):
            self.device = device

        def __enter__(self):
            selected.append(self.device)

        def __exit__(self, *exc):
            selected.pop()

    class Library:
        def __getattr__(self, name):
            def entry(*args):
                log.append((name, selected[-1]))
                if name == "rbp_results":  # no unconverged shots
                    ct.c_int32.from_address(args[8]).value = 0
                return nat.RBP_OK

            return entry

    library = Library()
    monkeypatch.setattr(nat, "lib", lambda: library)
    monkeypatch.setattr(torch.cuda, "device", Select)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: SimpleNamespace(cuda_stream=0))
    return log


def _on_tensor_device(log, names):
    assert {n for n, _ in log} >= set(names)
    assert all(device == DEV for name, device in log if name in names), log


def test_result_arrays_and_queue_order(calls):
    found, wfix = torch.ones(4, dtype=torch.int32), torch.zeros(4, dtype=torch.int64)
    finish_results(found, wfix, 1)
    queue_order(found, torch.zeros(1, dtype=torch.int32))
    _on_tensor_device(calls, ("rbp_results", "rbp_queue_order"))


def test_gf2_products_and_failure_counts(calls):
    A = _DeviceCSR(sp.csr_matrix(np.eye(C, V)), DEV)
    x, n = torch.zeros(4, V, dtype=torch.uint8), torch.ones(4, dtype=torch.int32)
    A.apply(x)
    A.failures(x, x, n, n)
    _on_tensor_device(calls, ("rbp_gf2_matvec", "rbp_gf2_failures"))


@pytest.mark.parametrize("gate,fused", [(False, False), (True, False), (True, True)])
def test_learned_decode(calls, gate, fused):
    native = SimpleNamespace(_dec=ct.c_void_p(), decode=lambda *args: None)
    dec = SimpleNamespace(C=C, V=V, algo="relay", num_gpus=1, num_sets=2, gamma_dist_interval=(-0.24, 0.66),
                          gamma0=0.65, pre_iter=3, stop_nconv=1, parity_first=2, device_ids=[1], _native={1: native},
                          new_state=lambda B: torch.zeros(B, 64, dtype=torch.uint8))
    net = SimpleNamespace(device=DEV, propose_into=lambda *args, **kw: None)
    learned = LearnedRelayBPDecoder(dec, net, learned_legs=1, gate=gate, fused=fused, graph=False)
    learned.decode(torch.zeros(4, C, dtype=torch.uint8))
    _on_tensor_device(calls, ("rbp_results", "rbp_queue_order"))

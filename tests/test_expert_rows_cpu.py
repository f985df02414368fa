"""How many routed rows the grouped product is told to expect, on a fake kernel library."""
import ctypes

import pytest
import torch

from tensorrt_edge_llm_b200.ops import cuda as cu


@pytest.fixture
def calls(monkeypatch):
    seen = {}

    class Library:
        def __getattr__(self, name):
            return lambda *a: seen.setdefault(name, a) and 0

    monkeypatch.setattr(cu, "lib", Library)
    monkeypatch.setattr(cu, "_p", lambda t: None)
    monkeypatch.setattr(cu, "_stream", lambda: ctypes.c_void_p(0))
    monkeypatch.setattr(cu.Workspace, "get", classmethod(lambda cls, device: type("W", (), {"status": None})))
    return seen


@pytest.mark.parametrize("tokens,top_k,experts,lo,hi,share,rows", [
    (32, 8, 128, 0, 128, None, 256), (32, 8, 128, 32, 64, None, 64), (1, 1, 64, 0, 1, None, 1), (512, 1, 16, 0, 16, 0.125, 64)])
def test_grouped_product_expects_the_slots_routed_here(calls, tokens, top_k, experts, lo, hi, share, rows):
    """Of the slots of a step a rank with part of the experts gets that part, and of a receive buffer one rank's share."""
    ws = cu.moe_align(torch.zeros(tokens, top_k, dtype=torch.int32), experts, lo, hi, share)
    assert ws.dst_row.numel() == tokens * top_k
    local = hi - lo
    acts = cu.QuantActs(torch.zeros(ws.rows_pad, 64, dtype=torch.uint8), torch.zeros(16, dtype=torch.uint8), (ws.rows_pad, 128), torch.float16)
    cu.gemm_grouped(acts, torch.zeros(local * 128, 64, dtype=torch.uint8), ws, local, w_sf=None)
    assert calls["telb_gemm_nvfp4_grouped"][-2].value == rows

"""The MLP's fused product leaves out its projection module only where nothing watches it."""
import pytest
import torch


@pytest.mark.parametrize("act", ["silu", "relu2"])
def test_mlp_calls_a_projection_that_is_watched(act, monkeypatch):
    """The product with the activation in its epilogue passes the projection module by: not where hooks or a replaced forward wait for the call."""
    from tensorrt_edge_llm_b200.config import hybrid_nemotron_config, qwen3_8b_config
    from tensorrt_edge_llm_b200.models import default
    cfg = (hybrid_nemotron_config if act == "relu2" else qwen3_8b_config)(hidden_size=64, intermediate_size=128, num_hidden_layers=1, vocab_size=64)
    cfg.hidden_act = act
    mlp = default.MLP(cfg, "model.layers.0.mlp")
    for p in mlp.parameters():
        torch.nn.init.normal_(p, std=0.1)

    class OnGpu(torch.Tensor):
        is_cuda = True

    taken, seen = [], []
    monkeypatch.setattr(default.ops, "linear_act", lambda x, w, a: taken.append(a) or x.new_zeros(x.shape[0], 128))
    x = torch.randn(3, 64, dtype=cfg.compute_dtype)
    run = lambda: mlp(x.as_subclass(OnGpu))
    monkeypatch.setattr(default.Linear, "forward", lambda self, v: torch.nn.functional.linear(v.as_subclass(torch.Tensor), self.weight))
    run()
    assert taken == ["relu2" if act == "relu2" else "swiglu"]
    for attach in ("register_forward_hook", "register_forward_pre_hook"):
        handle = getattr(mlp.gate_up_proj, attach)(lambda *a: seen.append(attach))
        run()
        handle.remove()
    mlp.gate_up_proj.forward = lambda v: seen.append("own") or torch.nn.functional.linear(v.as_subclass(torch.Tensor), mlp.gate_up_proj.weight)
    run()
    assert len(taken) == 1 and seen == ["register_forward_hook", "register_forward_pre_hook", "own"]

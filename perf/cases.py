"""Work that a serving program has this framework do, as measurable cases.

A case of the 16-bit stacks is one step of a model through ``ModelRunner`` (prompts, and prompt portions beside decode rows) or one
replay of a captured model step (decode, tree verification).  The stacks are the benchmark's own: the Qwen3-8B shape and the Mamba2 /
gated DeltaNet / attention hybrid, each cut to a part of its layers, and its vocabulary to the same part, so that the head keeps its
share of the time.  Weights, prompts and cached rows are random.

A case of the NVFP4 stacks (the Qwen3-8B shape, and the Qwen3-30B-A3B shape with NVFP4 experts) is the blocks of its layers that work on
NVFP4 rows: norm and q / k / v projection, output projection, norm and MLP or experts.  Every block has an input of its own: rounding
activations to four bits turns a last-bit difference in front of it into one of some per cent behind it, so that the end of
a chain of such layers says nothing about whether they were computed rightly.
"""
from __future__ import annotations

import math
import zlib

import torch

PAGE = 64
#: layers and vocabulary kept (dense 6 of 36, mixture 6 of 48, hybrid 12 of 52)
STACKS = {
    "dense": dict(layers=6, vocab=25344, hidden=4096, hq=32, hkv=8, inter=12288, eps=1e-6, theta=1e6, qk_norm=True),
    "moe": dict(layers=6, vocab=19008, hidden=2048, hq=32, hkv=4, inter=768, eps=1e-6, theta=1e6, qk_norm=True, experts=128, top_k=8),
    "hybrid": dict(layers=12, vocab=30272, hidden=4096, hq=32, hkv=8, inter=16384, eps=1e-5, theta=1e4, qk_norm=False),
}
HD = 128                                              # head size of every attention layer
SSM = dict(heads=64, dim=64, state=128, groups=8, taps=4, limit=50.0)
GDN = dict(heads=16, dim=128, taps=4)
INPUT_SCALE = 1.0 / 448.0


def listed():
    bf16 = dict(model="dense", weights="bf16")
    fp4 = dict(model="dense", weights="nvfp4", phase="rows", batch=1)
    moe = dict(model="moe", weights="nvfp4", phase="rows", batch=1)
    hyb = dict(model="hybrid", weights="bf16")
    none = dict(past=0, new=1, spread=0.0, rows=0)
    return [
        # NVFP4 projections: one user's token, where launches and weight reads are all there is; the headline benchmark's 64 users; its
        # prompt step of 8 x 1024 tokens
        dict(none, name="fp4_token", **fp4),
        dict(none, name="fp4_batch64", **dict(fp4, new=64)),
        dict(none, name="fp4_prompts", **dict(fp4, new=8192)),
        # NVFP4 experts: decode step and prompts of the benchmark's shape
        dict(none, name="experts_token", **dict(moe, new=32)),
        dict(none, name="experts_prompts", **dict(moe, new=8000)),
        # decode of 64 users, 1024 tokens and a bit each
        dict(none, name="batch64_token", phase="decode", batch=64, past=1088, **bf16),
        # many long conversations, lengths apart
        dict(none, name="long_token", phase="decode", batch=30, past=4000, spread=0.6, **bf16),
        # in-flight batching: decode rows of other users beside a portion of a new prompt
        dict(none, name="mixed_step", phase="mixed", batch=47, past=1100, spread=0.5, new=983, **bf16),
        # one long document
        dict(none, name="long_prompt", phase="prefill", batch=1, new=8129, **bf16),
        # EAGLE-3: 60 tree rows for each of 4 users
        dict(none, name="tree_verify", phase="verify", batch=4, past=2048, rows=60, **bf16),
        # recurrent hybrid: decode of 16 long sequences, and prompts
        dict(none, name="hybrid_token", phase="decode", batch=16, past=8192, **hyb),
        dict(none, name="hybrid_prompt", phase="prefill", batch=3, new=2700, spread=0.3, **hyb),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another step of the same stacks: 1 to 8192 rows, batches of 1 to 64, up to 131072 cached tokens."""
    model, weights, phase = rng.choice([
        ("dense", "nvfp4", "rows"), ("dense", "nvfp4", "rows"), ("moe", "nvfp4", "rows"), ("moe", "nvfp4", "rows"), ("dense", "bf16", "prefill"),
        ("dense", "bf16", "decode"), ("dense", "bf16", "decode"), ("dense", "bf16", "mixed"), ("dense", "bf16", "verify"),
        ("hybrid", "bf16", "decode"), ("hybrid", "bf16", "prefill")])
    c = dict(model=model, weights=weights, phase=phase, batch=1, past=0, new=1, rows=0, spread=0.0)
    if phase == "rows":
        c["new"] = _log(rng, 1, 8192)
        return c
    c["spread"] = round(rng.choice([0.0, rng.uniform(0.1, 0.8)]), 3)
    if phase == "prefill":
        c["new"] = _log(rng, 100, 8129)
        c["batch"] = rng.randint(1, max(1, min(16, 8129 // c["new"])))
    elif phase == "verify":
        c["batch"], c["past"], c["rows"] = rng.randint(1, 8), _log(rng, 100, 4096), rng.choice([16, 31, 60])
    else:
        c["batch"] = _log(rng, 1, 64) if model == "dense" else _log(rng, 1, 32)
        c["past"] = _log(rng, 100, min(8192, 131072 // c["batch"]))
        if phase == "mixed":
            c["new"] = _log(rng, 64, 4096)
    return c


def _lens(c, longest):
    """Lengths of a batch: the longest, and the others shorter by up to ``spread``."""
    return [max(1, int(round(longest * (1.0 - c["spread"] * ((i * 0.6180339887) % 1.0))))) for i in range(c["batch"])]


def _steps(c):
    """(cached tokens, new rows) of every sequence of the step."""
    if c["phase"] in ("prefill", "rows"):
        return [(0, n) for n in _lens(c, c["new"])]
    if c["phase"] == "verify":
        return [(p, c["rows"]) for p in _lens(c, c["past"])]
    decode = [(p, 1) for p in _lens(c, c["past"])]
    return decode + [(PAGE, c["new"])] if c["phase"] == "mixed" else decode       # the portion goes on behind a cached page


def _kinds(model):
    """Mixer of every layer."""
    if model != "hybrid":
        return ["attention"] * STACKS[model]["layers"]
    kinds, seen = [], 0
    for i in range(STACKS[model]["layers"]):
        if (i + 1) % 6 == 0:
            kinds.append("attention")
        else:
            seen += 1
            kinds.append("gdn" if seen % 4 == 0 else "mamba")
    return kinds


# ---- weights and inputs, drawn by name from the seed ---------------------------------------------------------------------------------


def _dtype(c):
    """NVFP4 rows go with fp16, as in the headline benchmark."""
    return torch.float16 if c["weights"] == "nvfp4" else torch.bfloat16


class _Source:
    """Checkpoint tensors by name, each drawn on the GPU from the seed and its name."""

    def __init__(self, c, seed):
        self.c, self.seed, self.s, self.dt = c, seed, STACKS[c["model"]], _dtype(c)

    def normal(self, name, shape, std=1.0):
        g = torch.Generator(device="cuda").manual_seed((self.seed * 1000003 + zlib.crc32(name.encode())) % (1 << 62))
        return torch.randn(shape, generator=g, device="cuda") * std

    def is_fp4(self, name):
        if self.c["weights"] != "nvfp4":
            return False
        return ".experts." in name if self.c["model"] == "moe" else ".layers." in name

    def shape(self, name):
        s, leaf = self.s, name.rsplit(".", 1)[-1]
        h, q, kv = s["hidden"], s["hq"] * HD, s["hkv"] * HD
        d_in, gn = SSM["heads"] * SSM["dim"], SSM["groups"] * SSM["state"]
        vd = GDN["heads"] * GDN["dim"]
        if leaf in ("lm_head", "embed_tokens"):
            return 64 if self.c["phase"] == "rows" else s["vocab"], h
        return {"q_proj": (q, h), "k_proj": (kv, h), "v_proj": (kv, h), "o_proj": (h, q), "gate_proj": (s["inter"], h), "up_proj": (s["inter"], h),
                "down_proj": (h, s["inter"]), "gate": (s.get("experts", 0), h),
                "in_proj": (2 * d_in + 2 * gn + SSM["heads"], h), "in_proj_qkv": (3 * vd, h), "in_proj_z": (vd, h), "in_proj_b": (GDN["heads"], h),
                "in_proj_a": (GDN["heads"], h), "out_proj": (h, d_in if ".mamba" in name else vd)}[leaf]

    def raw(self, name):
        return self.normal(name, self.shape(name), 0.02)

    def linear(self, name):
        """Checkpoint tensors of one linear layer (NVFP4: E2M1 pairs, an E4M3 scale per 16 inputs, a scale per tensor)."""
        w = self.raw(name)
        if not self.is_fp4(name):
            return {"weight": w.to(self.dt)}
        codes, sf, gs = _fp4(w, w.abs().amax() / (6.0 * 448.0))
        return {"weight": (codes[:, 0::2] | (codes[:, 1::2] << 4)).contiguous(), "weight_scale": sf, "weight_scale_2": gs,
                "input_scale": torch.tensor(INPUT_SCALE, device="cuda")}

    def dense64(self, name):
        """The same weight as 64-bit numbers."""
        w = self.raw(name)
        if not self.is_fp4(name):
            return w.to(self.dt).double()
        return _fp4_round(w, w.abs().amax() / (6.0 * 448.0))

    def conv(self, name, channels):
        return self.normal(name, (channels, 4), 0.3).to(self.dt)

    def small(self, name, n):
        """Decay rates and step-size offsets of a recurrent layer."""
        u = torch.sigmoid(self.normal(name, (n,), 1.5))
        return torch.log(u * 3 + 1) if name.endswith("A_log") else u - 2.0

    def cached(self, i, layers, hkv, past):
        """Cached keys and values of sequence ``i``: ``[layers, 2, kv heads, past, head]``."""
        return self.normal(f"kv.{i}", (layers, 2, hkv, past, HD)).to(self.dt)

    def block_inputs(self, i):
        """What the blocks of layer ``i`` read: projection outputs and residual rows in front of both norms, and attention outputs."""
        s, t, p = self.s, self.c["new"], f"in.{i}."
        x = {n: self.normal(p + n, (t, s["hidden"])).to(self.dt) for n in ("h1", "r1", "h2", "r2")}
        x["a"] = self.normal(p + "a", (t, s["hq"] * HD), 0.5).to(self.dt)
        return x

    def tokens(self):
        g = torch.Generator().manual_seed(self.seed * 7919 + 17)
        return [torch.randint(0, self.s["vocab"], (n,), generator=g).tolist() for _, n in _steps(self.c)]

    def parents(self):
        """A draft tree per sequence: row 0 is the root, every other row hangs below an earlier one."""
        g = torch.Generator().manual_seed(self.seed * 104729 + 3)
        b, r = self.c["batch"], self.c["rows"]
        u = torch.rand(b, r, generator=g)
        return torch.stack([torch.full((b,), -1, dtype=torch.int64)] + [(u[:, j] * min(j, 10)).long() + max(0, j - 10) for j in range(1, r)], 1)


_LEVELS = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0)


def _fp4(x, gs):
    """E2M1 codes, E4M3 block scales and the tensor's scale; ties to even."""
    b = x.reshape(x.shape[0], -1, 16)
    sf = (b.abs().amax(-1) / 6.0 / gs).clamp(max=448.0).to(torch.float8_e4m3fn)
    step = (sf.to(x.dtype) * gs)[..., None]
    a = torch.where(step > 0, b / step.clamp(min=1e-30), torch.zeros_like(b))
    m = a.abs()
    code = torch.zeros_like(m, dtype=torch.uint8)
    for i, (edge, up) in enumerate(zip((0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0), (0, 1, 0, 1, 0, 1, 0))):
        code += ((m >= edge) if up else (m > edge)).to(torch.uint8)
    code |= torch.signbit(a).to(torch.uint8) << 3
    return code.reshape(x.shape), sf, gs.float()


def _fp4_round(x, gs):
    """``x`` rounded to NVFP4, in 64 bits."""
    code, sf, gs = _fp4(x, gs if isinstance(gs, torch.Tensor) else torch.tensor(gs, dtype=x.dtype, device=x.device))
    lv = torch.tensor(_LEVELS, dtype=torch.float64, device=x.device)
    v = lv[(code & 7).long()] * (1.0 - 2.0 * (code >> 3).double())
    return (v.reshape(x.shape[0], -1, 16) * (sf.double() * gs.double())[..., None]).reshape(x.shape)


# ---- the program: model, cache, runner -----------------------------------------------------------------------------------------------


def _config(c):
    from tensorrt_edge_llm_b200.config import QUANT_NVFP4, QuantConfig, hybrid_nemotron_config, qwen3_30b_a3b_config, qwen3_8b_config
    s = STACKS[c["model"]]
    kw = dict(num_hidden_layers=s["layers"], vocab_size=64 if c["phase"] == "rows" else s["vocab"], dtype="float16" if _dtype(c) == torch.float16 else "bfloat16")
    if c["model"] == "hybrid":
        return hybrid_nemotron_config(**kw)
    if c["model"] == "moe":
        return qwen3_30b_a3b_config(quant=QuantConfig(quant_type=QUANT_NVFP4, group_size=16, excluded=["*self_attn*", "*mlp.gate", "lm_head"]), **kw)
    return qwen3_8b_config(quant=QuantConfig(quant_type=QUANT_NVFP4, group_size=16) if c["weights"] == "nvfp4" else QuantConfig(), **kw)


def _load(model, src):
    """Fill the model as its checkpoint loader does, from drawn tensors."""
    from tensorrt_edge_llm_b200.models.linear import LinearBase
    kinds = _kinds(src.c["model"])
    stack = {}

    def full(name):
        i = int(name.split(".")[2]) if name.startswith("model.layers.") else -1
        return name.replace(".mixer.", f".{kinds[i]}.") if i >= 0 else name

    def experts(name):
        p, e, leaf, field = name.rsplit(".", 3)
        if (p, leaf) not in stack:
            parts = [src.linear(f"{p}.{j}.{leaf}") for j in range(src.s["experts"])]
            stack[p, leaf] = parts
        return stack[p, leaf][int(e)].get(field)

    def fetch(name):
        name = full(name)
        if ".experts." in name:
            return experts(name)
        if name.endswith("conv1d.weight"):
            return src.conv(name, 6144 if ".gdn" in name or ".mamba" in name else 0)
        if name.endswith(("A_log", "dt_bias")):
            return src.small(name, SSM["heads"] if ".mamba" in name else GDN["heads"])
        return None

    with torch.no_grad():
        for name, mod in model.named_modules():
            if isinstance(mod, LinearBase):
                parent, _, leaf = name.rpartition(".")
                mod.load_from([src.linear(full(f"{parent}.{s}" if parent else s)) for s in (mod.sources or [leaf])])
        for _, mod in model.named_modules():
            if hasattr(mod, "load_checkpoint") and not isinstance(mod, LinearBase):
                mod.load_checkpoint(fetch)
                stack.clear()
        model.model.embed_tokens.weight.copy_(src.raw("model.embed_tokens").to(src.dt))
    model.finalize()


def _fill_cache(c, src, kv, steps):
    layers = sum(k == "attention" for k in _kinds(c["model"]))
    for i, (past, new) in enumerate(steps):
        kv.reserve(i, past + new)
        if past:
            n = -(-past // PAGE)
            buf = torch.zeros(layers, 2, src.s["hkv"], n * PAGE, HD, dtype=src.dt, device="cuda")
            buf[:, :, :, :past] = src.cached(i, layers, src.s["hkv"], past)
            pages = torch.tensor(kv.pages_of(i)[:n], device="cuda")
            kv.pool[:, pages] = buf.view(layers, 2, src.s["hkv"], n, PAGE, HD).permute(0, 3, 1, 2, 4, 5)
            kv.commit(i, past)


def _state_draw(src, kind, i, what, shape):
    """State of one recurrent layer behind a long past."""
    std = {"conv": 1.2, "ssm": 0.3, "gdn": 0.1}[what]
    t = src.normal(f"state.{kind}.{i}.{what}", shape, std)
    return t.to(src.dt) if what == "conv" else t


def _fill_state(c, src, kv):
    if kv.recurrent is None or c["phase"] == "prefill":
        return
    for what in ("conv", "ssm", "gdn"):
        for i, t in getattr(kv.recurrent, what).items():
            t.copy_(_state_draw(src, _kinds(c["model"])[i], i, what, tuple(t.shape)))


def _state_pools(kv):
    r = kv.recurrent
    return [] if r is None else [d[i] for d in (r.conv, r.ssm, r.gdn) for i in sorted(d)]


def _blocks(st):
    """The blocks of every layer on NVFP4 rows, as a decoder layer runs them."""
    from tensorrt_edge_llm_b200 import ops
    out = []
    for layer, x in zip(st["model"].model.layers, st["inputs"]):
        at, mlp, y = layer.self_attn, layer.mlp, {}
        n1, n2 = layer.input_layernorm, layer.post_attention_layernorm
        if st["case"]["model"] == "dense":
            xn, y["r1"] = ops.add_rmsnorm(x["h1"], x["r1"], n1.weight, n1.eps, at.qkv_proj.fused_input_scale())
            y["qkv"], y["o"] = at.qkv_proj(xn), at.o_proj(x["a"])
            xn, y["r2"] = ops.add_rmsnorm(x["h2"], x["r2"], n2.weight, n2.eps, mlp.gate_up_proj.fused_input_scale())
        else:
            xn, y["r2"] = ops.add_rmsnorm(x["h2"], x["r2"], n2.weight, n2.eps)
        y["mlp"] = mlp(xn)
        out.append(y)
    return out


def _capture(fn):
    """One warm run on a side stream, then the same work as a CUDA graph: ``(graph, its outputs)``."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        fn()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        out = fn()
    return graph, out


GRAPH_ROWS = 512            # steps of up to so many rows replay from a graph, as decode and verification steps do


@torch.no_grad()
def prepare(case, seed):
    from tensorrt_edge_llm_b200.model import AutoModel
    from tensorrt_edge_llm_b200.ops import build_step_meta, eagle_tree_meta
    from tensorrt_edge_llm_b200.runtime.kv_cache import KVCacheManager
    from tensorrt_edge_llm_b200.runtime.runner import ModelRunner
    c, src, steps = case, _Source(case, seed), _steps(case)
    cfg = _config(c)
    model = AutoModel.from_config(cfg, device="cuda")
    _load(model, src)
    if c["phase"] == "rows":
        st = dict(case=c, model=model, inputs=[src.block_inputs(i) for i in range(src.s["layers"])])
        if c["new"] <= GRAPH_ROWS:
            st["graph"], st["blocks"] = _capture(lambda: _blocks(st))
        return st
    pages = [-(-(p + n) // PAGE) for p, n in steps]
    kv = KVCacheManager(cfg, num_pages=sum(pages), page_size=PAGE, max_seats=len(steps), max_pages_per_seq=max(pages), device="cuda")
    _fill_cache(c, src, kv, steps)
    runner = ModelRunner(model, kv, device="cuda", max_num_tokens=8192)
    toks, seats = src.tokens(), list(range(len(steps)))
    st = dict(case=c, runner=runner, kv=kv, tokens=toks, seats=seats)
    if c["phase"] in ("decode", "verify"):
        # as the runner's decode graph and the speculative decoder do: the step's state on the device, the model step captured once
        more = {}
        if c["phase"] == "verify":
            base = torch.tensor([p for p, _ in steps], dtype=torch.int32, device="cuda")
            mask, _, pos = eagle_tree_meta(src.parents().to("cuda", torch.int32), base, 0, 0)
            more = dict(tree_mask=mask, positions=pos, logits_all=True)
        meta = build_step_meta([n for _, n in steps], [p for p, _ in steps], kv.table_rows(seats), PAGE, slot_ids=seats, device="cuda", **more)
        meta.host_lens, meta.max_seq_len = None, max(pages) * PAGE
        st["pinned"] = torch.tensor([t for ts in toks for t in ts], dtype=torch.int32).pin_memory()
        st["ids"] = st["pinned"].to("cuda")
        st["graph"], st["logits"] = _capture(lambda: model(st["ids"], meta, runner.cache))
        st["meta"] = meta
    _fill_state(c, src, kv)
    return st


@torch.no_grad()
def run(st):
    if st["case"]["phase"] == "rows":
        if "graph" not in st:
            return _blocks(st)
        st["graph"].replay()
        return st["blocks"]
    if "graph" in st:
        st["ids"].copy_(st["pinned"], non_blocking=True)
        st["graph"].replay()
        out = {"logits": st["logits"]}
    else:
        out = {"logits": st["runner"].step(st["seats"], st["tokens"], commit=False), "kv": st["kv"].pool}
    out["state"] = _state_pools(st["kv"])
    return out


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------------------


def work(case):
    c, s, steps = case, STACKS[case["model"]], _steps(case)
    kinds = _kinds(c["model"])
    t = sum(n for _, n in steps)
    rows = t if c["phase"] == "verify" else len(steps)
    h, q, kvw = s["hidden"], s["hq"] * HD, s["hkv"] * HD
    fp4 = 0.5 + 1.0 / 16
    wb = fp4 if c["weights"] == "nvfp4" and c["model"] == "dense" else 2.0
    nbytes, flops = rows * s["vocab"] * 2 + s["vocab"] * h * 2.0 + t * h * 2, 2.0 * rows * s["vocab"] * h
    blocks = c["phase"] == "rows"
    if blocks:
        nbytes, flops = 0.0, 0.0
    for kind in kinds:
        if blocks:
            nbytes += t * h * 2 * 4                          # rows and residual rows in, residual rows and the block's rows out
            if c["model"] == "dense":
                n = (q + 2 * kvw) * h + h * q
                nbytes += n * wb + t * 2 * (3 * h + q + 2 * kvw + q + h)
                flops += 2.0 * t * n
        elif kind == "attention":
            n = (q + 2 * kvw) * h + h * q
            nbytes += n * wb + sum(p + m for p, m in steps) * 2 * kvw * 2
            flops += 2.0 * t * n + sum(4.0 * q * (m * p + m * (m + 1) / 2) for p, m in steps)
        elif kind == "mamba":
            d, gn = SSM["heads"] * SSM["dim"], SSM["groups"] * SSM["state"]
            n = (2 * d + 2 * gn + SSM["heads"]) * h + h * d
            nbytes += n * 2 + len(steps) * d * SSM["state"] * 4 * (1 if c["phase"] == "prefill" else 2)
            flops += 2.0 * t * n + 6.0 * t * d * SSM["state"]
        else:
            d = GDN["heads"] * GDN["dim"]
            n = (4 * d + 2 * GDN["heads"]) * h + h * d
            nbytes += n * 2 + len(steps) * d * GDN["dim"] * 4 * (1 if c["phase"] == "prefill" else 2)
            flops += 2.0 * t * n + 8.0 * t * d * GDN["dim"]
        if c["model"] == "moe":
            e, k, n = s["experts"], s["top_k"], 3 * s["inter"] * h
            nbytes += e * h * 2 + e * (1 - (1 - k / e) ** t) * n * fp4      # experts that random routing reaches
            flops += 2.0 * t * (e * h + k * n)
        else:
            n = (2 if c["model"] == "hybrid" else 3) * s["inter"] * h
            nbytes += n * wb
            flops += 2.0 * t * n
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """16-bit stacks: the roundings of a step add up to 0.02 against 64 bits, states of the last layers to 0.03.  NVFP4 blocks: sums in
    another order move a 16-bit rounding here and there, and some of those cross an edge of the four-bit rounding behind it."""
    return {"rel": 0.03, "max": 0.99}


# ---- the same steps in 64 bits -------------------------------------------------------------------------------------------------------


def _norm(x, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


class _Exact:
    def __init__(self, c, seed):
        self.c, self.src, self.s, self.steps = c, _Source(c, seed), STACKS[c["model"]], _steps(c)
        self.starts = [0]
        for _, n in self.steps:
            self.starts.append(self.starts[-1] + n)
        self.past = [p for p, _ in self.steps]
        layers = sum(k == "attention" for k in _kinds(c["model"]))
        self.cache = [self.src.cached(i, layers, self.s["hkv"], p).double() if p else None for i, p in enumerate(self.past)]
        self.kv_rows, self.state = [], {}
        if c["phase"] == "verify":
            par = self.src.parents()
            b, r = par.shape
            self.mask = torch.zeros(b, r, r, dtype=torch.bool, device="cuda")
            depth = torch.zeros(b, r, dtype=torch.int64)
            for i in range(b):
                for j in range(r):
                    k = j
                    while k >= 0:
                        self.mask[i, j, k] = True
                        k = int(par[i, k])
                        depth[i, j] += k >= 0
            self.pos = torch.cat([p + depth[i] for i, p in enumerate(self.past)]).cuda()
        else:
            self.mask = None
            self.pos = torch.cat([torch.arange(p, p + n) for p, n in self.steps]).cuda()

    def lin(self, x, name, quant=None):
        if self.src.is_fp4(name):
            x = _fp4_round(x, INPUT_SCALE) if quant is None else quant
        return x @ self.src.dense64(name).t()

    def rope(self, x):
        f = self.s["theta"] ** (-torch.arange(0, HD, 2, dtype=torch.float64, device="cuda") / HD)
        a = self.pos.double()[:, None, None] * f
        x1, x2 = x[..., :HD // 2], x[..., HD // 2:]
        return torch.cat([x1 * a.cos() - x2 * a.sin(), x2 * a.cos() + x1 * a.sin()], -1)

    def attention(self, x, p, layer):
        s, t = self.s, x.shape[0]
        q, k, v = (self.lin(x, f"{p}.{n}_proj").view(t, -1, HD) for n in "qkv")
        if s["qk_norm"]:
            q, k = _norm(q, s["eps"]), _norm(k, s["eps"])
        q, k = self.rope(q), self.rope(k)
        self.kv_rows.append((k, v))
        out, g = torch.empty_like(q), s["hq"] // s["hkv"]
        for i, (past, n) in enumerate(self.steps):
            a, b = self.starts[i], self.starts[i + 1]
            for hk in range(s["hkv"]):
                kk, vv = k[a:b, hk], v[a:b, hk]
                if past:
                    kk, vv = (torch.cat([self.cache[i][layer, w, hk], z]) for w, z in ((0, kk), (1, vv)))
                for r0 in range(0, n, 2048):
                    r1 = min(n, r0 + 2048)
                    end = past + (n if self.mask is not None else r1)
                    sc = torch.einsum("qhd,kd->hqk", q[a + r0:a + r1, hk * g:(hk + 1) * g], kk[:end]) * HD ** -0.5
                    if self.mask is not None:
                        sc[:, :, past:].masked_fill_(~self.mask[i][None], float("-inf"))
                    elif n > 1:
                        seen = torch.arange(end, device="cuda")[None] <= past + torch.arange(r0, r1, device="cuda")[:, None]
                        sc.masked_fill_(~seen[None], float("-inf"))
                    out[a + r0:a + r1, hk * g:(hk + 1) * g] = torch.einsum("hqk,kd->qhd", torch.softmax(sc, -1), vv[:end])
        return self.lin(out.reshape(t, -1), f"{p}.o_proj")

    def conv(self, x, p, kind, i):
        """Short causal convolution and silu; keeps the last inputs as state."""
        w, ch = self.src.conv(f"{p}.conv1d.weight", x.shape[1]).double(), x.shape[1]
        hist = _state_draw(self.src, kind, i, "conv", (len(self.steps), ch, 3)).double() if self.past[0] else torch.zeros(len(self.steps), ch, 3, dtype=x.dtype, device="cuda")
        out, last = torch.empty_like(x), torch.empty_like(hist)
        for j in range(len(self.steps)):
            a, b = self.starts[j], self.starts[j + 1]
            seq = torch.cat([hist[j], x[a:b].t()], 1)
            out[a:b] = sum(w[:, d:d + 1] * seq[:, d:d + b - a] for d in range(4)).t()
            last[j] = seq[:, -3:]
        self.state["conv", i] = last
        return _silu(out)

    def by_time(self, n):
        """Row of every sequence at time ``n`` (sequences that have ended repeat their last row) and which are alive."""
        lens = torch.tensor([m for _, m in self.steps], device="cuda")
        return torch.tensor(self.starts[:-1], device="cuda") + torch.clamp(lens - 1, max=n), n < lens

    def mamba(self, x, p, i):
        m, t, nseq = SSM, x.shape[0], len(self.steps)
        d, gn = m["heads"] * m["dim"], m["groups"] * m["state"]
        z, xbc, dt = self.lin(x, f"{p}.in_proj").split([d, d + 2 * gn, m["heads"]], -1)
        xs, bm, cm = self.conv(xbc, p, "mamba", i).split([d, gn, gn], -1)
        dt = torch.nn.functional.softplus(dt + self.src.small(f"{p}.dt_bias", m["heads"]).double()).clamp(max=m["limit"])
        decay = torch.exp(-torch.exp(self.src.small(f"{p}.A_log", m["heads"]).double()) * dt)
        xs, rep = xs.reshape(t, m["heads"], m["dim"]), m["heads"] // m["groups"]
        bm, cm = (v.reshape(t, m["groups"], m["state"]).repeat_interleave(rep, 1) for v in (bm, cm))
        shape = (nseq, m["heads"], m["dim"], m["state"])
        hst = _state_draw(self.src, "mamba", i, "ssm", shape).double() if self.past[0] else torch.zeros(shape, dtype=x.dtype, device="cuda")
        y, dx = torch.empty_like(xs), dt[..., None] * xs
        for n in range(max(m for _, m in self.steps)):
            r, alive = self.by_time(n)
            new = hst * decay[r][..., None, None] + dx[r][..., None] * bm[r][:, :, None]
            hst = torch.where(alive[:, None, None, None], new, hst)
            y[r] = torch.einsum("bhdn,bhn->bhd", hst, cm[r])
        self.state["ssm", i] = hst
        y = (y + xs).reshape(t, d) * _silu(z)
        y = _norm(y.reshape(t, m["groups"], -1), self.s["eps"]).reshape(t, d)
        return self.lin(y, f"{p}.out_proj")

    def gdn(self, x, p, i):
        t, h, d, nseq = x.shape[0], GDN["heads"], GDN["dim"], len(self.steps)
        qkv = self.conv(self.lin(x, f"{p}.in_proj_qkv"), p, "gdn", i)
        q, k, v = (z.reshape(t, h, d) for z in qkv.split(h * d, -1))
        q, k = (z * torch.rsqrt(z.pow(2).sum(-1, keepdim=True) + 1e-6) for z in (q, k))
        q = q * d ** -0.5
        a = self.lin(x, f"{p}.in_proj_a") + self.src.small(f"{p}.dt_bias", h).double()
        decay = torch.exp(-torch.exp(self.src.small(f"{p}.A_log", h).double()) * torch.nn.functional.softplus(a))
        beta = torch.sigmoid(self.lin(x, f"{p}.in_proj_b"))
        shape = (nseq, h, d, d)
        hst = _state_draw(self.src, "gdn", i, "gdn", shape).double() if self.past[0] else torch.zeros(shape, dtype=x.dtype, device="cuda")
        o = torch.empty_like(v)
        for n in range(max(m for _, m in self.steps)):
            r, alive = self.by_time(n)
            new = hst * decay[r][..., None, None]
            delta = beta[r][..., None] * (v[r] - torch.einsum("bhkv,bhk->bhv", new, k[r]))
            new = new + k[r][..., None] * delta[:, :, None]
            hst = torch.where(alive[:, None, None, None], new, hst)
            o[r] = torch.einsum("bhkv,bhk->bhv", hst, q[r])
        self.state["gdn", i] = hst
        return self.lin(_norm(o, self.s["eps"]).reshape(t, h * d) * _silu(self.lin(x, f"{p}.in_proj_z")), f"{p}.out_proj")

    def mlp(self, x, p):
        if self.c["model"] == "hybrid":
            return self.lin(torch.relu(self.lin(x, f"{p}.up_proj")).pow(2), f"{p}.down_proj")
        if self.c["model"] == "dense":
            quant = _fp4_round(x, INPUT_SCALE) if self.src.is_fp4(f"{p}.up_proj") else None
            return self.lin(_silu(self.lin(x, f"{p}.gate_proj", quant)) * self.lin(x, f"{p}.up_proj", quant), f"{p}.down_proj")
        # the experts are chosen by logits of the activations' type: two that it does not tell apart are not told apart in 64 bits either
        logits = self.lin(x.to(self.src.dt).double(), f"{p}.gate").to(self.src.dt).double()
        probs = torch.softmax(logits, -1)
        w, idx = probs.topk(self.s["top_k"], -1)
        w = w / w.sum(-1, keepdim=True)
        xq, out = _fp4_round(x, INPUT_SCALE), torch.zeros_like(x)
        for e in range(self.s["experts"]):
            rows, slot = (idx == e).nonzero(as_tuple=True)
            if rows.numel():
                a = xq[rows]
                g, u = (self.lin(a, f"{p}.experts.{e}.{n}_proj", a) for n in ("gate", "up"))
                out.index_add_(0, rows, self.lin(_silu(g) * u, f"{p}.experts.{e}.down_proj") * w[rows, slot][:, None])
        return out

    def blocks(self, i):
        p, x, y = f"model.layers.{i}.", {k: v.double() for k, v in self.src.block_inputs(i).items()}, {}
        if self.c["model"] == "dense":
            y["r1"] = x["h1"] + x["r1"]
            xn = _fp4_round(_norm(y["r1"], self.s["eps"]), INPUT_SCALE)
            y["qkv"] = torch.cat([self.lin(xn, f"{p}self_attn.{n}_proj", xn) for n in "qkv"], 1)
            y["o"] = self.lin(x["a"], f"{p}self_attn.o_proj")
        y["r2"] = x["h2"] + x["r2"]
        y["mlp"] = self.mlp(_norm(y["r2"], self.s["eps"]), f"{p}mlp")
        return y

    def __call__(self):
        s, c = self.s, self.c
        if c["phase"] == "rows":
            return [self.blocks(i) for i in range(s["layers"])]
        ids = torch.tensor([t for ts in self.src.tokens() for t in ts], device="cuda")
        x = self.src.raw("model.embed_tokens").to(self.src.dt).double()[ids]
        layer = 0
        for i, kind in enumerate(_kinds(c["model"])):
            name = f"model.layers.{i}." + (kind if c["model"] == "hybrid" else "self_attn")
            xn = _norm(x, s["eps"])
            if kind == "attention":
                x, layer = x + self.attention(xn, name, layer), layer + 1
            else:
                x = x + getattr(self, kind)(xn, name, i)
            x = x + self.mlp(_norm(x, s["eps"]), f"model.layers.{i}.mlp")
        if c["phase"] != "verify":
            x = x[torch.tensor(self.starts[1:], device="cuda") - 1]
        out = {"logits": _norm(x, s["eps"]) @ self.src.dense64("lm_head").t()}
        if c["phase"] in ("prefill", "mixed"):
            out["kv"] = self.pool()
        out["state"] = [self.state[w, i] for w, i in sorted(self.state, key=lambda z: (("conv", "ssm", "gdn").index(z[0]), z[1]))]
        return out

    def pool(self):
        """The cache in its pages, handed out in order: ``[layers, pages, 2, kv heads, 64, head]``."""
        layers = []
        for li, (k, v) in enumerate(self.kv_rows):
            pages = []
            for i, (past, n) in enumerate(self.steps):
                new = torch.stack([k[self.starts[i]:self.starts[i + 1]], v[self.starts[i]:self.starts[i + 1]]]).transpose(1, 2)   # [2, kv heads, n, head]
                rows = torch.cat([self.cache[i][li], new], 2) if past else new
                m = -(-(past + n) // PAGE)
                rows = torch.nn.functional.pad(rows, (0, 0, 0, m * PAGE - past - n))
                pages.append(rows.reshape(2, self.s["hkv"], m, PAGE, HD).permute(2, 0, 1, 3, 4))
            layers.append(torch.cat(pages))
        return torch.stack(layers)


@torch.no_grad()
def exact(case, seed):
    return _Exact(case, seed)()

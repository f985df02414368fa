"""Kernels of prompt and decode steps at the sizes where a tile, a ring or a split ends: against the plain statements of the same ops, or
bit for bit against another kernel of the same products in the same order."""
import pytest
import torch

from tensorrt_edge_llm_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cu():
    from tensorrt_edge_llm_b200.ops import cuda
    cuda.lib()
    return cuda


def _check_status(cu):
    torch.cuda.synchronize()
    cu.Workspace.get(torch.device("cuda", 0)).check_status()


def _nvfp4_operands(cu, m, n, k, dtype):
    g = torch.Generator(device="cuda").manual_seed(m * 7 + n * 3 + k)
    x = torch.randn(m, k, device="cuda", generator=g).to(dtype)
    wq, wsf, wgs = ref.nvfp4_quantize(torch.randn(n, k, device="cuda", generator=g) * 0.05)
    gs = torch.full((1,), 1.0 / 448, device="cuda")
    xq, xsf = cu.nvfp4_quantize(x, gs)
    alpha = wgs * gs * (0.5 + torch.rand(n, device="cuda", generator=g))
    extra = dict(bias=torch.randn(n, device="cuda", generator=g).to(dtype), residual=torch.randn(m, n, device="cuda", generator=g).to(dtype))
    return xq, xsf, wq, cu.nvfp4_swizzle_scales(wsf), alpha.contiguous(), extra


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,n,k", [(129, 256, 32), (200, 264, 288), (257, 520, 1056), (385, 3000, 768), (1920, 4096, 1024), (19000, 272, 512)])
def test_gemm_nvfp4_tile_equals_the_128_wide_kernel(cu, m, n, k, dtype):
    """128 x 256 tiles: ragged rows, columns and K steps, row pitches that no 32-byte store fits, more tiles than CTAs; with and without
    bias and residual.  Both kernels add the same products in the same order."""
    xq, xsf, wq, w_sf, alpha, extra = _nvfp4_operands(cu, m, n, k, dtype)
    L = cu.lib()
    old = L.telb_set_nvfp4_wide_mode(0)
    try:
        outs = []
        for mode in (0, 1):
            L.telb_set_nvfp4_wide_mode(mode)
            outs.append([cu.gemm_nvfp4(xq, xsf, wq, w_sf, alpha, dtype, mode=1), cu.gemm_nvfp4(xq, xsf, wq, w_sf, alpha, dtype, mode=1, **extra)])
    finally:
        L.telb_set_nvfp4_wide_mode(old)
    _check_status(cu)
    for a, b in zip(*outs):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,inter,k", [(130, 128, 256), (300, 192, 320), (700, 1088, 512)])
def test_gemm_nvfp4_tile_swiglu_equals_the_128_wide_kernel(cu, m, inter, k, dtype):
    """SwiGLU and quantisation in the epilogue, with a half tile at the end of the columns."""
    xq, xsf, wq, w_sf, alpha, _ = _nvfp4_operands(cu, m, 2 * inter, k, dtype)
    acts = cu.QuantActs(xq, xsf, (m, k), dtype)
    gs = torch.full((1,), 0.004, device="cuda")
    L = cu.lib()
    old = L.telb_set_nvfp4_wide_mode(0)
    try:
        outs = []
        for mode in (0, 1):
            L.telb_set_nvfp4_wide_mode(mode)
            outs.append(cu.gemm_nvfp4_swiglu(acts, wq, w_sf, alpha, gs))
    finally:
        L.telb_set_nvfp4_wide_mode(old)
    _check_status(cu)
    assert torch.equal(outs[0].xq, outs[1].xq)
    eye = torch.eye(inter, device="cuda", dtype=dtype)[:min(inter, 256)]
    wi, wi_sf, wi_gs = ref.nvfp4_quantize(eye)
    one = torch.full((eye.shape[0],), 1.0, device="cuda") * wi_gs
    rows = [cu.gemm_nvfp4(o.xq, o.sf, wi, cu.nvfp4_swizzle_scales(wi_sf), one, dtype) for o in outs]      # the scales, read as a GEMM reads them
    assert torch.equal(rows[0], rows[1])


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,n,k,world", [(130, 256, 64, 2), (300, 544, 288, 2), (1000, 1056, 512, 4), (385, 288, 1056, 3)])
def test_gemm_nvfp4_tile_scatters_rows_to_their_ranks(cu, m, n, k, world, dtype):
    """The reduce-scatter form: every row leaves for its owner's buffer with the bits of the plain product, and nothing else is written.  The
    ranks' buffers all lie on this GPU, and nothing waits."""
    xq, xsf, wq, w_sf, alpha, extra = _nvfp4_operands(cu, m, n, k, dtype)
    rpr, rank = -(-m // world), world - 1
    parts = [torch.full((world * rpr, n), float("nan"), device="cuda", dtype=dtype) for _ in range(world)]
    f = cu.GemmFusion()
    for d in range(world):
        f.rs_out[d] = parts[d].data_ptr()
    f.rs_world, f.rs_rank, f.rs_rows_per_rank = world, rank, rpr
    cu.gemm_fused(cu.QuantActs(xq, xsf, (m, k), dtype), wq, f, w_sf=w_sf, alpha=alpha, bias=extra["bias"])
    want = cu.gemm_nvfp4(xq, xsf, wq, w_sf, alpha, dtype, bias=extra["bias"], mode=1)
    _check_status(cu)
    for d in range(world):
        rows = want[d * rpr:(d + 1) * rpr]
        assert torch.equal(parts[d][rank * rpr:rank * rpr + rows.shape[0]], rows)
        parts[d][rank * rpr:rank * rpr + rows.shape[0]] = float("nan")
        assert parts[d].isnan().all()


@pytest.mark.parametrize("tokens,inter", [(600, 256), (1500, 192), (9, 256)])
def test_grouped_swiglu_tiles_equal_the_separate_pass(cu, tokens, inter, monkeypatch):
    """SwiGLU and quantisation in the epilogue of the 128 x 256 expert tiles, half a tile of columns at an expert's end, against the product
    and its pass, and against the 128-wide kernel."""
    from tensorrt_edge_llm_b200.config import QuantConfig, qwen3_30b_a3b_config
    from tensorrt_edge_llm_b200.models.qwen3_moe import MoEBlock
    cfg = qwen3_30b_a3b_config(num_hidden_layers=1, hidden_size=512, moe_intermediate_size=inter, num_experts=72, num_experts_per_tok=4)
    cfg.quant = QuantConfig(quant_type="nvfp4")
    g = torch.Generator(device="cuda").manual_seed(tokens)
    x = torch.randn(tokens, 512, device="cuda", generator=g).bfloat16()
    L, outs = cu.lib(), []
    old = L.telb_set_nvfp4_wide_mode(0)
    try:
        for fused in ("1", "0"):
            monkeypatch.setenv("TELB_MOE_SWIGLU_FUSION", fused)
            blk = MoEBlock(cfg, "model.layers.0.mlp").cuda()
            blk.random_init(torch.Generator().manual_seed(3), std=0.05)
            blk.finalize()
            assert blk._w13_interleaved == (fused == "1")
            blk.input_scale.fill_(float(x.abs().max()) / (6.0 * 448.0))
            blk.down_input_scale.fill_(0.5 / (6.0 * 448.0))
            blk._refresh_alpha()
            for mode in (0, 1):
                L.telb_set_nvfp4_wide_mode(mode)
                outs.append(blk(x))
    finally:
        L.telb_set_nvfp4_wide_mode(old)
    _check_status(cu)
    assert outs[0].abs().max() > 0 and all(torch.equal(outs[0], o) for o in outs[1:])


def _step_meta(q_lens, pasts):
    from tensorrt_edge_llm_b200.ops import build_step_meta
    return build_step_meta(q_lens, pasts, torch.zeros(len(q_lens), 1, dtype=torch.int32), 64, slot_ids=list(range(len(q_lens)))[::-1]).to("cuda")


@pytest.mark.parametrize("width", [2, 3, 4])
@pytest.mark.parametrize("channels,ld", [(24, 40), (1040, 1040), (136, 137), (33, 33)])
@pytest.mark.parametrize("q_lens,pasts", [([1, 1, 1], [5, 0, 9]), ([2, 0, 17, 1, 33], [0, 3, 4, 1, 0]), ([4100], [7])])
def test_causal_conv1d_of_rows_in_wider_rows(cu, q_lens, pasts, channels, ld, width):
    """Every rows-per-thread split, sequences that end inside a thread's rows, a pitch that no 16-byte load fits, odd channels."""
    g = torch.Generator(device="cuda").manual_seed(channels + width)
    t = sum(q_lens)
    x = torch.randn(t, ld, device="cuda", generator=g).bfloat16()[:, ld - channels:]
    w, b = (torch.randn(*s, device="cuda", generator=g).bfloat16() for s in ((channels, width), (channels,)))
    st = torch.randn(len(q_lens), channels, width - 1, device="cuda", generator=g).bfloat16()
    st_ref, meta = st.clone(), _step_meta(q_lens, pasts)
    y, yr = cu.causal_conv1d(x, w, b, st, meta, True), ref.causal_conv1d(x, w, b, st_ref, meta, True)
    _check_status(cu)
    # one 16-bit rounding each side, fp32 sums of at most 5 terms
    assert (y.float() - yr.float()).abs().max() <= 2 ** -7 * yr.float().abs().max() and torch.equal(st, st_ref)


@pytest.mark.parametrize("hidden,groups", [(512, 2), (1024, 2), (768, 1), (1024, 1), (96, 3)])
@pytest.mark.parametrize("rows", [1, 9])
def test_gated_norms_of_rows_in_wider_rows(cu, rows, hidden, groups):
    g = torch.Generator(device="cuda").manual_seed(hidden + rows)
    x, z, w = (torch.randn(*s, device="cuda", generator=g).bfloat16() for s in ((rows, hidden), (rows, hidden + 24), (hidden,)))
    z = z[:, 8:8 + hidden]
    y, yr = cu.gated_group_rmsnorm(x, z, w, groups, 1e-5), ref.gated_group_rmsnorm(x, z, w, groups, 1e-5)
    assert (y.float() - yr.float()).norm() < 2 ** -7 * yr.float().norm()        # two 16-bit roundings
    for dim in (64, 128, 256, 32):
        if hidden % dim == 0:
            h = x.view(rows, hidden // dim, dim)
            y, yr = cu.rmsnorm_gate(h, z, w[:dim], 1e-5), ref.rmsnorm_gate(h, z, w[:dim], 1e-5)
            assert (y.float() - yr.float()).norm() < 2 ** -7 * yr.float().norm()
    _check_status(cu)


@pytest.mark.parametrize("offset", [1, 3, 8])
@pytest.mark.parametrize("rows,dim", [(1, 64), (1, 128), (5, 128), (1, 256)])
def test_gated_head_norm_of_rows_that_start_anywhere(cu, rows, dim, offset):
    """A row cut out of a wider one is contiguous for torch wherever it starts; gates of another type take the generic form."""
    g = torch.Generator(device="cuda").manual_seed(dim + offset)
    r = torch.randn(3, rows * 2 * dim + 16, device="cuda", generator=g).bfloat16()
    x, w = r[0, offset:offset + rows * 2 * dim].view(rows, 2, dim), r[1, offset:offset + dim]
    z = torch.randn(rows, 2 * dim + 24, device="cuda", generator=g).bfloat16()[:, offset:offset + 2 * dim]
    for gate in (z, z.float()):
        y, yr = cu.rmsnorm_gate(x, gate, w, 1e-5), ref.rmsnorm_gate(x, gate, w, 1e-5)
        assert (y.float() - yr.float()).norm() < 2 ** -7 * yr.float().norm()        # two 16-bit roundings
    _check_status(cu)


@pytest.mark.parametrize("q_lens,pasts", [([1, 1, 1], [5, 0, 9]), ([3, 1], [0, 4]), ([37, 130], [0, 64]), ([300], [2])])
def test_recurrences_read_parts_of_wider_rows(cu, q_lens, pasts):
    """x, B, C (q, k, v) and the step sizes as views into one projection's rows give the bits of packed copies."""
    g = torch.Generator(device="cuda").manual_seed(sum(q_lens))
    t, meta = sum(q_lens), _step_meta(q_lens, pasts)
    r = torch.randn(t, 4 * 64 + 2 * 256 + 16, device="cuda", generator=g).bfloat16()
    xs, B, C = r[:, :256].reshape(t, 4, 64), r[:, 256:512].reshape(t, 2, 128), r[:, 512:768].reshape(t, 2, 128)
    dt, A = r[:, 768:772], torch.rand(4, device="cuda", generator=g)
    st = torch.randn(len(q_lens), 4, 64, 128, device="cuda", generator=g)
    D, db = torch.ones(4, device="cuda"), torch.zeros(4, device="cuda")
    st2 = st.clone()
    y = cu.ssm_scan(xs, dt, A, B, C, D, db, st, meta, a_log=True)
    y2 = cu.ssm_scan(xs.contiguous(), dt.contiguous(), -torch.exp(A.double()).float(), B.contiguous(), C.contiguous(), D, db, st2, meta)
    assert torch.equal(y, y2) and torch.equal(st, st2)
    r = torch.randn(t, 6 * 128, device="cuda", generator=g).bfloat16()
    q, k, v = (r[:, i * 256:(i + 1) * 256].reshape(t, 2, 128) for i in range(3))
    a, b = torch.randn(2, t, 2, device="cuda", generator=g).bfloat16()
    st = torch.randn(len(q_lens), 2, 128, 128, device="cuda", generator=g) * 0.1
    st2 = st.clone()
    y = cu.gated_delta_rule(q, k, v, a, b, A[:2], db[:2], st, meta)
    y2 = cu.gated_delta_rule(q.contiguous(), k.contiguous(), v.contiguous(), a, b, A[:2], db[:2], st2, meta)
    assert torch.equal(y, y2) and torch.equal(st, st2)
    _check_status(cu)


def _paged_step(q_lens, past_lens, hq, hkv, page, dtype, rows_masked=False):
    from tensorrt_edge_llm_b200.ops import build_step_meta
    g = torch.Generator(device="cuda").manual_seed(sum(q_lens) + hq)
    n, most = len(q_lens), max((q + p + page - 1) // page for q, p in zip(q_lens, past_lens)) + 1
    perm = torch.randperm(n * most + 3, generator=torch.Generator().manual_seed(hq))
    table = torch.full((n, most), -1, dtype=torch.int32)
    for i in range(n):
        need = (q_lens[i] + past_lens[i] + page - 1) // page
        table[i, :need] = perm[i * most:i * most + need].to(torch.int32)
    kv = torch.randn(n * most + 3, 2, hkv, page, 128, device="cuda", generator=g).to(dtype)
    q = torch.randn(sum(q_lens), hq, 128, device="cuda", generator=g).to(dtype)
    more = {}
    if rows_masked:
        words = (max(q_lens) + 31) // 32
        bits = torch.randint(-2 ** 31, 2 ** 31, (sum(q_lens), words), generator=torch.Generator().manual_seed(1))
        r = 0
        for ql in q_lens:
            for i in range(ql):
                bits[r, i // 32] |= (1 << (i % 32)) if i % 32 < 31 else -(1 << 31)       # every row sees itself
                r += 1
        more = dict(tree_mask=bits.to(torch.int32).cuda(), positions=torch.zeros(sum(q_lens), dtype=torch.int32), logits_all=True)
    return q, kv, build_step_meta(q_lens, past_lens, table, page, device="cuda", **more)


@pytest.mark.parametrize("q_lens,past_lens,hq,hkv,page,dtype", [
    ([63, 64, 65], [0, 1, 127], 32, 8, 64, torch.bfloat16), ([1, 0, 129, 1], [300, 5, 64, 0], 8, 2, 64, torch.float16),
    ([1] * 40 + [200], [70] * 40 + [3], 4, 1, 128, torch.bfloat16), ([257], [1000], 4, 4, 64, torch.bfloat16),
    ([5, 40], [600, 2049], 16, 1, 128, torch.float16), ([3], [200], 128, 1, 64, torch.bfloat16)])
def test_two_tile_attention(cu, q_lens, past_lens, hq, hkv, page, dtype):
    """Blocks that end inside a tile, one-row sequences beside longer ones, key tiles across pages and past the end; causal, windowed,
    unmasked; one split, several, and splits without a key."""
    q, kv, meta = _paged_step(q_lens, past_lens, hq, hkv, page, dtype)
    for kw in (dict(), dict(sliding_window=100), dict(causal=False)):
        want = ref.paged_attention(q, kv, meta, 128 ** -0.5, **kw)
        for splits in (1, 3, 7):
            got = cu.paged_attention(q, kv, meta, 128 ** -0.5, splits=splits, **kw)
            # probabilities and outputs rounded to 16 bits (2^-8 each) over sums of weights of one sign
            assert (got.float() - want.float()).norm() < 8e-3 * want.float().norm(), (kw, splits)
    _check_status(cu)


@pytest.mark.parametrize("q_lens,past_lens", [([60, 60], [2048, 100]), ([16], [0]), ([33, 7, 64, 90], [63, 640, 65, 31])])
def test_two_tile_attention_of_tree_rows(cu, q_lens, past_lens):
    q, kv, meta = _paged_step(q_lens, past_lens, 32, 8, 64, torch.bfloat16, rows_masked=True)
    want = ref.paged_attention(q, kv, meta, 128 ** -0.5)
    for splits in (None, 1, 4):
        got = cu.paged_attention(q, kv, meta, 128 ** -0.5, splits=splits)
        assert (got.float() - want.float()).norm() < 8e-3 * want.float().norm(), splits
    _check_status(cu)


@pytest.mark.parametrize("page", [64, 128])
@pytest.mark.parametrize("q_lens,past_lens", [([60, 60], [2048, 100]), ([33, 7, 64, 90], [63, 640, 65, 301]), ([1, 200], [700, 0])])
def test_two_tile_attention_of_tree_rows_in_a_window(cu, q_lens, past_lens, page):
    """A row sees the keys that its bits and the window both allow: windows shorter than the tree, of several tiles, and longer than the rest."""
    q, kv, meta = _paged_step(q_lens, past_lens, 32, 8, page, torch.bfloat16, rows_masked=True)
    for window in (20, 40, 100, 200, 5000):
        want = ref.paged_attention(q, kv, meta, 128 ** -0.5, sliding_window=window)
        for kw in (dict(), dict(splits=1), dict(splits=4), dict(kernel="tile")):
            got = cu.paged_attention(q, kv, meta, 128 ** -0.5, sliding_window=window, **kw)
            assert (got.float() - want.float()).norm() < 8e-3 * want.float().norm(), (window, kw)
    _check_status(cu)


@pytest.mark.parametrize("q_lens,past_lens", [([256], [700]), ([40, 300], [1000, 707]), ([90], [164])])
def test_two_tile_attention_reads_no_page_that_a_window_retired(cu, q_lens, past_lens):
    """Table entries before the window are -1; page 0, which another sequence may own, holds NaN and must not reach any row."""
    q, kv, meta = _paged_step(q_lens, past_lens, 32, 8, 64, torch.bfloat16)
    kv = torch.cat([torch.full_like(kv[:1], float("nan")), kv])
    meta.page_table = torch.where(meta.page_table >= 0, meta.page_table + 1, meta.page_table)
    want = ref.paged_attention(q, kv, meta, 128 ** -0.5, sliding_window=100)
    for i, past in enumerate(past_lens):
        meta.page_table[i, :(past - 100 + 1) // 64] = -1
    for splits in (None, 1, 3):
        got = cu.paged_attention(q, kv, meta, 128 ** -0.5, sliding_window=100, splits=splits)
        assert (got.float() - want.float()).norm() < 8e-3 * want.float().norm(), splits
    _check_status(cu)


@pytest.mark.parametrize("q_lens,past_lens,hq,hkv,one_tile", [
    ([256], [0], 32, 8, True), ([257], [0], 32, 8, False), ([33] * 20, [223] * 20, 32, 8, True), ([33] * 20, [224] * 20, 32, 8, False),
    ([32] * 20, [736] * 20, 32, 8, True), ([32] * 20, [737] * 20, 32, 8, False), ([60], [2000], 8, 1, True), ([96], [3000], 32, 8, False), ([64], [4000], 8, 1, True), ([31], [0], 32, 8, True),
    ([96], [900], 32, 8, True), ([97], [900], 32, 8, False), ([100], [0], 16, 16, False), ([1] * 20 + [200], [50] * 21, 32, 8, False),
    ([1024], [0], 16, 16, False)])
def test_prompt_attention_on_both_sides_of_the_route(cu, q_lens, past_lens, hq, hkv, one_tile):
    q, kv, meta = _paged_step(q_lens, past_lens, hq, hkv, 64, torch.bfloat16)
    want = ref.paged_attention(q, kv, meta, 128 ** -0.5)
    got, tile = cu.paged_attention(q, kv, meta, 128 ** -0.5), cu.paged_attention(q, kv, meta, 128 ** -0.5, kernel="tile")
    assert (got.float() - want.float()).norm() < 8e-3 * want.float().norm()
    assert torch.equal(got, tile) == one_tile
    _check_status(cu)


@pytest.mark.parametrize("q_lens,past_lens,hq,hkv", [([300, 90], [1000, 290], 32, 8), ([200], [333], 16, 16), ([40, 130], [120, 7], 8, 1)])
def test_two_tile_attention_of_infinite_and_missing_scores(cu, q_lens, past_lens, hq, hkv):
    """Scores of minus infinity weigh nothing, NaN and plus infinity spread to the rows that see them and to no other; under a window of 40
    keys most rows find their block's first key tile masked, and most of 7 splits hold no key of theirs or none at all."""
    q, kv, meta = _paged_step(q_lens, past_lens, hq, hkv, 64, torch.bfloat16)
    q[:, :, 0] = q[:, :, 0].abs() + 1.0
    for s, (ql, past) in enumerate(zip(q_lens, past_lens)):
        for at, value in ((past // 2, -3e38), (past + ql // 3, float("nan")), (past + 2 * ql // 3, 3e38)):
            kv[int(meta.page_table[s, at // 64]), 0, :, at % 64, 0] = value
    q[:, :, 0] *= 4.0
    for kw in (dict(), dict(sliding_window=40)):
        want = ref.paged_attention(q, kv, meta, 128 ** -0.5, **kw)
        for splits in (1, 3, 7):
            got = cu.paged_attention(q, kv, meta, 128 ** -0.5, splits=splits, **kw)
            assert torch.equal(got.isnan(), want.isnan()), (kw, splits)
            ok = ~want.isnan()
            assert ok.any() and (got[ok].float() - want[ok].float()).norm() < 8e-3 * want[ok].float().norm(), (kw, splits)
    _check_status(cu)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,n,k", [(129, 264, 8), (256, 512, 64), (257, 1040, 136), (700, 3000, 200), (5000, 2064, 520)])
def test_pair_gemm_equals_the_single_cta_kernel(cu, m, n, k, dtype):
    """256 x 256 tiles: ragged rows, columns and K steps, more tiles than pairs; bias, scale and residual; SwiGLU and squared ReLU in the
    epilogue.  Both kernels add the same products in the same order."""
    from tensorrt_edge_llm_b200.ops.cuda import _check, _p, _stream, c_int
    g = torch.Generator(device="cuda").manual_seed(m + n)
    x, w = torch.randn(m, k, device="cuda", generator=g).to(dtype), torch.randn(n, k, device="cuda", generator=g).to(dtype)
    bias, res = torch.randn(n, device="cuda", generator=g).to(dtype), torch.randn(m, n, device="cuda", generator=g).to(dtype)
    alpha = torch.rand(n, device="cuda", generator=g)

    def pair(cols, epi, b=None, a=None, r=None):
        out = torch.full((m, cols), float("nan"), device="cuda", dtype=dtype)
        _check(cu.lib().telb_gemm_pair(_p(x), _p(w), _p(out), c_int(m), c_int(cols), c_int(k), _p(b), _p(a), _p(r), c_int(epi),
                                       c_int(int(dtype == torch.bfloat16)), _p(cu.Workspace.get(x.device).status), _stream()), "gemm_pair")
        return out

    plain = cu.gemm(x, w, mode=1)
    assert torch.equal(pair(n, 0), plain)
    assert torch.equal(pair(n, 0, bias, alpha, res), cu.gemm(x, w, bias, alpha, res, mode=1))
    assert torch.equal(pair(n // 2, 1), cu.swiglu(plain)) if n % 16 == 0 else True
    assert torch.equal(pair(n, 2), cu.relu2(plain))
    for act in ("swiglu", "relu2"):
        if act == "relu2" or n % 16 == 0:
            assert torch.equal(cu.gemm_act(x, w, act), getattr(cu, act)(plain))
    _check_status(cu)


@pytest.mark.parametrize("tokens,experts,top_k,hidden,inter", [(1, 8, 2, 256, 128), (40, 16, 4, 544, 384), (33, 128, 8, 2048, 256), (700, 4, 2, 1056, 640), (300, 3, 1, 288, 192)])
def test_grouped_gemm_tiles_equal_the_128_wide_kernel(cu, tokens, experts, top_k, hidden, inter):
    """128 x 256 tiles over experts: few rows, full tiles and tails, unused tiles, half a tile of columns at an expert's end."""
    g = torch.Generator(device="cuda").manual_seed(tokens + experts)
    x = torch.randn(tokens, hidden, device="cuda", generator=g).half()
    idx = torch.rand(tokens, experts, device="cuda", generator=g).topk(top_k, 1).indices.int()
    n = 2 * inter
    wq, sf, _ = ref.nvfp4_quantize(torch.randn(experts * n, hidden, device="cuda", generator=g) * 0.05)
    w_sf, alpha = cu.nvfp4_swizzle_scales(sf), torch.rand(experts * n, device="cuda", generator=g) * 1e-3
    L, outs = cu.lib(), []
    old = L.telb_set_nvfp4_wide_mode(0)
    lo, hi = (1, experts) if experts == 3 else (0, experts)
    try:
        for mode in (0, 1):
            L.telb_set_nvfp4_wide_mode(mode)
            ws = cu.moe_align(idx, experts, lo, hi)
            a = cu.moe_gather(x, ws, top_k, torch.full((1,), 1.0 / 448, device="cuda"))
            rows = ws.dst_row.clone()
            ws.dst_row = torch.empty(10 ** 6, dtype=torch.int32, device="cuda")         # as many routed rows as take the wide tiles
            y = cu.gemm_grouped(a, wq[lo * n:], ws, hi - lo, alpha=alpha[lo * n:], w_sf=cu.nvfp4_swizzle_scales(sf[lo * n:]))
            outs.append(torch.where(rows[:, None] >= 0, y[rows.clamp(min=0).long()], torch.zeros((), dtype=y.dtype, device="cuda")))
    finally:
        L.telb_set_nvfp4_wide_mode(old)
    _check_status(cu)
    assert torch.equal(*outs) and outs[0].abs().max() > 0


@pytest.mark.parametrize("hidden", [16, 64, 560, 2048, 4112])
@pytest.mark.parametrize("tokens,top_k,experts,lo,hi", [(1, 1, 4, 0, 4), (37, 3, 8, 2, 6), (1025, 8, 128, 0, 128)])
def test_moe_tables_gather_and_combine(cu, tokens, top_k, experts, lo, hi, hidden):
    """Slot counts that are no multiple of four, experts of other ranks, rows whose scales end inside a word; all against their plain statement."""
    g = torch.Generator(device="cuda").manual_seed(hidden + tokens)
    x = torch.randn(tokens, hidden, device="cuda", generator=g).bfloat16()
    idx = torch.rand(tokens, experts, device="cuda", generator=g).topk(top_k, 1).indices.int()
    ws = cu.moe_align(idx, experts, lo, hi)
    dst, flat = ws.dst_row.long(), idx.reshape(-1).long()
    on = (flat >= lo) & (flat < hi)
    assert torch.equal(dst >= 0, on) and dst[on].unique().numel() == int(on.sum())
    assert torch.equal(ws.tile_expert[dst[on] // 128].long(), flat[on] - lo)
    gs = torch.full((1,), 1.0 / 448, device="cuda")
    a = cu.moe_gather(x, ws, top_k, gs)
    xq, sf = cu.nvfp4_quantize(x, gs)
    # the two kernels scale by a product and by a quotient: values on an edge of the four-bit grid may fall either way
    assert (a.xq[dst[on]] != xq.repeat_interleave(top_k, 0)[on]).sum() <= 1 + 0.02 * on.sum() * hidden // 2
    assert torch.equal(a.xq[dst[on]], cu.moe_gather(x.repeat_interleave(top_k, 0), ws, 1, gs).xq[dst[on]])
    k64 = cu.lib().telb_nvfp4_k64_pad(hidden)

    def scales(buf, rows):
        kb = torch.arange(hidden // 16, device="cuda")
        r = rows[:, None]
        return buf.reshape(-1).view(torch.uint8)[((r // 128) * k64 + kb // 4) * 512 + (r % 32) * 16 + (r % 128) // 32 * 4 + kb % 4]

    assert torch.equal(scales(a.sf, dst[on]), scales(sf, torch.arange(tokens, device="cuda").repeat_interleave(top_k)[on]))
    w = torch.rand(tokens, top_k, device="cuda", generator=g)
    y = cu.moe_gather(x, ws, top_k, None)
    want = (x.float()[:, None] * (w * on.view(tokens, top_k))[:, :, None]).sum(1)
    assert (cu.moe_combine(y, ws, w).float() - want).norm() <= 2 ** -8 * want.norm() + 1e-6     # one rounding of an fp32 sum
    _check_status(cu)


@pytest.mark.parametrize("hidden", [48, 2048])
@pytest.mark.parametrize("tokens,top_k", [(128, 8), (129, 8), (64, 8), (65, 8), (1500, 2), (1500, 1)])
def test_moe_gather_by_slot_and_by_token(cu, tokens, top_k, hidden):
    """Both sides of the sizes where a CTA per slot gives way to one per token; one expert in eight is here, so most tokens have no slot.  A
    row per slot, gathered one slot a token, says what every row holds."""
    g = torch.Generator(device="cuda").manual_seed(hidden + tokens)
    x = torch.randn(tokens, hidden, device="cuda", generator=g).bfloat16()
    ws = cu.moe_align(torch.rand(tokens, 16, device="cuda", generator=g).topk(top_k, 1).indices.int(), 16, 4, 6)
    dst = ws.dst_row.long()
    on, gs = dst >= 0, torch.full((1,), 1.0 / 448, device="cuda")
    one, rows = x.repeat_interleave(top_k, 0), dst[dst >= 0]
    a, b = cu.moe_gather(x, ws, top_k, gs), cu.moe_gather(one, ws, 1, gs)
    assert torch.equal(a.xq[rows], b.xq[rows])
    kb = torch.arange(hidden // 16, device="cuda")
    at = ((rows[:, None] // 128) * cu.lib().telb_nvfp4_k64_pad(hidden) + kb // 4) * 512 + (rows[:, None] % 32) * 16 + (rows[:, None] % 128) // 32 * 4 + kb % 4
    assert torch.equal(a.sf.reshape(-1).view(torch.uint8)[at], b.sf.reshape(-1).view(torch.uint8)[at])
    assert torch.equal(cu.moe_gather(x, ws, top_k, None)[rows], one[on])
    _check_status(cu)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("tokens,top_k", [(8191, 1), (8195, 1), (4096, 2), (2730, 3), (2731, 3), (1639, 5)])
def test_moe_tables_and_sums_by_slot_count(cu, tokens, top_k, dtype):
    """Slot counts around those where the tables are built four slots at a time, with and without a remainder; every batch of the sum."""
    g = torch.Generator(device="cuda").manual_seed(tokens)
    idx = torch.rand(tokens, 24, device="cuda", generator=g).topk(top_k, 1).indices.int()
    ws = cu.moe_align(idx, 24, 3, 21)
    dst, flat = ws.dst_row.long(), idx.reshape(-1).long()
    on = (flat >= 3) & (flat < 21)
    assert torch.equal(dst >= 0, on) and dst[on].unique().numel() == int(on.sum())
    assert torch.equal(ws.tile_expert[dst[on] // 128].long(), flat[on] - 3)
    y, w = torch.randn(ws.rows_pad, 72, device="cuda", generator=g).to(dtype), torch.rand(tokens, top_k, device="cuda", generator=g)
    want = (torch.where(on[:, None], y[dst.clamp(min=0)].double(), 0.0) * w.double().reshape(-1, 1)).view(tokens, top_k, 72).sum(1)
    eps = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -11
    assert (cu.moe_combine(y, ws, w).double() - want).norm() <= eps * want.norm()             # one rounding of an fp32 sum
    _check_status(cu)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,n,k,ranks", [(129, 128, 8, 1), (256, 4096, 4096, 0), (200, 1000, 1032, 3), (240, 520, 12288, 8), (131, 6, 256, 2), (255, 3000, 520, 1)])
def test_split_gemm_of_129_to_256_rows(cu, m, n, k, ranks, dtype):
    """One token tile of 256: ragged tokens, features and K steps, every way out of the epilogue; bias, scale and residual."""
    g = torch.Generator(device="cuda").manual_seed(m + n)
    x, w = torch.randn(m, k, device="cuda", generator=g).to(dtype), (torch.randn(n, k, device="cuda", generator=g) * k ** -0.5).to(dtype)
    bias, res = torch.randn(n, device="cuda", generator=g).to(dtype), torch.randn(m, n, device="cuda", generator=g).to(dtype)
    alpha, exact = torch.rand(n, device="cuda", generator=g), x.double() @ w.double().t()
    for kw, want in ((dict(), exact), (dict(alpha=alpha, bias=bias, residual=res), exact * alpha.double() + bias.double() + res.double())):
        got = cu.gemm_skinny(x, w, ranks=ranks, **kw)
        eps = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -11
        assert ((got.double() - want).abs() <= eps * want.abs() + 1e-5 * want.abs().max()).all()      # one rounding of an fp32 sum
        assert ((cu.gemm(x, w, **kw).double() - want).abs() <= eps * want.abs() + 1e-5 * want.abs().max()).all()
    _check_status(cu)


@pytest.mark.parametrize("seqs,past", [(1, 9000), (3, 2300), (9, 1100), (20, 2100), (25, 2100), (40, 300)])
def test_decode_attention_with_chosen_splits(cu, seqs, past):
    q, kv, meta = _paged_step([1] * seqs, [past - 37 * i for i in range(seqs)] if past > 37 * seqs else [past] * seqs, 32, 8, 64, torch.bfloat16)
    want = ref.paged_attention(q, kv, meta, 128 ** -0.5)
    got = cu.paged_attention(q, kv, meta, 128 ** -0.5)
    assert (got.float() - want.float()).norm() < 8e-3 * want.float().norm()       # probabilities and outputs rounded to 16 bits
    _check_status(cu)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("seqs,past,hq,hkv", [(1, 700, 32, 8), (3, 130, 16, 2), (8, 1, 32, 4), (20, 300, 32, 8), (20, 2500, 32, 8)])
def test_decode_attention_of_steps_planned_for_longer_sequences(cu, seqs, past, hq, hkv, fp8):
    """A captured step plans its splits for the table's capacity; splits that find no keys add nothing, whatever the scratch held before."""
    q, kv, meta = _paged_step([1] * seqs, [past + i % 3 for i in range(seqs)], hq, hkv, 64, torch.bfloat16)
    want = ref.paged_attention(q.to(torch.float8_e4m3fn).bfloat16() if fp8 else q, kv.to(torch.float8_e4m3fn).bfloat16() if fp8 else kv, meta, 128 ** -0.5)
    sinks = torch.zeros(hq, device="cuda")
    meta.host_lens, meta.max_seq_len = None, 8192
    ws = cu.Workspace.get(q.device)
    for splits in (None, 3, 19, 32):
        ws.attn_ws.fill_(float("nan"))
        if fp8:
            got = cu.paged_attention_decode_fp8(q.to(torch.float8_e4m3fn), kv.to(torch.float8_e4m3fn), meta, 128 ** -0.5, None, torch.ones(2, device="cuda"),
                                                torch.bfloat16, splits=splits)
        else:
            got = cu.paged_attention(q, kv, meta, 128 ** -0.5, splits=splits)
        # probabilities rounded to 16 bits (E4M3: 2^-4 each), outputs to 16, over values of either sign
        assert (got.float() - want.float()).norm() < (2 ** -4 if fp8 else 8e-3) * want.float().norm(), splits
        if not fp8:
            ws.attn_ws.fill_(float("nan"))
            got = cu.paged_attention(q, kv, meta, 128 ** -0.5, splits=splits, sinks=sinks)
            more = ref.paged_attention(q, kv, meta, 128 ** -0.5, sinks=sinks)
            assert (got.float() - more.float()).norm() < 8e-3 * more.float().norm(), splits
    ws.attn_ws.zero_()
    _check_status(cu)


def test_decode_splits_of_known_and_unknown_lengths(cu):
    """148 to 197 items are split in three only where the step's own lengths are known, and long."""
    for past, known, fp8, splits in ((2500, True, False, 3), (2500, False, False, 1), (1900, True, False, 1), (2500, True, True, 1), (3100, True, True, 3)):
        _, _, meta = _paged_step([1] * 20, [past] * 20, 8, 8, 64, torch.bfloat16)
        meta.host_lens = meta.host_lens if known else None
        assert cu._decode_splits(meta, 8, fp8=fp8) == splits


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("tokens,hq,hkv,norm", [(256, 4, 1, True), (300, 5, 5, False), (700, 32, 8, True), (5000, 3, 1, True)])
def test_rope_rows_of_several_heads_a_warp(cu, tokens, hq, hkv, norm, dtype):
    """Head counts that end inside a group of four, one to all groups a warp, sequences and pages that end anywhere."""
    from tensorrt_edge_llm_b200.ops import build_step_meta, rope_cos_sin
    g = torch.Generator(device="cuda").manual_seed(tokens)
    q_lens, pasts = [tokens - 101, 1, 100], [3, 70, 0]
    n = [-(-(a + b) // 64) for a, b in zip(q_lens, pasts)]
    table = torch.full((3, max(n)), -1, dtype=torch.int32)
    for i in range(3):
        table[i, :n[i]] = torch.arange(sum(n[:i]), sum(n[:i + 1]), dtype=torch.int32)
    meta = build_step_meta(q_lens, pasts, table, 64, device="cuda")
    qkv = torch.randn(tokens, (hq + 2 * hkv) * 128, device="cuda", generator=g).to(dtype)
    w = [(torch.rand(128, device="cuda", generator=g) + 0.5).to(dtype) if norm else None for _ in range(2)]
    cs = rope_cos_sin(8192, 128, 1e6, device="cuda")
    kv, kv_ref = (torch.zeros(sum(n), 2, hkv, 64, 128, device="cuda", dtype=dtype) for _ in range(2))
    q = cu.rope_kv_write(qkv, kv, meta, cs, hq, hkv, 128, *w, 1e-6)
    q_ref = ref.rope_kv_write(qkv, kv_ref, meta, cs, hq, hkv, 128, *w, 1e-6)
    _check_status(cu)
    eps = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -11
    for a, b in ((q, q_ref), (kv, kv_ref)):
        assert (a.float() - b.float()).norm() < 2 * eps * b.float().norm()          # up to three 16-bit roundings, two of which may flip
    assert torch.equal(kv == 0, kv_ref == 0)

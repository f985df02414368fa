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

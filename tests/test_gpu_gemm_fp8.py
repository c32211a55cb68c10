"""GPU parity tests of the FP8 e4m3 tcgen05 GEMM against the CPU oracle (fp64 contraction), through the C ABI.
Stated tolerance: relative Frobenius error <= 1e-2 of the bf16/fp16 output (the reference arithmetic is a closed
library; the measured error is in fact near bf16 rounding, ~2e-3), and element-wise |d| <= 2 output ulps + 1e-2*|y|."""

import pytest
import torch

from oracle import gemm, quant, workloads
from tests.util import assert_bit_equal, check_status, cu, rel_err

pytestmark = pytest.mark.gpu

REL_TOL = 1e-2


@pytest.fixture(scope="module")
def ops():
    from lyradiff_b200 import ops as _ops
    return _ops


@pytest.fixture(params=[0, 2561, 1281, 2562], ids=["auto", "1cta_n256", "1cta_n128", "pair_n256"])
def tile(request):
    from lyradiff_b200 import _lib
    assert _lib.lib().lyraq_debug_force_gemm_tile(request.param) == 0
    yield request.param
    _lib.lib().lyraq_debug_force_gemm_tile(0)


def _run(ops, f, dtype, bias=True, residual=False, gelu=False, alpha=1.0, beta=1.0):
    m, k = f["qx"].shape
    n = f["qw"].shape[0]
    y = torch.empty(m, n, dtype=dtype, device="cuda")
    b = f["bias"].to(dtype) if bias else None
    r = f["residual"].to(dtype) if residual else None
    ops.gemm_with_residual_and_bias_fp8(cu(f["qw"]), cu(f["s_w"]), cu(f["qx"]), cu(f["s_x"]), y, bias=cu(b), residual=cu(r),
                                        alpha=alpha, beta=beta, is_gelu=gelu)
    want = gemm.fp8_gemm(f["qx"], f["qw"], f["s_x"], f["s_w"], out_dtype=dtype, bias=b, residual=r, alpha=alpha, beta=beta,
                         gelu=gelu)
    return y, want


def _check(y, want, dtype):
    assert rel_err(y, want) <= REL_TOL
    ulp = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -20}[dtype]
    d = (y.cpu().double() - want.double()).abs()
    bound = 2 * ulp * want.double().abs() + 1e-2 * want.double().abs() + 1e-3
    assert bool((d <= bound).all()), float((d - bound).max())


@pytest.mark.parametrize("m,n,k", [(128, 256, 128), (128, 128, 256), (130, 72, 144), (1, 8, 16), (300, 1000, 3072),
                                   (256, 384, 12288)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_plain_and_bias(ops, tile, m, n, k, dtype):
    f = workloads.fp8_linear(m, k, n, seed=m + n, with_residual=True)
    for bias in (False, True):
        y, want = _run(ops, f, dtype, bias=bias)
        _check(y, want, dtype)
    check_status()


def test_exact_on_small_integers(ops, tile):
    """Operands that are small integers in e4m3 and unit scales give integer sums below 2**24: fp32 accumulation
    must then be exact, whatever the order."""
    g = torch.Generator().manual_seed(4)
    xi = torch.randint(-8, 9, (200, 512), generator=g).float()
    wi = torch.randint(-8, 9, (136, 512), generator=g).float()
    one = torch.ones(1)
    qx, qw = quant.fp8_quant(xi, one), quant.fp8_quant(wi, one)
    y = torch.empty(200, 136, dtype=torch.float32, device="cuda")
    ops.gemm_with_residual_and_bias_fp8(cu(qw), cu(one), cu(qx), cu(one), y)
    assert torch.equal(y.cpu(), xi @ wi.t())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gelu_and_residual_epilogues(ops, tile, dtype):
    f = workloads.fp8_linear(260, 512, 392, seed=21, with_residual=True)
    for kw in ({"gelu": True}, {"gelu": True, "bias": False}, {"residual": True}, {"residual": True, "beta": 0.5, "alpha": 2.0}):
        y, want = _run(ops, f, dtype, **kw)
        _check(y, want, dtype)
    check_status()


def test_golden_vectors(ops, golden):
    z = golden("fp8")
    f = {k: z[k] for k in ("qx", "qw", "s_x", "s_w", "bias", "residual")}
    for key, kw in (("y_plain", {}), ("y_gelu", {"gelu": True}), ("y_residual", {"residual": True})):
        y, _ = _run(ops, f, torch.bfloat16, **kw)
        _check(y, z[key], torch.bfloat16)


def test_quantize_then_gemm_matches_unquantized_linear(ops):
    f = workloads.fp8_linear(512, 3072, 640, seed=2)
    x, w = cu(f["x"]), cu(f["w"])
    sx = torch.zeros(1, dtype=torch.float32, device="cuda")
    sw = torch.zeros(1, dtype=torch.float32, device="cuda")
    ops.invoke_get_fp8_weight_scale(sx, x)
    ops.invoke_get_fp8_weight_scale(sw, w)
    qx = torch.empty(512, 3072, dtype=torch.uint8, device="cuda")
    qw = torch.empty(640, 3072, dtype=torch.uint8, device="cuda")
    ops.invoke_cuda_d2d_scale_cpy_convert(qx, x, sx)
    ops.invoke_cuda_d2d_scale_cpy_convert(qw, w, sw)
    assert torch.equal(qx.cpu(), f["qx"]) and torch.equal(qw.cpu(), f["qw"])
    y = torch.empty(512, 640, dtype=torch.bfloat16, device="cuda")
    ops.gemm_with_residual_and_bias_fp8(qw, sw, qx, sx, y, bias=cu(f["bias"]))
    ref = f["x"].float() @ f["w"].float().t() + f["bias"].float()
    assert rel_err(y, ref) < 0.05  # e4m3 quantization noise of both operands


@pytest.mark.parametrize("name,k,n,gelu,residual", workloads.FLUX_FP8_LINEARS)
def test_full_size_flux_linears(ops, name, k, n, gelu, residual):
    """The FLUX FP8 linears at full size (M=4608): a strided sample of rows against the oracle, and the
    row-checksum property sum_n Y[m,n] == s * X[m,:] . sum_n W[n,:] (fp32 output, no epilogue)."""
    m = workloads.FLUX_TOKENS
    f = workloads.fp8_linear(m, k, n, seed=7, with_bias=True, with_residual=residual)
    qx, qw, sx, sw = cu(f["qx"]), cu(f["qw"]), cu(f["s_x"]), cu(f["s_w"])
    y = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    ops.gemm_with_residual_and_bias_fp8(qw, sw, qx, sx, y, bias=cu(f["bias"]), residual=cu(f["residual"]), is_gelu=gelu)
    rows = torch.arange(0, m, 149)
    want = gemm.fp8_gemm(f["qx"][rows], f["qw"], f["s_x"], f["s_w"], bias=f["bias"],
                         residual=None if f["residual"] is None else f["residual"][rows], gelu=gelu)
    _check(y[rows.cuda()], want, torch.bfloat16)
    y32 = torch.empty(m, n, dtype=torch.float32, device="cuda")
    ops.gemm_with_residual_and_bias_fp8(qw, sw, qx, sx, y32)
    wsum = quant.fp8_dequant(f["qw"]).double().sum(dim=0)
    check = (quant.fp8_dequant(f["qx"]).double() @ wsum) * float(f["s_x"]) * float(f["s_w"])
    got = y32.double().sum(dim=1).cpu()
    scale = (quant.fp8_dequant(f["qx"]).double().abs() @ quant.fp8_dequant(f["qw"]).double().abs().sum(dim=0)) * float(f["s_x"]) * float(f["s_w"])
    assert float(((got - check).abs() / scale).max()) < 1e-5
    check_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,n,k", [(260, 520, 512), (128, 256, 3072), (130, 72, 144)])
def test_fused_output_quantize(ops, tile, dtype, m, n, k):
    """The GEMM epilogue that also quantizes its result for the next FP8 linear equals GEMM -> T -> e4m3 quantize.
    A one-ulp difference of the T value (fp32 vs fp64 accumulation) can move an e4m3 code by one step: stated tolerance
    |code distance| <= 1 on <= 2 % of the outputs, everything else identical."""
    f = workloads.fp8_linear(m, k, n, seed=m + 3 * n, with_residual=True)
    y_scale = torch.tensor([0.037], dtype=torch.float32)
    for kw in ({"gelu": True}, {"residual": True}, {}):
        b = f["bias"].to(dtype)
        r = f["residual"].to(dtype) if kw.get("residual") else None
        yq = torch.empty(m, n, dtype=torch.uint8, device="cuda")
        ops.gemm_fp8_quant_out(cu(f["qw"]), cu(f["s_w"]), cu(f["qx"]), cu(f["s_x"]), yq, cu(y_scale), dtype, bias=cu(b),
                               residual=cu(r), is_gelu=bool(kw.get("gelu")))
        y = gemm.fp8_gemm(f["qx"], f["qw"], f["s_x"], f["s_w"], out_dtype=dtype, bias=b, residual=r, gelu=bool(kw.get("gelu")))
        want = quant.fp8_quant(y, y_scale)
        got = yq.cpu()
        same_sign = ((got ^ want) & 0x80) == 0
        dist = ((got & 0x7F).to(torch.int32) - (want & 0x7F).to(torch.int32)).abs()
        zeroish = ((got & 0x7F) <= 1) & ((want & 0x7F) <= 1)   # +-0 and the smallest subnormal may swap sign
        assert bool(((dist <= 1) & (same_sign | zeroish)).all())
        assert float((got != want).float().mean()) <= 0.02
    check_status()


@pytest.mark.parametrize("m", [1, 2, 7, 15, 16, 17])
@pytest.mark.parametrize("n,k", [(8, 16), (130, 272), (128, 1024), (264, 3072), (264, 4112), (3072, 6144)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_few_tokens(ops, m, n, k, dtype):
    """The few-token kernel: row counts up to its width and past it, and around the share of them each CTA of a cluster sums, ragged n and k,
    one, two, four and eight CTAs along k; the larger row counts of the first three shapes, and 17, are the dense kernel's.  An fp32 sum of k products in any order is within k 2^-24 of the sum of their magnitudes; the
    epilogue adds a few fp32 roundings (GELU's approximate tanh: 2^-10 of its argument's magnitude) and one to the output type."""
    f = workloads.fp8_linear(m, k, n, seed=m + n + k, with_residual=True)
    mags = (quant.fp8_dequant(f["qx"]).double().abs() @ quant.fp8_dequant(f["qw"]).double().abs().t()) * float(f["s_x"]) * float(f["s_w"])
    eps = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -22}[dtype]
    for kw in (dict(bias=False), dict(residual=True, beta=0.5, alpha=1.25), dict(gelu=True)):
        y, want = _run(ops, f, dtype, **kw)
        terms = 1.25 * mags + f["bias"].double().abs()[None, :] + f["residual"].double().abs() + 1.0
        bound = eps * want.double().abs() + k * 2.0 ** -24 * terms + 2.0 ** -22 * terms + (2.0 ** -10 * want.double().abs() + 2.0 ** -10 if "gelu" in kw else 0.0)
        d = (y.cpu().double() - want.double()).abs()
        assert bool((d <= bound).all()), (kw, float((d / bound).max()))
    check_status()


@pytest.mark.parametrize("m,n,k,stalled", [(16, 264, 4096, 0), (16, 264, 4096, 5), (1, 8192, 3072, 3), (16, 15360, 3072, 1)])
def test_few_tokens_store_nothing_when_a_cluster_rank_gives_up(ops, m, n, k, stalled):
    """Eight, four and two CTAs along k: one of each cluster loads nothing and its wait runs out; the
    others have whole partial products of their own, but no sum to store."""
    from lyradiff_b200 import _lib
    lib = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(n)
    qw, qx = (torch.randint(0, 0x78, (r, k), generator=g, dtype=torch.uint8, device="cuda") for r in (n, m))   # no NaN codes
    scale = torch.full((1,), 0.001, device="cuda")
    good, out = (torch.full((m, n), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    ops.gemm_with_residual_and_bias_fp8(qw, scale, qx, scale, good)
    check_status()
    assert lib.lyraq_debug_skinny_wait_test(stalled, 50) == 0
    try:
        ops.gemm_with_residual_and_bias_fp8(qw, scale, qx, scale, out)   # the launch itself succeeds
        torch.cuda.synchronize()
        status, detail = ops.last_status()
    finally:
        assert lib.lyraq_debug_skinny_wait_test(-1, 0) == 0
    assert status == 4 and 0x4000 <= detail < 0x5000, (status, hex(detail))
    assert bool((out == 7.0).all()), "a timed-out cluster must not store results"
    assert ops.last_status()[0] == 0                                     # reading the status cleared it
    ops.gemm_with_residual_and_bias_fp8(qw, scale, qx, scale, out)
    check_status()
    assert_bit_equal(out, good.cpu(), "after a timed-out launch")


@pytest.mark.parametrize("m", [1, 4, 5, 7, 15, 16])
@pytest.mark.parametrize("n,k", [(264, 4096), (4224, 4096), (4352, 4096), (3072, 3072), (9088, 2048), (9216, 2048), (18944, 1024), (19072, 1024),
                                 (130, 16), (256, 256), (4096, 512), (9216, 8192)])
def test_few_tokens_with_every_split_of_k(ops, m, n, k):
    """Both sides of the rows at which the dense kernel takes over (small k; 128 KB of X with many tiles).  One, two, four and eight CTAs along k, and both sides of the tile counts at which fewer are taken (33, 71 and 148 tiles of 128).
    Operands of 0, 1, -1 and 2 make every partial sum an integer below 2^24, so the fp32 results are exact in any order."""
    g = torch.Generator(device="cuda").manual_seed(n + m)
    codes = torch.tensor([0x00, 0x38, 0xB8, 0x40], dtype=torch.uint8, device="cuda")
    values = torch.tensor([0.0, 1.0, -1.0, 2.0], dtype=torch.float64, device="cuda")
    iw, ix = (torch.randint(0, 4, (r, k), generator=g, device="cuda") for r in (n, m))
    one = torch.ones(1, device="cuda")
    y = torch.empty(m, n, dtype=torch.float32, device="cuda")
    ops.gemm_with_residual_and_bias_fp8(codes[iw], one, codes[ix], one, y)
    check_status()
    assert_bit_equal(y, (values[ix] @ values[iw].t()).float().cpu())

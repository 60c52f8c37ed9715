"""GPU numerics: every sm_100a kernel against the fp32 PyTorch oracle (ml_b200.ops.ref) on the same inputs,
including odd shapes that take the scalar / SIMT paths and rows with tgt = -1."""
import ctypes
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from ml_b200.ops import ref


def nat():
    from ml_b200.ops import native
    return native


def dev():
    return torch.device("cuda:0")


def rnd(*shape, scale=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, device=dev(), dtype=torch.float32) * scale).to(dtype)


def close(a, b, rtol=2e-2, atol=2e-2, name="", fro=None):
    """Two bounds.  Max norm: no single element is off by more than atol + rtol * max|ref|.  Relative Frobenius norm:
    ||a - ref|| / ||ref|| <= fro, which catches what the first cannot - an error confined to small-magnitude elements, a
    bias of a percent of the peak, a wrong low-order bit pattern spread over the tensor.  Default fro: 4e-3 for bf16
    outputs (one bf16 rounding is 2^-9 relative at worst, ~1.1e-3 rms), 1e-3 for fp32 outputs."""
    if fro is None:
        fro = 4e-3 if a.dtype == torch.bfloat16 else 1e-3
    a, b = a.float(), b.float()
    err = (a - b).abs().max().item()
    ref_mag = b.abs().max().item()
    assert torch.isfinite(a).all(), f"{name}: non-finite output"
    assert err <= atol + rtol * ref_mag, f"{name}: max err {err} vs ref magnitude {ref_mag}"
    den = b.double().norm().item()
    if den > 0:
        rel = (a.double() - b.double()).norm().item() / den
        assert rel <= fro, f"{name}: relative Frobenius error {rel:.3e} > {fro:.1e}"


@pytest.fixture(autouse=True)
def _no_kernel_error():
    yield
    torch.cuda.synchronize()
    e = nat().get_error()
    nat().clear_error()
    assert e == 0, f"kernel error word {e:#x}"


# ------------------------------------------------------------------ GEMM with SwiGLU epilogue
@pytest.mark.parametrize("M,I,K", [(1024, 2048, 768), (392, 256, 128), (4096 + 200, 384, 264), (512, 128, 64)])
def test_linear_fwd_swiglu_epilogue(M, I, K):
    """gate|up product with silu(gate) * up formed in the epilogue: both outputs against the fp32 oracle, and the fused
    activation bit-equal to the separate SwiGLU kernel run on the fused kernel's own [gate | up] output."""
    torch.manual_seed(M + I)
    x, W = rnd(M, K), rnd(2 * I, K, scale=K ** -0.5)
    gu = torch.full((M, 2 * I), float("nan"), device=dev(), dtype=torch.bfloat16)
    sw = torch.full((M, I), float("nan"), device=dev(), dtype=torch.bfloat16)
    assert nat().linear_fwd_swiglu(gu, sw, x, W)
    egu = torch.empty(M, 2 * I, device=dev())
    ref.linear_fwd(egu, x, W)
    close(gu, egu, name="gate|up")
    esw = torch.empty(M, I, device=dev())
    ref.swiglu_fwd(esw, egu)
    close(sw, esw, name="swiglu", fro=6e-3)        # two roundings (gate / up, then the product) against none
    sep = torch.empty_like(sw)
    nat().swiglu_fwd(sep, gu)
    assert torch.equal(sep, sw)
    # shapes the epilogue form does not take are declined without a launch
    assert not nat().linear_fwd_swiglu(torch.empty(64, 2 * I, device=dev(), dtype=torch.bfloat16),
                                       torch.empty(64, I, device=dev(), dtype=torch.bfloat16), x[:64], W)
    assert not nat().linear_fwd_swiglu(torch.empty(M, 200, device=dev(), dtype=torch.bfloat16),
                                       torch.empty(M, 100, device=dev(), dtype=torch.bfloat16), x, W[:200])


@pytest.mark.parametrize("M,N,K,period", [(392, 768, 768, 196), (1024, 256, 128, 64), (300, 520, 264, 100)])
def test_linear_fwd_posembed_epilogue(M, N, K, period):
    """Patch embedding with the learned positions added in the GEMM epilogue (fp32 accumulators + position, one
    rounding) against the fp32 oracle of product + add."""
    torch.manual_seed(M)
    x, W, pos = rnd(M, K), rnd(N, K, scale=K ** -0.5), rnd(period, N, scale=0.5)
    out = torch.full((M, N), float("nan"), device=dev(), dtype=torch.bfloat16)
    assert nat().linear_fwd_posembed(out, x, W, pos, period)
    exp = torch.empty(M, N, device=dev())
    ref.linear_fwd(exp, x, W)
    exp += pos.float().repeat((M + period - 1) // period, 1)[:M]
    close(out, exp, name="patch embed + pos")
    assert not nat().linear_fwd_posembed(torch.empty(64, N, device=dev(), dtype=torch.bfloat16), x[:64], W, pos, period)


# ------------------------------------------------------------------ GEMM
GEMM_SHAPES = [(256, 256, 128), (384, 768, 768), (1024, 2304, 768), (512, 4096, 768), (300, 520, 264), (128, 128, 64),
               (2048, 768, 2048), (256, 1000, 512), (4096 + 136, 776, 392)]


@pytest.fixture(params=[(1, 1, 1), (1, 0, 0), (0, 0, 0), (1, 1, 2)],
                ids=["cta_pair", "cta_pair_tma_epilogue_splitk", "single_cta", "cta_pair_ungrouped_streamk_m_first"])
def gemm_mode(request):
    """Large products have two tcgen05 kernels: a 256x256 tile shared by a CTA pair (cta_group::2) whose epilogue either
    writes coalesced rows itself or hands slabs to TMA (weight gradients: equal k-block ranges per cluster, or a fixed
    split count), or 128x256 per CTA."""
    nat().lib().mlb_gemm_use_pairs(request.param[0])
    nat().lib().mlb_gemm_epilogue_mode(request.param[1])
    nat().lib().mlb_gemm_streamk(1 if request.param[2] else 0)
    nat().lib().mlb_gemm_streamk_groups(0 if request.param[2] == 2 else 1)
    nat().lib().mlb_gemm_tile_order(1 if request.param[2] == 2 else 0)
    yield request.param
    nat().lib().mlb_gemm_use_pairs(1)
    nat().lib().mlb_gemm_epilogue_mode(1)
    nat().lib().mlb_gemm_streamk(1)
    nat().lib().mlb_gemm_streamk_groups(1)
    nat().lib().mlb_gemm_tile_order(0)


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES)
def test_linear_fwd(M, N, K, gemm_mode):
    torch.manual_seed(0)
    x, W = rnd(M, K), rnd(N, K, scale=0.05)
    out, exp = torch.empty(M, N, device=dev(), dtype=torch.bfloat16), torch.empty(M, N, device=dev())
    nat().linear_fwd(out, x, W)
    ref.linear_fwd(exp, x, W)
    close(out, exp, name="linear_fwd")


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES)
def test_linear_dx(M, N, K, gemm_mode):
    torch.manual_seed(1)
    dout, W = rnd(M, N), rnd(N, K, scale=0.05)
    dx, exp = torch.empty(M, K, device=dev(), dtype=torch.bfloat16), torch.empty(M, K, device=dev())
    nat().linear_dx(dx, dout, W)
    ref.linear_dx(exp, dout, W)
    close(dx, exp, name="linear_dx")


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES + [(16384, 768, 768)])
def test_linear_dw_accumulates(M, N, K, gemm_mode):
    torch.manual_seed(2)
    dout, x = rnd(M, N, scale=0.1), rnd(M, K)
    dW = torch.randn(N, K, device=dev())
    exp = dW.clone()
    nat().linear_dw(dW, dout, x)
    ref.linear_dw(exp, dout, x)
    close(dW, exp, rtol=1e-2, atol=1e-2, name="linear_dw")


@pytest.mark.parametrize("a_mn", [False, True])
@pytest.mark.parametrize("b_mn", [False, True])
@pytest.mark.parametrize("acc", [False, True])
def test_gemm_general_entry_all_layouts(a_mn, b_mn, acc, gemm_mode):
    """D = A.B^T with either operand stored transposed, bf16 store or fp32 accumulate."""
    torch.manual_seed(5)
    M, N, K = 640, 520, 328
    A = rnd(K, M) if a_mn else rnd(M, K)
    B = rnd(K, N, scale=0.05) if b_mn else rnd(N, K, scale=0.05)
    exp = (A.t() if a_mn else A).float() @ (B if b_mn else B.t()).float()
    if acc:
        out = torch.randn(M, N, device=dev())
        exp = exp + out
    else:
        out = torch.empty(M, N, device=dev(), dtype=torch.bfloat16)
    nat().gemm(out, A, B, a_mn, b_mn, acc)
    close(out, exp, name="gemm")


def test_linear_fwd_with_rope_epilogue_matches_separate_rope():
    """QKV product with the rotation applied in the GEMM epilogue vs product, then the in-place RoPE kernel."""
    torch.manual_seed(8)
    B, T, H, hd = 3, 160, 4, 64
    C = H * hd
    x, W = rnd(B * T, C), rnd(3 * C, C, scale=0.05)
    cos, sin = ref.rope_tables(T, hd, 10000.0, dev())
    fused = torch.empty(B * T, 3 * C, device=dev(), dtype=torch.bfloat16)
    assert nat().linear_fwd_rope(fused, x, W, cos, sin, T, 2 * C) is True
    exp = torch.empty(B * T, 3 * C, device=dev())
    ref.linear_fwd(exp, x, W)
    ref.rope_fwd(exp, cos, sin, B, T, H, hd)
    close(fused, exp, name="qkv + rope")
    # V columns are untouched by the rotation
    plain = torch.empty_like(fused)
    nat().linear_fwd(plain, x, W)
    assert torch.equal(plain[:, 2 * C:], fused[:, 2 * C:])
    # a shape that does not take the CTA-pair path reports it instead of launching
    small = torch.empty(64, 3 * C, device=dev(), dtype=torch.bfloat16)
    assert nat().linear_fwd_rope(small, x[:64], W, cos, sin, T, 2 * C) is False


def test_gemm_simt_path_odd_shape():
    torch.manual_seed(3)
    M, N, K = 130, 100, 100   # C=100-style odd sizes: no 16-byte pitch, SIMT kernel
    x, W = rnd(M, K), rnd(N, K, scale=0.1)
    out, exp = torch.empty(M, N, device=dev(), dtype=torch.bfloat16), torch.empty(M, N, device=dev())
    nat().linear_fwd(out, x, W)
    ref.linear_fwd(exp, x, W)
    close(out, exp, name="simt fwd")
    dout = rnd(M, N)
    dx, expx = torch.empty(M, K, device=dev(), dtype=torch.bfloat16), torch.empty(M, K, device=dev())
    nat().linear_dx(dx, dout, W)
    ref.linear_dx(expx, dout, W)
    close(dx, expx, name="simt dx")
    dW = torch.zeros(N, K, device=dev())
    expw = torch.zeros(N, K, device=dev())
    nat().linear_dw(dW, dout, x)
    ref.linear_dw(expw, dout, x)
    close(dW, expw, name="simt dw")


def test_gemm_tc_matches_simt():
    """Same inputs through the tcgen05 kernel and the SIMT kernel."""
    torch.manual_seed(4)
    M, N, K = 512, 768, 256
    x, W = rnd(M, K), rnd(N, K, scale=0.05)
    a = torch.empty(M, N, device=dev(), dtype=torch.bfloat16)
    b = torch.empty_like(a)
    nat().linear_fwd(a, x, W)
    nat().lib().mlb_gemm_force_simt(1)
    try:
        nat().linear_fwd(b, x, W)
    finally:
        nat().lib().mlb_gemm_force_simt(0)
    close(a, b, rtol=1e-2, atol=1e-2, name="tc vs simt")


# ------------------------------------------------------------------ attention
ATTN_CASES = [(2, 128, 2, 64), (1, 256, 3, 64), (2, 384, 2, 64), (2, 192, 2, 64), (2, 64, 4, 64), (1, 1024, 2, 64),
              (1, 256, 2, 128), (2, 320, 1, 128), (2, 64, 4, 32), (1, 100, 2, 16)]


@pytest.fixture(params=[True, False], ids=["fused_bwd", "split_bwd"])
def bwd_mode(request):
    """Head size 64 has two backward implementations: one fused kernel, or separate dK/dV and dQ kernels."""
    old = nat().FUSED_ATTN_BWD
    nat().FUSED_ATTN_BWD = request.param
    yield request.param
    nat().FUSED_ATTN_BWD = old


@pytest.mark.parametrize("B,T,H", [(2, 384, 2), (3, 1024, 4), (1, 128, 1), (16, 512, 12)])
def test_attn_dynamic_work_counter_equals_static_schedule(B, T, H):
    """Work items drawn from the device counter instead of the host-built table: the same bits out of forward and
    backward (who computes an item does not enter its arithmetic), twice in a row (the last CTA resets the counter)."""
    torch.manual_seed(B * T + H)
    hd, C = 64, H * 64
    qkv, dout = rnd(B * T, 3 * C), rnd(B * T, C)
    outs = []
    for dyn in (False, True, True):
        nat().attn_dynamic(dyn)
        try:
            out = torch.full((B * T, C), float("nan"), device=dev(), dtype=torch.bfloat16)
            lse = torch.empty(B, H, T, device=dev())
            dqkv = torch.full((B * T, 3 * C), float("nan"), device=dev(), dtype=torch.bfloat16)
            nat().attn_fwd(out, lse, qkv, B, T, H, hd)
            nat().attn_bwd(dqkv, dout, qkv, out, lse, B, T, H, hd)
            torch.cuda.synchronize()
        finally:
            nat().attn_dynamic(False)
        outs.append((out, lse, dqkv))
    for o in outs[1:]:
        assert torch.equal(o[0], outs[0][0]) and torch.equal(o[1], outs[0][1]) and torch.equal(o[2], outs[0][2])



@pytest.mark.parametrize("B,T,H,hd", [c for c in ATTN_CASES if c[3] == 64] + [(3, 640, 2, 64), (1, 1100, 1, 64), (4, 1024, 12, 64)])
@pytest.mark.parametrize("rows", [1, 2, 3, 0], ids=["thread_per_row", "thread_per_row_lazy_rescale", "thread_per_row_one_pass", "four_threads_per_row"])
@pytest.mark.parametrize("qscale", [1.0, 3.0], ids=["unit_scale", "peaked_scores"])
def test_attn_fwd_variants_hd64(B, T, H, hd, rows, qscale):
    """Head size 64 has four forward kernels: thread-per-row over tile pairs (P kept in TMEM) with O folded into
    registers every key block; the same with O accumulated in TMEM and rescaled only when a row maximum grows by more
    than 2^8; that with the row maximum tracked inside the exponential pass (a block is redone when the threshold is
    passed); and four threads per row.  With inputs three times as large the scores are peaked (standard deviation 13
    in log2 units), so running maxima jump by more than the threshold and the in-place rescale / the redo run.  The
    largest case has more tile pairs than the GPU has SMs, so the host's balanced work schedule is in use."""
    torch.manual_seed(15)
    C = H * hd
    qkv = rnd(B * T, 3 * C, scale=qscale)
    out = torch.empty(B * T, C, device=dev(), dtype=torch.bfloat16)
    lse = torch.empty(B, H, T, device=dev())
    nat().lib().mlb_attn_fwd_mode(rows)
    try:
        nat().attn_fwd(out, lse, qkv, B, T, H, hd)
    finally:
        nat().lib().mlb_attn_fwd_mode(3)
    eo, el = torch.empty(B * T, C, device=dev()), torch.empty(B, H, T, device=dev())
    ref.attn_fwd(eo, el, qkv, B, T, H, hd)
    close(out, eo, name="attn out")
    close(lse, el, rtol=1e-3, atol=2e-2, name="attn lse")


# the last two cases have more work items than the GPU has SMs: the persistent kernels walk the host's balanced schedule
@pytest.mark.parametrize("B,T,H,hd", ATTN_CASES + [(4, 1024, 12, 64), (3, 640, 13, 64)])
def test_attn_fwd_bwd(B, T, H, hd, bwd_mode):
    if hd != 64 and not bwd_mode:
        pytest.skip("only one backward implementation for this head size")
    torch.manual_seed(5)
    C = H * hd
    qkv = rnd(B * T, 3 * C, scale=1.0)
    out = torch.empty(B * T, C, device=dev(), dtype=torch.bfloat16)
    lse = torch.empty(B, H, T, device=dev())
    nat().attn_fwd(out, lse, qkv, B, T, H, hd)
    eo, el = torch.empty(B * T, C, device=dev()), torch.empty(B, H, T, device=dev())
    ref.attn_fwd(eo, el, qkv, B, T, H, hd)
    close(out, eo, name="attn out")
    close(lse, el, rtol=1e-3, atol=2e-2, name="attn lse")
    dout = rnd(B * T, C)
    dqkv = torch.empty(B * T, 3 * C, device=dev(), dtype=torch.bfloat16)
    fused = nat().attn_bwd(dqkv, dout, qkv, out, lse, B, T, H, hd)
    assert fused is False
    ed = torch.empty(B * T, 3 * C, device=dev())
    ref.attn_bwd(ed, dout, qkv, eo.to(torch.bfloat16), el, B, T, H, hd)
    d5, e5 = dqkv.view(B, T, 3, C), ed.view(B, T, 3, C)
    for i, nm in enumerate(("dq", "dk", "dv")):
        close(d5[:, :, i], e5[:, :, i], rtol=3e-2, atol=3e-2, name=nm)


def test_attn_bwd_fused_rope_matches_separate(bwd_mode):
    torch.manual_seed(6)
    B, T, H, hd = 2, 256, 2, 64
    C = H * hd
    qkv, dout = rnd(B * T, 3 * C), rnd(B * T, C)
    out = torch.empty(B * T, C, device=dev(), dtype=torch.bfloat16)
    lse = torch.empty(B, H, T, device=dev())
    nat().attn_fwd(out, lse, qkv, B, T, H, hd)
    cos, sin = ref.rope_tables(T, hd, 10000.0, dev())
    a = torch.empty(B * T, 3 * C, device=dev(), dtype=torch.bfloat16)
    b = torch.empty_like(a)
    assert nat().attn_bwd(a, dout, qkv, out, lse, B, T, H, hd, rope=(cos, sin)) is True
    nat().attn_bwd(b, dout, qkv, out, lse, B, T, H, hd)
    nat().rope_bwd(b, cos, sin, B, T, H, hd)
    close(a, b, rtol=2e-2, atol=2e-2, name="fused rope bwd")


# ------------------------------------------------------------------ elementwise
@pytest.mark.parametrize("rows,C", [(64, 768), (33, 128), (17, 100), (8, 2048), (5, 1024)])
def test_rmsnorm_fwd_bwd(rows, C):
    torch.manual_seed(7)
    x, b2, w = rnd(rows, C), rnd(rows, C), (1 + 0.1 * torch.randn(C, device=dev())).to(torch.bfloat16)
    out, rstd = torch.empty_like(x), torch.empty(rows, device=dev())
    eo, er = torch.empty(rows, C, device=dev()), torch.empty(rows, device=dev())
    nat().rmsnorm_fwd(out, rstd, x, w, 1e-5)
    ref.rmsnorm_fwd(eo, er, x, w, 1e-5)
    close(out, eo, name="rmsnorm out")
    close(rstd, er, rtol=1e-4, atol=1e-5, name="rstd")
    resid, out2, rstd2 = torch.empty_like(x), torch.empty_like(x), torch.empty(rows, device=dev())
    e_res, e_out, e_r = torch.empty(rows, C, device=dev()), torch.empty(rows, C, device=dev()), torch.empty(rows, device=dev())
    nat().add_rmsnorm_fwd(resid, out2, rstd2, x, b2, w, 1e-5)
    ref.add_rmsnorm_fwd(e_res, e_out, e_r, x, b2, w, 1e-5)
    close(resid, e_res, name="resid")
    close(out2, e_out, name="add_rmsnorm out")
    for add in (None, b2):
        dy = rnd(rows, C)
        dx, dw = torch.empty_like(x), torch.randn(C, device=dev())
        edx, edw = torch.empty(rows, C, device=dev()), dw.clone()
        nat().rmsnorm_bwd(dx, dw, dy, x, w, rstd, add)
        ref.rmsnorm_bwd(edx, edw, dy, x, w, er, add)
        close(dx, edx, name="rmsnorm dx")
        close(dw, edw, rtol=1e-3, atol=1e-3, name="rmsnorm dw")


def test_rmsnorm_bwd_deterministic_and_many_rows():
    torch.manual_seed(8)
    rows, C = 4096, 768
    x, dy, w = rnd(rows, C), rnd(rows, C), rnd(C)
    rstd = torch.rand(rows, device=dev()) + 0.5
    res = []
    for _ in range(2):
        dx, dw = torch.empty_like(x), torch.zeros(C, device=dev())
        nat().rmsnorm_bwd(dx, dw, dy, x, w, rstd, None)
        res.append((dx.clone(), dw.clone()))
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])
    edx, edw = torch.empty(rows, C, device=dev()), torch.zeros(C, device=dev())
    ref.rmsnorm_bwd(edx, edw, dy, x, w, rstd, None)
    close(res[0][1], edw, rtol=2e-3, atol=1e-2, name="dw many rows")


@pytest.mark.parametrize("B,T,H,hd", [(2, 64, 4, 32), (1, 128, 12, 64), (2, 32, 2, 128), (1, 16, 3, 6)])
def test_rope(B, T, H, hd):
    torch.manual_seed(9)
    C = H * hd
    cos, sin = ref.rope_tables(T, hd, 10000.0, dev())
    qkv = rnd(B * T, 3 * C)
    a, e = qkv.clone(), qkv.clone()
    nat().rope_fwd(a, cos, sin, B, T, H, hd)
    ref.rope_fwd(e, cos, sin, B, T, H, hd)
    close(a, e, name="rope fwd")
    nat().rope_bwd(a, cos, sin, B, T, H, hd)
    close(a, qkv, rtol=2e-2, atol=3e-2, name="rope round trip")


@pytest.mark.parametrize("rows,I", [(64, 2048), (10, 192), (7, 100)])
def test_swiglu(rows, I):
    torch.manual_seed(10)
    gu, d = rnd(rows, 2 * I, scale=2.0), rnd(rows, I)
    out, eo = torch.empty(rows, I, device=dev(), dtype=torch.bfloat16), torch.empty(rows, I, device=dev())
    nat().swiglu_fwd(out, gu)
    ref.swiglu_fwd(eo, gu)
    close(out, eo, name="swiglu fwd")
    dgu, edgu = torch.empty_like(gu), torch.empty(rows, 2 * I, device=dev())
    nat().swiglu_bwd(dgu, d, gu)
    ref.swiglu_bwd(edgu, d, gu)
    close(dgu, edgu, name="swiglu bwd")


@pytest.mark.parametrize("smem_row", [1, 0], ids=["row_in_smem", "two_pass"])
def test_token_ids_outside_the_vocabulary_are_reported_not_followed(smem_row):
    """A token id or a target >= V (a token file made with a larger vocabulary) must not become an address: the kernels
    check the index first, give such a row zeros / no gradient / loss 0, and record MLB_ERR_BOUNDS with the kernel's tag
    in the error word; every other row is computed as usual."""
    torch.manual_seed(17)
    B, T, C, V = 2, 16, 96, 56
    bounds = lambda tag: (3 << 24) | tag
    wte = rnd(V, C)
    ids = torch.randint(0, V, (B * T,), device=dev(), dtype=torch.int32)
    bad = torch.tensor([5, 20], device=dev())
    ids[5], ids[20] = V + 5, -3
    good = torch.ones(B * T, dtype=torch.bool, device=dev())
    good[bad] = False
    assert nat().get_error() == 0
    out = torch.full((B * T, C), 7.0, device=dev(), dtype=torch.bfloat16)
    nat().embed_fwd(out, wte, ids)
    torch.cuda.synchronize()
    assert nat().get_error() == bounds(0xE1)
    nat().clear_error()
    assert torch.equal(out[good], wte[ids[good].long()]) and (out[bad] == 0).all()
    d = rnd(B * T, C)
    dw, edw = torch.zeros(V, C, device=dev()), torch.zeros(V, C, device=dev())
    nat().embed_bwd(dw, d, ids, T, 0)
    torch.cuda.synchronize()
    assert nat().get_error() == bounds(0xE2)
    nat().clear_error()
    edw.index_add_(0, ids[good].long(), d[good].float())
    close(dw, edw, rtol=1e-4, atol=1e-4, name="embed bwd, bad rows dropped")
    rows = 12
    logits = rnd(rows, V, scale=3.0)
    tgt = torch.randint(0, V, (rows,), device=dev(), dtype=torch.int32)
    tgt[3] = V + 7
    a, la = logits.clone(), torch.full((rows,), 9.0, device=dev())
    nat().lib().mlb_ce_mode(smem_row)
    try:
        nat().ce_fwd_bwd(la, a, tgt, 0.25)
        torch.cuda.synchronize()
    finally:
        nat().lib().mlb_ce_mode(0)
    assert nat().get_error() == bounds(0xCE)
    nat().clear_error()
    ok = tgt < V
    e, le = logits.float().clone(), torch.empty(rows, device=dev())
    ref.ce_fwd_bwd(le, e, torch.where(ok, tgt, torch.full_like(tgt, -1)), 0.25)
    close(la, le, rtol=1e-3, atol=1e-3, name="ce loss with one bad target")
    close(a, e, rtol=2e-2, atol=1e-4, name="dlogits with one bad target")
    assert la[3] == 0 and (a[3] == 0).all()


@pytest.mark.parametrize("rows,V", [(64, 50304), (16, 512), (9, 1001)])
@pytest.mark.parametrize("smem_row", [1, 0], ids=["row_in_smem", "two_pass"])
def test_cross_entropy(rows, V, smem_row):
    """Two kernels: the row parked in shared memory (one exponential per logit; needs V % 8 == 0), or two passes over
    global memory."""
    nat().lib().mlb_ce_mode(smem_row)
    try:
        _check_cross_entropy(rows, V)
    finally:
        nat().lib().mlb_ce_mode(0)


def _check_cross_entropy(rows, V):
    torch.manual_seed(11)
    logits = rnd(rows, V, scale=3.0)
    tgt = torch.randint(0, V, (rows,), device=dev(), dtype=torch.int32)
    tgt[::4] = -1
    dscale = 1.0 / 37
    a, e = logits.clone(), logits.float().clone()
    la, le = torch.empty(rows, device=dev()), torch.empty(rows, device=dev())
    nat().ce_fwd_bwd(la, a, tgt, dscale)
    ref.ce_fwd_bwd(le, e, tgt, dscale)
    close(la, le, rtol=1e-3, atol=1e-3, name="ce loss")
    close(a, e, rtol=2e-2, atol=1e-4, name="dlogits")
    assert (a[::4] == 0).all() and (la[::4] == 0).all()


@pytest.mark.parametrize("rows,V,chunk", [(64, 1024, 256), (37, 1000, 384), (5, 130, 130), (33, 257, 64)])
def test_cross_entropy_over_vocabulary_chunks(rows, V, chunk):
    """ce_chunk_stats / ce_chunk_grad (the LM head without a [rows, V] logits buffer) against the fp32 oracle of the same
    two ops, and against the fused whole-row cross-entropy: widths that divide V and that do not, ignored rows."""
    torch.manual_seed(13)
    logits = rnd(rows, V, scale=3.0)
    tgt = torch.randint(0, V, (rows,), device=dev(), dtype=torch.int32)
    tgt[::4] = -1
    dscale = 1.0 / 29
    mk = lambda: (torch.full((rows,), float("-inf"), device=dev()), torch.zeros(rows, device=dev()), torch.zeros(rows, device=dev()))
    m, s, zt = mk()
    em, es, ezt = mk()
    for off in range(0, V, chunk):
        c = logits[:, off:off + chunk].clone()     # (a full-width slice is the tensor itself)
        nat().ce_chunk_stats(m, s, zt, c, tgt, off)
        ref.ce_chunk_stats(em, es, ezt, c.float(), tgt, off)
    v = tgt >= 0
    close(m[v], em[v], rtol=0, atol=0, name="row max")
    close(s[v], es[v], rtol=1e-3, atol=1e-4, name="row sum")
    close(zt[v], ezt[v], rtol=0, atol=0, name="target logit")
    la, d = torch.empty(rows, device=dev()), torch.empty_like(logits)
    for off in range(0, V, chunk):
        c = logits[:, off:off + chunk].clone()     # (a full-width slice is the tensor itself)
        nat().ce_chunk_grad(la, c, tgt, m, s, zt, off, dscale)
        d[:, off:off + chunk] = c
    e, le = logits.float().clone(), torch.empty(rows, device=dev())
    ref.ce_fwd_bwd(le, e, tgt, dscale)
    close(la, le, rtol=1e-3, atol=1e-3, name="chunked ce loss")
    close(d, e, rtol=2e-2, atol=1e-4, name="chunked dlogits")
    assert (d[::4] == 0).all() and (la[::4] == 0).all()


@pytest.mark.parametrize("scale", [1.0, 8.0, 0.37])
def test_e4m3_rounding_kernel(scale):
    """fp8_qdq against the oracle (torch's float8_e4m3fn conversion after the same saturation): normal range,
    subnormals, saturation, zeros, both signs."""
    torch.manual_seed(14)
    x = torch.cat([rnd(4096, scale=1.0), rnd(2048, scale=300.0), rnd(2048, scale=2e-3),
                   torch.tensor([0.0, -0.0, 448.0, -448.0, 1e4, -1e4, 2.0 ** -9, 2.0 ** -10], device=dev()).bfloat16()])
    out = torch.empty_like(x)
    nat().fp8_qdq(out, x, scale)
    exp = torch.empty(x.numel(), device=dev())
    ref.fp8_qdq(exp, x, scale)
    # the kernel's result is rounded to bf16; with a power-of-two scale that is exact
    close(out, exp.bfloat16(), rtol=0 if scale in (1.0, 8.0) else 8e-3, atol=0 if scale in (1.0, 8.0) else 1e-6, name="e4m3 rounding")


@pytest.mark.parametrize("n", [4096 * 3, 1001])
def test_adamw(n):
    torch.manual_seed(12)
    master = torch.randn(n, device=dev())
    g = torch.randn(n, device=dev())
    m, v = torch.rand(n, device=dev()) * 0.1, torch.rand(n, device=dev()) * 0.01
    p = torch.empty(n, device=dev(), dtype=torch.bfloat16)
    em, emm, ev = master.clone(), m.clone(), v.clone()
    args = (1e-3, 0.9, 0.95, 1e-8, 0.1, 1 - 0.9 ** 3, 1 - 0.95 ** 3, 0.25)
    nat().adamw(master, p, g, m, v, *args)
    ref.adamw(em, None, g, emm, ev, *args)
    close(master, em, rtol=1e-5, atol=1e-6, name="adamw master")
    close(m, emm, rtol=1e-5, atol=1e-7, name="adamw m")
    close(v, ev, rtol=1e-5, atol=1e-7, name="adamw v")
    assert torch.equal(p, master.to(torch.bfloat16))


def test_embedding_and_prefix():
    torch.manual_seed(13)
    B, T, C, V, n_pre = 2, 16, 96, 50, 4
    wte = rnd(V, C)
    ids = torch.randint(0, V, (B * T,), device=dev(), dtype=torch.int32)
    out = torch.empty(B * T, C, device=dev(), dtype=torch.bfloat16)
    nat().embed_fwd(out, wte, ids)
    assert torch.equal(out, wte[ids.long()])
    prefix = rnd(B * n_pre, C)
    nat().set_prefix(out, prefix, B, T, n_pre)
    assert torch.equal(out.view(B, T, C)[:, :n_pre], prefix.view(B, n_pre, C))
    d = rnd(B * T, C)
    dw, edw = torch.zeros(V, C, device=dev()), torch.zeros(V, C, device=dev())
    nat().embed_bwd(dw, d, ids, T, n_pre)
    ref.embed_bwd(edw, d, ids, T, n_pre)
    close(dw, edw, rtol=1e-4, atol=1e-4, name="embed bwd")
    g = torch.empty(B * n_pre, C, device=dev(), dtype=torch.bfloat16)
    nat().gather_prefix_grad(g, d, B, T, n_pre)
    assert torch.equal(g.view(B, n_pre, C), d.view(B, T, C)[:, :n_pre])


@pytest.mark.parametrize("BT,C,shift", [(1, 8, 0), (5, 768, 0), (4098, 132, 0), (301, 102, 0), (9, 20, 0), (66, 128, 2), (7, 1, 0)])
def test_embedding_rows_and_widths(BT, C, shift):
    """Rows past the last whole block, widths of whole vectors or not, gradients from a place where vectors may not be loaded, prefix positions left out."""
    torch.manual_seed(BT + C)
    V, T, n_pre = 37, BT if BT % 3 else BT // 3, 0 if BT < 5 else 2
    wte, ids = rnd(V, C), torch.randint(0, V, (BT,), device=dev(), dtype=torch.int32)
    out = torch.full((BT + 1, C), 7.0, device=dev(), dtype=torch.bfloat16)
    nat().embed_fwd(out[:BT], wte, ids)
    assert torch.equal(out[:BT], wte[ids.long()]) and (out[BT] == 7).all()
    d, dw = rnd(BT * C + shift).view(-1)[shift:].view(BT, C), torch.ones(V, C, device=dev())
    nat().embed_bwd(dw, d, ids, T, n_pre)
    live = torch.arange(BT, device=dev()) % T >= n_pre
    e = torch.ones(V, C, device=dev(), dtype=torch.float64).index_add_(0, ids[live].long(), d[live].double())
    # at most BT additions in any order, each rounding a partial sum of at most 1 + sum |d|
    bound = BT * 2.0 ** -24 * torch.ones(V, C, device=dev(), dtype=torch.float64).index_add_(0, ids[live].long(), d[live].double().abs())
    assert ((dw - e).abs() <= bound).all()


# (forward a block per row: items >= 128 in up to 1184 rows and 2^21 elements; backward: 128 items in up to 1024 rows, 2048 of single additions)
@pytest.mark.parametrize("BT,C,shift", [(1, 768, 0), (1024, 512, 0), (1025, 512, 0), (1184, 1024, 0), (1185, 1024, 0), (1025, 2048, 0), (3, 4104, 0), (2048, 513, 0),
                                        (2049, 513, 0), (1024, 129, 0), (1025, 127, 0), (40, 1024, 1), (40, 1020, 2)])
def test_embedding_either_side_of_its_lines(BT, C, shift):
    """A warp and a block per row, whole and partial trips of four items a thread."""
    test_embedding_rows_and_widths(BT, C, shift)


def test_vision_helpers_and_casts():
    torch.manual_seed(14)
    B, g = 2, 3
    for P in (16, 8, 4):        # eight pixels per thread where the patch edge allows it, else one
        px = torch.randn(B, 3, g * P, g * P, device=dev())
        out = torch.empty(B * g * g, 3 * P * P, device=dev(), dtype=torch.bfloat16)
        e = torch.empty(B * g * g, 3 * P * P, device=dev())
        nat().patchify(out, px, P)
        ref.patchify(e, px, P)
        assert torch.equal(out, e.to(torch.bfloat16)), P
    NP, vC, n_patch = B * 9, 96, 9
    x, pos = rnd(NP, vC), rnd(n_patch, vC)
    a, ee = x.clone(), x.clone()
    nat().add_posembed(a, pos, n_patch)
    ref.add_posembed(ee, pos, n_patch)
    close(a, ee, name="posembed")
    dpos, edpos = torch.zeros(n_patch, vC, device=dev()), torch.zeros(n_patch, vC, device=dev())
    nat().posembed_grad(dpos, x, n_patch)
    ref.posembed_grad(edpos, x, n_patch)
    close(dpos, edpos, rtol=1e-4, atol=1e-4, name="posembed grad")
    r = torch.empty_like(x)
    nat().residual_add(r, x, a)
    close(r, x.float() + a.float(), name="residual")
    f = torch.randn(1003, device=dev())
    bb = torch.empty(1003, device=dev(), dtype=torch.bfloat16)
    nat().cast(bb, f)
    assert torch.equal(bb, f.to(torch.bfloat16))
    ff = torch.empty(1003, device=dev())
    nat().cast(ff, bb, 0.5)
    close(ff, bb.float() * 0.5, rtol=1e-6, atol=1e-6, name="cast back")


# ------------------------------------------------------------------ 8-bit forward (E4M3 storage + tcgen05 kind::f8f6f4)
def _e4m3(x_f32, scale):
    """torch's own E4M3 conversion after the kernels' saturation (+-448), as bytes."""
    return (x_f32 * scale).clamp(-448.0, 448.0).to(torch.float8_e4m3fn).view(torch.uint8)


def _bytes_close(a8, e8, max_flip_frac=2e-3):
    """Two E4M3 byte tensors: equal, except that a value computed in a different fp32 operation order may land on the
    neighbouring code (byte +-1); such flips must be rare."""
    a, e = a8.view(torch.int8).int(), e8.view(torch.int8).int()
    d = (a - e).abs()
    zero_signs = ((a8 & 0x7f) == 0) & ((e8 & 0x7f) == 0)          # +0 and -0 are the same value
    d = torch.where(zero_signs, torch.zeros_like(d), d)
    assert int(d.max()) <= 1, f"E4M3 codes differ by {int(d.max())}"
    assert float((d != 0).float().mean()) <= max_flip_frac, float((d != 0).float().mean())


@pytest.mark.parametrize("M,N,K", [(1024, 2304, 768), (512, 768, 2048), (300, 520, 272), (4096, 1024, 256)])
def test_linear_fwd_fp8_against_dequantised_product(M, N, K):
    """E4M3 x E4M3 product on the tensor cores against the fp32 product of the same bytes read back as numbers."""
    torch.manual_seed(N)
    x, W = rnd(M, K), rnd(N, K, scale=0.05)
    sa, sw = 4.0, 64.0
    x8 = torch.empty(M, K, device=dev(), dtype=torch.uint8)
    W8 = torch.empty(N, K, device=dev(), dtype=torch.uint8)
    nat().cast_bf16_fp8(x8, x, sa)
    nat().cast_bf16_fp8(W8, W, sw)
    assert torch.equal(x8, _e4m3(x.float(), sa)) and torch.equal(W8, _e4m3(W.float(), sw))
    out = torch.full((M, N), float("nan"), device=dev(), dtype=torch.bfloat16)
    assert nat().linear_fwd_fp8(out, x8, W8, 1.0 / (sa * sw))
    exp = (x8.view(torch.float8_e4m3fn).float() @ W8.view(torch.float8_e4m3fn).float().t()) / (sa * sw)
    close(out, exp, name="fp8 linear")
    # and against the unquantised product: E4M3 keeps 3 mantissa bits, so a few percent in norm
    full = x.float() @ W.float().t()
    assert ((out.float() - full).norm() / full.norm()).item() < 0.06
    # shapes the 8-bit kernel does not take are declined without a launch
    assert not nat().linear_fwd_fp8(torch.empty(64, N, device=dev(), dtype=torch.bfloat16), x8[:64], W8, 1.0)


def test_linear_fwd_fp8_epilogues():
    """The 8-bit product with the rotary-embedding epilogue and with the SwiGLU epilogue, against the plain 8-bit
    product followed by the separate kernels."""
    torch.manual_seed(3)
    B, T, H, hd, I = 2, 256, 4, 64, 512
    C = H * hd
    M = B * T
    x8 = _e4m3(rnd(M, C).float(), 2.0)
    Wq8 = _e4m3(rnd(3 * C, C, scale=0.05).float(), 32.0)
    Wg8 = _e4m3(rnd(2 * I, C, scale=0.05).float(), 32.0)
    cos, sin = ref.rope_tables(T, hd, 10000.0, dev())
    plain = torch.empty(M, 3 * C, device=dev(), dtype=torch.bfloat16)
    assert nat().linear_fwd_fp8(plain, x8, Wq8, 1 / 64.0)
    roped = torch.empty_like(plain)
    assert nat().linear_fwd_fp8_rope(roped, x8, Wq8, 1 / 64.0, cos, sin, T, 2 * C)
    nat().rope_fwd(plain, cos, sin, B, T, H, hd)
    close(roped, plain.float(), name="fp8 qkv + rope", fro=6e-3)      # rotation of fp32 accumulators vs of bf16 outputs
    gu = torch.empty(M, 2 * I, device=dev(), dtype=torch.bfloat16)
    assert nat().linear_fwd_fp8(gu, x8, Wg8, 1 / 64.0)
    gu2, sw2 = torch.empty_like(gu), torch.empty(M, I, device=dev(), dtype=torch.bfloat16)
    assert nat().linear_fwd_fp8_swiglu(gu2, sw2, x8, Wg8, 1 / 64.0)
    assert torch.equal(gu2, gu)
    sw = torch.empty_like(sw2)
    nat().swiglu_fwd(sw, gu)
    assert torch.equal(sw2, sw)


@pytest.mark.parametrize("rows,C", [(512, 768), (100, 264), (33, 100)])
def test_fp8_producers_write_e4m3_copies(rows, C):
    """Norms / SwiGLU / AdamW with an additional E4M3 output: the bf16 outputs equal the plain kernels', the bytes equal
    torch's conversion of the fp32 values (up to rare neighbouring-code flips)."""
    torch.manual_seed(rows)
    x, b, w = rnd(rows, C), rnd(rows, C), rnd(C, scale=0.2) + 1.0
    sa = 8.0
    out, rstd = torch.empty_like(x), torch.empty(rows, device=dev())
    out2, rstd2, out8 = torch.empty_like(x), torch.empty(rows, device=dev()), torch.empty(rows, C, device=dev(), dtype=torch.uint8)
    nat().rmsnorm_fwd(out, rstd, x, w, 1e-5)
    nat().rmsnorm_fwd_fp8(out2, out8, rstd2, x, w, 1e-5, sa)
    assert torch.equal(out, out2) and torch.equal(rstd, rstd2)
    y = x.float() * torch.rsqrt(x.float().pow(2).mean(-1, keepdim=True) + 1e-5) * w.float()
    _bytes_close(out8, _e4m3(y, sa))
    res, res2 = torch.empty_like(x), torch.empty_like(x)
    nat().add_rmsnorm_fwd(res, out, rstd, x, b, w, 1e-5)
    nat().add_rmsnorm_fwd_fp8(res2, out2, out8, rstd2, x, b, w, 1e-5, sa)
    assert torch.equal(out, out2) and torch.equal(res, res2)
    s = x.float() + b.float()
    _bytes_close(out8, _e4m3(s * torch.rsqrt(s.pow(2).mean(-1, keepdim=True) + 1e-5) * w.float(), sa))
    if C % 8 == 0:
        I = C
        gu = rnd(rows, 2 * I)
        sw, sw2, sw8 = torch.empty(rows, I, device=dev(), dtype=torch.bfloat16), torch.empty(rows, I, device=dev(), dtype=torch.bfloat16), \
            torch.empty(rows, I, device=dev(), dtype=torch.uint8)
        nat().swiglu_fwd(sw, gu)
        nat().swiglu_fwd_fp8(sw2, sw8, gu, sa)
        assert torch.equal(sw, sw2)
        g, u = gu[:, :I].float(), gu[:, I:].float()
        _bytes_close(sw8, _e4m3(g * torch.sigmoid(g) * u, sa), max_flip_frac=2e-2)     # __expf vs torch's sigmoid
    n = rows * C
    master, grads = torch.randn(n, device=dev()) * 0.02, torch.randn(n, device=dev()) * 1e-3
    m, v = torch.zeros(n, device=dev()), torch.zeros(n, device=dev())
    m2, v2, master2 = m.clone(), v.clone(), master.clone()
    p, p2, p8 = torch.empty(n, device=dev(), dtype=torch.bfloat16), torch.empty(n, device=dev(), dtype=torch.bfloat16), \
        torch.empty(n, device=dev(), dtype=torch.uint8)
    nat().adamw(master, p, grads, m, v, 1e-3, 0.9, 0.95, 1e-8, 0.1, 0.1, 0.05)
    nat().adamw_fp8(master2, p2, p8, grads, m2, v2, 1e-3, 0.9, 0.95, 1e-8, 0.1, 0.1, 0.05, 1.0, 32.0)
    assert torch.equal(master, master2) and torch.equal(p, p2) and torch.equal(m, m2) and torch.equal(v, v2)
    assert torch.equal(p8, _e4m3(master2, 32.0))


# ------------------------------------------------------------------ LayerNorm, bidirectional attention (vision encoder)
@pytest.mark.parametrize("rows,C", [(1000, 768), (37, 100), (8, 2048)])
def test_layernorm_fwd_bwd(rows, C):
    torch.manual_seed(rows)
    x, w, b, dy = rnd(rows, C), rnd(C, scale=0.3) + 1.0, rnd(C, scale=0.2), rnd(rows, C)
    out, mean, rstd = torch.empty_like(x), torch.empty(rows, device=dev()), torch.empty(rows, device=dev())
    nat().layernorm_fwd(out, mean, rstd, x, w, b, 1e-5)
    eo, em, er = torch.empty(rows, C, device=dev()), torch.empty(rows, device=dev()), torch.empty(rows, device=dev())
    ref.layernorm_fwd(eo, em, er, x, w, b, 1e-5)
    close(out, eo, name="layernorm out")
    close(mean, em, rtol=1e-4, atol=1e-5, name="mean")
    close(rstd, er, rtol=1e-4, atol=1e-5, name="rstd")
    dx = torch.empty_like(x)
    dw, db = torch.zeros(C, device=dev()), torch.zeros(C, device=dev())
    nat().layernorm_bwd(dx, dw, db, dy, x, w, mean, rstd)
    edx, edw, edb = torch.empty(rows, C, device=dev()), torch.zeros(C, device=dev()), torch.zeros(C, device=dev())
    ref.layernorm_bwd(edx, edw, edb, dy, x, w, em, er)
    close(dx, edx, name="layernorm dx", fro=6e-3)
    close(dw, edw, rtol=1e-3, atol=1e-3, name="layernorm dw")
    close(db, edb, rtol=1e-3, atol=1e-3, name="layernorm db")


@pytest.mark.parametrize("B,T,H,hd", [(2, 197, 4, 64), (3, 50, 2, 32), (1, 17, 3, 24)])
def test_bidirectional_attention_fwd_bwd(B, T, H, hd):
    torch.manual_seed(T)
    C = H * hd
    qkv, dout = rnd(B * T, 3 * C), rnd(B * T, C)
    out, lse = torch.empty(B * T, C, device=dev(), dtype=torch.bfloat16), torch.empty(B, H, T, device=dev())
    nat().attn_bidir_fwd(out, lse, qkv, B, T, H, hd)
    eo, el = torch.empty(B * T, C, device=dev()), torch.empty(B, H, T, device=dev())
    ref.attn_bidir_fwd(eo, el, qkv, B, T, H, hd)
    close(out, eo, name="bidir attn out")
    close(lse, el, rtol=1e-3, atol=2e-2, name="bidir lse")
    dqkv = torch.empty_like(qkv)
    nat().attn_bidir_bwd(dqkv, dout, qkv, out, lse, B, T, H, hd)
    e = torch.empty(B * T, 3 * C, device=dev())
    ref.attn_bidir_bwd(e, dout, qkv, eo, el, B, T, H, hd)
    close(dqkv, e, rtol=3e-2, atol=3e-2, name="bidir dqkv", fro=1.5e-2)


def test_vit_encoder_gpu_against_cpu():
    from ml_b200.models.vit import ViTEncoder
    torch.manual_seed(2)
    cpu = ViTEncoder(image_size=64, patch=16, C=128, L=2, H=2, I=256, out_dim=96, device="cpu")
    gpu = ViTEncoder(image_size=64, patch=16, C=128, L=2, H=2, I=256, out_dim=96, device="cuda:0")
    with torch.no_grad():
        for (n, p), (_, q) in zip(cpu.named_parameters(), gpu.named_parameters()):
            q.copy_(p.to(q.dtype))
    px = torch.randn(4, 3, 64, 64)
    oc = cpu(px)
    og = gpu(px.cuda())
    oc.square().sum().backward()
    og.float().square().sum().backward()
    assert ((og.float().cpu() - oc).norm() / oc.norm()).item() < 3e-2
    for (n, p), (_, q) in zip(cpu.named_parameters(), gpu.named_parameters()):
        d = (q.grad.float().cpu() - p.grad).norm() / (p.grad.norm() + 1e-8)
        assert d.item() < 8e-2, (n, d.item())


def test_gemm_autotune_plan_cache():
    """Autotune on: the first call of a shape times this library's forms and caches a plan, later calls reuse it; every
    form computes the same product (bf16 outputs within rounding of each other, the add-reduce form really adds once)."""
    torch.manual_seed(5)
    M, N, K = 1024, 768, 512
    x, W, dy = rnd(M, K), rnd(N, K, scale=K ** -0.5), rnd(M, N)
    base, dW0 = torch.empty(M, N, device=dev(), dtype=torch.bfloat16), torch.ones(N, K, device=dev())
    nat().linear_fwd(base, x, W)
    nat().linear_dw(dW0, dy, x)
    n0 = len(nat().gemm_plans())
    nat().gemm_autotune(True)
    try:
        out, dW = torch.empty_like(base), torch.ones(N, K, device=dev())
        nat().linear_fwd(out, x, W)
        nat().linear_dw(dW, dy, x)              # tuned into a scratch output: the accumulator gets the product exactly once
        plans = nat().gemm_plans()
        assert len(plans) == n0 + 2
        nat().linear_fwd(out, x, W)
        assert len(nat().gemm_plans()) == n0 + 2
    finally:
        nat().gemm_autotune(False)
    e = torch.empty(M, N, device=dev())
    ref.linear_fwd(e, x, W)
    close(out, e, name="tuned forward")
    edw = torch.ones(N, K, device=dev())
    ref.linear_dw(edw, dy, x)
    close(dW, edw, rtol=2e-2, atol=2e-2, name="tuned dW")
    close(dW0, edw, rtol=2e-2, atol=2e-2, name="untuned dW")


@pytest.mark.parametrize("B,T,H,N", [(2, 256, 4, 256), (3, 200, 3, 192), (16, 1024, 12, 768)])
def test_linear_dx_delta_epilogue(B, T, H, N):
    """Input gradient of the attention output projection with delta = rowsum(dO * O) per head from its epilogue: the
    product against the fp32 oracle, delta against the fp32 row dots, and the attention backward fed with that delta
    against the one that runs its own pass over dO and O."""
    torch.manual_seed(B * T + H)
    C, hd, M = H * 64, 64, B * T
    dy, W = rnd(M, N), rnd(N, C, scale=N ** -0.5)
    qkv = rnd(M, 3 * C)
    out = torch.empty(M, C, device=dev(), dtype=torch.bfloat16)
    lse = torch.empty(B, H, T, device=dev())
    nat().attn_fwd(out, lse, qkv, B, T, H, hd)
    dx = torch.full((M, C), float("nan"), device=dev(), dtype=torch.bfloat16)
    assert nat().linear_dx_delta(dx, dy, W, out, B, T, H)
    e = torch.empty(M, C, device=dev())
    ref.linear_dx(e, dy, W)
    close(dx, e, name="dx")
    delta = nat().scratch("attn_delta", B * H * T, torch.float32, torch.device(dev()))[:B * H * T].view(B, H, T).clone()
    ed = (e.view(B, T, H, 64) * out.float().view(B, T, H, 64)).sum(-1).permute(0, 2, 1)
    close(delta, ed, rtol=1e-2, atol=1e-2, name="delta", fro=5e-3)
    a = torch.empty(M, 3 * C, device=dev(), dtype=torch.bfloat16)
    b = torch.empty_like(a)
    nat().attn_bwd(a, dx, qkv, out, lse, B, T, H, hd, have_delta=True)
    nat().attn_bwd(b, dx, qkv, out, lse, B, T, H, hd)
    close(a, b.float(), name="attention backward with the epilogue's delta", fro=6e-3)


def _attn64(qkv, dout, B, T, H, hd, causal):
    """out, lse, dqkv of plain attention in 64 bits."""
    x = qkv.double().view(B, T, 3, H, hd).permute(2, 0, 3, 1, 4).contiguous().requires_grad_(True)
    s = x[0] @ x[1].transpose(-1, -2) / hd ** 0.5
    if causal:
        s = s.masked_fill(torch.ones(T, T, dtype=torch.bool, device=s.device).triu(1), float("-inf"))
    out = (torch.softmax(s, -1) @ x[2]).transpose(1, 2).reshape(B * T, H * hd)
    (g,) = torch.autograd.grad(out, x, dout.double())
    return out.detach(), torch.logsumexp(s, -1).detach(), g.permute(1, 3, 0, 2, 4).reshape(B * T, 3 * H * hd)


def _attn_bwd_bound64(qkv, dout, B, T, H, hd):
    """How far each element of causal attention's dqkv may be from 64 bits before its last rounding.  Rounding to bf16 costs 2^-9 of a value, twice that is
    allowed for what is not written out (exponentials, sums in 32 bits).  P is rounded for dV, dS for dQ and dK, dQ's partial sums once more; the forward's P
    is cut off (2^-7), and what that and its rounding do to O reaches dS through delta = rowsum(dO O)."""
    q, k, v = qkv.double().view(B, T, 3, H, hd).permute(2, 0, 3, 1, 4)
    g = dout.double().view(B, T, H, hd).transpose(1, 2)
    sc = hd ** -0.5
    P = torch.softmax((q @ k.transpose(-1, -2) * sc).masked_fill(torch.ones(T, T, dtype=torch.bool, device=q.device).triu(1), float("-inf")), -1)
    O = P @ v
    dS = P * (g @ v.transpose(-1, -2) - (g * O).sum(-1, keepdim=True))
    d_delta = (g.abs() * (2 ** -7 * (P @ v.abs()) + 2 ** -8 * O.abs())).sum(-1, keepdim=True)
    E = 2 ** -8 * dS.abs() + P * d_delta
    bq = sc * (E + 2 ** -8 * dS.abs()) @ k.abs()
    bk = sc * E.transpose(-1, -2) @ q.abs()
    bv = 2 ** -8 * P.transpose(-1, -2) @ g.abs()
    return torch.stack((bq, bk, bv)).permute(1, 3, 0, 2, 4).reshape(B * T, 3 * H * hd).contiguous()


def _rel(a, e):
    return ((a.double() - e).norm() / e.norm()).item()


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("T,hd", [(1, 16), (17, 32), (63, 64), (64, 48), (65, 64), (127, 128), (128, 16), (129, 80), (197, 64), (257, 32), (321, 112)])
def test_attention_with_split_probabilities(T, hd, causal):
    """Edges of the 128-row tiles and 64-row blocks and every padded head size.  Results are rounded to bf16 once (at most 2^-9
    per element), P and dS carry 2^-17; delta comes from the bf16 output, whose rounding adds up to 2^-9 of the delta term."""
    if causal and hd in (64, 128):
        pytest.skip("those head sizes have their own causal kernels")
    torch.manual_seed(T * 131 + hd)
    B, H = 2, 3
    qkv, dout = rnd(B * T, 3 * H * hd), rnd(B * T, H * hd)
    out, lse, dqkv = rnd(B * T, H * hd), torch.empty(B, H, T, device=dev()), torch.zeros(B * T, 3 * H * hd, device=dev(), dtype=torch.bfloat16)
    n = nat()
    if causal:
        n.attn_fwd(out, lse, qkv, B, T, H, hd)
        assert n.attn_bwd(dqkv, dout, qkv, out, lse, B, T, H, hd) is False
    else:
        n.attn_bidir_fwd(out, lse, qkv, B, T, H, hd)
        n.attn_bidir_bwd(dqkv, dout, qkv, out, lse, B, T, H, hd)
    eo, el, ed = _attn64(qkv, dout, B, T, H, hd, causal)
    assert _rel(out, eo) < 2 ** -9 and _rel(lse, el) < 1e-6
    if T > 1:
        assert _rel(dqkv, ed) < 2 ** -8
    # a sample full of infinities leaves its neighbour alone (its rows lie right behind the other's last, partial block)
    qkv2 = qkv.clone()
    qkv2[T:] = float("inf")
    out2 = torch.empty_like(out)
    (n.attn_fwd if causal else n.attn_bidir_fwd)(out2, lse, qkv2, B, T, H, hd)
    assert torch.equal(out2[:T], out[:T])


@pytest.mark.parametrize("B,T,H", [(2, 1, 3), (2, 64, 1), (1, 128, 2), (2, 130, 3), (1, 257, 2), (2, 384, 2), (1, 640, 3), (12, 384, 16), (1, 2048, 2)])
def test_causal_attention_head_size_128(B, T, H):
    """One and two query tiles per pair, partial tiles, few items and more items than SMs.  P and the result are bf16 (at most 2^-9 per
    element each): below 2^-8.  In backward dS is, and it carries the rounding of O through delta besides: twice that."""
    torch.manual_seed(T + 7 * B)
    hd = 128
    qkv, dout = rnd(B * T, 3 * H * hd), rnd(B * T, H * hd)
    out, lse, dqkv = rnd(B * T, H * hd), torch.empty(B, H, T, device=dev()), torch.zeros(B * T, 3 * H * hd, device=dev(), dtype=torch.bfloat16)
    n = nat()
    n.attn_fwd(out, lse, qkv, B, T, H, hd)
    n.attn_bwd(dqkv, dout, qkv, out, lse, B, T, H, hd)
    eo, el, ed = _attn64(qkv, dout, B, T, H, hd, True)
    assert _rel(out, eo) < 2 ** -8 and _rel(lse, el) < 1e-6
    assert _rel(dqkv, ed) < 2 ** -7
    again = torch.empty_like(dqkv)
    n.attn_bwd(again, dout, qkv, out, lse, B, T, H, hd)
    assert torch.equal(again, dqkv)
    # scores that grow along the keys: the running maximum is passed again and again
    qkv.view(B, T, 3, H, hd)[:, :, 1] *= torch.linspace(0.1, 8, T, device=dev()).bfloat16().view(1, T, 1, 1)
    n.attn_fwd(out, lse, qkv, B, T, H, hd)
    eo, el, _ = _attn64(qkv, dout, B, T, H, hd, True)
    assert _rel(out, eo) < 2 ** -8 and _rel(lse, el) < 1e-6


@pytest.mark.parametrize("rows,V", [(1, 8), (5, 1001), (300, 512), (33, 50304)])
def test_ce_mean_and_scale(rows, V):
    torch.manual_seed(rows)
    logits = rnd(rows, V, scale=2.0)
    keep = logits.clone()
    tgt = torch.randint(0, V, (rows,), device=dev(), dtype=torch.int32)
    if rows > 2:
        tgt[1] = -1
    loss, losses, d = torch.empty((), device=dev()), torch.empty(rows, device=dev()), torch.empty_like(logits)
    nat().ce_mean(loss, losses, d, logits, tgt)
    assert torch.equal(logits, keep)
    z = logits.double().requires_grad_(True)
    e = torch.nn.functional.cross_entropy(z, tgt.long(), ignore_index=-1)
    (g,) = torch.autograd.grad(e, z)
    assert abs(loss.item() - e.item()) < 1e-5 * max(1.0, e.item())
    assert _rel(d, g) < 2 ** -8
    l2 = torch.empty_like(loss)
    nat().ce_mean(l2, losses, None, logits, tgt)
    assert torch.equal(l2, loss)
    s = torch.tensor(0.37, device=dev())
    nat().scale_dev(logits, d, s)
    assert torch.equal(logits, (d.float() * s).bfloat16())
    view = rnd(rows * V + 1, 1)[1:].view(rows, V)      # rows that start two bytes off a 16-byte boundary
    nat().ce_mean(loss, losses, d, view, tgt)
    assert abs(loss.item() - torch.nn.functional.cross_entropy(view.double(), tgt.long(), ignore_index=-1).item()) < 1e-4


@pytest.mark.parametrize("B,T,H,Hkv,hd", [(2, 65, 4, 2, 64), (1, 33, 6, 1, 32), (2, 17, 3, 3, 128), (1, 9, 4, 2, 24)])
def test_rope_copy_with_grouped_heads(B, T, H, Hkv, hd):
    torch.manual_seed(hd)
    x = rnd(B * T, (H + 2 * Hkv) * hd)
    cos, sin = ref.rope_tables(T, hd, 10000.0, dev())
    out, e = rnd(B * T, 3 * H * hd), torch.empty(B * T, 3 * H * hd, device=dev())
    nat().rope_copy(out, x, cos, sin, B, T, H, hd, Hkv)
    ref.rope_copy(e, x, cos, sin, B, T, H, hd, Hkv)
    assert _rel(out, e.double()) < 2 ** -9
    back, eb = torch.empty_like(x), torch.empty_like(x)
    nat().kv_group_sum(back, out, B, T, H, hd, Hkv)
    ref.kv_group_sum(eb, out, B, T, H, hd, Hkv)
    assert _rel(back, eb.double()) < 2 ** -8      # (the two round the same sums, in another order)


@pytest.mark.parametrize("M,N,K", [(64, 96, 64), (200, 264, 136), (1003, 768, 768), (3000, 2304, 256), (50, 1024, 2048)])
def test_linear_bias_dw_cast(M, N, K):
    torch.manual_seed(M)
    x, W, b, d = rnd(M, K), rnd(N, K, scale=0.1), rnd(N), rnd(M, N)
    out, dW = rnd(M, N), rnd(N, K)
    nat().linear_bias_fwd(out, x, W, b)
    assert _rel(out, x.double() @ W.double().T + b.double()) < 2 ** -8      # twice rounded where the epilogue does not take the shape
    nat().linear_dw_cast(dW, d, x)
    assert _rel(dW, d.double().T @ x.double()) < 2 ** -9


def test_first_call_of_a_thread_may_be_a_product():
    """A worker thread whose memory comes out of the allocator's cache has no context bound when it asks for a tensor map."""
    import threading
    x, W, out = rnd(136, 72), rnd(200, 72), rnd(136, 200)
    torch.cuda.synchronize()
    errs = []

    def work():
        try:
            nat().linear_fwd(out, x, W)
        except Exception as e:      # noqa: BLE001
            errs.append(e)
    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert not errs, errs
    assert _rel(out, x.double() @ W.double().T) < 2 ** -9


@pytest.mark.parametrize("M,N", [(1, 8), (64, 96), (200, 264), (1003, 768), (3000, 2304), (50, 1024)])
def test_colsum(M, N):
    torch.manual_seed(M)
    d, db = rnd(M, N), rnd(N)
    nat().colsum(db, d)
    assert _rel(db, d.double().sum(0)) < 2 ** -8


@pytest.mark.parametrize("rows,C", [(1, 256), (7, 768), (100, 1024), (37, 1536), (1000, 2048), (9, 100)])
def test_norm_backward_with_cast_column_sums(rows, C):
    torch.manual_seed(rows)
    x, dy, add, w, b = rnd(rows, C), rnd(rows, C), rnd(rows, C), 1 + rnd(C, scale=0.1), rnd(C)
    o, mean, rstd, dx, dw, db = torch.empty_like(x), *(torch.empty(rows, device=dev()) for _ in range(2)), torch.empty_like(x), rnd(C), rnd(C)
    xd, wd, bd = (t.double().requires_grad_(True) for t in (x, w, b))
    nat().rmsnorm_fwd(o, rstd, x, w, 1e-5)
    nat().rmsnorm_bwd_cast(dx, dw, dy, x, w, rstd, add)
    y = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-5) * wd
    gx, gw = torch.autograd.grad(y, [xd, wd], dy.double())
    assert _rel(dx, gx + add.double()) < 2 ** -8 and _rel(dw, gw) < 2 ** -8
    acc = torch.ones(C, device=dev())
    nat().rmsnorm_bwd(dx, acc, dy, x, w, rstd, None)
    assert _rel(dx, gx) < 2 ** -8 and _rel(acc - 1, gw) < 1e-4
    nat().layernorm_fwd(o, mean, rstd, x, w, b, 1e-5)
    nat().layernorm_bwd_cast(dx, dw, db, dy, x, w, mean, rstd)
    y = torch.nn.functional.layer_norm(xd, (C,), wd, bd, 1e-5)
    gx, gw, gb = torch.autograd.grad(y, [xd, wd, bd], dy.double())
    assert _rel(dx, gx) < 2 ** -8 and _rel(dw, gw) < 2 ** -8 and _rel(db, gb) < 2 ** -8


def test_attention_work_tables_are_bounded():
    """More shapes than tables are kept: results of a shape whose table was given back, and of a graph that holds one, stay the same.
    The first calls run on a stream of their own (its copy of the table is waited for)."""
    n, B, hd = nat(), 160, 64
    qkv = rnd(B * 300, 3 * hd)

    def run(T):
        out, lse = torch.empty(B * T, hd, device=dev(), dtype=torch.bfloat16), torch.empty(B, 1, T, device=dev())
        n.attn_fwd(out, lse, qkv[:B * T], B, T, 1, hd)
        return out, lse
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        first, _ = run(131)
    side.synchronize()
    assert _rel(first, _attn64(qkv[:B * 131], qkv[:B * 131, :hd], B, 131, 1, hd, True)[0]) < 2 ** -8
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        held, _ = run(131)
    run(132)
    for T in range(1, 300):
        run(T)
    assert 200 < n.lib().mlb_attn_schedule_count() <= 256
    graph.replay()
    assert torch.equal(held, first) and torch.equal(run(131)[0], first)
    assert torch.equal(run(132)[0], run(132)[0])


@pytest.mark.parametrize("T,H,hd", [(384, 6, 64), (384, 4, 128), (200, 6, 32)])
def test_backwards_on_two_streams_keep_apart(T, H, hd):
    """Attention and norm backward on two streams at once, from two threads: bit for bit what each gives alone."""
    import threading
    n, B, C = nat(), 4, H * hd
    torch.manual_seed(hd)
    W = rnd(C, C, scale=C ** -0.5)

    def work(seed, rounds, results):
        g = torch.Generator(device=dev()).manual_seed(seed)
        r = lambda *s: torch.randn(*s, generator=g, device=dev()).bfloat16()
        qkv, dy, x, w = r(B * T, 3 * C), r(B * T, C), r(B * T, 256), r(256)
        out, lse, rstd = torch.empty(B * T, C, device=dev(), dtype=torch.bfloat16), torch.empty(B, H, T, device=dev()), torch.rand(B * T, device=dev(), generator=g)
        n.attn_fwd(out, lse, qkv, B, T, H, hd)
        for _ in range(rounds):
            dqkv, dx, dw, d = torch.zeros_like(qkv), torch.empty_like(x), torch.zeros(256, device=dev()), torch.empty_like(out)
            have = hd == 64 and n.linear_dx_delta(d, dy, W, out, B, T, H)
            n.attn_bwd(dqkv, d if have else dy, qkv, out, lse, B, T, H, hd, have_delta=bool(have))
            n.rmsnorm_bwd(dx, dw, x, x, w, rstd)
            results.append((dqkv, dx, dw))
    alone = [[], []]
    for i in (0, 1):
        work(i, 1, alone[i])
    torch.cuda.synchronize()
    got = [[], []]

    def on_stream(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            work(i, 20, got[i])
            torch.cuda.current_stream().synchronize()
    threads = [threading.Thread(target=on_stream, args=(i,)) for i in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i in (0, 1):
        assert len(got[i]) == 20
        for r in got[i]:
            assert all(torch.equal(a, b) for a, b in zip(r, alone[i][0]))


def test_norm_backward_in_graphs_whose_first_one_never_ran():
    """The ticket of the one-launch norm backward is part of its graph: zero at every replay, whatever other graphs have done."""
    n, rows, C = nat(), 300, 768
    x, dy, w, rstd = rnd(rows, C), rnd(rows, C), rnd(C), torch.rand(rows, device=dev())
    e, dx = torch.zeros(C, device=dev()), torch.empty_like(x)
    n.rmsnorm_bwd(dx, e, dy, x, w, rstd)
    graphs, dws = [], []
    for _ in range(2):
        dw = torch.zeros(C, device=dev())
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            n.rmsnorm_bwd(dx, dw, dy, x, w, rstd)
        graphs.append(g)
        dws.append(dw)
    graphs[1].replay()
    n.rmsnorm_bwd(dx, dws[0], dy, x, w, rstd)
    assert torch.equal(dws[1], e) and torch.equal(dws[0], e)
    graphs[1].replay()
    assert torch.equal(dws[1], e + e)


@pytest.mark.parametrize("order", [0, 1, 2])
@pytest.mark.parametrize("M,N,K", [(2048, 2304, 2304), (2100, 2312, 2200), (2048, 1536, 9472), (2048, 2560, 5504), (4160, 2048, 2432)])
def test_linear_dw_whole_waves_then_shared_tiles(M, N, K, order):
    """Weight gradients of 76 to 222 tiles on 74 clusters: whole waves, then q tiles shared by q + 1 clusters (q = 1, 2), none
    left over (222), ragged rows, columns and reductions, both tile orders, and every tile cut up (the hook off).  Added to what
    is there, in fp32: products of bf16 are exact, sums of <= 4160 terms in any order are off by less than 4160 * 2^-24 of their
    terms' norm (1e-5 of the result here).  From zero, two runs agree bit for bit."""
    torch.manual_seed(N + K)
    n = nat()
    x, d = rnd(M, K), rnd(M, N)
    e = d.double().T @ x.double() + 1
    L = n.lib()
    try:
        L.mlb_gemm_tile_order(order)
        for whole in (1, 0):
            L.mlb_gemm_streamk_whole(whole)
            dW = torch.ones(N, K, device=dev())
            n.linear_dw(dW, d, x)
            assert _rel(dW, e) < 1e-5
            runs = [torch.zeros(N, K, device=dev()) for _ in range(3)]
            for r in runs:
                n.linear_dw(r, d, x)
            assert torch.equal(runs[0], runs[1]) and torch.equal(runs[0], runs[2])
    finally:
        L.mlb_gemm_tile_order(0)
        L.mlb_gemm_streamk_whole(1)


@pytest.mark.parametrize("B,T,H,Hkv,hd", [(2, 130, 4, 2, 64), (1, 257, 8, 2, 128), (2, 65, 6, 1, 32), (1, 40, 4, 2, 24)])
def test_grouped_heads_through_autograd(B, T, H, Hkv, hd):
    """Rotary embedding, repeated heads, attention and back, against 64 bits.  bf16: the rotated Q and K, P, dS and the result are rounded
    once each (2^-9 at most, and the rotated ones enter squared scores): below 2^-6."""
    from ml_b200.ops import autograd as F
    torch.manual_seed(T)
    cos, sin = ref.rope_tables(T, hd, 10000.0, dev())
    x = rnd(B * T, (H + 2 * Hkv) * hd).requires_grad_(True)
    dout = rnd(B * T, H * hd)
    out = F.rope_causal_attention(x, cos, sin, B, T, H, hd, Hkv)
    (g,) = torch.autograd.grad(out, x, dout)
    xd = x.detach().double().requires_grad_(True)
    q, k, v = xd.view(B, T, H + 2 * Hkv, hd).transpose(1, 2).split([H, Hkv, Hkv], 1)
    c, s = cos.double(), sin.double()
    rot = lambda t: torch.cat([t[..., :hd // 2] * c - t[..., hd // 2:] * s, t[..., hd // 2:] * c + t[..., :hd // 2] * s], -1)
    k, v = (t.repeat_interleave(H // Hkv, 1) for t in (rot(k), v))
    a = rot(q) @ k.transpose(-1, -2) / hd ** 0.5
    a = torch.softmax(a.masked_fill(torch.ones(T, T, dtype=torch.bool, device=dev()).triu(1), float("-inf")), -1)
    e = (a @ v).transpose(1, 2).reshape(B * T, H * hd)
    (eg,) = torch.autograd.grad(e, xd, dout.double())
    assert _rel(out, e) < 2 ** -6 and _rel(g, eg) < 2 ** -6
    with pytest.raises(ValueError):
        nat().rope_copy(torch.empty(B * T, 3 * H * hd, device=dev(), dtype=torch.bfloat16), x.detach(), cos, sin, B, T, H, hd, H + 1)


@pytest.mark.parametrize("T,spread", [(640, 4.0), (1000, 2.0)])
def test_causal_attention_128_rounds_no_row_maximum(T, spread):
    """P is rounded to bf16 against the maximum of the keys seen so far, so a row's largest probability is exact.  The same roundings
    in 64-bit torch (P per 128-key block, then the result) are as far from the unrounded result as the kernel's, to 3 %; with a
    maximum that may be stale the kernel is 11 to 13 % further off at these spreads of the scores."""
    torch.manual_seed(T)
    B, H, hd = 1, 6, 128
    qkv = torch.randn(T, 3 * H * hd, device=dev())
    qkv[:, :2 * H * hd] *= spread ** 0.5
    qkv = qkv.bfloat16()
    out, lse = torch.empty(T, H * hd, device=dev(), dtype=torch.bfloat16), torch.empty(B, H, T, device=dev())
    nat().attn_fwd(out, lse, qkv, B, T, H, hd)
    q, k, v = qkv.double().view(T, 3, H, hd).permute(1, 2, 0, 3)
    s = (q @ k.transpose(-1, -2) / hd ** 0.5).masked_fill(torch.ones(T, T, dtype=torch.bool, device=dev()).triu(1), float("-inf"))
    m, o, l = torch.full((H, T, 1), float("-inf"), device=dev(), dtype=torch.float64), 0.0, 0.0
    for j in range(0, T, 128):
        mn = torch.maximum(m, s[..., j:j + 128].amax(-1, keepdim=True))
        p, a = torch.exp(s[..., j:j + 128] - mn), torch.exp(m - mn)
        o, l, m = o * a + p.float().bfloat16().double() @ v[:, j:j + 128], l * a + p.sum(-1, keepdim=True), mn
    e = (torch.softmax(s, -1) @ v).transpose(0, 1).reshape(T, H * hd)
    same = (o / l).float().bfloat16().double().transpose(0, 1).reshape(T, H * hd)
    assert _rel(out, e) < 1.03 * _rel(same, e)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("T,hd", [(64, 32), (200, 48), (197, 64), (150, 112)])
@pytest.mark.parametrize("where,value", [("v", float("inf")), ("k", float("-inf")), ("q", float("inf")), ("dout", float("inf")), ("v", float("nan")),
                                         ("k", float("nan"))])
def test_split_attention_keeps_infinities_where_they_belong(causal, T, hd, where, value):
    """One non-finite value in one token's V, K, Q or dO: what it reaches and what it leaves alone (the rows that do not see it, under
    the causal mask) is what the scalar kernels give, NaN, infinite or finite."""
    if causal and hd == 64:
        pytest.skip("that head size has its own causal kernels")
    torch.manual_seed(T + hd)
    B, H, at = 2, 2, T - T // 4
    qkv, dout = rnd(B * T, 3 * H * hd), rnd(B * T, H * hd)
    if where == "dout":
        dout[T // 3, hd + 3] = value
    else:
        qkv.view(B, T, 3, H, hd)[0, at, "qkv".index(where), 1, 5] = value
    n = nat()

    def run():
        out, lse = rnd(B * T, H * hd), torch.empty(B, H, T, device=dev())
        dqkv = torch.zeros(B * T, 3 * H * hd, device=dev(), dtype=torch.bfloat16)
        if causal:
            n.attn_fwd(out, lse, qkv, B, T, H, hd)
            n.attn_bwd(dqkv, dout, qkv, out, lse, B, T, H, hd)
        else:
            n.attn_bidir_fwd(out, lse, qkv, B, T, H, hd)
            n.attn_bidir_bwd(dqkv, dout, qkv, out, lse, B, T, H, hd)
        return out, lse, dqkv
    got = run()
    n.lib().mlb_attn_force_simt(1)
    try:
        e = run()
    finally:
        n.lib().mlb_attn_force_simt(0)
    for a, b in zip(got, e):
        assert torch.equal(a.isnan(), b.isnan())
        assert torch.equal(a.isinf(), b.isinf()) and torch.equal(a[a.isinf()], b[b.isinf()])
        assert _rel(a[a.isfinite()], b[b.isfinite()].double()) < 2 ** -7
    if causal and where != "dout":
        assert got[0][:at].isfinite().all()


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("T,hd", [(513, 16), (577, 64), (260, 80), (400, 96), (577, 128)])
def test_split_attention_over_many_blocks(T, hd, causal):
    """Five to ten key blocks, at every padded head size: the products of the loop and of its prologue are separate code.  Bounds as for
    the short sequences: one rounding to bf16 (2^-9), the backward's delta another."""
    if causal and hd in (64, 128):
        pytest.skip("those head sizes have their own causal kernels")
    torch.manual_seed(T + hd)
    B, H, n = 2, 2, nat()
    qkv, dout = rnd(B * T, 3 * H * hd), rnd(B * T, H * hd)
    out, lse, dqkv = rnd(B * T, H * hd), torch.empty(B, H, T, device=dev()), torch.zeros(B * T, 3 * H * hd, device=dev(), dtype=torch.bfloat16)
    (n.attn_fwd if causal else n.attn_bidir_fwd)(out, lse, qkv, B, T, H, hd)
    (n.attn_bwd if causal else n.attn_bidir_bwd)(dqkv, dout, qkv, out, lse, B, T, H, hd)
    eo, el, ed = _attn64(qkv, dout, B, T, H, hd, causal)
    assert _rel(out, eo) < 2 ** -9 and _rel(lse, el) < 1e-6 and _rel(dqkv, ed) < 2 ** -8


@pytest.mark.parametrize("rows,V", [(1, 8), (37, 250), (300, 4104), (1200, 512)])
@pytest.mark.parametrize("factor", [1.0, 0.37])
def test_cross_entropy_gradient_in_place_and_not(rows, V, factor):
    """The saved gradient is scaled in place at its last use only: a kept graph, a pack hook that holds on to the tensor and a plain pass
    give the same bits, and what the hook holds stays as it was."""
    from ml_b200.ops import autograd as F
    torch.manual_seed(rows + V)
    x, tgt = rnd(rows, V, scale=2.0), torch.randint(0, V, (rows,), device=dev(), dtype=torch.int32)
    leaf = x.clone().requires_grad_(True)
    assert _native(F.cross_entropy(leaf, tgt))
    (F.cross_entropy(leaf, tgt) * factor).backward()
    z = x.clone().requires_grad_(True)
    loss = F.cross_entropy(z, tgt) * factor
    first, = torch.autograd.grad(loss, z, retain_graph=True)
    again, = torch.autograd.grad(loss, z, retain_graph=True)
    last, = torch.autograd.grad(loss, z)
    held = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: held.append(t) or t, lambda t: t):
        hooked = F.cross_entropy(z, tgt) * factor
    keep = [t.clone() for t in held]
    through, = torch.autograd.grad(hooked, z)
    assert held and all(torch.equal(a, b) for a, b in zip(held, keep))
    for g in (again, last, through, leaf.grad):
        assert torch.equal(first, g)
    e = x.double().requires_grad_(True)
    eg, = torch.autograd.grad(torch.nn.functional.cross_entropy(e, tgt.long()) * factor, e)
    assert _rel(first, eg) < 2 ** -7      # (two roundings to bf16)


def _forms(rows, C):
    """A [rows, C] operand as programs hold it: dense, the transpose of its transpose, every other row, every other column, off a
    16-byte boundary."""
    yield "dense", lambda: rnd(rows, C)
    yield "transposed", lambda: rnd(C, rows).t()
    yield "rows", lambda: rnd(2 * rows, C)[::2]
    yield "columns", lambda: rnd(rows, 2 * C)[:, ::2]
    yield "offset", lambda: rnd(1, rows * C + 8).view(-1)[3:3 + rows * C].view(rows, C)


@pytest.mark.parametrize("form", ["dense", "transposed", "rows", "columns", "offset"])
@pytest.mark.parametrize("rows,C,N", [(1, 256, 8), (37, 256, 512), (130, 768, 384), (300, 264, 512), (200, 512, 77 * 8)])
def test_plain_calls_are_what_the_functions_give(form, rows, C, N):
    """The extension module and the Python Functions run the same kernels in the same order: the same bits, for every form of the operands
    and of the incoming gradient that either takes (weight gradients with the reduction uncut, which makes their sums repeatable)."""
    from ml_b200.ops import autograd as F
    torch.manual_seed(rows + C + N)
    L = nat().lib()

    def both(fast, slow, leaves, shape):
        outs = []
        dout = dict(_forms(*shape))[form]()
        for fn in (fast, slow):
            ls = [t.detach().requires_grad_(True) if t is not None else None for t in leaves]
            y = fn(*ls)
            assert _native(y) == (fn is fast and form != "offset")      # (the module takes no unaligned operand)
            gs = torch.autograd.grad(y, [t for t in ls if t is not None], dout)
            with torch.no_grad():
                outs.append([y.detach(), fn(*ls), *gs])
        for a, b in zip(*outs):
            assert a.shape == b.shape and a.dtype == b.dtype and torch.equal(a, b), form

    mk = dict(_forms(rows, C))[form]
    L.mlb_gemm_set_splits(1)
    try:
        for b in (None, rnd(1, N).view(-1)):
            both(lambda x, W, b: F.linear(x, W, b), lambda x, W, b: F.Linear.apply(x, W, b), [mk(), dict(_forms(N, C))[form](), b], (rows, N))
    finally:
        L.mlb_gemm_set_splits(0)
    if form != "offset" and C % 256 == 0:      # (the norms and SwiGLU read whole vectors: such rows were never theirs; other widths are not the module's)
        w, b = rnd(1, C).view(-1), rnd(1, C).view(-1)
        both(lambda x, w: F.rmsnorm(x, w, 1e-5), lambda x, w: F.RMSNorm.apply(x, w, 1e-5), [mk(), w], (rows, C))
        both(lambda x, w, b: F.layer_norm(x, w, b, 1e-5), lambda x, w, b: F.LayerNorm.apply(x, w, b, 1e-5), [mk(), w, b], (rows, C))
        both(F.swiglu, F.SwiGLU.apply, [mk()], (rows, C // 2))


@pytest.mark.parametrize("B,T,H,Hkv,hd", [(1, 1, 1, 1, 64), (2, 130, 4, 2, 64), (1, 257, 2, 2, 128), (2, 65, 6, 1, 32), (3, 40, 4, 4, 16)])
def test_plain_attention_calls_are_what_the_functions_give(B, T, H, Hkv, hd):
    from ml_b200.ops import autograd as F
    torch.manual_seed(T)
    cos, sin = ref.rope_tables(T, hd, 10000.0, dev())
    for width, fast, slow in (((H + 2 * Hkv) * hd, lambda x: F.rope_causal_attention(x, cos, sin, B, T, H, hd, Hkv),
                               lambda x: F.RopeCausalAttention.apply(x, cos, sin, B, T, H, hd, Hkv)),
                              (3 * H * hd, lambda x: F.bidir_attention(x, B, T, H, hd), lambda x: F.BidirAttention.apply(x, B, T, H, hd))):
        x = rnd(B * T, width).requires_grad_(True)
        for dout in (rnd(B * T, H * hd), rnd(H * hd, B * T).t()):
            a, b = fast(x), slow(x)
            assert _native(a) and not _native(b)
            assert torch.equal(a, b) and torch.equal(*(torch.autograd.grad(y, x, dout)[0] for y in (a, b)))
        with torch.no_grad():
            assert torch.equal(fast(x), slow(x))


def test_what_the_extension_module_declines():
    """Anything but plain tensors of the current GPU goes to the Python Functions, with their errors."""
    from torch.utils.checkpoint import checkpoint
    from ml_b200.ops import autograd as F
    m, x, W = nat().bridge(), rnd(16, 256), rnd(64, 256)
    assert isinstance(m.linear(x, W, None), torch.Tensor)
    for a in ((x.float(), W, None), (x, W.float(), None), (x.cpu(), W, None), (x, rnd(64, 248), None), (x[:0], W, None), (x.view(-1), W, None),
              (x, W, rnd(1, 63).view(-1)), (x, None, None), (3, W, None), (x.as_subclass(type("T", (torch.Tensor,), {})), W, None)):
        assert m.linear(*a) is NotImplemented
    assert m.rmsnorm(rnd(4, 264), rnd(1, 264).view(-1), 1e-5) is NotImplemented      # (its backward is another kernel)
    with pytest.raises(AssertionError):
        F.linear(x.float(), W)
    with pytest.raises(AssertionError):
        nat().linear_fwd(rnd(16, 64), x.float(), W)
    with pytest.raises(AssertionError):
        nat().rmsnorm_fwd(None, torch.empty(16, device=dev()), x, W[0], 1e-5)
    with torch.autograd.forward_ad.dual_level(), pytest.raises(Exception):
        F.linear(torch.autograd.forward_ad.make_dual(x, x), W)
    y = checkpoint(lambda t: F.swiglu(F.linear(t, W)), x.requires_grad_(True), use_reentrant=False)
    assert _native(y)
    g, = torch.autograd.grad(y, x, torch.ones_like(y))
    e, = torch.autograd.grad(F.SwiGLU.apply(F.Linear.apply(x, W, None)), x, torch.ones_like(y := y.detach()))
    assert torch.equal(g, e)


def test_entry_points_through_ctypes_and_through_the_module(monkeypatch):
    """Every entry point that the extension module has, called through it and through ctypes (all there is where the module cannot be built): the
    same bits, the same refusals."""
    n, seen = nat(), set()
    B, T, H, hd, C, I, V = 2, 192, 4, 64, 256, 384, 512
    M = B * T
    cos, sin = ref.rope_tables(T, hd, 10000.0, dev())

    class Spy:
        def __init__(self, entries):
            self.entries = entries

        def __getattr__(self, name):
            seen.add(name)
            return getattr(self.entries, name)

    def work():
        torch.manual_seed(0)
        made = []
        e = lambda *sh, dtype=torch.bfloat16, fill=0: made.append(torch.full(sh, fill, device=dev(), dtype=dtype)) or made[-1]
        f32, u8 = dict(dtype=torch.float32), dict(dtype=torch.uint8)
        x, y, w, b = rnd(M, C), rnd(M, C), rnd(1, C).view(-1), rnd(1, C).view(-1)
        Wq, Wgu, Wo, dq, dgu = rnd(3 * C, C), rnd(2 * I, C), rnd(C, C), rnd(M, 3 * C), rnd(M, 2 * I)
        ids = torch.randperm(V, device=dev())[:M].int()
        n.linear_fwd(e(M, 3 * C), x, Wq)
        assert n.linear_fwd_posembed(e(M, 3 * C), x, Wq, rnd(7, 3 * C), 7) and n.linear_fwd_rope(e(M, 3 * C), x, Wq, cos, sin, T, 2 * C)
        assert n.linear_fwd_swiglu(e(M, 2 * I), e(M, I), x, Wgu)
        n.linear_dx(e(M, C), dq, Wq)
        n.linear_dw(e(3 * C, C, **f32), dq, x)
        n.linear_dw_cast(e(3 * C, C), dq, x)
        n.gemm(e(M, 3 * C), x, Wq)
        n._entries().mlb_cast_f2b(e(M, C), x.float(), x.numel(), 0.5)
        n.zero_(e(M, C, fill=1))
        n.colsum(e(3 * C), dq)
        n.rmsnorm_fwd(e(M, C), rstd := e(M, **f32), x, w, 1e-5)
        n.add_rmsnorm_fwd(e(M, C), e(M, C), e(M, **f32), x, y, w, 1e-5)
        x8 = e(M, C, **u8)
        n.rmsnorm_fwd_fp8(e(M, C), x8, e(M, **f32), x, w, 1e-5, 1.0)
        W8 = e(3 * C, C, **u8)
        n.cast_bf16_fp8(W8, Wq, 16.0)
        assert n.linear_fwd_fp8(e(M, 3 * C), x8, W8, 1 / 16)
        n.rmsnorm_bwd(e(M, C), e(C, **f32), y, x, w, rstd, y)
        n.rmsnorm_bwd_cast(e(M, C), e(C), y, x, w, rstd)
        n.layernorm_fwd(e(M, C), mean := e(M, **f32), rs := e(M, **f32), x, w, b, 1e-5)
        n.layernorm_bwd_cast(e(M, C), e(C), e(C), y, x, w, mean, rs)
        n.swiglu_fwd(e(M, I), dgu)
        n.swiglu_fwd_fp8(e(M, I), e(M, I, **u8), dgu, 1.0)
        n.swiglu_bwd(e(M, 2 * I), rnd(M, I), dgu)
        q = rnd(M, 3 * C)
        n.rope_fwd(made.append(q.clone()) or made[-1], cos, sin, B, T, H, hd)
        n.rope_copy(qr := e(M, 3 * C), rnd(M, 2 * C), cos, sin, B, T, H, hd, 2)
        n.kv_group_sum(e(M, 2 * C), q, B, T, H, hd, 2)
        n.attn_fwd(o := e(M, C), lse := e(B, H, T, **f32), qr, B, T, H, hd)
        assert n.linear_dx_delta(do := e(M, C), rnd(M, C), Wo, o, B, T, H)
        assert n.attn_bwd(e(M, 3 * C), do, qr, o, lse, B, T, H, hd, (cos, sin), have_delta=True)
        assert n.attn_bwd(e(M, 3 * C), do, qr, o, lse, B, T, H, hd, (cos, sin))
        n.attn_bidir_fwd(o := e(M, C), lse := e(B, H, T, **f32), qr, B, T, H, hd)
        n.attn_bidir_bwd(e(M, 3 * C), do, qr, o, lse, B, T, H, hd)
        n.ce_mean(e(1, **f32), e(M, **f32), e(M, V), z := rnd(M, V), ids)
        n.ce_fwd_bwd(e(M, **f32), made.append(z.clone()) or made[-1], ids, 0.5)
        n.scale_dev(e(M, V), z, e(1, fill=0.7, **f32))
        n.embed_fwd(e(M, C), t := rnd(V, C), ids)
        n.embed_bwd(e(V, C, **f32), y, ids, T, 0)
        g = torch.randn(V * C, device=dev())
        n.adamw(e(V * C, fill=1, **f32), e(V * C), g, e(V * C, **f32), e(V * C, **f32), 1e-3, 0.9, 0.95, 1e-8, 0.1, 0.1, 0.05)
        n.sum_scale(e(1, **f32), g, 0.25)
        with pytest.raises(AssertionError):
            n.linear_fwd(e(M, 3 * C), x.float(), Wq)
        with pytest.raises(AssertionError):
            n.rmsnorm_fwd(e(M, C), e(M, **f32), x.t(), w, 1e-5)
        return made

    n.lib().mlb_gemm_set_splits(1)
    outs = []
    try:
        for entries in (n._Ctypes(), n.bridge()):
            seen.clear()
            monkeypatch.setattr(n, "_E", Spy(entries))
            outs.append(work())
            assert seen | {"mlb_capture_id"} == {"mlb_" + k for k in n._KINDS}      # (that one is asked through ctypes)
            assert [getattr(entries, f)(*a) for f, a in (("mlb_capture_id", ()), ("mlb_gemm_dw_direct", (768, 768, 1003)))] == [
                0, n.lib().mlb_gemm_dw_direct(768, 768, 1003)]
    finally:
        n.lib().mlb_gemm_set_splits(0)
    assert len(outs[0]) == len(outs[1])
    for i, (p, q) in enumerate(zip(*outs)):
        assert torch.equal(p, q), i


@pytest.mark.parametrize("ways", [2, 4, 8])
@pytest.mark.parametrize("M,N,K", [(1, 8, 1024), (127, 136, 520), (136, 128, 1000), (304, 264, 2056), (64, 768, 11008)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
def test_products_whose_reduction_a_cluster_shares(ways, M, N, K, a_mn, b_mn):
    """Edges of the tile, reductions that the ways do not divide, fewer k-blocks per CTA than stages and more.  fp32 sums and one rounding
    (2^-9 at most); the order of the sums is fixed, so a second run gives the same bits."""
    if a_mn and M % 8:
        pytest.skip("such an operand has no 16-byte rows")
    torch.manual_seed(M + K)
    A, B, n = rnd(*((K, M) if a_mn else (M, K))), rnd(*((K, N) if b_mn else (N, K))), nat()
    e = (A.t() if a_mn else A).double() @ (B if b_mn else B.t()).double()
    n.lib().mlb_gemm_splitk(ways)
    try:
        outs = [torch.full((M, N), float("nan"), device=dev(), dtype=torch.bfloat16) for _ in range(2)]
        for o in outs:
            n.gemm(o, A, B, a_mn, b_mn)
        assert torch.equal(*outs) and _rel(outs[0], e) < 2 ** -8.5
        if not a_mn and not b_mn:
            pos, o = rnd(3, N), torch.empty_like(outs[0])
            assert n.linear_fwd_posembed(o, A, B, pos, 3)
            assert _rel(o, e + pos.double()[torch.arange(M, device=dev()) % 3]) < 2 ** -8.5
    finally:
        n.lib().mlb_gemm_splitk(-1)


@pytest.mark.parametrize("rows", [1, 64, 200, 1003])
@pytest.mark.parametrize("C,I", [(128, 384), (768, 2048), (2048, 5504)])
def test_products_of_few_rows_by_cost(rows, C, I):
    """Whatever form the estimate picks for a layer's products at few rows: forward, both gradients, and the add-reduce form into what was there."""
    torch.manual_seed(rows + C)
    n = nat()
    for N, K in ((3 * C, C), (2 * I, C), (C, I)):
        x, W, dout = rnd(rows, K), rnd(N, K, scale=K ** -0.5), rnd(rows, N)
        out, dx, dW, acc = rnd(rows, N), rnd(rows, K), rnd(N, K), torch.randn(N, K, device=dev())
        before = acc.double()
        n.linear_fwd(out, x, W)
        n.linear_dx(dx, dout, W)
        n.linear_dw_cast(dW, dout, x)
        n.linear_dw(acc, dout, x)
        ew = dout.double().t() @ x.double()
        assert _rel(out, x.double() @ W.double().t()) < 2 ** -8.5 and _rel(dx, dout.double() @ W.double()) < 2 ** -8.5
        assert _rel(dW, ew) < 2 ** -8.5 and _rel(acc, before + ew) < 1e-5


@pytest.mark.parametrize("rows,C", [(1, 8), (3, 128), (256, 128), (257, 128), (300, 248), (2500, 64), (40, 256), (33, 768), (9, 264)])
@pytest.mark.parametrize("add", [False, True])
def test_rmsnorm_backward_of_few_or_narrow_rows(rows, C, add):
    """One partial row per block up to 32 blocks and their sum by the last one, rows narrower than a warp's vectors, and the two-level sum beyond: dx to one
    rounding (2^-9), dw in fp32 added to what was there, the same on a second run."""
    torch.manual_seed(rows + C)
    n = nat()
    x, dy, w, a = rnd(rows, C), rnd(rows, C), 1 + rnd(1, C, scale=0.1).view(-1), rnd(rows, C) if add else None
    out, rstd = torch.empty_like(x), torch.empty(rows, device=dev())
    n.rmsnorm_fwd(out, rstd, x, w, 1e-5)
    dw0 = torch.randn(C, device=dev())
    runs = []
    for _ in range(2):
        dx, dw = torch.empty_like(x), dw0.clone()
        n.rmsnorm_bwd(dx, dw, dy, x, w, rstd, a)
        runs.append((dx, dw))
    xd, wd = x.double().requires_grad_(True), w.double().requires_grad_(True)
    e = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-5) * wd
    gx, gw = torch.autograd.grad(e, [xd, wd], dy.double())
    assert _rel(runs[0][0], gx + (a.double() if add else 0)) < 2 ** -8 and _rel(runs[0][1], dw0.double() + gw) < 1e-5
    if C % 256 == 0 or C < 256:      # (other widths add up in shared memory as it comes)
        assert torch.equal(runs[0][0], runs[1][0]) and torch.equal(runs[0][1], runs[1][1])


@pytest.mark.parametrize("rows,C,shift", [(1, 256, 0), (25, 512, 0), (2369, 256, 0), (7200, 768, 0), (25, 512, 1), (9, 768, 8), (3, 256, 4),
                                          (4096, 256, 0), (4097, 256, 0), (1024, 512, 0), (1025, 512, 0), (455, 768, 0), (456, 768, 0)])
def test_rmsnorm_backward_of_whole_vectors_of_columns(rows, C, shift):
    """A row per warp and rows that share a block's threads, either side of the line, past one round of the groups, and the same widths from a place where
    vectors may not be loaded."""
    torch.manual_seed(rows + C)
    big = rnd(rows * C + 8)
    x, dy, w, a = big[shift:shift + rows * C].view(rows, C), rnd(rows, C), 1 + rnd(1, C, scale=0.1).view(-1), rnd(rows, C)
    rstd = torch.rand(rows, device=dev()) + 0.5
    dx, dw = torch.empty_like(a), torch.ones(C, device=dev())
    nat().rmsnorm_bwd(dx, dw, dy, x, w, rstd, a)
    xd, dd, wd, r = x.double(), dy.double(), w.double(), rstd.double()[:, None]
    ex = a.double() + r * wd * dd - xd * r ** 3 / C * (dd * wd * xd).sum(1, keepdim=True)
    assert _rel(dx, ex) < 2 ** -8 and _rel(dw, 1 + (dd * xd * r).sum(0)) < 1e-5


@pytest.mark.parametrize("rows", [1, 7, 300])
@pytest.mark.parametrize("C", [256, 512, 768, 1024, 1280, 1536, 1792, 2048, 264, 40])
@pytest.mark.parametrize("bias", [False, True])
def test_layernorm_forward_widths(rows, C, bias):
    """Every width that stays in registers and two that do not, rows that do not fill a block: one rounding (2^-9), statistics in fp32."""
    torch.manual_seed(rows + C)
    x, w, b = rnd(rows, C) + 2, 1 + rnd(1, C, scale=0.1).view(-1), rnd(1, C).view(-1) if bias else None
    out, mean, rstd = torch.empty_like(x), torch.empty(rows, device=dev()), torch.empty(rows, device=dev())
    nat().layernorm_fwd(out, mean, rstd, x, w, b, 1e-5)
    xd = x.double()
    e = torch.nn.functional.layer_norm(xd, (C,), w.double(), b.double() if bias else None, 1e-5)
    assert _rel(out, e) < 2 ** -8.5 and _rel(mean, xd.mean(-1)) < 1e-5
    assert _rel(rstd, torch.rsqrt(xd.var(-1, unbiased=False) + 1e-5)) < 1e-5


@pytest.mark.parametrize("rows", [1, 7, 301])
@pytest.mark.parametrize("C", [256, 512, 768, 1024, 1280, 1536, 1792, 2048])
@pytest.mark.parametrize("bias", [False, True])
def test_layernorm_forward_adds_in_one_order(rows, C, bias):
    """Rows read as vectors and rows off a 16-byte boundary, read element by element, are added up in the same order: the same bits."""
    torch.manual_seed(rows + C)
    w, b, flat = 1 + rnd(1, C, scale=0.1).view(-1), rnd(1, C).view(-1) if bias else None, rnd(1, rows * C + 8).view(-1) + 0.3
    outs = []
    for x in (flat[1:1 + rows * C].clone().view(rows, C), flat[1:1 + rows * C].view(rows, C)):
        o = torch.empty_like(x), torch.empty(rows, device=dev()), torch.empty(rows, device=dev())
        nat().layernorm_fwd(*o, x, w, b, 1e-5)
        outs.append(o)
    for a, e in zip(*outs):
        assert torch.equal(a, e)


@pytest.mark.parametrize("rows", [1, 9, 250, 1003, 2369, 9000])
@pytest.mark.parametrize("C", [256, 768])
def test_column_sums_fold_in_one_order(rows, C):
    """Eight slices of every eighth partial row, added in order: exactly that, in 32 bits, from one partial row up to the most there are."""
    torch.manual_seed(rows)
    n = nat()
    L, x, dy, w = n.lib(), rnd(rows, C), rnd(rows, C), rnd(1, C).view(-1)
    o, mean, rstd, dx = torch.empty_like(x), torch.empty(rows, device=dev()), torch.empty(rows, device=dev()), torch.empty_like(x)
    n.layernorm_fwd(o, mean, rstd, x, w, None, 1e-5)
    part, d = torch.empty(L.mlb_rmsnorm_bwd_blocks(rows), 2 * C, device=dev()), torch.zeros(2 * C, device=dev())
    p = lambda t: t.data_ptr()
    assert L.mlb_layernorm_bwd2(p(dx), p(d), p(d[C:]), 0, p(dy), p(x), p(w), p(mean), p(rstd), rows, C, p(part), n._st()) == 0
    total = None
    for q in range(8):
        s = torch.zeros(2 * C, device=dev())
        for row in part[q::8]:
            s += row
        total = s if total is None else total + s
    assert torch.equal(d, total)


@pytest.mark.parametrize("rows", [640, 641, 648, 2367])
def test_column_sums_fold_at_a_trips_end(rows):
    """80 partial rows are the most that eight warps take in one trip; one more, and 32 warps load them."""
    test_column_sums_fold_in_one_order(rows, 256)


@pytest.mark.parametrize("B,T,H,hd", [(11, 1000, 12, 64), (33, 125, 16, 128)])
def test_attention_backward_of_many_rows_is_that_of_each_sample(B, T, H, hd):
    """From 2^20 vectors on a thread sums two of them for rowsum(dO * O), the last block not full: the gradients are those of one sample at a time, bit for bit."""
    torch.manual_seed(B)
    n = nat()
    qkv, dout = rnd(B * T, 3 * H * hd), rnd(B * T, H * hd)
    out, lse, d = torch.empty_like(dout), torch.empty(B, H, T, device=dev()), torch.empty_like(qkv)
    n.attn_fwd(out, lse, qkv, B, T, H, hd)
    n.attn_bwd(d, dout, qkv, out, lse, B, T, H, hd)
    for b in (0, B // 2, B - 1):
        r, e = slice(b * T, (b + 1) * T), torch.empty(T, 3 * H * hd, device=dev(), dtype=torch.bfloat16)
        n.attn_bwd(e, dout[r], qkv[r], out[r], lse[b:b + 1], 1, T, H, hd)
        assert torch.equal(d[r], e)


@pytest.mark.parametrize("rows,V", [(3, 8), (700, 512), (40, 1016), (7, 1024), (7, 1032), (40, 2056)])
def test_cross_entropy_either_side_of_its_block_sizes(rows, V):
    torch.manual_seed(V)
    n, z = nat(), rnd(rows, V, scale=3.0)
    tgt = torch.randint(0, V, (rows,), device=dev(), dtype=torch.int32)
    tgt[rows // 2] = -1
    zd, live = z.double(), (tgt >= 0).double()
    lse, zt = torch.logsumexp(zd, -1), zd.gather(1, tgt.clamp(min=0).long()[:, None])[:, 0]
    loss, losses, dz = torch.empty((), device=dev()), torch.empty(rows, device=dev()), torch.empty_like(z)
    n.ce_mean(loss, losses, dz, z, tgt)
    # fp32 sums of at most 16 terms a thread and nine levels over the threads, the exponentials off by 2 ulp: below 2^-17 of the sum
    assert ((losses - (lse - zt) * live).abs() < 2 ** -17 + 2 ** -22 * lse.abs()).all()
    g = (zd - lse[:, None]).exp()
    g[torch.arange(rows, device=dev()), tgt.clamp(min=0).long()] -= 1
    assert _rel(dz, g * (live / live.sum())[:, None]) < 2 ** -8
    in_place, ls = z.clone(), torch.empty(rows, device=dev())
    n.ce_fwd_bwd(ls, in_place, tgt, 1.0 / float(live.sum()))
    assert torch.equal(ls, losses) and torch.equal(in_place, dz)


def _native_nodes():
    """name -> (operands, call through the public entry point), each a plain call of the extension module: for tests of its autograd nodes."""
    from ml_b200.ops import autograd as F
    B, T, H, Hkv, hd, rows, C, N = 2, 72, 4, 2, 64, 40, 256, 128
    v = lambda n: rnd(1, n).view(-1)
    cos, sin = ref.rope_tables(T, hd, 10000.0, dev())
    tgt = torch.randint(0, N, (rows,), device=dev(), dtype=torch.int32)
    return {
        "linear": ([rnd(rows, C), rnd(N, C), v(N)], F.linear),
        "rmsnorm": ([rnd(rows, C), v(C)], lambda x, w: F.rmsnorm(x, w, 1e-5)),
        "layer_norm": ([rnd(rows, C), v(C), v(C)], lambda x, w, b: F.layer_norm(x, w, b, 1e-5)),
        "swiglu": ([rnd(rows, 2 * N)], F.swiglu),
        "rope_causal_attention": ([rnd(B * T, (H + 2 * Hkv) * hd)], lambda x: F.rope_causal_attention(x, cos, sin, B, T, H, hd, Hkv)),
        "rope_causal_attention_128": ([rnd(B * T // 2, 3 * H * 128)],
                                      lambda x, r=ref.rope_tables(T, 128, 10000.0, dev()): F.rope_causal_attention(x, *r, 1, T, H, 128)),
        "bidir_attention": ([rnd(B * T, 3 * H * hd)], lambda x: F.bidir_attention(x, B, T, H, hd)),
        "cross_entropy": ([rnd(rows, N)], lambda z: F.cross_entropy(z, tgt)),
    }


NATIVE_NODES = ["linear", "rmsnorm", "layer_norm", "swiglu", "rope_causal_attention", "rope_causal_attention_128", "bidir_attention", "cross_entropy"]


def _native(y):
    return "CppNode" in y.grad_fn.name()


def _strided(t):      # the same values behind other strides
    u = torch.empty(*t.shape[::-1], 2, dtype=t.dtype, device=t.device)[..., 0]
    return u.permute(*reversed(range(t.dim()))).copy_(t)


def _offset(t):       # ... one element off the start of a buffer
    return torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view(t.shape).copy_(t)


@pytest.mark.parametrize("name", NATIVE_NODES)
def test_saved_tensors_come_back_in_another_form(name):
    """What a saved-tensor hook returns is not checked by torch.  The same values in another layout or off a 16-byte boundary give the same
    gradients; another type, device or size is refused on the host, in front of the launches, as the entry points refuse it."""
    from torch.autograd.graph import saved_tensors_hooks
    torch.manual_seed(3)
    ops_, call = _native_nodes()[name]
    leaves = [t.requires_grad_(True) for t in ops_]
    nat().lib().mlb_gemm_set_splits(1)      # (repeatable weight gradients)

    def grads(change):
        with saved_tensors_hooks(lambda t: t, change):
            y = call(*leaves)
        assert _native(y)
        torch.manual_seed(4)
        return torch.autograd.grad(y, leaves, rnd(1, *y.shape, dtype=y.dtype)[0])

    try:
        want = grads(lambda t: t)
        for same in (_strided, _offset, lambda t: _strided(_offset(t)), lambda t: t.cpu().cuda()):
            for a, b in zip(want, grads(same)):
                assert torch.equal(a, b)
        launched = nat().get_error()
        for other in (torch.Tensor.float, torch.Tensor.double, torch.Tensor.half, torch.Tensor.cpu, lambda t: t[:-1], lambda t: t.view(-1), lambda t: t[None]):
            changed = lambda t: other(t).dtype != t.dtype or other(t).device != t.device or other(t).shape != t.shape
            # (a tensor that this changes nothing about is left as it is)
            with pytest.raises(AssertionError, match="saved tensor"):
                assert grads(lambda t: other(t) if changed(t) else t) is None
        assert nat().get_error() == launched == 0
        for a, b in zip(want, grads(lambda t: t)):
            assert torch.equal(a, b)
    finally:
        nat().lib().mlb_gemm_set_splits(0)


@pytest.mark.parametrize("name", NATIVE_NODES)
def test_transforms_and_modes_take_the_functions(name):
    """Under a transform of torch.func, a trace or a dispatch mode the extension module declines (its tensors may have no memory) and the Python
    Function runs, with its results and its errors."""
    from torch.utils._python_dispatch import TorchDispatchMode
    ops_, call = _native_nodes()[name]
    assert _native(call(*(t.requires_grad_(True) for t in ops_)))
    ops_ = [t.detach() for t in ops_]
    want = call(*ops_)
    with pytest.raises(RuntimeError, match="autograd.Function with functorch"):      # (the Functions do not support them)
        torch.func.grad(lambda x: call(x, *ops_[1:]).float().sum())(ops_[0])
    with pytest.raises(RuntimeError, match="autograd.Function with functorch"):
        torch.vmap(lambda x: call(x, *ops_[1:]))(torch.stack([ops_[0], ops_[0]]))
    with pytest.raises(RuntimeError, match="autograd.Function with functorch"):      # (nor a level that is about other tensors)
        torch.func.grad(lambda z: (call(*ops_).float() * z).sum())(torch.ones(1, device=dev()))

    class Seen(TorchDispatchMode):
        ops = []

        def __torch_dispatch__(self, fn, types, args=(), kwargs=None):
            self.ops.append(str(fn))
            return fn(*args, **(kwargs or {}))

    with Seen() as seen:
        got = call(*ops_)
    assert torch.equal(got, want) and any("new_empty" in o for o in seen.ops)      # (the module allocates without the dispatcher's modes looking on)
    graph = torch.jit.trace(lambda *a: call(*a), tuple(ops_), check_trace=False).graph
    assert any(n.kind() == "prim::PythonOp" for n in graph.nodes()), graph


@pytest.mark.parametrize("native", [True, False])
def test_workspace_of_the_attention_backward_is_bounded_when_it_runs(native, monkeypatch):
    """FUSED_ATTN_BWD and FUSED_ATTN_BWD_MAX_SCRATCH hold at the time of backward, whatever they were in forward, and take any number: through the
    extension module as through the Function."""
    from ml_b200.ops import autograd as F
    B, T, H, hd, n = 1, 2048, 4, 64, nat()
    cos, sin = ref.rope_tables(T, hd, 10000.0, dev())
    x, dout = rnd(B * T, 3 * H * hd).requires_grad_(True), rnd(B * T, H * hd)
    need = n.lib().mlb_attn_bwd_scratch_bytes(B, T, H, hd)
    torch.autograd.grad(F.RopeCausalAttention.apply(x, cos, sin, B, T, H, hd, None), x, dout)

    def backward(**late):
        with monkeypatch.context() as mp:
            y = F.rope_causal_attention(x, cos, sin, B, T, H, hd) if native else F.RopeCausalAttention.apply(x, cos, sin, B, T, H, hd, None)
            assert _native(y) == native
            for k, v in late.items():
                mp.setattr(n, k, v)
            torch.cuda.synchronize()
            torch.cuda.reset_peak_memory_stats()
            before = torch.cuda.memory_allocated()
            g, = torch.autograd.grad(y, x, dout)
            return g, torch.cuda.max_memory_allocated() - before

    fused, most = backward()
    apart, least = backward(FUSED_ATTN_BWD=False)
    assert need > 8 << 20 and least < most - need // 2      # (what else comes and goes meanwhile is smaller than that)
    for limit, fits in ((need, True), (need - 1, False), (1 << 70, True), (float("inf"), True), (-(1 << 70), False)):
        g, used = backward(FUSED_ATTN_BWD_MAX_SCRATCH=limit)
        assert torch.equal(g, fused if fits else apart) and (used > most - need // 2) == fits, limit
    with monkeypatch.context() as mp:      # (in forward it asks for nothing)
        mp.setattr(n, "FUSED_ATTN_BWD_MAX_SCRATCH", 1 << 70)
        y = F.rope_causal_attention(x, cos, sin, B, T, H, hd)
    assert torch.equal(torch.autograd.grad(y, x, dout)[0], fused)


@pytest.mark.parametrize("together", [False, True])
@pytest.mark.parametrize("factor", [1.0, 0.37])
def test_cross_entropy_backward_replayed(together, factor):
    """A captured backward gives the same gradient at each of its replays, behind one replay of its forward; captured with its forward it does
    so too."""
    from ml_b200.ops import autograd as F
    torch.manual_seed(1)
    z, tgt = rnd(37, 264, scale=2.0).requires_grad_(True), torch.randint(0, 264, (37,), device=dev(), dtype=torch.int32)
    want, = torch.autograd.grad(F.cross_entropy(z, tgt) * factor, z)
    fwd, bwd, s = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph(), torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        torch.autograd.grad(F.cross_entropy(z, tgt) * factor, z)
        with torch.cuda.graph(fwd, stream=s):
            loss = F.cross_entropy(z, tgt) * factor
            if together:
                g, = torch.autograd.grad(loss, z)
        if not together:
            with torch.cuda.graph(bwd, pool=fwd.pool(), stream=s):
                g, = torch.autograd.grad(loss, z)
    torch.cuda.current_stream().wait_stream(s)
    for _ in range(2):
        fwd.replay()
        for _ in range(1 if together else 3):
            if not together:
                bwd.replay()
            assert torch.equal(g, want)


@pytest.mark.parametrize("name", NATIVE_NODES)
def test_nodes_run_on_the_stream_they_are_called_on(name):
    """Forward and backward on a side stream, behind operands that arrive late there; and from two threads at once, each on a stream of its own: the
    bits of a call by itself."""
    import threading
    ops_, call = _native_nodes()[name]
    nat().lib().mlb_gemm_set_splits(1)

    def one(values, wait=0):
        late = [torch.zeros_like(v) for v in values]
        if wait:
            torch.cuda._sleep(wait)
        for t, v in zip(late, values):
            t.copy_(v)
        leaves = [t.requires_grad_(True) for t in late]
        y = call(*leaves)
        assert _native(y)
        return [y.detach(), *torch.autograd.grad(y, leaves, torch.ones_like(y))]

    try:
        sets = [ops_, [t * 0.5 + 0.25 for t in ops_]]
        want = [one(v) for v in sets]
        streams = [torch.cuda.Stream() for _ in sets]
        torch.cuda.synchronize()
        with torch.cuda.stream(streams[0]):
            got = one(sets[0], wait=20_000_000)      # (10 ms)
        streams[0].synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want[0]))
        outs = [[], []]

        def work(i):
            with torch.cuda.stream(streams[i]):
                for _ in range(10):
                    outs[i].append(one(sets[i], wait=20_000))
                streams[i].synchronize()

        threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join(60)
        for i in range(2):
            assert len(outs[i]) == 10
            for got in outs[i]:
                assert all(torch.equal(a, b) for a, b in zip(got, want[i]))
    finally:
        nat().lib().mlb_gemm_set_splits(0)


@pytest.mark.parametrize("T", [1, 31, 33, 96, 127, 129, 161, 255, 300, 385])
@pytest.mark.parametrize("B,H,hd", [(1, 2, 64), (40, 6, 64), (1, 2, 128), (24, 8, 128)])
def test_causal_backward_at_tile_edges_with_rope(B, T, H, hd):
    """Gradients through RoPE where a tile's last 32 rows are whole (they leave by TMA), cut (by row) or not there, with one item per CTA and with
    several.  Against 64 bits; the bound is that of the test without RoPE: P, dS and the result in bf16, the rounding of O in delta."""
    torch.manual_seed(T + hd + B)
    qkv, dout = rnd(B * T, 3 * H * hd), rnd(B * T, H * hd)
    cos, sin = ref.rope_tables(T, hd, 10000.0, dev())
    n = nat()
    rot = qkv.clone()
    n.rope_fwd(rot, cos, sin, B, T, H, hd)
    out, lse, dqkv = rnd(B * T, H * hd), torch.empty(B, H, T, device=dev()), torch.full_like(qkv, float("nan"))
    n.attn_fwd(out, lse, rot, B, T, H, hd)
    assert n.attn_bwd(dqkv, dout, rot, out, lse, B, T, H, hd, rope=(cos, sin))
    _, _, ed = _attn64(rot, dout, B, T, H, hd, True)
    e = ed.view(B, T, 3, H, 2, hd // 2).clone()
    c, s = cos.double().view(1, T, 1, 1, hd // 2), sin.double().view(1, T, 1, 1, hd // 2)
    d0, d1 = e[:, :, :2, :, 0].clone(), e[:, :, :2, :, 1].clone()
    e[:, :, :2, :, 0], e[:, :, :2, :, 1] = d0 * c + d1 * s, d1 * c - d0 * s
    assert _rel(dqkv, e.view_as(dqkv)) < 2 ** -7
    # and each element, so that no row of one head can be another's: the norm above would let one pass
    b = _attn_bwd_bound64(rot, dout, B, T, H, hd).view(B, T, 3, H, 2, hd // 2)
    b0, b1 = b[:, :, :2, :, 0].clone(), b[:, :, :2, :, 1].clone()
    b[:, :, :2, :, 0], b[:, :, :2, :, 1] = b0 * c.abs() + b1 * s.abs(), b1 * c.abs() + b0 * s.abs()
    b += 2 ** -8 * e.abs()
    far = ((dqkv.double().view_as(e) - e).abs() / (b + 1e-30)).amax((0, 1, 3, 4, 5))
    assert (far <= 1).all(), far.tolist()


@pytest.mark.parametrize("hd,B,T,H", [(64, 640, 16, 16), (64, 320, 130, 16), (128, 640, 16, 16), (128, 320, 130, 16)])
def test_attention_with_more_items_than_a_block_keeps_at_hand(hd, B, T, H):
    """A block takes its first 48 (64) work items from shared memory and later ones from the schedule: with 69 and more to a block on 148 SMs each sample is
    still what it is alone, one item to a block, bit for bit.  Head size 64: from the device's counter too, through a ring of 64."""
    assert B * H * ((T + 127) // 128) > 64 * torch.cuda.get_device_properties(0).multi_processor_count
    torch.manual_seed(T + hd)
    n = nat()
    qkv, dout = rnd(B * T, 3 * H * hd), rnd(B * T, H * hd)
    rope = ref.rope_tables(T, hd, 10000.0, dev())

    def run(r, samples):
        q, g = qkv[r], dout[r]
        out, lse, d = torch.empty_like(g), torch.empty(samples, H, T, device=dev()), torch.full_like(q, float("nan"))
        n.attn_fwd(out, lse, q, samples, T, H, hd)
        assert n.attn_bwd(d, g, q, out, lse, samples, T, H, hd, rope=rope)
        return out.view(samples, T, -1), lse, d.view(samples, T, -1)

    alone = [run(slice(b * T, (b + 1) * T), 1) for b in range(0, B, 7)]
    want = [torch.cat(x) for x in zip(*alone)]
    for dynamic in (False, True) if hd == 64 else (False,):
        n.attn_dynamic(dynamic)
        try:
            got = run(slice(None), B)
            torch.cuda.synchronize()
        finally:
            n.attn_dynamic(False)
        assert n.get_error() == 0
        assert all(torch.equal(x[::7], w) for x, w in zip(got, want))
        assert not got[2].isnan().any()


def test_a_block_whose_waits_run_out_gives_up_and_says_which():
    """Waits on a barrier that nobody arrives on, 2 ms at most: all of them end, with the number of one that ran out as the block's word.  Later waits return
    without waiting for their own limit and leave the word alone, one whose barrier is complete is still answered, and a block's word is what the error word
    holds.  The context stays usable."""
    n, blocks, warps = nat(), 592, 8
    out = torch.zeros(blocks, 32 * warps, 4, device=dev(), dtype=torch.int32)
    probe = n.lib().mlb_attn_wait_probe
    probe.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
    try:
        assert probe(out.data_ptr(), blocks, torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        err = n.get_error()
    finally:
        n.clear_error()
    answers, word, last, again_us = out.cpu().unbind(-1)
    assert (answers == 4).all()
    assert (word >= 1).all() and (word <= warps).all()
    assert (last == last[:, :1]).all() and (last >= 1).all() and (last <= warps).all()
    assert err >> 24 == 1 and (err & 0xFFFFFF) in set(last[:, 0].tolist())
    assert int(again_us.max()) < 2000
    x = rnd(64, 128)
    y = torch.empty_like(x)
    n.rmsnorm_fwd(y, torch.empty(64, device=dev()), x, torch.ones(128, device=dev(), dtype=torch.bfloat16), 1e-6)
    torch.cuda.synchronize()
    assert n.get_error() == 0

"""Numerics of the sm_100a kernels against the plain-PyTorch fp32 definitions."""
import math

import pytest
import torch

from cosmos_b200 import ops
from cosmos_b200.ops import reference as ref

pytestmark = pytest.mark.gpu

DEV = "cuda"
GELU = 7     # EPI_GELU of the kernels


def _rand(*shape, scale=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, device=DEV, dtype=torch.float32) * scale).to(dtype)


def _close(got, want, atol, rtol, what=""):
    got = got.float()
    want = want.float()
    err = (got - want).abs()
    tol = atol + rtol * want.abs()
    bad = (err > tol).sum().item()
    assert bad == 0, f"{what}: {bad}/{err.numel()} elements off, max err {err.max().item():.4g}"


@pytest.fixture(autouse=True)
def _status_clean():
    ops.load_extension()
    yield
    torch.cuda.synchronize()
    ops.check_status()


def test_extension_is_loaded():
    assert ops.load_extension(), "kernel library must load on a GPU host"
    assert hasattr(torch.ops.cosmos_b200, "gemm")


@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (256, 512, 256), (1000, 768, 320), (77, 136, 72),
                                    (4096, 4096, 1024), (300, 6144, 4096)])
def test_gemm_plain(m, n, k):
    torch.manual_seed(0)
    a = _rand(m, k)
    w = _rand(n, k, scale=1 / math.sqrt(k))
    got = ops.gemm(a, w)
    want = a.float() @ w.float().t()
    _close(got, want, 2e-2, 2e-2, f"gemm {m}x{n}x{k}")


def test_gemm_bias_and_strided_a():
    torch.manual_seed(1)
    m, n, k = 513, 384, 256
    big = _rand(m, k + 64)
    a = big[:, :k]
    w = _rand(n, k, scale=1 / math.sqrt(k))
    bias = _rand(n)
    got = ops.gemm(a, w, bias)
    want = a.float() @ w.float().t() + bias.float()
    _close(got, want, 2e-2, 2e-2, "gemm+bias")


@pytest.mark.parametrize("m,dff,k", [(256, 512, 128), (700, 1536, 512), (130, 200, 64)])
def test_gemm_swiglu(m, dff, k):
    torch.manual_seed(2)
    a = _rand(m, k)
    w = _rand(2 * dff, k, scale=1 / math.sqrt(k))
    got = ops.gemm(a, w, epi=ops.EPI_SWIGLU)
    want = ref.gemm(a.float(), w.float(), epi=ops.EPI_SWIGLU)
    assert got.shape == (m, dff)
    _close(got, want, 2e-2, 2e-2, "gemm swiglu")


@pytest.mark.parametrize("m,n,k,rpb", [(512, 256, 128, 256), (600, 520, 192, 300), (384, 1024, 512, 384)])
def test_gemm_gated_residual(m, n, k, rpb):
    torch.manual_seed(3)
    a = _rand(m, k)
    w = _rand(n, k, scale=1 / math.sqrt(k))
    r = _rand(m, n)
    gate = _rand(m // rpb, n)
    got = ops.gemm(a, w, None, ops.EPI_GATED_RESID, r, gate, rpb)
    want = ref.gemm(a.float(), w.float(), None, ops.EPI_GATED_RESID, r.float(), gate.float(), rpb)
    _close(got, want, 3e-2, 2e-2, "gemm gated residual")
    got2 = ops.gemm(a, w, None, ops.EPI_GATED_RESID, r, None, rpb)
    want2 = r.float() + a.float() @ w.float().t()
    _close(got2, want2, 3e-2, 2e-2, "gemm residual without gate")


@pytest.mark.parametrize("m,hq,hk", [(256, 4, 2), (333, 8, 2)])
def test_gemm_qkv_rope(m, hq, hk):
    torch.manual_seed(4)
    k = 256
    n = (hq + 2 * hk) * 128
    a = _rand(m, k)
    w = _rand(n, k, scale=1 / math.sqrt(k))
    ang = torch.rand(m, 64, device=DEV) * 6.28
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    gq = (1 + 0.1 * torch.randn(128, device=DEV)).bfloat16()
    gk = (1 + 0.1 * torch.randn(128, device=DEV)).bfloat16()
    got = ops.gemm_qkv_rope(a, w, None, cos, sin, gq, gk, hq, hk, 1e-6)
    want = ref.gemm_qkv_rope(a.float(), w.float(), None, cos, sin, gq.float(), gk.float(), hq, hk, 1e-6)
    _close(got, want, 3e-2, 2e-2, "qkv rope epilogue")


def test_gemm_qkv_rope_routed():
    """Head chunks written through the routing table land where the table says."""
    torch.manual_seed(5)
    m, k, hq, hk = 256, 128, 2, 1
    n = (hq + 2 * hk) * 128
    a = _rand(m, k)
    w = _rand(n, k, scale=1 / math.sqrt(k))
    bufs = [torch.zeros(m, 128, device=DEV, dtype=torch.bfloat16) for _ in range(n // 128)]
    ptr = torch.tensor([b.data_ptr() for b in bufs], device=DEV, dtype=torch.int64)
    ld = torch.full((n // 128,), 128, device=DEV, dtype=torch.int64)
    ops.gemm_qkv_rope(a, w, None, None, None, None, None, hq, hk, 1e-6, ptr, ld)
    want = (a.float() @ w.float().t())
    for i, b in enumerate(bufs):
        _close(b, want[:, i * 128:(i + 1) * 128], 2e-2, 2e-2, f"routed chunk {i}")


@pytest.mark.parametrize("b,sq,skv,hq,hkv,mask", [
    (1, 256, 256, 1, 1, ops.MASK_FULL),
    (1, 512, 1024, 4, 1, ops.MASK_FULL),
    (2, 300, 777, 4, 2, ops.MASK_FULL),
    (1, 1024, 1024, 2, 1, ops.MASK_CAUSAL),
    (1, 500, 500, 4, 2, ops.MASK_CAUSAL),
    (1, 200, 456, 2, 2, ops.MASK_CAUSAL),
    (1, 2048, 2304, 8, 2, ops.MASK_FULL),
])
def test_attention(b, sq, skv, hq, hkv, mask):
    torch.manual_seed(6)
    q = _rand(b, sq, hq, 128)
    k = _rand(b, skv, hkv, 128)
    v = _rand(b, skv, hkv, 128)
    got, lse = ops.attention(q, k, v, mask=mask, return_lse=True)
    want, lse_ref = ref.attention(q.float(), k.float(), v.float(), None, mask, 0, True)
    _close(got, want, 2e-2, 2e-2, "attention out")
    _close(lse, lse_ref, 2e-2, 1e-3, "attention lse")


def test_attention_mot_mask():
    torch.manual_seed(7)
    s, n_ar = 640, 200
    q = _rand(1, s, 4, 128)
    k = _rand(1, s, 2, 128)
    v = _rand(1, s, 2, 128)
    got, _ = ops.attention(q, k, v, mask=ops.MASK_MOT, n_ar=n_ar)
    want, _ = ref.attention(q.float(), k.float(), v.float(), None, ops.MASK_MOT, n_ar)
    _close(got, want, 2e-2, 2e-2, "attention MoT mask")


def test_attention_large_scores_rescale():
    """Scores whose running max grows block after block exercise the lazy O rescale."""
    torch.manual_seed(8)
    sq, skv = 256, 1024
    q = _rand(1, sq, 1, 128)
    k = _rand(1, skv, 1, 128)
    ramp = torch.linspace(0.2, 3.0, skv, device=DEV)[None, :, None, None]
    k = (k.float() * ramp).bfloat16()
    v = _rand(1, skv, 1, 128)
    got, _ = ops.attention(q, k, v, scale=1.0)
    want, _ = ref.attention(q.float(), k.float(), v.float(), 1.0)
    _close(got, want, 3e-2, 3e-2, "attention with growing max")


def test_attention_strided_qkv_views():
    """q/k/v as views into one fused [S, (Hq+2Hkv)*128] projection buffer."""
    torch.manual_seed(9)
    s, hq, hkv = 384, 4, 1
    qkv = _rand(1, s, (hq + 2 * hkv) * 128)
    q = qkv[..., :hq * 128].view(1, s, hq, 128)
    k = qkv[..., hq * 128:(hq + hkv) * 128].view(1, s, hkv, 128)
    v = qkv[..., (hq + hkv) * 128:].view(1, s, hkv, 128)
    got, _ = ops.attention(q, k, v)
    want, _ = ref.attention(q.float(), k.float(), v.float())
    _close(got, want, 2e-2, 2e-2, "attention on strided views")


def test_attention_routed_output():
    torch.manual_seed(10)
    s, h, parts = 512, 2, 4
    q, k, v = _rand(1, s, h, 128), _rand(1, s, h, 128), _rand(1, s, h, 128)
    rows = s // parts
    bufs = [torch.zeros(1, rows, h, 128, device=DEV, dtype=torch.bfloat16) for _ in range(parts)]
    ptr = torch.tensor([b.data_ptr() for b in bufs], device=DEV, dtype=torch.int64)
    ops.attention(q, k, v, dest_ptr=ptr, rows_per_dest=rows, out=bufs[0])
    want, _ = ref.attention(q.float(), k.float(), v.float())
    for i, bfr in enumerate(bufs):
        _close(bfr, want[:, i * rows:(i + 1) * rows], 2e-2, 2e-2, f"routed rows {i}")


@pytest.mark.parametrize("rows,d", [(64, 128), (1000, 512), (333, 4096), (50, 5120)])
def test_rmsnorm(rows, d):
    torch.manual_seed(11)
    x, g, r = _rand(rows, d), _rand(d), _rand(rows, d)
    y, _ = ops.rmsnorm(x, g, 1e-6)
    want, _ = ref.rmsnorm(x.float(), g.float(), 1e-6)
    _close(y, want, 2e-2, 1e-2, "rmsnorm")
    y2, res = ops.rmsnorm(x, g, 1e-6, r)
    w2, wres = ref.rmsnorm(x.float(), g.float(), 1e-6, r.float())
    _close(y2, w2, 2e-2, 1e-2, "rmsnorm+res")
    _close(res, wres, 2e-2, 1e-2, "residual out")


def test_adaln_rmsnorm():
    torch.manual_seed(12)
    b, s, d = 2, 300, 512
    x = _rand(b * s, d)
    mod = _rand(b, 6 * d, scale=0.3)
    shift, scale = mod[:, :d], mod[:, d:2 * d]
    y = ops.adaln_rmsnorm(x, None, shift, scale, s, 1e-6)
    want = ref.adaln_rmsnorm(x.float(), None, shift.float(), scale.float(), s, 1e-6)
    _close(y, want, 2e-2, 1e-2, "adaln")


def test_mrope_and_qknorm():
    torch.manual_seed(13)
    s, h = 500, 6
    x = _rand(s, h, 128)
    ang = torch.rand(s, 64, device=DEV) * 6.28
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    g = (1 + 0.1 * torch.randn(128, device=DEV)).bfloat16()
    want = ref.mrope(x.float(), cos, sin, g.float(), 1e-6)
    got = ops.mrope(x.clone(), cos, sin, g, 1e-6)
    _close(got, want, 2e-2, 1e-2, "mrope")


def test_gated_residual_and_swiglu():
    torch.manual_seed(14)
    b, s, d = 2, 200, 256
    x, f, gate = _rand(b * s, d), _rand(b * s, d), _rand(b, d)
    _close(ops.gated_residual(x, f, gate, s), ref.gated_residual(x.float(), f.float(), gate.float(), s),
           2e-2, 1e-2, "gated residual")
    gu = _rand(b * s, 2 * d)
    _close(ops.swiglu(gu), ref.swiglu(gu.float()), 2e-2, 1e-2, "swiglu")


@pytest.mark.parametrize("normalize", [False, True])
def test_cfg_euler_step(normalize):
    torch.manual_seed(15)
    rows, d = 1000, 64
    x = torch.randn(rows, d, device=DEV)
    vc, vu = _rand(rows, d), _rand(rows, d)
    want = ref.cfg_euler_step(x.clone(), vc, vu, 7.0, -0.03, normalize)
    got = ops.cfg_euler_step(x.clone(), vc, vu, 7.0, -0.03, normalize)
    _close(got, want, 1e-5, 1e-5, "cfg euler step")


@pytest.mark.parametrize("b,hq,hkv,page,lens,splits", [
    (2, 4, 1, 16, [100, 37], 1),
    (3, 8, 2, 32, [700, 1, 333], 4),
    (4, 4, 4, 16, [513, 512, 511, 64], 3),
    (2, 8, 1, 16, [2000, 1500], None),
    (3, 4, 2, 8, [1000, 129, 128], 2),
    (2, 32, 8, 128, [3000, 4097], None),
])
@pytest.mark.parametrize("impl", [0, 1])
def test_paged_decode(b, hq, hkv, page, lens, splits, impl):
    """impl 0: TMA + tcgen05 kernel, impl 1: CUDA-core kernel; both against the fp32 definition."""
    torch.manual_seed(16)
    max_pages = (max(lens) + page - 1) // page + 1
    n_pages = b * max_pages + 3
    kc = _rand(n_pages, hkv, page, 128)
    vc = _rand(n_pages, hkv, page, 128)
    perm = torch.randperm(n_pages, device=DEV)[:b * max_pages].view(b, max_pages).int()
    sl = torch.tensor(lens, device=DEV, dtype=torch.int32)
    q = _rand(b, hq, 128)
    got = ops.paged_decode(q, kc, vc, perm, sl, n_splits=splits, max_len=max(lens), impl=impl)
    torch.cuda.synchronize()
    ops.check_status()
    want = ops.paged_decode_ref(q.float(), kc.float(), vc.float(), perm, sl)
    _close(got, want, 2e-2, 2e-2, "paged decode")


@pytest.mark.parametrize("b,hq,hkv,page", [(5, 4, 1, 16), (32, 32, 8, 16), (3, 8, 2, 4)])
def test_decode_qkv_post(b, hq, hkv, page):
    """The fused decode glue (q/k norm + rotary + cache write) against the fp32 definition of each step."""
    torch.manual_seed(18)
    n_pages = 2 * b + 1
    qkv = _rand(b, hq + 2 * hkv, 128)
    ang = torch.rand(b, 64, device=DEV) * 6.0
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    gq, gk = (1 + 0.1 * torch.randn(128, device=DEV)).bfloat16(), (1 + 0.1 * torch.randn(128, device=DEV)).bfloat16()
    slots = (torch.randperm(n_pages * page, device=DEV)[:b]).long()
    kc, vc = _rand(n_pages, hkv, page, 128), _rand(n_pages, hkv, page, 128)
    kc0, vc0 = kc.clone(), vc.clone()
    q = ops.decode_qkv_post(qkv, hq, cos, sin, gq, gk, 1e-6, slots, kc, vc)
    torch.cuda.synchronize()
    ops.check_status()
    f = qkv.float()
    q_want = ref.mrope(f[:, :hq], cos, sin, gq.float(), 1e-6)
    k_want = ref.mrope(f[:, hq:hq + hkv], cos, sin, gk.float(), 1e-6)
    _close(q, q_want, 2e-2, 2e-2, "q")
    pg, off = slots // page, slots % page
    _close(kc[pg, :, off], k_want, 2e-2, 2e-2, "k rows")
    assert torch.equal(vc[pg, :, off], qkv[:, hq + hkv:])
    # every other cache row is untouched
    mask = torch.ones(n_pages, page, dtype=torch.bool, device=DEV)
    mask[pg, off] = False
    assert torch.equal(kc.transpose(1, 2)[mask], kc0.transpose(1, 2)[mask])
    assert torch.equal(vc.transpose(1, 2)[mask], vc0.transpose(1, 2)[mask])


@pytest.mark.parametrize("epi", [ops.EPI_PLAIN, ops.EPI_SWIGLU, ops.EPI_GATED_RESID])
def test_gemm_grouped_two_segments(epi):
    """MoT routing: an AR segment and a DM segment with their own weights in one launch."""
    torch.manual_seed(17)
    k, n = 256, 512
    m0, m1 = 200, 1100
    a0, a1 = _rand(m0, k), _rand(2, m1 // 2, k)
    w0, w1 = _rand(n, k, scale=1 / 16), _rand(n, k, scale=1 / 16)
    n_out = n // 2 if epi == ops.EPI_SWIGLU else n
    r0 = r1 = g1 = None
    if epi == ops.EPI_GATED_RESID:
        r0, r1, g1 = _rand(m0, n_out), _rand(2, m1 // 2, n_out), _rand(2, n_out)
    c0, c1 = ops.gemm_grouped2(a0, w0, a1, w1, epi, r0, r1, None, g1, m0, m1 // 2)
    f = lambda t: None if t is None else t.float()  # noqa: E731
    want0 = ref.gemm(a0.float(), w0.float(), None, epi, f(r0), None, m0)
    want1 = ref.gemm(a1.float(), w1.float(), None, epi, f(r1), f(g1), m1 // 2)
    assert c0.shape == want0.shape and c1.shape == want1.shape
    _close(c0, want0, 3e-2, 2e-2, "grouped segment 0")
    _close(c1, want1, 3e-2, 2e-2, "grouped segment 1")


@pytest.mark.parametrize("m,n,k,epi", [(32, 768, 4096, ops.EPI_PLAIN), (32, 3072, 4096, ops.EPI_SWIGLU),
                                        (32, 4096, 1536, ops.EPI_GATED_RESID), (7, 512, 1024, ops.EPI_PLAIN),
                                        (64, 1000, 2048, ops.EPI_PLAIN),
                                        # more than one 128-row tile: split-K on CTA pairs
                                        (256, 6144, 4096, ops.EPI_PLAIN), (200, 4096, 12288, ops.EPI_GATED_RESID),
                                        (384, 1024, 4096, ops.EPI_PLAIN), (256, 24576, 4096, ops.EPI_SWIGLU)])
def test_gemm_skinny_split_k(m, n, k, epi):
    """Decode-sized problems take the split-K path (fp32 partials + reduce/epilogue kernel)."""
    torch.manual_seed(18)
    a = _rand(m, k)
    w = _rand(n, k, scale=1 / math.sqrt(k))
    r = _rand(m, n) if epi == ops.EPI_GATED_RESID else None
    got = ops.gemm(a, w, None, epi, r, None, m)
    want = ref.gemm(a.float(), w.float(), None, epi, None if r is None else r.float(), None, m)
    _close(got, want, 3e-2, 2e-2, f"skinny gemm {m}x{n}x{k} epi {epi}")


@pytest.mark.parametrize("cin,cout", [(64, 128), (64, 64), (128, 32), (64, 256), (128, 384)])
def test_conv3d_implicit_gemm_matches_conv3d(cin, cout):
    """One causal 3x3x3 convolution on a padded channels-last volume vs F.conv3d (64 / 128 output channels and fewer
    run narrower MMAs; 384 takes two n tiles)."""
    import torch.nn.functional as F
    torch.manual_seed(19)
    t, h, w = 5, 12, 20
    x = _rand(1, cin, t, h, w)
    wt = _rand(cout, cin, 3, 3, 3, scale=1 / math.sqrt(27 * cin))
    b = _rand(cout)
    r = _rand(1, cout, t, h, w)
    want = F.conv3d(F.pad(x.float(), (1, 1, 1, 1, 2, 0)), wt.float(), b.float()) + r.float()
    vol = torch.zeros(t + 2, h + 2, w + 2, cin, device=DEV, dtype=torch.bfloat16)
    vol[2:, 1:-1, 1:-1] = x[0].permute(1, 2, 3, 0)
    rv = torch.zeros(t + 2, h + 2, w + 2, cout, device=DEV, dtype=torch.bfloat16)
    rv[2:, 1:-1, 1:-1] = r[0].permute(1, 2, 3, 0)
    wp = wt.permute(0, 2, 3, 4, 1).reshape(cout, 27 * cin).contiguous()
    out = torch.zeros(t + 2, h + 2, w + 2, cout, device=DEV, dtype=torch.bfloat16)
    torch.ops.cosmos_b200.conv3d_cl(vol, wp, b, rv, out, 2)
    got = out[2:, 1:-1, 1:-1].permute(3, 0, 1, 2)[None]
    _close(got, want, 3e-2, 2e-2, "implicit-GEMM conv3d")
    assert out[:2].abs().max() == 0 and out[:, 0].abs().max() == 0 and out[:, :, -1].abs().max() == 0


@pytest.mark.parametrize("cin,cout,tpad", [(64, 64, 2), (128, 320, 2), (64, 256, 1), (64, 32, 0)])
def test_conv3d_cl_writes_the_interior_only(cin, cout, tpad):
    """Border cells and the frames before `tpad` keep what they hold; the interior has the bits of the form that zeroes its border."""
    torch.manual_seed(24)
    k = torch.ops.cosmos_b200
    vol = torch.zeros(6, 14, 22, cin, device=DEV, dtype=torch.bfloat16)
    vol[:, 1:-1, 1:-1] = _rand(6, 12, 20, cin)
    wp, b = _rand(cout, 27 * cin, scale=1 / math.sqrt(27 * cin)), _rand(cout)
    out = torch.full((6, 14, 22, cout), 7.0, device=DEV, dtype=torch.bfloat16)
    k.conv3d_cl(vol, wp, b, None, out, tpad)
    full = torch.empty_like(out)
    k.conv3d_fused(vol, wp, b, None, None, full, None, None, 1e-6, 0, 0, 0)
    lo = max(tpad, 2)
    assert torch.equal(out[lo:, 1:-1, 1:-1], full[lo:, 1:-1, 1:-1])
    assert (out[tpad:, 1:-1, 1:-1] != 7).any(-1).all()
    out[tpad:, 1:-1, 1:-1] = 7.0
    assert (out == 7).all()


def test_vae_channels_last_decoder_matches_pytorch():
    from cosmos_b200.models.vae import CausalVideoVAE
    from cosmos_b200.models.vae_cuda import CLDecoder
    torch.manual_seed(20)
    vae = CausalVideoVAE(16, (64, 128, 256, 256)).to(DEV).float().eval()
    z = torch.randn(1, 16, 3, 6, 8, device=DEV)
    with torch.no_grad():
        want = CausalVideoVAE.to_uint8(vae.decode(z))
    dec = CLDecoder(vae)
    got = dec.decode(z, chunk_latents=2)
    assert got.shape == want.shape == (1, 9, 48, 64, 3)
    diff = (got.int() - want.int()).abs()
    assert diff.float().mean() < 1.5 and (diff > 8).float().mean() < 0.01, (diff.float().mean(), diff.max())
    one = dec.decode(z, chunk_latents=3)
    assert (one.int() - got.int()).abs().max() <= 1  # chunking does not change the result


@pytest.mark.parametrize("m,n,k", [(256, 512, 384), (300, 264, 1000), (1024, 4096, 2048)])
def test_gemm_operand_majors(m, n, k):
    """Backward-pass GEMMs read transposed operands in place (MN-major shared-memory tiles)."""
    torch.manual_seed(21)
    dy = _rand(m, n)                       # [tokens, out]
    w = _rand(n, k, scale=1 / math.sqrt(n))  # [out, in]
    x = _rand(m, k)                        # [tokens, in]
    dx = torch.ops.cosmos_b200.gemm_ex(dy, w, False, True, None)       # dY @ W
    _close(dx, dy.float() @ w.float(), 3e-2, 2e-2, "dX = dY W")
    dw = torch.ops.cosmos_b200.gemm_ex(dy, x, True, True, None)        # dY^T @ X
    _close(dw, (dy.float().t() @ x.float()) / 1.0, 6e-2, 3e-2, "dW = dY^T X")


def test_linear_autograd_on_own_kernels():
    from cosmos_b200.ops import autograd as own
    torch.manual_seed(22)
    x = _rand(2, 300, 256).requires_grad_(True)
    w = _rand(512, 256, scale=1 / 16).requires_grad_(True)
    y = own.linear(x, w)
    g = _rand(2, 300, 512)
    y.backward(g)
    xf, wf = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    (xf @ wf.t()).backward(g.float())
    _close(y, xf @ wf.t(), 3e-2, 2e-2, "linear fwd")
    _close(x.grad, xf.grad, 3e-2, 2e-2, "linear dX")
    _close(w.grad, wf.grad, 8e-2, 3e-2, "linear dW")


@pytest.mark.parametrize("materialized", [False, True])
@pytest.mark.parametrize("b,sq,skv,hq,hkv,mask,n_ar", [
    (1, 384, 384, 4, 2, ops.MASK_FULL, 0), (1, 300, 300, 2, 1, ops.MASK_CAUSAL, 0),
    (1, 256, 520, 2, 2, ops.MASK_FULL, 0), (2, 640, 640, 8, 2, ops.MASK_MOT, 200),
    (1, 130, 700, 4, 1, ops.MASK_CAUSAL, 0), (2, 1024, 1024, 4, 4, ops.MASK_FULL, 0)])
def test_attention_autograd_on_own_kernels(b, sq, skv, hq, hkv, mask, n_ar, materialized, monkeypatch):
    from cosmos_b200.ops import autograd as own
    monkeypatch.setattr(own, "_MATERIALIZED", materialized)
    if materialized and b * hq > 8:
        pytest.skip("the per-head variant is covered by the smaller cases")
    torch.manual_seed(23)
    q = _rand(b, sq, hq, 128).requires_grad_(True)
    k = _rand(b, skv, hkv, 128).requires_grad_(True)
    v = _rand(b, skv, hkv, 128).requires_grad_(True)
    g = _rand(b, sq, hq, 128)
    o = own.attention(q, k, v, None, mask, n_ar)
    o.backward(g)
    torch.cuda.synchronize()
    ops.check_status()
    qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    of, _ = ref.attention(qf, kf, vf, None, mask, n_ar)
    of.backward(g.float())
    _close(o, of, 2e-2, 2e-2, "attention fwd")
    _close(q.grad, qf.grad, 3e-2, 3e-2, "dQ")
    _close(k.grad, kf.grad, 3e-2, 3e-2, "dK")
    _close(v.grad, vf.grad, 3e-2, 3e-2, "dV")


@pytest.mark.parametrize("sq,skv", [(1, 1), (128, 129), (129, 512), (385, 128), (256, 897), (1025, 641)])
def test_attention_backward_rings(sq, skv):
    """One to nine tiles through rings of two and three slots, with full and ragged last tiles. bf16 P and dS as in the
    case above, whose bounds hold for fewer terms too."""
    from cosmos_b200.ops import autograd as own
    torch.manual_seed(29)
    t = [_rand(2, s, h, 128) for s, h in ((sq, 4), (skv, 2), (skv, 2))]
    g = _rand(2, sq, 4, 128)
    a = [x.clone().requires_grad_(True) for x in t]
    own.attention(*a, None, ops.MASK_FULL, 0).backward(g)
    torch.cuda.synchronize()
    ops.check_status()
    f = [x.float().requires_grad_(True) for x in t]
    ref.attention(*f, None, ops.MASK_FULL, 0)[0].backward(g.float())
    for x, y, n in zip(a, f, ("dQ", "dK", "dV")):
        _close(x.grad, y.grad, 3e-2, 3e-2, n)


@pytest.mark.parametrize("b,s,h", [(1, 1, 1), (2, 33, 3), (1, 130, 32)])
def test_attention_backward_delta(b, s, h):
    o, do = _rand(b, s, h, 128), _rand(b, h, s, 128).transpose(1, 2)
    flat = torch.empty(o.numel() + 1, dtype=o.dtype, device=o.device)
    odd = flat[1:].view_as(o).copy_(o)   # starts at an odd element
    want = (do.double() * o.double()).sum(-1).permute(0, 2, 1)
    bound = 128 * 2 ** -24 * (do.double() * o.double()).abs().sum(-1).permute(0, 2, 1)   # exact products, 128 sums in fp32
    same = (do.contiguous().float() * o.float()).sum(-1).permute(0, 2, 1)
    for x in (o, odd):
        got = torch.ops.cosmos_b200.attn_bwd_delta(do, x)
        assert ((got.double() - want).abs() <= bound).all()
        assert b * s * h < 16 or torch.equal(got, same)


@pytest.mark.parametrize("b,d,unused", [(1, 4096, ()), (2, 1032, (1,)), (7, 8, (0, 5))])
def test_dm_modulation(b, d, unused):
    """The bits of the expressions that it stands for: a sum rounded once, gradients that are copies, and a sum over the batch in
    fp32 that is rounded once (its order is the reduction's up to four entries; beyond, two spacings of bf16)."""
    from cosmos_b200.models.mot import dm_modulation
    t, tab = _rand(b, 6 * d), _rand(6, d)
    want = [(t.view(b, 6, d).float() + tab.float()[None]).to(t.dtype)[:, i] for i in range(6)]
    odd = torch.empty(tab.numel() + 1, dtype=tab.dtype, device=tab.device)[1:].view_as(tab).copy_(tab)
    for table in (tab, odd):
        assert all(torch.equal(x, y) for x, y in zip(dm_modulation(t, table), want))
    t1, tab1 = t.clone().requires_grad_(True), tab.clone().requires_grad_(True)
    t2, tab2 = t.clone().requires_grad_(True), tab.clone().requires_grad_(True)
    g = [_rand(b, d) for _ in range(6)]
    use = [i for i in range(6) if i not in unused]
    got = dm_modulation(t1, tab1)
    torch.autograd.backward([got[i] for i in use], [g[i] for i in use])
    m = (t2.view(b, 6, d).float() + tab2.float()[None]).to(t.dtype)
    torch.autograd.backward([m[:, i] for i in use], [g[i] for i in use])
    assert torch.equal(t1.grad, t2.grad)
    if b <= 4:
        assert torch.equal(tab1.grad, tab2.grad)
    assert ((tab1.grad - tab2.grad).abs() <= 2 ** -7 * tab2.grad.abs()).all()


def test_dm_modulation_of_an_empty_batch():
    """The table's gradient is the sum over no entries. Deterministic algorithms fill new memory with NaN, so that a result that
    nobody wrote shows."""
    from cosmos_b200.models.mot import dm_modulation
    t, tab = torch.empty(0, 6 * 64, device=DEV, dtype=torch.bfloat16).requires_grad_(True), _rand(6, 64).requires_grad_(True)
    rows = dm_modulation(t, tab)
    assert all(r.shape == (0, 64) for r in rows)
    torch.use_deterministic_algorithms(True)
    try:
        torch.autograd.backward(rows, [torch.empty_like(r) for r in rows])
    finally:
        torch.use_deterministic_algorithms(False)
    assert t.grad.shape == t.shape and tab.grad.shape == tab.shape and not tab.grad.any()


def _modulation_expressions(t, tab):
    b, d = t.shape[0], tab.shape[-1]
    m = (t.view(b, 6, d).float() + tab.float()[None]).to(t.dtype)
    return [m[:, i].contiguous() for i in range(6)]


@pytest.mark.parametrize("b", [1, 3])
def test_dm_modulation_under_transforms(b):
    """What looks through the operations sees the expressions: forward mode, functorch, fake tensors, a second derivative."""
    from torch._subclasses.fake_tensor import FakeTensorMode
    from torch.autograd import forward_ad as fw
    from cosmos_b200.models.mot import dm_modulation
    t, tab, dt, dtab = _rand(b, 6 * 16), _rand(6, 16), _rand(b, 6 * 16), _rand(6, 16)
    with fw.dual_level():
        got = [fw.unpack_dual(x).tangent for x in dm_modulation(fw.make_dual(t, dt), fw.make_dual(tab, dtab))]
    assert all(torch.equal(x, y) for x, y in zip(got, _modulation_expressions(dt, dtab)))
    vm = torch.func.vmap(lambda x: tuple(dm_modulation(x, tab)))(torch.stack([t, dt]))
    assert all(torch.equal(x[1], y) for x, y in zip(vm, _modulation_expressions(dt, tab)))
    want = torch.func.vjp(lambda x, y: torch.stack(_modulation_expressions(x, y)), t, tab)[1](_rand(6, b, 16).fill_(0.5))
    got = torch.func.vjp(lambda x, y: torch.stack(dm_modulation(x, y)), t, tab)[1](_rand(6, b, 16).fill_(0.5))
    assert all(torch.equal(x, y) for x, y in zip(got, want))
    with FakeTensorMode():
        rows = dm_modulation(torch.empty(b, 96, device=DEV, dtype=torch.bfloat16), torch.empty(6, 16, device=DEV, dtype=torch.bfloat16))
        assert all(r.shape == (b, 16) for r in rows)
    second = []
    for f in (dm_modulation, _modulation_expressions):
        p, q = t.clone().requires_grad_(True), tab.clone().requires_grad_(True)
        first = torch.autograd.grad(sum((r * r).sum() for r in f(p, q)), (p, q), create_graph=True)
        second.append(first + torch.autograd.grad(sum((x * x).sum() for x in first), (p, q)))
    assert all(torch.equal(x, y) for x, y in zip(*second))


def test_dm_modulation_of_other_forms():
    from cosmos_b200.models.mot import dm_modulation
    t, one = _rand(2, 6 * 16), _rand(1, 16)
    assert all(torch.equal(x, y) for x, y in zip(dm_modulation(t, one), _modulation_expressions(t, one)))   # one row for all six
    with pytest.raises(RuntimeError):
        dm_modulation(t, _rand(6, 16).cpu())
    assert all(r.shape == (2, 0) for r in dm_modulation(_rand(2, 0), _rand(6, 0)))
    p, q = t.clone().requires_grad_(True), _rand(6, 16).requires_grad_(True)
    rows = dm_modulation(p, q)
    rows[1].mul_(3)                       # rows of their own: the others do not see it
    torch.stack(rows).sum().backward()
    want = torch.ones(2, 6, 16, device=DEV)
    want[:, 1] = 3
    assert torch.equal(p.grad.float(), want.view(2, 96)) and torch.equal(q.grad.float(), want.sum(0))


@pytest.mark.parametrize("b,one,n,rows,h", [(1, False, 1, 3, 2), (2, True, 77, 317, 8), (3, False, 5, 5, 1), (2, False, 0, 4, 2)])
@pytest.mark.parametrize("form", ["contiguous", "view of a projection", "odd start"])
def test_copy_prefix(b, one, n, rows, h, form):
    bp = 1 if one else b
    if form == "view of a projection":
        qkv = _rand(bp, n, 3 * h, 128)
        k, v = qkv[:, :, h:2 * h], qkv[:, :, 2 * h:]
    elif form == "odd start":
        k, v = (_rand(bp * n * h * 128 + 1)[1:].view(bp, n, h, 128) for _ in range(2))
    else:
        k, v = _rand(bp, n, h, 128), _rand(bp, n, h, 128)
    kb, vb = _rand(b, rows, h, 128), _rand(b, rows, h, 128)
    wk, wv = kb.clone(), vb.clone()
    wk[:, :n], wv[:, :n] = k, v
    torch.ops.cosmos_b200.copy_prefix(k, v, kb, vb)
    assert torch.equal(kb, wk) and torch.equal(vb, wv)


@pytest.mark.parametrize("form", ["one head", "fp32", "keys alone of one head"])
def test_workspace_prefix_of_other_forms(form):
    """Prefixes that the copies into the workspace spread over the heads or cast: the keys and values that `attend` gets."""
    from cosmos_b200.config import get_model_config
    from cosmos_b200.models.mot import WorkspaceAttn
    cfg = get_model_config("tiny128")
    b, s, n, hk, hd = 2, 5, 3, cfg.n_kv_heads, cfg.head_dim
    h, w = _rand(b, s, cfg.d_model), _rand(cfg.q_dim + 2 * cfg.kv_dim, cfg.d_model, scale=0.05)
    ang = torch.rand(s, 64, device=DEV)
    norm = torch.ones(hd, device=DEV, dtype=torch.bfloat16)
    wide, one = (_rand(b, n, hk, hd), _rand(b, n, hk, hd)), (_rand(b, n, 1, hd), _rand(b, n, 1, hd))
    prefix = {"one head": one, "fp32": (wide[0].float(), wide[1].float()), "keys alone of one head": (one[0], wide[1])}[form]
    with torch.no_grad():
        _, k, v = WorkspaceAttn().qkv_project(h, w, ang.cos(), ang.sin(), norm, norm, cfg, prefix=prefix)
    for got, p in ((k, prefix[0]), (v, prefix[1])):
        assert got.shape == (b, n + s, hk, hd) and torch.equal(got[:, :n], p.bfloat16().expand(b, n, hk, hd))


@pytest.mark.parametrize("n,theta,section", [(1, 5.0e5, (24, 20, 20)), (333, 1.0e4, (24, 20, 20)), (2001, 5.0e6, (10, 11, 11))])
def test_rope_tables(n, theta, section):
    """The bits of the expressions in fp64, for positions up to a million and in any layout."""
    from cosmos_b200.models import rope
    pos = torch.randint(0, 10 ** 6, (n, 3), generator=torch.Generator().manual_seed(n)).t()   # [3, n], rows strided
    want = rope.rope_tables(pos, 2 * sum(section), theta, section)
    for p in (pos.cuda(), pos.cuda().contiguous()):
        got = rope.rope_tables(p, 2 * sum(section), theta, section)
        for x, y in zip(got, want):   # the CPU's own library: half a spacing of fp32 at most
            assert (x.cpu() - y).abs().max() <= 2 ** -24


@pytest.mark.parametrize("head_dim,section", [(129, (24, 20, 20)), (7, (3, 0, 0)), (6, (1, 1, 1)), (600, (100, 100, 100)), (1, (0, 0, 0))])
def test_rope_tables_of_other_sizes(head_dim, section):
    """Odd head sizes (half of them has a frequency), sizes above the kernel's, none at all: as the expressions on the CPU."""
    from cosmos_b200.models import rope
    pos = torch.arange(33).expand(3, -1)
    for x, y in zip(rope.rope_tables(pos.cuda(), head_dim, 1.0e4, section), rope.rope_tables(pos, head_dim, 1.0e4, section)):
        assert x.shape == y.shape and (x.cpu() - y).abs().le(2 ** -24).all()


def test_rope_tables_other_forms():
    from cosmos_b200.models import rope
    pos = torch.arange(9, device=DEV).expand(3, -1)
    want = rope.rope_tables(pos, 6, 1.0e4, (1, 1, 1))
    got = torch.func.vmap(lambda p: rope.rope_tables(p, 6, 1.0e4, (1, 1, 1)))(torch.stack([pos, pos + 1]))
    tensor = rope.rope_tables(pos, 6, torch.tensor(1.0e4, dtype=torch.float64, device=DEV), (1, 1, 1))
    for x, y, z in zip(got, want, tensor):
        assert (x[0] - y).abs().max() <= 2 ** -24 and (z - y).abs().max() <= 2 ** -24
    for bad in ((3,), (1, 2), (1, 1, 1, 0)):    # three sections, whatever they add up to
        with pytest.raises(ValueError):
            rope.rope_tables(pos, 6, 1.0e4, bad)


@pytest.mark.parametrize("b,d,page,delta,inc", [(1, 64, 16, False, False), (3, 4096, 32, True, True), (70, 1032, 16, True, False)])
def test_decode_begin(b, d, page, delta, inc):
    from types import SimpleNamespace
    from cosmos_b200.serve.decoder import TPDecoder
    g = torch.Generator(device="cuda").manual_seed(b)
    ids = lambda hi, *s: torch.randint(0, hi, s, generator=g, device="cuda")  # noqa: E731
    dec = SimpleNamespace(lens=ids(20 * page, b).int(), tokens=ids(1000, b), table=ids(5000, b, 20).int(), page_size=page, embed=_rand(1000, d),
                          inv_freq=torch.rand(64, generator=g, device="cuda"), pos_delta=-ids(7, b) if delta else None,
                          step_inc=ids(2, b).int() if inc else None)
    lens = dec.lens.clone()
    got = torch.ops.cosmos_b200.decode_begin(lens, dec.step_inc, dec.pos_delta, dec.inv_freq, dec.table, page, dec.tokens, dec.embed)
    want = TPDecoder._begin_step(dec)
    assert torch.equal(got[0], want[0]) and torch.equal(got[3], want[3]) and torch.equal(lens, dec.lens)
    for x, y in zip(got[1:3], want[1:3]):
        assert (x - y).abs().max() <= 2 ** -22   # two spacings of the functions' results
    torch.cuda.synchronize()
    ops.check_status()


@pytest.mark.parametrize("b,v,stride", [(1, 151936, 151936), (33, 1000, 1000), (2, 7, 7), (3, 4097, 5001), (1, 1, 1)])
def test_greedy_pick(b, v, stride):
    x = _rand(b, stride)[:, :v]
    x[0, v // 2:] = x[0].max() + 1          # ties: the smallest index
    if b > 2:
        x[1] = -float("inf")
        x[2, v - 1] = float("nan")          # counts as the largest
    nxt = torch.full((b,), -1, device="cuda")
    torch.ops.cosmos_b200.greedy_pick(x, 0, v - 1, nxt)
    assert torch.equal(nxt, x.float().max(dim=-1)[1])
    torch.ops.cosmos_b200.greedy_pick(x, 3, 5, nxt)
    assert torch.equal(nxt, (x.float().max(dim=-1)[1] + 3).clamp(max=5))


def test_early_launches_under_capture():
    """Kernels that start behind the end of the one before them, as nodes of a graph: behind a copy, behind a kernel of torch, as the first
    node of a joined side stream and behind one another. Each replay sees what that replay's kernels wrote."""
    x, w1, w2, gam = _rand(300, 1024), _rand(1024, 1024) * 0.05, _rand(1024, 1024) * 0.05, _rand(1024)
    src = _rand(300, 1024)

    def work(side):
        x.copy_(src)                                           # a copy, then a norm
        h, _ = ops.rmsnorm(x, gam, 1e-6)
        a = ops.gemm(h, w1)                                    # on CTA pairs
        y = ops.gemm(a, w2, None, ops.EPI_GATED_RESID, x, None, 300)
        cur = torch.cuda.current_stream()
        side.wait_stream(cur)
        with torch.cuda.stream(side):
            z = ops.gemm(y[:16], w1)                           # single CTAs, split-K, first on its stream
        cur.wait_stream(side)
        q = ops.gemm(y, w1).view(1, 300, 8, 128)
        o, _ = ops.attention(q, q[:, :, :2], q[:, :, 2:4])
        return ops.rmsnorm((o.view(300, 1024) @ w2.t()) * 2, gam, 1e-6)[0], z

    side, cap = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(cap):
        work(side)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=cap):
            out = work(side)
    for seed in range(3):
        torch.manual_seed(seed)
        src.copy_(torch.randn(300, 1024, device=DEV))
        g.replay()
        got = [t.clone() for t in out]
        want = work(side)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    ops.check_status()


def _grads_close(own_in, ref_in, names, atol=4e-2, rtol=4e-2):
    for a, b, n in zip(own_in, ref_in, names):
        assert a.grad is not None, f"no gradient for {n}"
        _close(a.grad, b.grad, atol, rtol, f"d{n}")


@pytest.mark.parametrize("b,s,d", [(2, 300, 512), (1, 200, 4096), (3, 64, 1024)])
def test_norm_autograd_on_own_kernels(b, s, d):
    """AdaLN-RMSNorm and plain RMSNorm: forward and backward kernels against fp32 autograd."""
    from cosmos_b200.ops import autograd as own
    torch.manual_seed(31)
    x = _rand(b, s, d).requires_grad_(True)
    gamma = (1 + 0.1 * torch.randn(d, device=DEV)).bfloat16().requires_grad_(True)
    mod = (0.3 * torch.randn(b, 2, d, device=DEV)).bfloat16().requires_grad_(True)
    g = _rand(b, s, d)
    y = own.adaln_rmsnorm(x, gamma, mod[:, 0], mod[:, 1], s, 1e-6)
    y.backward(g)
    xf, gf, mf = (t.detach().float().requires_grad_(True) for t in (x, gamma, mod))
    yf = ref.adaln_rmsnorm(xf, gf, mf[:, 0], mf[:, 1], s, 1e-6)
    yf.backward(g.float())
    _close(y, yf, 3e-2, 3e-2, "adaln fwd")
    _grads_close((x, mod), (xf, mf), ("x", "mod"))
    _close(gamma.grad, gf.grad, 0.5, 5e-2, "dgamma")  # sums over b*s rows of bf16-rounded terms
    x2 = _rand(b * s, d).requires_grad_(True)
    gamma2 = (1 + 0.1 * torch.randn(d, device=DEV)).bfloat16().requires_grad_(True)
    y2 = own.rmsnorm(x2, gamma2, 1e-6)
    y2.backward(g.reshape(b * s, d))
    x2f, g2f = x2.detach().float().requires_grad_(True), gamma2.detach().float().requires_grad_(True)
    y2f, _ = ref.rmsnorm(x2f, g2f, 1e-6)
    y2f.backward(g.reshape(b * s, d).float())
    _close(y2, y2f, 3e-2, 3e-2, "rmsnorm fwd")
    _close(x2.grad, x2f.grad, 4e-2, 4e-2, "rmsnorm dx")
    _close(gamma2.grad, g2f.grad, 0.5, 5e-2, "rmsnorm dgamma")
    ops.check_status()


def test_qkv_post_autograd_on_own_kernels():
    from cosmos_b200.ops import autograd as own
    torch.manual_seed(32)
    rows, hq, hk, rr = 70, 4, 2, 35
    qkv = _rand(rows, hq + 2 * hk, 128).requires_grad_(True)
    ang = torch.rand(rr, 64, device=DEV) * 6.0
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    gq = (1 + 0.1 * torch.randn(128, device=DEV)).bfloat16().requires_grad_(True)
    gk = (1 + 0.1 * torch.randn(128, device=DEV)).bfloat16().requires_grad_(True)
    go = [_rand(rows, h, 128) for h in (hq, hk, hk)]
    q, k, v = own.qkv_post(qkv, hq, cos, sin, gq, gk, 1e-6)
    torch.autograd.backward([q, k, v], go)
    f, gqf, gkf = (t.detach().float().requires_grad_(True) for t in (qkv, gq, gk))
    qf = ref.mrope(f[:, :hq], cos, sin, gqf, 1e-6)
    kf = ref.mrope(f[:, hq:hq + hk], cos, sin, gkf, 1e-6)
    vf = f[:, hq + hk:]
    torch.autograd.backward([qf, kf, vf], [t.float() for t in go])
    _close(q, qf, 3e-2, 3e-2, "q")
    _close(k, kf, 3e-2, 3e-2, "k")
    assert torch.equal(v, qkv.detach()[:, hq + hk:])
    _close(qkv.grad, f.grad, 4e-2, 4e-2, "dqkv")
    _close(gq.grad, gqf.grad, 0.3, 5e-2, "dgamma_q")
    _close(gk.grad, gkf.grad, 0.3, 5e-2, "dgamma_k")
    ops.check_status()


@pytest.mark.parametrize("rows,hq,hk", [(1, 1, 1), (9, 3, 1), (70, 5, 2), (1300, 7, 1)])
def test_qkv_post_head_counts(rows, hq, hk):
    """Heads that do not fill the last group of four, of one head and of several rows a warp. The norm weights' gradient comes out
    the same every time."""
    kern = torch.ops.cosmos_b200
    torch.manual_seed(rows)
    qkv, go = _rand(rows, hq + 2 * hk, 128), [_rand(rows, h, 128) for h in (hq, hk, hk)]
    ang = torch.rand(rows, 64, device=DEV) * 6.0
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    gq, gk = ((1 + 0.1 * torch.randn(128, device=DEV)).bfloat16() for _ in range(2))
    out = kern.qkv_post_fwd(qkv, hq, cos, sin, gq, gk, 1e-6)
    f, gqf, gkf = (t.float().requires_grad_(True) for t in (qkv, gq, gk))
    want = ref.mrope(f[:, :hq], cos, sin, gqf, 1e-6), ref.mrope(f[:, hq:hq + hk], cos, sin, gkf, 1e-6), f[:, hq + hk:]
    torch.autograd.backward(want, [t.float() for t in go])
    for x, y in zip(out, want):
        assert ((x.float() - y).abs() <= 2 ** -8 * y.abs() + 1e-5).all()       # one rounding to bf16
    d, part = kern.qkv_post_bwd(qkv, *go, cos, sin, gq, gk, 1e-6)
    assert ((d.float() - f.grad).abs() <= 2 ** -8 * f.grad.abs() + 1e-5).all()
    assert (part.sum(0)[0] - gqf.grad).abs().max() <= 1e-5 * rows * hq and (part.sum(0)[1] - gkf.grad).abs().max() <= 1e-5 * rows * hk
    assert torch.equal(part, kern.qkv_post_bwd(qkv, *go, cos, sin, gq, gk, 1e-6)[1])


def test_swiglu_and_gated_residual_autograd_on_own_kernels():
    from cosmos_b200.ops import autograd as own
    torch.manual_seed(33)
    gu = _rand(100, 512).requires_grad_(True)
    g = _rand(100, 256)
    y = own.swiglu(gu)
    y.backward(g)
    guf = gu.detach().float().requires_grad_(True)
    yf = ref.swiglu(guf)
    yf.backward(g.float())
    _close(y, yf, 3e-2, 3e-2, "swiglu fwd")
    _close(gu.grad, guf.grad, 4e-2, 4e-2, "swiglu bwd")
    b, s, d = 2, 150, 1024
    x, f = _rand(b * s, d).requires_grad_(True), _rand(b * s, d).requires_grad_(True)
    gate = (0.5 * torch.randn(b, d, device=DEV)).bfloat16().requires_grad_(True)
    go = _rand(b * s, d)
    y = own.gated_residual(x, f, gate, s)
    y.backward(go)
    xf, ff, gf = (t.detach().float().requires_grad_(True) for t in (x, f, gate))
    yf = ref.gated_residual(xf, ff, gf, s)
    yf.backward(go.float())
    _close(y, yf, 3e-2, 3e-2, "gated residual fwd")
    _grads_close((x, f), (xf, ff), ("x", "f"))
    _close(gate.grad, gf.grad, 0.5, 5e-2, "dgate")
    ops.check_status()


def test_training_step_own_kernels_match_library_baseline(monkeypatch):
    """One optimizer step of a small head_dim-128 model: the autograd path on this package's kernels
    against the PyTorch / library path (same seeds), compared on loss, gradient norm and parameters."""
    from cosmos_b200.config import ParallelConfig, tiny128_config
    from cosmos_b200.models.mot import MoTModel
    from cosmos_b200.parallel.mesh import Mesh
    from cosmos_b200.train import TrainConfig, Trainer

    def run(library):
        if library:
            monkeypatch.setenv("COSMOS_TRAIN_LIBRARY_BACKWARD", "1")
        else:
            monkeypatch.delenv("COSMOS_TRAIN_LIBRARY_BACKWARD", raising=False)
        cfg = tiny128_config(max_text_len=32, n_layers=2)
        model = MoTModel(cfg, dtype=torch.bfloat16, device=DEV, pad_to=128)
        model.init_weights(seed=3)
        tr = Trainer(model, Mesh(ParallelConfig(), 1, 0), TrainConfig(lr=1e-3, max_grad_norm=0.5))
        g = torch.Generator(device=DEV).manual_seed(100)
        lat = torch.randn(1, 16, 3, 16, 16, generator=g, device=DEV, dtype=torch.bfloat16)
        ids = torch.randint(0, cfg.vocab_size, (1, 32), generator=g, device=DEV)
        t = torch.rand(1, generator=g, device=DEV)
        eps = torch.randn(lat.shape, generator=g, device=DEV, dtype=torch.bfloat16)
        log = tr.train_step(lat, ids, t=t, eps=eps)
        torch.cuda.synchronize()
        ops.check_status()
        return log, tr.fsdp.full_state()

    log_o, st_o = run(False)
    log_l, st_l = run(True)
    assert abs(log_o["loss"] - log_l["loss"]) < 2e-2 * max(1.0, abs(log_l["loss"]))
    assert abs(log_o["grad_norm"] - log_l["grad_norm"]) < 5e-2 * max(1.0, log_l["grad_norm"])
    worst = max((st_o[k].float() - st_l[k].float()).abs().max().item() for k in st_l)
    assert worst < 2e-2, f"parameters differ by {worst}"


@pytest.mark.parametrize("m,n,k", [(32, 4096, 4096), (1, 4096, 12288), (7, 1024, 2048), (300, 512, 256),
                                   (256, 4096, 12288), (130, 4096, 4096)])
def test_gemm_reduce_rmsnorm(m, n, k):
    """Output projection + residual + RMS-norm (the split-K reduction pass does all three for skinny problems;
    the last shape takes the unfused fallback) against the fp32 definition."""
    torch.manual_seed(41)
    a = _rand(m, k)
    w = _rand(n, k, scale=1 / math.sqrt(k))
    resid = _rand(m, n)
    gamma = (1 + 0.1 * torch.randn(n, device=DEV)).bfloat16()
    h, x_new = ops.gemm_reduce_rmsnorm(a, w, resid, gamma, 1e-6)
    torch.cuda.synchronize()
    ops.check_status()
    xf = resid.float() + a.float() @ w.float().t()
    hf = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-6) * gamma.float()
    _close(x_new, xf, 3e-2, 2e-2, "x_new")
    _close(h, hf, 3e-2, 2e-2, "h")



def test_kernels_do_not_write_outside_their_outputs():
    """Canary check: outputs are views into larger buffers whose guard regions hold a bit pattern; after ragged
    GEMM, QKV-epilogue and attention launches the guards must be untouched."""
    torch.manual_seed(43)
    guard = 4096  # elements before and after

    def guarded(rows, cols):
        buf = torch.full((2 * guard + rows * cols,), -7.0, device=DEV, dtype=torch.bfloat16)
        return buf, buf[guard:guard + rows * cols].view(rows, cols)

    def intact(buf, what):
        assert bool((buf[:guard] == -7.0).all()) and bool((buf[-guard:] == -7.0).all()), f"{what}: guard region overwritten"

    for m, n, k in [(300, 264, 1000), (1, 512, 256), (129, 136, 72)]:
        a, w = _rand(m, k), _rand(n, k, scale=1 / math.sqrt(k))
        buf, out = guarded(m, n)
        ops.gemm(a, w, out=out)
        torch.cuda.synchronize()
        intact(buf, f"gemm {m}x{n}x{k}")
        _close(out, a.float() @ w.float().t(), 3e-2, 3e-2, "gemm into a guarded view")
    # SwiGLU epilogue writes N / 2 columns
    a, w = _rand(77, 512), _rand(1024, 512, scale=1 / math.sqrt(512))
    buf, out = guarded(77, 512)
    ops.gemm(a, w, epi=ops.EPI_SWIGLU, out=out)
    torch.cuda.synchronize()
    intact(buf, "gemm swiglu")
    # attention with ragged lengths writes exactly [B, Sq, Hq, 128]
    b, sq, skv, hq, hkv = 2, 300, 517, 4, 2
    q, kk, v = _rand(b, sq, hq, 128), _rand(b, skv, hkv, 128), _rand(b, skv, hkv, 128)
    buf, out = guarded(b * sq, hq * 128)
    o, _ = ops.attention(q, kk, v, out=out.view(b, sq, hq, 128))
    torch.cuda.synchronize()
    intact(buf, "attention")
    want, _ = ref.attention(q.float(), kk.float(), v.float())
    _close(o, want, 2e-2, 2e-2, "attention into a guarded view")
    ops.check_status()


@pytest.mark.parametrize("checked", [False, True])
def test_bounds_checked_build_selftest(checked):
    """The debug build with device-side index checks (cosmos_b200/_C_check.so): its check classifies good and
    bad indices and reports through the status word, and the checked kernels still match their definitions
    on valid inputs. Runs in a child process because the build is chosen when the library is loaded."""
    import json
    import os
    import subprocess
    import sys
    from pathlib import Path
    root = Path(__file__).resolve().parents[1]
    if checked and not (root / "cosmos_b200" / "_C_check.so").exists():
        pytest.skip("bounds-checked build not present (python -m cosmos_b200.ops._build --bounds-check)")
    env = dict(os.environ, COSMOS_BOUNDS_CHECK="1" if checked else "0", COSMOS_B200_NO_BUILD="1")
    r = subprocess.run([sys.executable, "-m", "cosmos_b200.ops.bounds_selftest"], cwd=root, env=env, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    res = json.loads(r.stdout.strip().splitlines()[-1])
    assert res["ok"] and res["bounds_check_build"] == checked
    assert res["selftest_verdicts"] == ([1, 1, 1, 0, 0, 0, 1] if checked else [1] * 7)



def test_gemm_result_does_not_depend_on_the_tile_to_cta_assignment():
    """Race check by schedule: the persistent GEMM is run with one CTA per SM, with 37 and with 3 CTAs, so
    that tiles land on other CTAs, in another order, and many tiles share one CTA's smem ring and TMEM
    double buffer. Accumulation order inside a tile and across split-K partials is fixed, so all runs
    must agree bit for bit."""
    torch.manual_seed(31)
    k = torch.ops.cosmos_b200
    cases = [
        (lambda: (_rand(1500, 512), _rand(1024, 512, scale=1 / 16)), dict(epi=ops.EPI_PLAIN)),
        (lambda: (_rand(700, 1024), _rand(2048, 1024, scale=1 / 16)), dict(epi=ops.EPI_SWIGLU)),
        (lambda: (_rand(8, 4096), _rand(512, 4096, scale=1 / 32)), dict(epi=ops.EPI_PLAIN)),   # split-K path
    ]
    try:
        for make, kw in cases:
            a, w = make()
            outs = []
            for limit in (0, 37, 3):
                k.gemm_set_grid_limit(limit)
                outs.append(ops.gemm(a, w, **kw).clone())
            torch.cuda.synchronize()
            ops.check_status()
            assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2]), kw
            want = ref.gemm(a.float(), w.float(), None, kw["epi"])
            _close(outs[0], want, 3e-2, 2e-2, "gemm")
    finally:
        k.gemm_set_grid_limit(0)


def test_attention_over_several_kv_sources_in_one_launch():
    """Ring-KV in the kernel: K/V given as separate buffers of different (ragged) lengths, visited in order by one
    launch, equals attention over their concatenation."""
    torch.manual_seed(5)
    b, sq, hq, hkv = 1, 700, 8, 2
    lens = [512, 300, 129, 77]
    q = torch.randn(b, sq, hq, 128, device="cuda").bfloat16()
    ks = [torch.randn(b, n, hkv, 128, device="cuda").bfloat16() for n in lens]
    vs = [torch.randn(b, n, hkv, 128, device="cuda").bfloat16() for n in lens]
    o = torch.ops.cosmos_b200.attn_fwd_sources(q, [t.data_ptr() for t in ks], [t.data_ptr() for t in vs], lens, hkv,
                                               128 ** -0.5, None)
    ref, _ = ops.ref.attention(q.float(), torch.cat(ks, 1).float(), torch.cat(vs, 1).float())
    assert (o.float() - ref).abs().max().item() < 2e-2
    one, _ = ops.attention(q, torch.cat(ks, 1), torch.cat(vs, 1))
    assert (o.float() - one.float()).abs().max().item() < 1e-2
    single = torch.ops.cosmos_b200.attn_fwd_sources(q, [ks[0].data_ptr()], [vs[0].data_ptr()], lens[:1], hkv, 128 ** -0.5, None)
    ref1, _ = ops.ref.attention(q.float(), ks[0].float(), vs[0].float())
    assert (single.float() - ref1).abs().max().item() < 2e-2


@pytest.mark.parametrize("normalize", [False, True])
def test_cfg_unipc_step_matches_the_sampler(normalize):
    """The fused CFG + UniPC kernel against the sampler's own fp32 step, over a whole schedule (first step without a
    corrector, later ones with it, the last one returning the prediction)."""
    from cosmos_b200.models import sampler as samplers
    torch.manual_seed(2)
    rows, d, steps = 300, 64, 6
    sig = samplers.shifted_sigmas(steps, 3.0, None, device="cpu")
    a, b = samplers.UniPCSampler(sig), samplers.UniPCSampler(sig)
    x = torch.randn(rows, d, device="cuda")
    xa, xb = x.clone(), x.clone()
    for i in range(steps):
        vc = torch.randn(rows, d, device="cuda").bfloat16()
        vu = torch.randn(rows, d, device="cuda").bfloat16()
        v = ops.ref.cfg_combine(vc, vu, 4.0, normalize)
        xa = a.step(xa, v)
        xb = ops.cfg_unipc_step(xb, vc, vu, 4.0, b, normalize)
        assert (xa - xb).abs().max().item() < 2e-4 * (1 + xa.abs().max().item()), i


@pytest.mark.parametrize("scheduler", ["euler", "unipc"])
def test_denoise_steps_through_a_cuda_graph_equal_the_eager_steps(scheduler):
    """Small sequences run the model evaluation of every denoise step from one CUDA graph captured at the first step
    of the generation; the latents must equal those of the eager steps, for both samplers and with a control stream."""
    from cosmos_b200.config import SamplingConfig, tiny128_config
    from cosmos_b200.models.generator import GeneratorEngine
    from cosmos_b200.models.mot import MoTModel

    cfg = tiny128_config(max_text_len=32, n_layers=2)
    model = MoTModel(cfg, dtype=torch.bfloat16, device=DEV)
    model.init_weights(seed=4)
    g = torch.Generator(device=DEV).manual_seed(9)
    ids_c = torch.randint(0, cfg.vocab_size, (1, 32), generator=g, device=DEV)
    ids_u = torch.randint(0, cfg.vocab_size, (1, 32), generator=g, device=DEV)
    outs = {}
    for limit in (0, 8192):
        eng = GeneratorEngine(model)
        eng.graph_max_tokens = limit
        st = eng.make_state(ids_c, ids_u, (3, 16, 16))
        st.control_tokens = torch.randn(1, st.n_video, cfg.patch_dim, generator=torch.Generator(device=DEV).manual_seed(3),
                                        device=DEV)
        sc = SamplingConfig(num_steps=4, guidance=4.0, shift=3.0, scheduler=scheduler, seed=5, control_guidance=1.5)
        outs[limit] = eng.sample(st, sc)
        assert (limit > 0) == bool(st.__dict__.get("_graphs"))
    assert torch.isfinite(outs[0]).all()
    assert (outs[0] - outs[8192]).abs().max().item() <= 1e-5 * (1 + outs[0].abs().max().item())


def test_attention_on_cta_pairs_matches_the_reference():
    """The CTA-pair variant of the forward kernel (cta_group::2 tiles; off by default) on shapes with an odd number of
    query blocks, causal and MoT masks, GQA and a batch."""
    k = torch.ops.cosmos_b200
    k.attn_set_cta_pair(True)
    try:
        torch.manual_seed(1)
        for (b, sq, skv, hq, hkv, mask, n_ar) in ((1, 777, 777, 4, 4, ops.MASK_CAUSAL, 0), (2, 600, 900, 2, 1, ops.MASK_FULL, 0),
                                                 (1, 1300, 1300, 4, 2, ops.MASK_MOT, 333)):
            q = torch.randn(b, sq, hq, 128, device=DEV).bfloat16()
            kk = torch.randn(b, skv, hkv, 128, device=DEV).bfloat16()
            v = torch.randn(b, skv, hkv, 128, device=DEV).bfloat16()
            o, lse = ops.attention(q, kk, v, mask=mask, n_ar=n_ar, return_lse=True)
            ro, rlse = ops.ref.attention(q.float(), kk.float(), v.float(), 128 ** -0.5, mask, n_ar, True)
            assert (o.float() - ro).abs().max().item() < 2e-2
            assert (lse - rlse).abs().max().item() < 1e-3
    finally:
        k.attn_set_cta_pair(False)


@pytest.mark.parametrize("b,v,flags", [(5, 151936, True), (3, 4097, True), (4, 1000, False), (2, 50, True)])
def test_sample_topk_selects_the_64_largest_penalised_logits(b, v, flags):
    """Radix-select kernel against torch.topk over the fp32 definition of the penalties. bf16 logits tie often, so the
    values are compared in order and every id is checked against the penalised row."""
    g = torch.Generator(device=DEV).manual_seed(v)
    logits = (torch.randn(b, v, device=DEV, generator=g) * 3).bfloat16()
    tokens = torch.randint(0, v, (b,), device=DEV, generator=g)
    any_ = (torch.rand(b, v, device=DEV, generator=g) < 0.3) if flags else None
    out_ = (any_ & (torch.rand(b, v, device=DEV, generator=g) < 0.5)) if flags else None
    pres = torch.rand(b, device=DEV, generator=g) * 2 if flags else None
    rep = 1 + torch.rand(b, device=DEV, generator=g) if flags else None
    off = 1000
    ref_any, ref_out = (any_.clone(), out_.clone()) if flags else (None, None)
    want = ops.sample_topk(logits.float(), ref_any, ref_out, tokens + off, pres, rep, off)      # PyTorch definition
    got = ops.sample_topk(logits, any_, out_, tokens + off, pres, rep, off)
    torch.cuda.synchronize()
    if flags:
        assert torch.equal(any_, ref_any) and torch.equal(out_, ref_out)
        assert out_[torch.arange(b), tokens].all()
    assert torch.equal(got[..., 0], want[..., 0])
    ids = got[..., 1].contiguous().view(torch.int32).long() - off
    k = min(64, v)
    pen = logits.float()
    if flags:
        pen = torch.where(ref_any, torch.where(pen > 0, pen / rep[:, None], pen * rep[:, None]), pen)
        pen = pen - pres[:, None] * ref_out.float()
    assert ((ids[:, :k] >= 0) & (ids[:, :k] < v)).all()
    assert torch.equal(pen.gather(1, ids[:, :k]), got[:, :k, 0])
    for r in range(b):
        assert ids[r, :k].unique().numel() == k


def test_sample_topk_with_all_logits_equal():
    logits = torch.full((2, 5000), 1.25, device=DEV, dtype=torch.bfloat16)
    got = ops.sample_topk(logits, None, None, None, None, None, 0)
    assert (got[..., 0] == 1.25).all()
    ids = got[..., 1].contiguous().view(torch.int32)
    assert all(ids[r].unique().numel() == 64 and ids[r].min() >= 0 and ids[r].max() < 5000 for r in range(2))


@pytest.mark.parametrize("n_src", [1, 2, 8])
def test_sample_pick_matches_the_definition(n_src):
    """Merge of the shards' candidates and the draw against the PyTorch definition on the same noise."""
    g = torch.Generator(device=DEV).manual_seed(n_src)
    b = 300
    vals = torch.randn(n_src, b, 64, device=DEV, generator=g).sort(dim=-1, descending=True).values * 2
    ids = torch.stack([torch.randperm(100000, device=DEV, generator=g)[:n_src * 64].view(n_src, 64) for _ in range(b)], 1)
    cand = torch.stack([vals, ids.to(torch.int32).view(torch.float32)], -1).view(n_src * b, 64, 2).contiguous()
    temp = torch.where(torch.rand(b, device=DEV, generator=g) < 0.2, torch.zeros(b, device=DEV),
                       0.3 + torch.rand(b, device=DEV, generator=g))
    top_k = torch.randint(1, 80, (b,), device=DEV, generator=g)
    top_p = 0.2 + 0.8 * torch.rand(b, device=DEV, generator=g)
    noise = torch.rand(b, 64, device=DEV, generator=g).clamp_min(1e-7)
    got = ops.sample_pick(cand, n_src, temp, top_k, top_p, noise, 90000, torch.empty(b, dtype=torch.long, device=DEV))
    want = ops.sample_pick(cand.cpu(), n_src, temp.cpu(), top_k.cpu(), top_p.cpu(), noise.cpu(), 90000,
                           torch.empty(b, dtype=torch.long))
    same = (got.cpu() == want).float().mean().item()
    assert same >= 0.99, f"only {same:.3f} of the draws agree"      # a nucleus boundary within rounding may differ
    greedy = temp.cpu() == 0
    assert torch.equal(got.cpu()[greedy], want[greedy]) and (got < 90000).all()


@pytest.mark.parametrize("b,hq,hkv,d", [(32, 32, 8, 4096), (1, 32, 8, 4096), (8, 8, 2, 1024), (300, 4, 4, 512)])
def test_gemm_decode_qkv_post_reduces_the_split_k_partials_in_the_glue_kernel(b, hq, hkv, d):
    """QKV projection + decode glue in two launches (partials reduced by the glue kernel) against the three-launch
    form (GEMM, split-K reduction, glue) and, through it, the fp32 definition."""
    torch.manual_seed(b)
    page, n_pages = 16, 2 * ((b + 15) // 16) + 1
    h = _rand(b, d)
    w = _rand((hq + 2 * hkv) * 128, d, scale=d ** -0.5)
    ang = torch.rand(b, 64, device=DEV) * 6.0
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    gq, gk = (1 + 0.1 * torch.randn(128, device=DEV)).bfloat16(), (1 + 0.1 * torch.randn(128, device=DEV)).bfloat16()
    slots = (torch.randperm(n_pages * page, device=DEV)[:b]).long()
    kc, vc = _rand(n_pages, hkv, page, 128), _rand(n_pages, hkv, page, 128)
    kc2, vc2 = kc.clone(), vc.clone()
    q = ops.gemm_decode_qkv_post(h, w, hq, cos, sin, gq, gk, 1e-6, slots, kc, vc)
    qkv = ops.gemm(h, w).view(b, hq + 2 * hkv, 128)
    q2 = ops.decode_qkv_post(qkv, hq, cos, sin, gq, gk, 1e-6, slots, kc2, vc2)
    torch.cuda.synchronize()
    _close(q, q2, 1e-2, 1e-2, "q")
    _close(kc, kc2, 1e-2, 1e-2, "k cache")
    _close(vc, vc2, 1e-2, 1e-2, "v cache")
    f = (h.float() @ w.float().t()).view(b, hq + 2 * hkv, 128)
    _close(q, ref.mrope(f[:, :hq], cos, sin, gq.float(), 1e-6), 4e-2, 4e-2, "q vs fp32")


def test_vae_channels_last_encoder_matches_pytorch():
    """Channels-last encoder (strided convolutions over parity planes, 1x1 skips as columns of the block's second convolution, chunked
    in time) against the fp32 PyTorch modules in one pass."""
    from cosmos_b200.models.vae import CausalVideoVAE
    from cosmos_b200.models.vae_cuda import CLEncoder
    torch.manual_seed(21)
    vae = CausalVideoVAE(16, (64, 128, 256, 256)).to(DEV).float().eval()
    video = torch.rand(1, 3, 17, 48, 64, device=DEV) * 2 - 1
    with torch.no_grad():
        want = vae.encode(video)
    enc = CLEncoder(vae)
    got = enc.encode(video, chunk_frames=8)
    assert got.shape == want.shape == (1, 16, 5, 6, 8)
    err = (got - want).abs()
    scale = want.abs().mean().item()
    assert err.mean().item() < 0.03 * scale and err.max().item() < 0.25 * want.abs().max().item(), \
        (err.mean().item(), err.max().item(), scale)
    other = enc.encode(video, chunk_frames=4)
    assert (other - got).abs().max().item() <= 0.02 * want.abs().max().item()   # chunking does not change the result


def test_vae_encoder_takes_frames_as_they_come():
    """Frames on the host, in fp64, cut out of a larger clip, of fewer or more channels than the tokenizer has (missing ones are
    zero, further ones ignored): the bits of the plain call."""
    from cosmos_b200.models.vae import CausalVideoVAE
    from cosmos_b200.models.vae_cuda import CLEncoder
    torch.manual_seed(22)
    enc = CLEncoder(CausalVideoVAE(16, (64, 64, 128, 128)).to(device=DEV, dtype=torch.bfloat16).eval())
    video = (torch.rand(1, 3, 9, 32, 40, device=DEV) * 2 - 1).bfloat16().float()
    want = enc.encode(video)
    big = torch.zeros(1, 5, 9, 40, 48, device=DEV)
    big[:, :3, :, 4:36, 4:44], big[:, 3:] = video, math.nan
    for what, v in {"host": video.cpu(), "host bf16": video.bfloat16().cpu(), "fp64": video.double(), "fp16": video.half(),
                    "cut": big[:, :3, :, 4:36, 4:44], "five channels": big[:, :, :, 4:36, 4:44]}.items():
        tol = 0 if what != "fp16" else 2 ** -8 * want.abs().max().item()    # bf16 values below 2^-14 are subnormal in fp16
        assert (enc.encode(v) - want).abs().max() <= tol, what
    grey = torch.zeros_like(video)
    grey[:, :1] = video[:, :1]
    assert torch.equal(enc.encode(video[:, :1]), enc.encode(grey))


def test_vae_encoder_is_enough_to_load_the_kernels():
    """A program that builds the encoder and calls nothing else before it."""
    import subprocess
    import sys
    code = ("import torch; from cosmos_b200.models.vae import CausalVideoVAE; from cosmos_b200.models.vae_cuda import CLEncoder; "
            "v = CausalVideoVAE(16, (64, 64, 64, 64)).cuda().bfloat16(); print(CLEncoder(v).encode(torch.zeros(1, 3, 1, 16, 16)).shape)")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "[1, 16, 1, 2, 2]" in r.stdout, r.stderr[-800:]


@pytest.mark.parametrize("channels", [1, 4])
def test_vae_encoder_of_other_input_channels(channels):
    """A tokenizer of 1 or 4 input channels against the fp32 modules; the bounds of three channels."""
    from cosmos_b200.models.vae import CausalVideoVAE
    from cosmos_b200.models.vae_cuda import CLEncoder
    torch.manual_seed(23)
    vae = CausalVideoVAE(16, (64, 128, 128, 128), in_channels=channels).to(DEV).float().eval()
    video = torch.rand(1, channels, 9, 32, 40, device=DEV) * 2 - 1
    with torch.no_grad():
        want = vae.encode(video)
    got = CLEncoder(vae).encode(video.cpu() if channels == 1 else video)
    err = (got - want).abs()
    assert got.shape == want.shape and err.mean() < 0.03 * want.abs().mean() and err.max() < 0.25 * want.abs().max()


@pytest.mark.parametrize("frames", [1, 2, 4, 8, 16])
def test_vae_tails_between_chunks_hold_little_memory(frames):
    """What stays allocated from one chunk to the next: for each convolution its two context frames, in a storage of at most
    three times that."""
    from cosmos_b200.models.vae import CausalVideoVAE
    from cosmos_b200.models.vae_cuda import CLDecoder, CLEncoder
    vae = CausalVideoVAE(16, (64, 64, 128, 128)).to(device=DEV, dtype=torch.bfloat16).eval()
    tails = {}, {}
    CLEncoder(vae).encode_chunk(torch.zeros(3, frames, 32, 32, device=DEV), tails[0], 1)
    CLDecoder(vae).decode_chunk(torch.zeros(16, frames, 4, 4, device=DEV), tails[1], False)
    assert tails[0] and tails[1]
    for name, t in [*tails[0].items(), *tails[1].items()]:
        assert t.shape[0] == 2 and t.untyped_storage().nbytes() <= 3 * t.numel() * t.element_size(), name


@pytest.mark.parametrize("n,off", [(4096, 0), (1003, 0), (2048, 3), (777, 8)])
def test_adamw_kernels_match_the_fp32_definition(n, off):
    """`rs_adamw` (gradients read from bf16 buffers, here one local source) and `adamw_shard` (fp32 reduced
    gradient): vector path, scalar tail and a source offset that rules the vector loads out."""
    k = torch.ops.cosmos_b200
    g = torch.Generator(device=DEV).manual_seed(n + off)
    full = torch.randn(off + n + 5, device=DEV, generator=g).bfloat16()
    lr, b1, b2, eps, wd, scale, step = 1e-2, 0.9, 0.95, 1e-8, 0.1, 0.5, 3

    def fresh():
        w = torch.randn(n, device=DEV, generator=torch.Generator(device=DEV).manual_seed(1))
        m = torch.randn(n, device=DEV, generator=torch.Generator(device=DEV).manual_seed(2)) * 0.1
        v = torch.rand(n, device=DEV, generator=torch.Generator(device=DEV).manual_seed(3)) * 0.1
        return w, m, v, torch.empty(n, device=DEV, dtype=torch.bfloat16)

    gr = full[off:off + n].float()
    w0, m0, v0, _ = fresh()
    gs = gr * scale
    m_ref = b1 * m0 + (1 - b1) * gs
    v_ref = b2 * v0 + (1 - b2) * gs * gs
    w_ref = w0 - lr * ((m_ref / (1 - b1 ** step)) / ((v_ref / (1 - b2 ** step)).sqrt() + eps) + wd * w0)
    ptrs = torch.tensor([full.data_ptr()], dtype=torch.int64, device=DEV)
    # pass 1: sum of squares (and the reduced gradient), pass 2: the update from the sources
    sq = torch.zeros(1, device=DEV)
    red = torch.empty(n, device=DEV)
    w, m, v, p = fresh()
    k.rs_adamw(ptrs, 1, off, w, m, v, p, 1.0, 0.0, b1, b2, eps, 0.0, step, 1, sq, red)
    assert torch.allclose(sq, (gr * gr).sum()[None], rtol=1e-4) and torch.equal(red, gr)
    k.rs_adamw(ptrs, 1, off, w, m, v, p, scale, lr, b1, b2, eps, wd, step, 0, None, None)
    for got, want in ((m, m_ref), (v, v_ref), (w, w_ref)):
        assert torch.allclose(got, want, rtol=1e-5, atol=1e-6)
    assert torch.equal(p, w.bfloat16())
    w, m, v, p = fresh()
    k.adamw_shard(gr.contiguous(), w, m, v, p, scale, lr, b1, b2, eps, wd, step)
    for got, want in ((m, m_ref), (v, v_ref), (w, w_ref)):
        assert torch.allclose(got, want, rtol=1e-5, atol=1e-6)
    assert torch.equal(p, w.bfloat16())


@pytest.mark.parametrize("sizes", [(1,), (8191, 8192, 8193), (100_003, 16, 65_536), (257,) * 70])
@pytest.mark.parametrize("shift", [0, 1])
def test_optimizer_list_kernels_match_the_definition(sizes, shift):
    """Norm and clipped AdamW over lists: chunk edges, more tensors than one launch takes, addresses that rule 16-byte
    accesses out (`shift`). fp32 arithmetic: a few roundings of values below 10 an element."""
    k = torch.ops.cosmos_b200
    g = torch.Generator(device=DEV).manual_seed(sum(sizes) + shift)
    cut = lambda n, dt: torch.randn(n + 8, device=DEV, generator=g).to(dt)[shift:shift + n]  # noqa: E731
    grads = [cut(n, torch.bfloat16) for n in sizes]
    w, m = ([cut(n, torch.float32) for n in sizes] for _ in range(2))
    v = [cut(n, torch.float32).abs() for n in sizes]
    p = [cut(n, torch.bfloat16) for n in sizes]
    w0, m0, v0 = ([t.double() for t in ts] for ts in (w, m, v))
    scale, lr, b1, b2, eps, wd, step = 0.5, 1e-2, 0.9, 0.95, 1e-8, 0.1, 3
    sq = torch.zeros(1, device=DEV, dtype=torch.float64)
    k.grad_sq_list(grads, scale, sq)
    norm = math.sqrt(sum(float((t.double() * scale).square().sum()) for t in grads))
    assert abs(math.sqrt(float(sq)) - norm) <= 1e-6 * norm
    for limit in (-1.0, 0.5 * norm, 2 * norm):
        for ts, t0 in ((w, w0), (m, m0), (v, v0)):
            for t, x in zip(ts, t0):
                t.copy_(x)
        k.adamw_list(grads, w, m, v, p, scale, sq, limit, lr, b1, b2, eps, wd, step)
        clip = limit / (norm + 1e-6) if 0 <= limit < norm else 1.0
        for i, gr in enumerate(grads):
            gd = gr.double() * scale * clip
            mr, vr = b1 * m0[i] + (1 - b1) * gd, b2 * v0[i] + (1 - b2) * gd * gd
            wr = w0[i] - lr * ((mr / (1 - b1 ** step)) / ((vr / (1 - b2 ** step)).sqrt() + eps) + wd * w0[i])
            for got, want in ((m[i], mr), (v[i], vr), (w[i], wr)):
                assert (got.double() - want).abs().max() <= 1e-5 + 1e-5 * want.abs().max()
            assert torch.equal(p[i], w[i].bfloat16())


@pytest.mark.parametrize("b1,b2", [(0.9, 0.999), (0.9, 0.95), (0.99, 0.9999)])
@pytest.mark.parametrize("step", [1, 2, 1000])
def test_optimizer_list_kernel_keeps_the_factors(b1, b2, step):
    """First and second moments against fp64: 1 - beta and the bias corrections carry no more than their rounding to fp32. A moment
    is a sum of two products (at most five roundings, 3.6e-7, where the terms have one sign); the update has about eight more."""
    k = torch.ops.cosmos_b200
    g = torch.Generator(device=DEV).manual_seed(step)
    n, lr, eps = 8192 + 100, 1e-2, 1e-8
    gr = torch.rand(n, device=DEV, generator=g).bfloat16() + 0.5
    m, v = (torch.rand(n, device=DEV, generator=g) * 1e-3 for _ in range(2))
    w, p = torch.zeros(n, device=DEV), torch.zeros(n, device=DEV, dtype=torch.bfloat16)
    gd = gr.double()
    mr, vr = b1 * m.double() + (1 - b1) * gd, b2 * v.double() + (1 - b2) * gd * gd
    wr = -lr * (mr / (1 - b1 ** step)) / ((vr / (1 - b2 ** step)).sqrt() + eps)
    k.adamw_list([gr], [w], [m], [v], [p], 1.0, torch.zeros(1, device=DEV, dtype=torch.float64), -1.0, lr, b1, b2, eps, 0.0, step)
    for got, want, bound in ((m, mr, 3.6e-7), (v, vr, 3.6e-7), (w, wr, 1e-6)):
        assert ((got.double() - want).abs() <= bound * want.abs()).all()


@pytest.mark.parametrize("sizes", [(8192 * 1500,), (8192 * 700 + 5, 3, 8192 * 900), (8192 * 20,) * 70])
def test_gradient_norm_is_the_same_bits_every_time(sizes):
    """Chunks of very different size, so that an fp64 sum shows its order: the ranks of a data-parallel step take this sum each by
    itself and must arrive at the same clip factor."""
    g = torch.Generator(device=DEV).manual_seed(len(sizes))
    grads = []
    for n in sizes:
        t = torch.randn(n, device=DEV, generator=g)
        grads.append((t * torch.exp2(-torch.arange(n, device=DEV).div(8192, rounding_mode="floor").mul(7).remainder(20).float())).bfloat16())
    seen = set()
    for _ in range(40):
        sq = torch.full((1,), 1e-3, device=DEV, dtype=torch.float64)
        torch.ops.cosmos_b200.grad_sq_list(grads, 0.5, sq)
        seen.add(sq.item())
    assert len(seen) == 1
    want = 1e-3 + 0.25 * sum(t.double().square().sum().item() for t in grads)
    assert abs(seen.pop() - want) <= 1e-6 * want     # fp32 sums of at most a few hundred squares a thread


def _volume(x):
    """[C, T, H, W] -> zero-bordered channels-last volume behind two zero context frames."""
    c, t, h, w = x.shape
    vol = torch.zeros(t + 2, h + 2, w + 2, c, device=DEV, dtype=torch.bfloat16)
    vol[2:, 1:-1, 1:-1] = x.permute(1, 2, 3, 0)
    return vol


@pytest.mark.parametrize("t,h,w", [(1, 8, 8), (3, 6, 10), (2, 34, 62)])
@pytest.mark.parametrize("cin,cout", [(64, 64), (64, 128), (128, 128), (256, 256), (320, 96), (128, 320)])
def test_conv3d_fused_forms(cin, cout, t, h, w):
    """Every layout a convolution writes, with residual, skip projection and norm, against fp64 convolutions of the same
    bf16 inputs (a CTA pair has one tile here; the schedules are the next test's): volumes smaller than a tile and with a remainder, channels in several blocks and output tiles. Bound:
    one bf16 rounding of the result (2^-9 relative), twice with the norm."""
    import torch.nn.functional as F
    k = torch.ops.cosmos_b200
    torch.manual_seed(cin + cout + t)
    x = _rand(cin, t, h, w)
    wt = _rand(cout, cin, 3, 3, 3, scale=1 / math.sqrt(27 * cin))
    b = torch.randn(cout, device=DEV)
    r, sk, sw = _rand(cout, t, h, w), _rand(64, t, h, w), _rand(cout, 64, scale=0.125)
    g = (1 + 0.1 * torch.randn(cout, device=DEV)).bfloat16()
    y = F.conv3d(F.pad(x[None].double(), (1, 1, 1, 1, 2, 0)), wt.double(), b.double())[0]
    wp = wt.permute(0, 2, 3, 4, 1).reshape(cout, 27 * cin).contiguous()
    vol = _volume(x)
    nan = lambda *s: torch.full(s, float("nan"), device=DEV, dtype=torch.bfloat16)  # noqa: E731

    def check(got, want, what, rel=2 ** -8):
        got, want = got.double(), want.permute(1, 2, 3, 0)
        assert (got - want).abs().max() <= rel * max(1.0, want.abs().max().item()), what

    def norm(v):
        v = v.bfloat16().double()
        z = v * torch.rsqrt(v.square().mean(0, keepdim=True) + 1e-6) * g.double()[:, None, None, None]
        return z * torch.sigmoid(z)

    def border(v):
        assert v[:, 0].abs().max() == 0 and v[:, -1].abs().max() == 0 and v[:, :, 0].abs().max() == 0 and v[:, :, -1].abs().max() == 0

    fused = cout in (64, 128, 256)
    out, on = nan(t + 2, h + 2, w + 2, cout), nan(t + 2, h + 2, w + 2, cout) if fused else None
    k.conv3d_fused(vol, wp, b, _volume(r), None, out, on, g if fused else None, 1e-6, 0, 0, 0)
    check(out[2:, 1:-1, 1:-1], y + r.double(), "residual")
    border(out[2:])
    assert out[:2].isnan().all()
    if fused:
        check(on[2:, 1:-1, 1:-1], norm(y + r.double()), "norm", 2 ** -6)
        border(on[2:])
        only = nan(*on.shape)
        k.conv3d_fused(vol, wp, b, _volume(r), None, None, only, g, 1e-6, 0, 0, 0)
        assert torch.equal(only[2:], on[2:])
    # skip projection, s2d layout
    s2d = nan(t + 2, 4, h // 2 + 1, w // 2 + 1, cout)
    k.conv3d_fused(vol, torch.cat([wp, sw], 1).contiguous(), b, None, _volume(sk), s2d, None, None, 1e-6, 1, 0, 0)
    flat = torch.empty(t, h + 2, w + 2, cout, device=DEV, dtype=torch.bfloat16)
    for i in range(4):
        flat[:, i >> 1::2, i & 1::2] = s2d[2:, i]
    check(flat[:, 1:-1, 1:-1], y + torch.einsum("oc,cthw->othw", sw.double(), sk.double()), "skip")
    border(flat)
    # nearest upsampling
    for tem, first in ((0, 0), (1, 0), (1, 1)):
        want = y.repeat_interleave(2, 2).repeat_interleave(2, 3)
        want = want.repeat_interleave(2, 1)[:, first:] if tem else want
        up = nan(want.shape[1] + 2, 2 * h + 2, 2 * w + 2, cout)
        k.conv3d_fused(vol, wp, b, None, None, up, None, None, 1e-6, 2, tem, first)
        check(up[2:, 1:-1, 1:-1], want, "upsampling")
        border(up[2:])
    # stride 2 over the s2d form of the input
    xs = torch.empty(t + 2, 4, h // 2 + 1, w // 2 + 1, cin, device=DEV, dtype=torch.bfloat16)
    for i in range(4):
        xs[:, i] = vol[:, i >> 1::2, i & 1::2]
    for first, step in ((0, 1), (0, 2), (1, 2)):
        want = y[:, first::step, ::2, ::2]
        if want.shape[1] == 0:
            continue
        down = nan(want.shape[1] + 2, h // 2 + 2, w // 2 + 2, cout)
        dn = nan(*down.shape) if fused else None
        k.conv3d_fused(xs, wp, b, None, None, down, dn, g if fused else None, 1e-6, 3, first, step)
        check(down[2:, 1:-1, 1:-1], want, "stride 2")
        border(down[2:])
        if fused:
            check(dn[2:, 1:-1, 1:-1], norm(want), "stride 2, norm", 2 ** -6)
            border(dn[2:])


@pytest.mark.parametrize("cin,cout", [(64, 64), (128, 128), (256, 256), (320, 96), (128, 320)])
def test_conv3d_results_do_not_depend_on_the_schedule(cin, cout):
    """4608 rows are 9 tiles of 512 (up to 128 output channels) or 18 of 256: one and three CTA pairs walk three to eighteen tiles
    each, through both accumulators, ring phases carried from tile to tile and both buffers of the norm's row sums. The same
    bits as with a pair for every tile, in every form."""
    k = torch.ops.cosmos_b200
    torch.manual_seed(cin + cout)
    t, h, w = 2, 34, 62
    fused = cout in (64, 128, 256)
    vol, resid, skip = _volume(_rand(cin, t, h, w)), _volume(_rand(cout, t, h, w)), _volume(_rand(64, t, h, w))
    wp = _rand(cout, 27 * cin, scale=1 / math.sqrt(27 * cin))
    ws = torch.cat([wp, _rand(cout, 64, scale=0.125)], 1).contiguous()
    b, g = torch.randn(cout, device=DEV), _rand(cout) if fused else None
    xs = torch.zeros(12, 4, h // 2 + 1, w // 2 + 1, cin, device=DEV, dtype=torch.bfloat16)    # 10 frames kept: 10 segments
    xs[2:] = _rand(10, 4, h // 2 + 1, w // 2 + 1, cin)
    x64, terms = _volume(_rand(64, t, h, w)), _rand(9, 27 * 64, scale=0.02)

    def run():
        new = lambda *s: torch.full((*s, cout), 7.0, device=DEV, dtype=torch.bfloat16)  # noqa: E731
        outs = [new(t + 2, h + 2, w + 2), new(t + 2, h + 2, w + 2), new(t + 2, 4, h // 2 + 1, w // 2 + 1),
                new(2 * t + 2, 2 * h + 2, 2 * w + 2), new(12, h // 2 + 2, w // 2 + 2), new(12, h // 2 + 2, w // 2 + 2)]
        k.conv3d_fused(vol, wp, b, resid, None, outs[0], outs[1] if fused else None, g, 1e-6, 0, 0, 0)
        k.conv3d_fused(vol, ws, b, None, skip, outs[2], None, None, 1e-6, 1, 0, 0)
        k.conv3d_fused(vol, wp, b, resid, None, outs[3], None, None, 1e-6, 2, 1, 0)
        k.conv3d_fused(xs, wp, b, None, None, outs[4], outs[5] if fused else None, g, 1e-6, 3, 0, 1)
        return outs + [k.conv3d_rgb(x64, terms, b[:3].contiguous())]

    want = run()
    try:
        for limit in (2, 6):
            k.gemm_set_grid_limit(limit)
            for i, (got, ref_) in enumerate(zip(run(), want)):
                assert torch.equal(got, ref_), (limit, i)
    finally:
        k.gemm_set_grid_limit(0)


@pytest.mark.parametrize("t", [1, 2, 4, 5, 9])
@pytest.mark.parametrize("cin,cout,h,w", [(64, 64, 34, 62), (128, 64, 6, 10), (192, 32, 20, 38)])
def test_conv3d_narrow_outputs_over_time(t, cin, cout, h, w):
    """At most 64 output channels: a CTA pair walks positions through time with three frames' sums in a ring of four accumulators. Frame
    counts around the ring's length, one to five tiles of 512 positions, and one and three pairs as well as one for every tile
    and time segment, so that the ring wraps at every place and is carried from tile to tile. Against fp64 (one bf16 rounding of the
    result), and the same bits whatever the schedule."""
    import torch.nn.functional as F
    k = torch.ops.cosmos_b200
    torch.manual_seed(t + cin)
    x, wt, b = _rand(cin, t, h, w), _rand(cout, cin, 3, 3, 3, scale=1 / math.sqrt(27 * cin)), torch.randn(cout, device=DEV)
    vol = _volume(x)
    vol[:2] = _rand(2, h + 2, w + 2, cin)
    vol[:2, 0], vol[:2, -1], vol[:2, :, 0], vol[:2, :, -1] = 0, 0, 0, 0
    full = vol.permute(3, 0, 1, 2)[None].double()
    want = F.conv3d(full, wt.double(), b.double())[0].permute(1, 2, 3, 0)
    wp = wt.permute(0, 2, 3, 4, 1).reshape(cout, 27 * cin).contiguous()
    x64, terms, rb = vol[..., :64].contiguous(), _rand(9, 27 * 64, scale=0.02), torch.randn(3, device=DEV) * 0.1
    wo = terms.double().view(3, 3, 3, 3, 3, 64).sum(0).permute(0, 4, 1, 2, 3)
    pix = (((F.conv3d(full[:, :64], wo, rb.double())[0]).clamp(-1, 1) + 1) * 127.5).permute(1, 2, 3, 0)

    def run():
        out = torch.full((t + 2, h + 2, w + 2, cout), 7.0, device=DEV, dtype=torch.bfloat16)
        k.conv3d_fused(vol, wp, b, None, None, out, None, None, 1e-6, 0, 0, 0)
        return out, k.conv3d_rgb(x64, terms, rb)

    first = run()
    assert (first[0][2:, 1:-1, 1:-1].double() - want).abs().max() <= 2 ** -8 * max(1.0, want.abs().max().item())
    assert (first[1].double() - pix).abs().max() <= 0.5 + 1e-3     # rounding, and fp32 sums of 1728 products
    try:
        for limit in (2, 6):
            k.gemm_set_grid_limit(limit)
            assert all(torch.equal(u, v) for u, v in zip(run(), first)), limit
    finally:
        k.gemm_set_grid_limit(0)


@pytest.mark.parametrize("t", [1, 2, 3, 4, 7])
@pytest.mark.parametrize("cin,cout", [(64, 64), (64, 128), (128, 256), (64, 32)])
def test_conv3d_chunk_is_conv3d_fused(t, cin, cout):
    """Volumes in two tensors (all frames but the last two, those) and the context in a third, or absent, against one volume with the
    context in front: the same bits in every form. 1 to 7 frames: nothing, nothing, one frame and more in the first tensor; the
    shape has tiles that cross from frame to frame in memory and a remainder."""
    from cosmos_b200.models.vae_cuda import Volume
    k = torch.ops.cosmos_b200
    torch.manual_seed(t + cin + cout)
    h, w = 14, 38
    fused = cout in (64, 128, 256)
    wp, sw = _rand(cout, 27 * cin, scale=1 / math.sqrt(27 * cin)), _rand(cout, 64, scale=0.125)
    ws, b, g = torch.cat([wp, sw], 1).contiguous(), torch.randn(cout, device=DEV), _rand(cout) if fused else None

    def full(c, s2d, ctx):
        shape = (t + 2, 4, h // 2 + 1, w // 2 + 1, c) if s2d else (t + 2, h + 2, w + 2, c)
        v = _rand(*shape)
        if not ctx:
            v[:2] = 0
        return v

    def split(v):
        vol = Volume(v.shape[0] - 2, v.shape[1:], DEV)
        for lo, hi, part in vol.pieces():
            part.copy_(v[2 + lo:2 + hi])
        return vol

    def new(frames, *shape):
        vol = Volume(frames, (*shape, cout), DEV)
        vol.body.fill_(7.0)
        vol.tail.fill_(7.0)
        return vol

    def same(vol, ref_):
        return all(torch.equal(part, ref_[2 + lo:2 + hi]) for lo, hi, part in vol.pieces())

    for ctx in (True, False):
        x, xs, r, sk = full(cin, False, ctx), full(cin, True, ctx), full(cout, False, True), full(64, False, True)
        forms = [(x, wp, r, None, 0, 0, 0, t, (h + 2, w + 2), fused), (x, ws, None, sk, 1, 0, 0, t, (4, h // 2 + 1, w // 2 + 1), False),
                 (x, wp, r, None, 2, 0, 0, t, (2 * h + 2, 2 * w + 2), False), (x, wp, r, None, 2, 1, 0, 2 * t, (2 * h + 2, 2 * w + 2), False),
                 (x, wp, r, None, 2, 1, 1, 2 * t - 1, (2 * h + 2, 2 * w + 2), False), (xs, wp, None, None, 3, 0, 1, t, (h // 2 + 2, w // 2 + 2), fused),
                 (xs, wp, None, None, 3, 0, 2, (t + 1) // 2, (h // 2 + 2, w // 2 + 2), fused)]
        if t > 1:
            forms.append((xs, wp, None, None, 3, 1, 2, t // 2, (h // 2 + 2, w // 2 + 2), fused))
        for v, wt, res, skip, mode, ma, mb, n, shape, norm in forms:
            want = [torch.full((n + 2, *shape, cout), 7.0, device=DEV, dtype=torch.bfloat16) for _ in range(2)]
            k.conv3d_fused(v, wt, b, res, skip, want[0], want[1] if norm else None, g, 1e-6, mode, ma, mb)
            got = [new(n, *shape), new(n, *shape)]
            k.conv3d_chunk(split(v).parts, v[:2].contiguous() if ctx else None, wt, b, split(res).parts if res is not None else [],
                           split(skip).parts if skip is not None else [], got[0].parts, got[1].parts if norm else [], g, 1e-6, mode, t, ma, mb)
            assert same(got[0], want[0]) and (not norm or same(got[1], want[1])), (ctx, mode, ma, mb)
            if n == 1:
                assert (got[0].tail[0] == 7.0).all()      # the frame before the only one is not this chunk's
        if cin == 64:
            terms, rb = _rand(9, 27 * 64, scale=0.02), torch.randn(3, device=DEV)
            assert torch.equal(k.conv3d_rgb_chunk(split(x).parts, x[:2].contiguous() if ctx else None, terms, rb, t), k.conv3d_rgb(x, terms, rb))


@pytest.mark.parametrize("t", [1, 2, 5])
@pytest.mark.parametrize("ctx", [True, False])
@pytest.mark.parametrize("cin,cout", [(64, 64), (128, 32), (128, 128), (256, 256), (128, 320)])
def test_conv3d_chunk_against_fp64(cin, cout, ctx, t):
    """The form that the tokenizer calls (volumes in two tensors, context frames in a third or absent) against fp64 convolutions of the
    same bf16 numbers, in every layout, and with one and three CTA pairs: the same bits. 2304 positions a frame are five tiles of 512
    or nine of 256. Bound: one bf16 rounding (2^-9 relative) and fp32 sums of up to 6976 products, together below 2^-8 of the larger of the
    result and 1."""
    import torch.nn.functional as F
    from cosmos_b200.models.vae_cuda import Volume
    k = torch.ops.cosmos_b200
    torch.manual_seed(t + cin + cout)
    h, w = 34, 62
    hp, wd = h + 2, w + 2
    fused = cout in (64, 128, 256)

    def full(c):
        v = torch.zeros(t + 2, hp, wd, c, device=DEV, dtype=torch.bfloat16)
        v[0 if ctx else 2:, 1:-1, 1:-1] = _rand(t + 2 if ctx else t, h, w, c)
        return v

    def split(v):
        vol = Volume(t, v.shape[1:], DEV)
        for lo, hi, part in vol.pieces():
            part.copy_(v[2 + lo:2 + hi])
        return vol.parts, v[:2].contiguous() if ctx else None

    def new(frames, *shape):
        vol = Volume(frames, (*shape, cout), DEV)
        vol.body.fill_(7.0)
        vol.tail.fill_(7.0)
        return vol

    def whole(vol):
        return torch.cat([part for _, _, part in vol.pieces()])

    def parity(v):
        return torch.stack([v[:, i::2, j::2] for i in (0, 1) for j in (0, 1)], dim=1).contiguous()

    def near(got, want):
        assert got.shape == want.shape and ((got.double() - want).abs() <= 2 ** -8 * want.abs().clamp(min=1.0)).all()

    x, res, sk = full(cin), full(cout), full(64)
    wt, sw, b = _rand(cout, cin, 3, 3, 3, scale=1 / math.sqrt(27 * cin)), _rand(cout, 64, scale=0.125), torch.randn(cout, device=DEV)
    g = _rand(cout) if fused else None
    wp = wt.permute(0, 2, 3, 4, 1).reshape(cout, 27 * cin).contiguous()
    ws = torch.cat([wp, sw], 1).contiguous()
    terms, rb = _rand(9, 27 * 64, scale=0.02), torch.randn(3, device=DEV) * 0.1
    x5 = x.permute(3, 0, 1, 2)[None].double()
    conv = F.conv3d(x5, wt.double(), b.double())[0].permute(1, 2, 3, 0)                          # [t, h, w, cout]
    down = F.conv3d(x5, wt.double(), b.double(), stride=(1, 2, 2))[0].permute(1, 2, 3, 0)
    inner = lambda v: v[2:, 1:-1, 1:-1].double()  # noqa: E731
    pad = lambda v: F.pad(v, (0, 0, 1, 1, 1, 1))  # noqa: E731
    twice = lambda v: v.repeat_interleave(2, 1).repeat_interleave(2, 2)  # noqa: E731
    xp, cx = split(x)
    xs, cs = split(parity(x))
    rp, sp = split(res)[0], split(sk)[0]

    def run():
        same, norm, s2d, up = new(t, hp, wd), new(t, hp, wd), new(t, 4, hp // 2, wd // 2), new(2 * t, 2 * h + 2, 2 * w + 2)
        up1, dn, dnorm = new(2 * t - 1, 2 * h + 2, 2 * w + 2), new((t + 1) // 2, h // 2 + 2, w // 2 + 2), new((t + 1) // 2, h // 2 + 2, w // 2 + 2)
        k.conv3d_chunk(xp, cx, wp, b, rp, [], same.parts, norm.parts if fused else [], g, 1e-6, 0, t, 0, 0)
        k.conv3d_chunk(xp, cx, ws, b, [], sp, s2d.parts, [], None, 1e-6, 1, t, 0, 0)
        k.conv3d_chunk(xp, cx, wp, b, rp, [], up.parts, [], None, 1e-6, 2, t, 1, 0)
        k.conv3d_chunk(xp, cx, wp, b, rp, [], up1.parts, [], None, 1e-6, 2, t, 1, 1)
        k.conv3d_chunk(xs, cs, wp, b, [], [], dn.parts, dnorm.parts if fused else [], g, 1e-6, 3, t, 0, 2)
        out = [whole(v) for v in (same, norm, s2d, up, up1, dn, dnorm)]
        return out + ([k.conv3d_rgb_chunk(split(x[..., :64].contiguous())[0], cx[..., :64].contiguous() if ctx else None, terms, rb, t)])

    got = run()
    plus = conv + inner(res)
    near(got[0], pad(plus))
    near(got[2], parity(pad(conv + inner(sk) @ sw.double().t())))
    near(got[3], pad(twice(plus.repeat_interleave(2, 0))))
    near(got[4], pad(twice(plus.repeat_interleave(2, 0)[1:])))
    near(got[5], pad(down[::2]))
    if fused:
        for raw, n in ((got[0], got[1]), (got[5], got[6])):
            y = raw.double()
            near(n, F.silu(y * torch.rsqrt((y * y).mean(-1, keepdim=True) + 1e-6) * g.double()))
    wo = terms.double().view(3, 3, 3, 3, 3, 64).sum(0).permute(0, 4, 1, 2, 3)
    pix = ((F.conv3d(x5[:, :64], wo, rb.double())[0].clamp(-1, 1) + 1) * 127.5).permute(1, 2, 3, 0)
    assert (got[7].double() - pix).abs().max() <= 0.5 + 1e-3
    try:
        for limit in (2, 6):
            k.gemm_set_grid_limit(limit)
            for i, (u, v) in enumerate(zip(run(), got)):
                assert torch.equal(u, v), (limit, i)
    finally:
        k.gemm_set_grid_limit(0)


@pytest.mark.parametrize("cin,cout,tpad", [(64, 64, 0), (64, 128, 1), (128, 32, 1), (64, 256, 0), (64, 64, 2)])
def test_conv3d_cl_of_weights_that_are_not_finite(cin, cout, tpad):
    """An infinite weight of an early tap meets the zeros in front of the first frame: NaN, as in the definition, in that channel."""
    import torch.nn.functional as F
    torch.manual_seed(cin + cout)
    x, wt = _rand(3, 8, 10, cin), _rand(cout, cin, 3, 3, 3, scale=0.02)
    wt[5, 3, 0, 1, 1] = math.inf
    out = torch.zeros(3, 8, 10, cout, device=DEV, dtype=torch.bfloat16)
    wp = wt.permute(0, 2, 3, 4, 1).reshape(cout, 27 * cin).contiguous()
    torch.ops.cosmos_b200.conv3d_cl(x, wp, None, None, out, tpad)
    xf = F.pad(x.permute(3, 0, 1, 2)[None].float(), (0, 0, 0, 0, 2, 0))
    want = F.conv3d(xf, wt.float())[0].permute(1, 2, 3, 0)[tpad:]
    got = out[tpad:, 1:-1, 1:-1].float()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isfinite(), want.isfinite())
    _close(got[..., :5], want[..., :5], 2e-2, 2e-2)


@pytest.mark.parametrize("part", ["dec_in", "enc_in", "enc_mid"])
def test_tokenizer_with_weights_that_are_not_finite(part):
    """An infinite weight of an early tap: whatever a clip's first chunk has NaN in with a context of zeros, it has without one."""
    from cosmos_b200.models.vae import CausalVideoVAE
    from cosmos_b200.models.vae_cuda import CLDecoder, CLEncoder
    torch.manual_seed(3)
    vae = CausalVideoVAE(widths=(64, 64, 64, 64)).to(DEV)
    conv = {"dec_in": vae.dec_in, "enc_in": vae.enc_in, "enc_mid": vae.enc_mid.c1}[part]
    conv.weight.data[5, 1, 0, 1, 1] = math.inf
    cl, key = CLDecoder(vae) if part == "dec_in" else CLEncoder(vae), "mid.c1" if part == "enc_mid" else "in"
    x = cl._volume(1, 6, 6, 64, zero=True)
    x.tail[1, 1:-1, 1:-1] = _rand(4, 4, 64)
    out, _ = cl._conv({}, key, x)
    assert out.tail[1, 1:-1, 1:-1, 5].isnan().all()
    assert out.tail[1, 1:-1, 1:-1, 6].isfinite().all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("t,h,w", [(1, 8, 8), (3, 10, 22)])
def test_conv3d_of_colours(dtype, t, h, w):
    """First layer of the encoder (packed taps) and last layer of the decoder (fp32 weights in three bf16 terms)."""
    import torch.nn.functional as F
    from cosmos_b200.models.vae_cuda import _bf16_terms
    k = torch.ops.cosmos_b200
    torch.manual_seed(t)
    src = torch.randn(3, t + 1, h, w, device=DEV).to(dtype)[:, 1:]      # channel stride of a slice
    wt = _rand(64, 3, 3, 3, 3, scale=1 / 9)
    p = torch.zeros(64, 3, 64, device=DEV, dtype=torch.bfloat16)
    p[:, :, :27] = wt.permute(0, 2, 3, 4, 1).reshape(64, 3, 27)
    vol = torch.zeros(t + 2, h + 2, w + 2, 64, device=DEV, dtype=torch.bfloat16)
    k.conv_pack_rgb(src, vol)
    out = torch.empty(t + 2, h + 2, w + 2, 64, device=DEV, dtype=torch.bfloat16)
    k.conv3d_fused(vol, p.view(64, 192), None, None, None, out, None, None, 1e-6, 0, 0, 0)
    want = F.conv3d(F.pad(src.bfloat16()[None].double(), (1, 1, 1, 1, 2, 0)), wt.double())[0].permute(1, 2, 3, 0)
    assert (out[2:, 1:-1, 1:-1].double() - want).abs().max() <= 2 ** -8 * max(1.0, want.abs().max().item())
    x, wo, b = _rand(64, t, h, w), torch.randn(3, 64, 3, 3, 3, device=DEV) / 40, torch.randn(3, device=DEV) * 0.1
    terms = _bf16_terms(wo.permute(0, 2, 3, 4, 1).reshape(3, 27 * 64))
    assert torch.equal(terms.float().view(3, 3, -1).sum(0), wo.permute(0, 2, 3, 4, 1).reshape(3, -1))
    got = k.conv3d_rgb(_volume(x), terms, b)
    y = F.conv3d(F.pad(x[None].double(), (1, 1, 1, 1, 2, 0)), wo.double(), b.double())[0]
    pix = ((y.clamp(-1, 1) + 1) * 127.5).permute(1, 2, 3, 0)
    assert (got.double() - pix).abs().max() <= 0.5 + 1e-3      # rounding, and fp32 sums of 1728 products below 4


@pytest.mark.parametrize("t,chunk", [(1, 2), (2, 2), (5, 2), (6, 1), (4, 8)])
def test_vae_decode_to_host_is_the_decode(t, chunk):
    from cosmos_b200.models.vae import CausalVideoVAE
    from cosmos_b200.models.vae_cuda import CLDecoder
    torch.manual_seed(t)
    dec = CLDecoder(CausalVideoVAE(16, (64, 128, 128, 128)).to(device=DEV, dtype=torch.bfloat16).eval())
    z = torch.randn(1, 16, t, 4, 6, device=DEV)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got = dec.decode_to_host(z, chunk_latents=chunk)
    assert torch.equal(got, dec.decode(z, chunk_latents=chunk)[0].cpu())


@pytest.mark.parametrize("m,n,k", [(129, 512, 64), (300, 768, 136), (513, 1032, 320), (700, 1536, 1088), (1024, 2048, 192),
                                    (257, 1024, 2048), (700, 3328, 1088)])
def test_gemm_wide_tiles(m, n, k):
    """Every tile shape (128x256 on single CTAs, 256x256 and 256x512 on pairs) on one and on two pairs, against the fp32
    definition, for each epilogue and operand order and for two problems in one launch; ragged rows, columns, k-blocks and an odd
    number of 256-column tiles. A tile's products are summed in the same order whoever computes it, so all give the same bits."""
    torch.manual_seed(41)
    kern = torch.ops.cosmos_b200
    a, w, r = _rand(m, k), _rand(n, k, scale=1 / math.sqrt(k)), _rand(m, n)
    bias, gate = _rand(n), _rand(2, n)
    rpb = (m + 1) // 2
    wt = w.t().contiguous()
    ang = torch.rand(m, 64, device=DEV) * 6.28
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    gamma = (1 + 0.1 * torch.randn(128, device=DEV)).bfloat16()
    calls = {
        "plain": lambda: ops.gemm(a, w, bias),
        "resid": lambda: ops.gemm(a, w, None, ops.EPI_GATED_RESID, r, gate, rpb),
        "b_mn": lambda: kern.gemm_ex(a, wt, False, True, None),
    }
    want = {"plain": a.float() @ w.float().t() + bias.float(),
            "resid": ref.gemm(a.float(), w.float(), None, ops.EPI_GATED_RESID, r.float(), gate.float(), rpb),
            "b_mn": a.float() @ w.float().t()}
    m2 = m // 2 + 1
    a2, w2, r2 = _rand(m2, k), _rand(n, k, scale=1 / math.sqrt(k)), _rand(m2, n)
    two = lambda epi, *rs: torch.cat(ops.gemm_grouped2(a, w, a2, w2, epi, *rs))  # noqa: E731
    ab, wb = (a.float(), a2.float()), (w.float(), w2.float())
    calls["gelu"] = lambda: ops.gemm(a, w, bias, GELU)
    want["gelu"] = torch.nn.functional.gelu(want["plain"])
    calls["two plain"] = lambda: two(ops.EPI_PLAIN)
    want["two plain"] = torch.cat([x @ y.t() for x, y in zip(ab, wb)])
    calls["two resid"] = lambda: two(ops.EPI_GATED_RESID, r, r2, None, gate, m, (m2 + 1) // 2)
    want["two resid"] = torch.cat([ref.gemm(a.float(), w.float(), None, ops.EPI_GATED_RESID, r.float(), None, m),
                                   ref.gemm(a2.float(), w2.float(), None, ops.EPI_GATED_RESID, r2.float(), gate.float(), (m2 + 1) // 2)])
    if n % 16 == 0:
        calls["two swiglu"] = lambda: two(ops.EPI_SWIGLU)
        want["two swiglu"] = torch.cat([ref.gemm(x, y, epi=ops.EPI_SWIGLU) for x, y in zip(ab, wb)])
        calls["swiglu"] = lambda: ops.gemm(a, w, epi=ops.EPI_SWIGLU)
        want["swiglu"] = ref.gemm(a.float(), w.float(), epi=ops.EPI_SWIGLU)
    if n % 128 == 0:
        hq, gf = n // 128 - 2, gamma.float()
        calls["qkv"] = lambda: ops.gemm_qkv_rope(a, w, bias, cos, sin, gamma, gamma, hq, 1, 1e-6)
        want["qkv"] = ref.gemm_qkv_rope(a.float(), w.float(), bias.float(), cos, sin, gf, gf, hq, 1, 1e-6)
        calls["qkv plain"] = lambda: ops.gemm_qkv_rope(a, w, None, None, None, None, None, hq, 1, 1e-6)
        want["qkv plain"] = want["b_mn"]
    if m % 8 == 0:
        at = a.t().contiguous()
        calls["a_mn"] = lambda: kern.gemm_ex(at, wt, True, True, None)
        want["a_mn"] = want["b_mn"]
    epi = {"swiglu": ops.EPI_SWIGLU, "two swiglu": ops.EPI_SWIGLU, "resid": ops.EPI_GATED_RESID, "two resid": ops.EPI_GATED_RESID,
           "gelu": GELU, "qkv": ops.EPI_QKV_ROPE, "qkv plain": ops.EPI_QKV_ROPE}
    try:
        for name, call in calls.items():
            first = None
            if name in ("plain", "resid", "gelu", "swiglu") and kern.gemm_pick_k_splits(m, n, k, epi.get(name, ops.EPI_PLAIN)) > 1:
                continue     # split-K launches have tiles of their own
            for tile in ((2, 2), (2, 1), (1, 1)):
                kern.gemm_set_tile(*tile)
                for limit in (2, 4):
                    kern.gemm_set_grid_limit(limit)
                    assert kern.gemm_pick_tile(m, n, k, epi.get(name, ops.EPI_PLAIN)) == tile
                    got = call().clone()
                    if first is None:
                        first = got
                        _close(got, want[name], 3e-2, 2e-2, f"{name} {m}x{n}x{k}")
                    assert torch.equal(got, first), (name, tile, limit)
    finally:
        kern.gemm_set_grid_limit(0)
        kern.gemm_set_tile(0, 0)


@pytest.mark.parametrize("m,n,k,side", [(129, 4096, 512, 2), (256, 768, 1024, 2), (257, 4096, 768, 1), (333, 4096, 1088, 1), (384, 4096, 512, 2),
                                        (384, 4096, 768, 1), (385, 3072, 1024, 2)])
def test_gemm_split_on_pairs_and_single_ctas(m, n, k, side):
    """Split-K launches of two to four row tiles, on the side that the number of rounds takes (single CTAs at 257 to 384 rows of a
    4096-wide projection in three splits, pairs elsewhere) and on either: the same sums."""
    kern = torch.ops.cosmos_b200
    assert kern.gemm_pick_k_splits(m, n, k, ops.EPI_GATED_RESID) > 1
    assert kern.gemm_pick_split_ctas(m, n, k, ops.EPI_GATED_RESID) == side
    a, w, r = _rand(m, k), _rand(n, k) * 0.05, _rand(m, n)
    got = ops.gemm(a, w, None, ops.EPI_GATED_RESID, r, None, m)
    _close(got, r.float() + a.float() @ w.float().t(), 3e-2, 2e-2, f"{m}x{n}x{k}")
    try:
        for ctas in (1, 2):
            kern.gemm_set_tile(ctas, 1)
            assert kern.gemm_pick_split_ctas(m, n, k, ops.EPI_GATED_RESID) == ctas
            assert torch.equal(got, ops.gemm(a, w, None, ops.EPI_GATED_RESID, r, None, m)), ctas
    finally:
        kern.gemm_set_tile(0, 0)
    torch.cuda.synchronize()
    ops.check_status()


def test_gemm_swiglu_keeps_the_limits_of_silu():
    """Gates beyond the range in which the quotient of silu is refined: large of both signs, tiny, zero, infinite. Two spacings of
    subnormal bf16 (9.2e-41) absolutely, far below every value that is checked."""
    k = 64
    g = torch.tensor([0.0, 1e-38, -1e-38, 1e-30, 79.0, -79.0, 81.0, -81.0, -87.0, -88.0, -89.0, -200.0, 3e38, -3e38, math.inf, 1.0])
    a = torch.zeros(300, k, device=DEV, dtype=torch.bfloat16)
    a[:, 0] = 1
    w = torch.zeros(32, k, device=DEV, dtype=torch.bfloat16)
    w[:16, 0] = g.to(DEV).bfloat16()
    w[16:, 0] = 1
    got = ops.gemm(a, w, epi=ops.EPI_SWIGLU)
    want = torch.nn.functional.silu(w[:16, 0].double())
    want[w[:16, 0].double() < -88.8] = 0.0    # exp(-gate) is beyond fp32
    fin = torch.isfinite(want)
    _close(got[:, fin], want[fin].float().expand(300, -1), 2e-40, 8e-3, "silu")
    assert (got[:, ~fin] == math.inf).all()


@pytest.mark.parametrize("first", range(0, 2 ** 32, 2 ** 30))
def test_silu_of_the_swiglu_epilogue_is_the_division(first):
    """Every fp32 gate: the epilogue's quotient has the bits of CUDA's division, signed zeros and both limits among them."""
    assert torch.ops.cosmos_b200.silu_selftest(first, 2 ** 30, torch.empty(0, device=DEV)).item() == 0


def test_silu_of_the_convolutions_is_the_division_in_bf16():
    """Every fp32 value: no bf16 result differs from the division's; in fp32 two do, by one spacing."""
    got = sum(torch.ops.cosmos_b200.conv_silu_selftest(i * 2 ** 30, 2 ** 30, torch.empty(0, device=DEV)) for i in range(4)).tolist()
    assert got[0] == 0 and got[1] <= 2 and got[2] <= got[1]


@pytest.mark.parametrize("m", [5, 300])
@pytest.mark.parametrize("n", [8, 24, 40, 264])
@pytest.mark.parametrize("shift", [1, 4])
def test_gemm_epilogues_take_views_that_start_anywhere(m, n, shift):
    """Residual, gate and output as views that rule 16-byte accesses out, and SwiGLU rows of an odd stride: the same bits as with
    aligned tensors, and nothing beside the view is written."""
    torch.manual_seed(59)
    a, w, w2 = _rand(m, 64), _rand(n, 64, scale=0.125), _rand(2 * n, 64, scale=0.125)
    r, gate, rpb = _rand(m, n), _rand(2, n), (m + 1) // 2
    ld = (n + shift + 7) // 8 * 8 + 8

    def moved(t):
        v = torch.empty(t.shape[0], ld, device=DEV, dtype=torch.bfloat16)[:, shift:shift + n]
        return v.copy_(t)

    flat = torch.empty(2 * n + 8, device=DEV, dtype=torch.bfloat16)[shift:shift + 2 * n].view(2, n).copy_(gate)
    for name, call in {"plain": lambda r, g, **o: ops.gemm(a, w, **o),
                       "gelu": lambda r, g, **o: ops.gemm(a, w, epi=GELU, **o),
                       "resid": lambda r, g, **o: ops.gemm(a, w, None, ops.EPI_GATED_RESID, r, g, rpb, **o),
                       "swiglu": lambda r, g, **o: ops.gemm(a, w2, epi=ops.EPI_SWIGLU, **o)}.items():
        want = call(r, gate)
        for stride in (ld, ld + 3) if name == "swiglu" else (ld,):
            big = torch.full((m, stride), 7.0, device=DEV, dtype=torch.bfloat16)
            call(moved(r), flat, out=big[:, shift:shift + n])
            assert torch.equal(big[:, shift:shift + n], want), (name, stride)
            assert (big[:, :shift] == 7).all() and (big[:, shift + n:] == 7).all(), (name, stride)


@pytest.mark.parametrize("batch,rows", [(1, 40), (2, 240), (3, 100), (5, 33), (9, 20), (40, 7)])
@pytest.mark.parametrize("hq,tile,limit", [(4, (0, 0), 0), (6, (2, 2), 0), (6, (2, 2), 2), (4, (2, 2), 4), (6, (2, 1), 2), (4, (1, 1), 2)])
def test_gemm_qkv_rope_routed_by_batch(batch, rows, hq, tile, limit):
    """One routing table per batch entry: the same bits in every buffer as one launch per entry, whichever tables a tile or
    a warp's 32 rows cross, for every tile shape (6 query heads make an odd number of 256-column tiles) and schedule; rows that
    belong to nobody stay untouched."""
    torch.manual_seed(43)
    k, hk, pre = 256, 2, 3
    a = _rand(batch, rows, k)
    w = _rand((hq + 2 * hk) * 128, k, scale=1 / math.sqrt(k))
    ang = torch.rand(rows, 64, device=DEV) * 6.28
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    gamma = (1 + 0.1 * torch.randn(128, device=DEV)).bfloat16()
    outs = []
    for merged in (False, True):
        q = torch.full((batch, rows, hq, 128), 7.0, device=DEV, dtype=torch.bfloat16)
        kv = torch.full((2, batch, pre + rows, hk, 128), 7.0, device=DEV, dtype=torch.bfloat16)
        ptr = torch.tensor([[q[b, :, j].data_ptr() for j in range(hq)] + [kv[i, b, pre:, j].data_ptr() for i in (0, 1) for j in range(hk)]
                            for b in range(batch)], device=DEV)
        ld = torch.tensor([[hq * 128] * hq + [hk * 128] * 2 * hk] * batch, device=DEV)
        if merged:
            try:
                torch.ops.cosmos_b200.gemm_set_tile(*tile)
                torch.ops.cosmos_b200.gemm_set_grid_limit(limit)
                ops.gemm_qkv_rope(a.view(batch * rows, k), w, None, cos, sin, gamma, gamma, hq, hk, 1e-6, ptr, ld, route_rows=rows)
            finally:
                torch.ops.cosmos_b200.gemm_set_tile(0, 0)
                torch.ops.cosmos_b200.gemm_set_grid_limit(0)
        else:
            for b in range(batch):
                ops.gemm_qkv_rope(a[b], w, None, cos, sin, gamma, gamma, hq, hk, 1e-6, ptr[b].contiguous(), ld[b].contiguous())
        outs.append((q, kv))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
    assert (outs[1][1][:, :, :pre] == 7).all()
    want = ref.gemm_qkv_rope(a[-1].float(), w.float(), None, cos, sin, gamma.float(), gamma.float(), hq, hk, 1e-6)
    _close(outs[1][0][-1].reshape(rows, -1), want[:, :hq * 128], 3e-2, 2e-2, "routed by batch")


@pytest.mark.parametrize("batch", [1, 2, 3])
def test_workspace_qkv_with_longer_rotary_tables(batch):
    """Tables for more positions than there are tokens: every batch entry takes the first rows. The operator refuses tables that
    would give the second entry other positions."""
    from cosmos_b200.config import get_model_config
    from cosmos_b200.models.mot import WorkspaceAttn
    torch.manual_seed(47)
    cfg = get_model_config("tiny128")
    rows, heads = 40, cfg.n_heads + 2 * cfg.n_kv_heads
    h, w = _rand(batch, rows, cfg.d_model), _rand(heads * 128, cfg.d_model, scale=1 / math.sqrt(cfg.d_model))
    ang = torch.rand(64, 64, device=DEV) * 6.28
    cos, sin, gamma = ang.cos(), ang.sin(), torch.ones(128, device=DEV, dtype=torch.bfloat16)
    with torch.no_grad():
        long = [t.clone() for t in WorkspaceAttn().qkv_project(h, w, cos, sin, gamma, gamma, cfg)]
        for b in range(batch):
            for got, want in zip(long, WorkspaceAttn().qkv_project(h[b:b + 1], w, cos[:rows], sin[:rows], gamma, gamma, cfg)):
                assert torch.equal(got[b:b + 1], want)
        buf = torch.empty(rows, heads * 128, device=DEV, dtype=torch.bfloat16)
        ptr = torch.full((batch, heads), buf.data_ptr(), device=DEV, dtype=torch.int64)
        ld = torch.full_like(ptr, heads * 128)
        with pytest.raises(RuntimeError, match="route_rows rows"):
            ops.gemm_qkv_rope(h.view(batch * rows, -1), w, None, cos, sin, gamma, gamma, cfg.n_heads, cfg.n_kv_heads, 1e-6, ptr, ld,
                              route_rows=rows)


@pytest.mark.parametrize("m", [1, 7, 8, 9, 16, 17, 100, 128])
@pytest.mark.parametrize("n,k", [(272, 72), (1024, 4096), (40000, 512)])
def test_gemm_of_a_partly_filled_row_tile(m, n, k):
    """Up to 16 rows only the rows that exist are staged, in eights: launches with and without split-K, one and several tiles a CTA. What lies
    behind the rows, infinities among it, reaches no result."""
    torch.manual_seed(53)
    big = torch.full((200, k), math.inf, device=DEV, dtype=torch.bfloat16)
    ops.gemm(big, _rand(1024, k))     # leaves infinities in shared memory
    a, w = _rand(m, k), _rand(n, k, scale=1 / math.sqrt(k))
    _close(ops.gemm(a, w), a.float() @ w.float().t(), 2e-2, 2e-2, f"gemm {m}x{n}x{k}")
    _close(ops.gemm(a, w, epi=ops.EPI_SWIGLU), ref.gemm(a.float(), w.float(), epi=ops.EPI_SWIGLU), 2e-2, 2e-2, "swiglu")

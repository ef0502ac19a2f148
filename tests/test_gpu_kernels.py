"""Numerics of the native sm_100a kernels against plain PyTorch fp32 references of the same op."""
import contextlib
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from tesseract_b200 import _native
    assert _native.available(), "native library missing on a GPU machine"
    _native.lib()
    return torch.device("cuda", 0)


def _status_ok():
    from tesseract_b200 import _native
    assert _native.read_status(torch.cuda.current_stream().cuda_stream) == 0


def test_probe(dev):
    from tesseract_b200 import _native
    out = torch.zeros(1, dtype=torch.int32, device=dev)
    _native.check(_native.lib().tsb_probe(out.data_ptr(), _native.stream_ptr(dev)), "probe")
    assert int(out.item()) == 100


def _rel_err(got, ref):
    return ((got.float() - ref.float()).norm() / ref.float().norm().clamp_min(1e-12)).item()


GEMM_SHAPES = [(64, 4096, 512), (256, 6144, 1024), (128, 128, 64), (128, 256, 128), (256, 512, 256), (384, 640, 192), (1024, 1024, 1024),
               (200, 264, 136), (4096, 768, 512), (64, 4096, 4096)]


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES)
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
def test_gemm_layouts(dev, M, N, K, a_mn, b_mn):
    from tesseract_b200.ops import gemm_bf16
    g = torch.Generator(device=dev).manual_seed(M * 7 + N * 3 + K)
    A = torch.randn(M, K, device=dev, generator=g).bfloat16()
    B = torch.randn(N, K, device=dev, generator=g).bfloat16()
    ref = A.float() @ B.float().t()
    a_in = A.t().contiguous() if a_mn else A
    b_in = B.t().contiguous() if b_mn else B
    out = gemm_bf16(a_in, b_in, a_mn=a_mn, b_mn=b_mn)
    torch.cuda.synchronize()
    _status_ok()
    assert _rel_err(out, ref) < 6e-3, (M, N, K, a_mn, b_mn)


@pytest.mark.parametrize("block_n", [32, 64, 128, 256])
def test_gemm_block_sizes_and_fp32_accumulate(dev, block_n):
    from tesseract_b200.ops import gemm_bf16
    M, N, K = 512, 768, 320
    A = torch.randn(M, K, device=dev).bfloat16()
    B = torch.randn(N, K, device=dev).bfloat16()
    ref = A.float() @ B.float().t()
    out = torch.ones(M, N, device=dev, dtype=torch.float32)
    gemm_bf16(A, B, out=out, accumulate=True, block_n=block_n)
    torch.cuda.synchronize()
    _status_ok()
    assert _rel_err(out - 1.0, ref) < 1e-3
    outb = torch.full((M, N), 2.0, device=dev, dtype=torch.bfloat16)
    gemm_bf16(A, B, out=outb, accumulate=True, block_n=block_n)
    assert _rel_err(outb.float() - 2.0, ref) < 2e-2


def test_gemm_persistent_many_tiles(dev):
    """More tiles than SMs: exercises the smem ring / TMEM double-buffer phase flips (on pairs of SMs; tiles of one SM: see below)."""
    from tesseract_b200.ops import gemm_bf16
    M, N, K = 4096, 4096, 1024
    A = torch.randn(M, K, device=dev).bfloat16() * 0.1
    B = torch.randn(N, K, device=dev).bfloat16() * 0.1
    out = gemm_bf16(A, B)
    ref = A.float() @ B.float().t()
    torch.cuda.synchronize()
    _status_ok()
    assert _rel_err(out, ref) < 6e-3
    out2 = gemm_bf16(A, B)
    assert torch.equal(out, out2), "GEMM is not run-to-run deterministic"


def test_linear_autograd(dev):
    from tesseract_b200 import ops
    x = torch.randn(3, 128, 256, device=dev).bfloat16().requires_grad_()
    w = (torch.randn(384, 256, device=dev) * 0.05).bfloat16().requires_grad_()
    y = ops.linear(x, w)
    dy = torch.randn_like(y)
    y.backward(dy)
    xr = x.detach().float().requires_grad_()
    wr = w.detach().float().requires_grad_()
    yr = torch.nn.functional.linear(xr, wr)
    yr.backward(dy.float())
    assert _rel_err(y, yr) < 6e-3
    assert _rel_err(x.grad, xr.grad) < 8e-3
    assert _rel_err(w.grad, wr.grad) < 8e-3


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,D", [(37, 256), (512, 4096), (5, 8192), (700, 3080), (700, 6152)])
def test_rmsnorm_fwd_bwd(dev, dtype, rows, D):
    from tesseract_b200 import ops
    x = torch.randn(rows, D, device=dev).to(dtype).requires_grad_()
    r = torch.randn(rows, D, device=dev).to(dtype).requires_grad_()
    w = (1 + 0.1 * torch.randn(D, device=dev)).to(dtype).requires_grad_()
    y, h = ops.rms_norm(x, w, 1e-5, residual=r)
    gy, gh = torch.randn_like(y), torch.randn_like(h)
    (y.float() * gy.float()).sum().add((h.float() * gh.float()).sum()).backward()
    xr, rr, wr = [t.detach().float().requires_grad_() for t in (x, r, w)]
    hr = (xr + rr).to(dtype).float() if dtype != torch.float32 else xr + rr
    hr_full = xr + rr
    yr = ops.rms_norm_ref(hr_full, wr, 1e-5)
    ((yr * gy.float()).sum() + (hr_full * gh.float()).sum()).backward()
    tol = 2e-2 if dtype == torch.bfloat16 else 1e-4
    assert _rel_err(y, yr) < tol and _rel_err(h, hr_full) < tol
    assert _rel_err(x.grad, xr.grad) < tol and _rel_err(r.grad, rr.grad) < tol
    assert _rel_err(w.grad, wr.grad) < tol


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_swiglu_fwd_bwd(dev, dtype):
    from tesseract_b200 import ops
    gu = torch.randn(77, 2 * 1376, device=dev).to(dtype).requires_grad_()
    out = ops.swiglu(gu)
    g = torch.randn_like(out)
    out.backward(g)
    gr = gu.detach().float().requires_grad_()
    outr = ops.swiglu_ref(gr)
    outr.backward(g.float())
    tol = 1.5e-2 if dtype == torch.bfloat16 else 1e-5
    assert _rel_err(out, outr) < tol and _rel_err(gu.grad, gr.grad) < tol


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_rope_qkv(dev, dtype):
    from tesseract_b200 import ops
    H, Hkv, D, S, B = 4, 2, 64, 48, 3
    cos, sin = ops.rope_tables(128, D, 10000.0, dev)
    qkv = torch.randn(B * S, (H + 2 * Hkv) * D, device=dev).to(dtype)
    ref = ops.rope_qkv(qkv.cpu().float(), cos.cpu(), sin.cpu(), num_heads=H, num_kv_heads=Hkv, head_dim=D, seq_len=S,
                       pos_offset=5)
    x = qkv.clone().requires_grad_()
    got = ops.rope_qkv(x * 1.0, cos, sin, num_heads=H, num_kv_heads=Hkv, head_dim=D, seq_len=S, pos_offset=5)
    tol = 1e-2 if dtype == torch.bfloat16 else 1e-5
    assert _rel_err(got.cpu(), ref) < tol
    # backward = inverse rotation: rotating the gradient back must return the upstream gradient's preimage
    g = torch.randn_like(got)
    got.backward(g)
    xr = qkv.cpu().float().requires_grad_()
    refr = ops.rope_qkv(xr, cos.cpu(), sin.cpu(), num_heads=H, num_kv_heads=Hkv, head_dim=D, seq_len=S, pos_offset=5)
    refr.backward(g.cpu().float())
    assert _rel_err(x.grad.cpu(), xr.grad) < tol


def test_embedding_fwd_bwd(dev):
    from tesseract_b200 import ops
    V, D = 1000, 256
    table = torch.randn(V, D, device=dev).bfloat16().requires_grad_()
    ids = torch.randint(0, V, (4, 33), device=dev)
    out = ops.embedding(ids, table)
    assert torch.equal(out, table.detach()[ids])
    g = torch.randn_like(out)
    out.backward(g)
    ref = torch.zeros(V, D, device=dev).index_add_(0, ids.reshape(-1), g.reshape(-1, D).float())
    assert _rel_err(table.grad, ref) < 1e-2


@pytest.mark.parametrize("dtype,V", [(torch.bfloat16, 4096), (torch.float32, 1000), (torch.bfloat16, 128256)])
def test_cross_entropy(dev, dtype, V):
    from tesseract_b200 import ops
    N = 64
    logits = (torch.randn(N, V, device=dev) * 3).to(dtype).requires_grad_()
    tgt = torch.randint(0, V, (N,), device=dev)
    loss = ops.cross_entropy(logits, tgt)
    loss.backward()
    lr = logits.detach().float().requires_grad_()
    ref = torch.nn.functional.cross_entropy(lr, tgt)
    ref.backward()
    assert abs(loss.item() - ref.item()) < 2e-3 * max(1.0, abs(ref.item()))
    tol = 2e-2 if dtype == torch.bfloat16 else 1e-4
    assert _rel_err(logits.grad, lr.grad) < tol


def test_vocab_parallel_ce_stats_merge(dev):
    from tesseract_b200 import ops
    N, V = 32, 2048
    logits = (torch.randn(N, V, device=dev) * 2).bfloat16()
    tgt = torch.randint(0, V, (N,), device=dev)
    halves = [logits[:, :1024].contiguous(), logits[:, 1024:].contiguous()]
    stats = ops.merge_ce_stats([ops.ce_stats(h, tgt, vocab_start=i * 1024) for i, h in enumerate(halves)])
    losses = ops.ce_loss_and_grad_(halves[0], tgt, stats, 1.0, vocab_start=0, write_grad=False)
    ref = torch.nn.functional.cross_entropy(logits.float(), tgt, reduction="none")
    assert torch.allclose(losses, ref, atol=2e-3, rtol=2e-3)


@pytest.mark.parametrize("use_arena", [True, False])
def test_adam_matches_reference_formula(dev, use_arena):
    from tesseract_b200.optim import Adam, ParamArena
    torch.manual_seed(0)
    ps = [torch.nn.Parameter(torch.randn(n, device=dev)) for n in (1000, 70001, 129)]
    ref = [p.detach().clone() for p in ps]
    m = [torch.zeros_like(p) for p in ref]
    v = [torch.zeros_like(p) for p in ref]
    arena = ParamArena(ps) if use_arena else None
    opt = Adam(arena if use_arena else ps, lr=1e-2)
    for t in range(1, 4):
        grads = [torch.randn_like(p) for p in ref]
        for p, g in zip(ps, grads):
            if use_arena:
                p.main_grad.copy_(g)
            else:
                p.grad = g.clone()
        opt.step()
        for i, g in enumerate(grads):
            m[i] = 0.9 * m[i] + 0.1 * g
            v[i] = 0.999 * v[i] + 0.001 * g * g
            ref[i] -= 1e-2 * (m[i] / (1 - 0.9 ** t)) / ((v[i] / (1 - 0.999 ** t)).sqrt() + 1e-8)
    for p, r in zip(ps, ref):
        assert torch.allclose(p.detach(), r, atol=1e-5, rtol=1e-5)


@pytest.mark.parametrize("master", [False, True])
def test_adam_flat_bf16_vector_path_and_tail(dev, master):
    """bf16 parameters and gradients through the 8-wide kernel plus its scalar tail, against the fp32 formula."""
    from tesseract_b200 import _native
    from tesseract_b200.optim import optimizers  # noqa: F401
    n = 8 * 4099 + 5
    g0 = torch.Generator(device=dev).manual_seed(4)
    w32 = torch.randn(n, device=dev, generator=g0)
    p = w32.bfloat16()
    mst = w32.clone() if master else None
    ref = w32.clone() if master else p.float()
    m = torch.zeros(n, device=dev)
    v = torch.zeros(n, device=dev)
    rm, rv = m.clone(), v.clone()
    lib = _native.lib()
    s = torch.cuda.current_stream().cuda_stream
    for t in range(1, 4):
        g = torch.randn(n, device=dev, generator=g0).bfloat16()
        bc1, bc2 = 1 - 0.9 ** t, 1 - 0.999 ** t
        _native.check(lib.tsb_adam_flat(p.data_ptr(), g.data_ptr(), m.data_ptr(), v.data_ptr(),
                                        mst.data_ptr() if master else None, n, 1e-2, 0.9, 0.999, 1e-8, bc1, bc2, 0.01,
                                        None, 1, 1, s), "tsb_adam_flat")
        gf = g.float()
        rm = 0.9 * rm + 0.1 * gf
        rv = 0.999 * rv + 0.001 * gf * gf
        ref = ref - 1e-2 * ((rm / bc1) / ((rv / bc2).sqrt() + 1e-8) + 0.01 * ref)
        if not master:
            ref = ref.bfloat16().float()          # without a master copy the weights round to bf16 every step
    assert torch.allclose(m, rm, atol=1e-6, rtol=1e-5) and torch.allclose(v, rv, atol=1e-7, rtol=1e-5)
    assert torch.allclose(p.float(), ref.bfloat16().float(), atol=2e-2, rtol=1e-2)
    if master:
        assert torch.allclose(mst, ref, atol=1e-5, rtol=1e-4)


@pytest.mark.parametrize("M,N,K", [(128, 128, 128), (300, 264, 512), (1024, 4096, 4096), (64, 6144, 1024)])
def test_fp8_blockscaled_gemm_and_quantisers(dev, M, N, K):
    """Quantisers against their torch restatement (same bytes, same scales) and the tcgen05 fp8 GEMM against the
    fp32 matmul of the dequantised operands."""
    from tesseract_b200.ops import fp8
    g = torch.Generator(device=dev).manual_seed(M + N)
    x = (torch.randn(M, K, device=dev, generator=g) * 3).bfloat16()
    w = (torch.randn(N, K, device=dev, generator=g) * 0.05).bfloat16()
    x[0, :128] = 0                                            # an all-zero block takes scale 1
    qa, sa = fp8.quantize_act(x)
    qb, sb = fp8.quantize_weight(w)
    qa_r, sa_r = fp8.quantize_act_ref(x)
    qb_r, sb_r = fp8.quantize_weight_ref(w)
    assert torch.allclose(sa, sa_r, rtol=1e-6) and torch.allclose(sb, sb_r, rtol=1e-6)
    # the device rounds x * (1 / scale), torch rounds x / scale: a few bytes may land on the neighbouring code
    assert float((qa != qa_r).float().mean()) < 0.02 and float((qb != qb_r).float().mean()) < 0.02
    da, ra = fp8.dequantize_act(qa, sa), fp8.dequantize_act(qa_r, sa_r)
    # at most one e4m3 step: 2^-3 relative for normal codes, scale * 2^-9 absolute in the subnormal range
    assert bool(((da - ra).abs() <= 0.13 * ra.abs() + float(sa.max()) * 2.0 ** -9 * 1.01).all())
    y = fp8.fp8_gemm(qa, sa, qb, sb)
    ref = fp8.dequantize_act(qa, sa) @ fp8.dequantize_weight(qb, sb).t()
    _status_ok()
    assert _rel_err(y, ref) < 5e-3                            # bf16 output rounding only
    assert _rel_err(y, x.float() @ w.float().t()) < 6e-2      # end-to-end fp8 quantisation error
    lin = fp8.Fp8Linear(w)
    assert _rel_err(lin(x.view(1, M, K)).view(M, N), ref) < 5e-3


def test_linear_with_unaligned_width_falls_back(dev):
    """A 4-wide projection (an MoE router with four experts) cannot use 16-byte aligned rows: forward and backward
    run through the library path instead of refusing."""
    from tesseract_b200.ops import linear
    x = torch.randn(33, 256, device=dev).bfloat16().requires_grad_(True)
    w = (torch.randn(4, 256, device=dev) * 0.1).bfloat16().requires_grad_(True)
    y = linear(x, w)
    y.float().sum().backward()
    assert _rel_err(y, x.float() @ w.float().t()) < 1e-2
    assert x.grad is not None and w.grad is not None and w.grad.shape == w.shape


@pytest.mark.parametrize("causal", [True, False])
def test_flash_forward_with_growing_row_maxima(dev, causal):
    """Scores that keep growing along the key axis (and rows whose first visible key comes late) force the
    forward kernel to rescale the output it accumulates in tensor memory several times per row."""
    from tesseract_b200.ops import attention_ref, flash_attention
    B, S, H, Hkv, D = 2, 700, 4, 2, 128
    g = torch.Generator(device=dev).manual_seed(12)
    q = torch.randn(B, S, H, D, device=dev, generator=g).bfloat16()
    k = torch.randn(B, S, Hkv, D, device=dev, generator=g)
    v = torch.randn(B, S, Hkv, D, device=dev, generator=g).bfloat16()
    ramp = torch.linspace(0.2, 6.0, S, device=dev).view(1, S, 1, 1)          # later keys score up to 30x higher
    k = (k * ramp).bfloat16()
    with torch.no_grad():
        got = flash_attention(q, k, v, causal=causal)
        ref = attention_ref(q.transpose(1, 2).float(), k.transpose(1, 2).float(), v.transpose(1, 2).float(),
                            causal=causal).transpose(1, 2)
    _status_ok()
    assert torch.isfinite(got.float()).all()
    assert _rel_err(got, ref) < 2e-2


def _online_softmax(q, k, v, causal):
    """softmax(q k^T / sqrt D) v of heads (q [N, Sq, D], k and v [N, Sk, D] in bf16) with the roundings that the kernel may make: key
    tiles of 128, exponents relative to the running maximum, P rounded to bf16; sums in fp32, those of masked tiles of the rounded P.
    Also by how much the rows' maxima rise after the first 128 keys."""
    (N, Sq, D), Sk = q.shape, k.shape[1]
    s = q.float() @ k.float().transpose(1, 2) * D ** -0.5
    row = torch.arange(Sq, device=q.device)[:, None] + Sk - Sq
    if causal:
        s = s.masked_fill(torch.arange(Sk, device=q.device) > row, float("-inf"))
    first = torch.arange(Sq, device=q.device)[:, None] // 128 * 128 + Sk - Sq             # position of the query tile's first row
    m, l, o = torch.full((N, Sq, 1), float("-inf"), device=q.device), 0.0, 0.0
    for t in range(0, Sk, 128):
        st = s[:, :, t:t + 128]
        top = torch.maximum(m, st.amax(2, keepdim=True))
        base = top.masked_fill(top == float("-inf"), 0.0)
        p, f = torch.exp(st - base), torch.exp(m - base)
        masked = (t + 127 > first) if causal else torch.full_like(row, t + 128 > Sk, dtype=torch.bool)
        l = l * f + torch.where(masked, p.bfloat16().float(), p).sum(2, keepdim=True)
        o, m = o * f + p.bfloat16().float() @ v[:, t:t + 128].float(), top
    return o / l, m - s[:, :, :128].amax(2, keepdim=True)


@pytest.mark.parametrize("B,H,Hkv", [(1, 4, 2), (20, 4, 2), (20, 3, 3)])      # a tile per CTA; two heads of a group; two tiles of a head
@pytest.mark.parametrize("Sq,Sk", [(700, 700), (300, 1200)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("width,grow", [(1.0, False), (3.0, False), (6.0, False), (1.0, True)])
def test_flash_forward_accuracy_over_score_widths(dev, B, H, Hkv, Sq, Sk, D, width, grow):
    """Scores of unit width, as wide as in trained models, and growing along the keys by more than 2^8 at a time: no further from 64
    bits than the arithmetic above (5 % for the order of sums and the exponential's last bits), whatever the output's scale in TMEM."""
    from tesseract_b200.ops import flash_attention
    g = torch.Generator(device=dev).manual_seed(Sq + D)
    q = (torch.randn(B, Sq, H, D, device=dev, generator=g) * width).bfloat16()
    k = torch.randn(B, Sk, Hkv, D, device=dev, generator=g)
    if grow:
        k = k * torch.linspace(0.2, 12.0, Sk, device=dev).view(1, Sk, 1, 1)
    k, v = k.bfloat16(), torch.randn(B, Sk, Hkv, D, device=dev, generator=g).bfloat16()
    rows = [t.repeat_interleave(n, 2).transpose(1, 2).flatten(0, 1) for t, n in ((q, 1), (k, H // Hkv), (v, H // Hkv))]
    for causal in (True, False):
        with torch.no_grad():
            got = flash_attention(q, k, v, causal=causal).transpose(1, 2).flatten(0, 1)
        torch.cuda.synchronize()
        _status_ok()
        s = rows[0].double() @ rows[1].double().transpose(1, 2) * D ** -0.5
        if causal:
            s = s.masked_fill(torch.arange(Sk, device=dev) > torch.arange(Sq, device=dev)[:, None] + Sk - Sq, float("-inf"))
        ref = torch.softmax(s, -1) @ rows[2].double()
        o, rise = _online_softmax(*rows, causal)
        assert not grow or float(rise.max()) > 8.0                 # (in units of e: more than 2^8)
        mine, theirs = (float((x.double() - ref).norm() / ref.norm()) for x in (got, o.bfloat16()))
        assert mine <= theirs * 1.05, (mine, theirs)


@pytest.mark.parametrize("M", [1, 2, 3, 4])
@pytest.mark.parametrize("N,K", [(1, 16), (7, 272), (149, 4096), (2049, 528), (33, 24576), (1000, 1040), (2049, 2304), (600, 4352), (5000, 272),
                                 (28672, 4096)])                              # (the last, and K = 16 with three rows on, by the tensor cores)
@pytest.mark.parametrize("pdl", [False, True])
def test_few_rows_gemv(dev, M, N, K, pdl):
    """One to four rows on CUDA cores: ends of rows, of K and of its share per warp, 1 to 16 warps per row. fp32 sums rounded to bf16 once: 0.0011 of a
    value in the mean. Rows of the result beside the written ones stay as they were."""
    from tesseract_b200.ops.gemm import stream_linear
    g = torch.Generator(device=dev).manual_seed(M * N + K)
    x = torch.randn(M, K + 8, device=dev, generator=g).bfloat16()[:, :K]
    w = (torch.randn(N, K + 8, device=dev, generator=g) * 0.05).bfloat16()[:, :K]
    out = torch.full((M, N + 3), 7.0, device=dev, dtype=torch.bfloat16)
    stream_linear(x, w, out=out[:, :N], pdl=pdl)
    torch.cuda.synchronize()
    _status_ok()
    assert _rel_err(out[:, :N], x.float() @ w.float().t()) < 3.5e-3
    assert bool((out[:, N:] == 7.0).all())


@pytest.mark.parametrize("M,N,K,split", [(64, 512, 512, 1), (64, 512, 512, 2), (256, 6144, 4096, 4), (37, 264, 1032, 8),
                                          (130, 4096, 14336, 8), (1, 128, 128, 2)])
def test_cluster_splitk_gemm(dev, M, N, K, split):
    """K slices reduced through the shared memory of a thread-block cluster, against the fp32 product."""
    from tesseract_b200 import _native
    from tesseract_b200.ops import gemm  # noqa: F401
    g = torch.Generator(device=dev).manual_seed(M + N + K)
    x = torch.randn(M, K, device=dev, generator=g).bfloat16()
    w = (torch.randn(N, K, device=dev, generator=g) * 0.05).bfloat16()
    out = torch.full((M, N), float("nan"), device=dev, dtype=torch.bfloat16)
    _native.check(_native.lib().tsb_gemm_cluster_splitk(x.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, x.stride(0),
                                                        w.stride(0), out.stride(0), split,
                                                        torch.cuda.current_stream().cuda_stream), "tsb_gemm_cluster_splitk")
    torch.cuda.synchronize()
    _status_ok()
    assert torch.isfinite(out.float()).all()
    assert _rel_err(out, x.float() @ w.float().t()) < 1e-2


@pytest.mark.parametrize("D", [128, 64])
@pytest.mark.parametrize("H,Hkv,copies", [(8, 2, 1), (8, 2, 3), (9, 3, 3)])   # a tile per CTA; two heads of a group; two tiles of a head
def test_flash_varlen_matches_per_sequence(dev, D, H, Hkv, copies):
    """Prompts of different lengths packed on one token axis, one launch, against per-sequence attention."""
    from tesseract_b200 import ops
    lens = [5, 300, 128, 1, 257, 64] * copies
    g = torch.Generator(device=dev).manual_seed(D)
    qkv = torch.randn(sum(lens), H + 2 * Hkv, D, device=dev, generator=g).bfloat16()
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=dev)
    got = ops.flash_attention_varlen_packed(qkv, cu, max(lens), H, Hkv)
    torch.cuda.synchronize()
    _status_ok()
    off = 0
    for n in lens:
        seg = qkv[off:off + n]
        q, k, v = seg[:, :H], seg[:, H:H + Hkv], seg[:, H + Hkv:]
        ref = ops.attention_ref(q.transpose(0, 1).unsqueeze(0).float(), k.transpose(0, 1).unsqueeze(0).float(),
                                v.transpose(0, 1).unsqueeze(0).float(), causal=True)[0].transpose(0, 1)
        assert _rel_err(got[off:off + n], ref) < 2e-2, n
        off += n


@pytest.mark.parametrize("M,N,K", [(128, 256, 128), (300, 264, 512), (1024, 2048, 512), (1024, 1024, 1024),
                                   (2048, 4096, 4096)])     # tile widths 64, 64, 128, 64, 256
def test_fp8_pertensor_gemm(dev, M, N, K):
    """Per-tensor-scaled E4M3 GEMM (whole K accumulated in tensor memory) against the fp32 product of the
    dequantised operands, and against the unquantised product within fp8 error."""
    from tesseract_b200.ops import fp8
    g = torch.Generator(device=dev).manual_seed(M + K)
    x = torch.randn(M, K, device=dev, generator=g).bfloat16()
    w = (torch.randn(N, K, device=dev, generator=g) * 0.05).bfloat16()
    qa, sa = fp8.quantize_tensor(x)
    qb, sb = fp8.quantize_tensor(w)
    assert abs(float(sa) - float(x.float().abs().max()) / 448.0) < 1e-6
    y = fp8.fp8_gemm_pertensor(qa, sa, qb, sb)
    _status_ok()
    ref = (qa.view(torch.float8_e4m3fn).float() * sa) @ (qb.view(torch.float8_e4m3fn).float() * sb).t()
    assert _rel_err(y, ref) < 5e-3
    assert _rel_err(y, x.float() @ w.float().t()) < 8e-2


def test_tiny_llama_train_step_matches_cpu(dev):
    """bf16 GPU step through every native kernel vs the fp32 CPU restatement of the same model."""
    from tesseract_b200.models import LlamaConfig, LlamaModel
    cfg = LlamaConfig(vocab_size=512, hidden_size=256, num_hidden_layers=2, num_attention_heads=4,
                      num_key_value_heads=2, intermediate_size=512, max_position_embeddings=128, dtype=torch.float32)
    cpu = LlamaModel(cfg, init_std=0.02, seed=3)
    cfg_g = LlamaConfig(**{**cfg.__dict__, "dtype": torch.bfloat16})
    gpu = LlamaModel(cfg_g, device=dev)
    gpu.load_hf_state_dict({k: v for k, v in cpu.hf_state_dict().items()})
    tok = torch.randint(0, 512, (2, 128))
    tgt = torch.randint(0, 512, (2, 128))
    lc = cpu.loss(tok, tgt)
    lc.backward()
    lg = gpu.loss(tok.to(dev), tgt.to(dev))
    lg.backward()
    _status_ok()
    assert abs(lc.item() - lg.item()) < 3e-2
    gc = dict(cpu.named_parameters())
    worst = 0.0
    for n, p in gpu.named_parameters():
        worst = max(worst, _rel_err(p.grad.cpu(), gc[n].grad))
    assert worst < 8e-2, worst


@pytest.mark.parametrize("M,N,K,pad", [(4864, 4096, 64, 0), (4872, 4104, 520, 0), (9000, 2312, 136, 0),      # pairs: halves of 192, and of 256
                                       (4864, 4096, 960, 0), (4872, 4104, 1032, 0), (9000, 2312, 1000, 3), (4864, 4096, 12288, 0),
                                       (4864, 4096, 12352, 0)])                                  # the last two: whole tiles of 256 x 384
@pytest.mark.parametrize("a_mn", [False, True])
@pytest.mark.parametrize("b_mn", [False, True])
@pytest.mark.parametrize("out,accumulate", [(torch.bfloat16, False), (torch.bfloat16, True), (torch.float32, True)])
def test_gemm_tiles_of_two_sms(dev, M, N, K, pad, a_mn, b_mn, out, accumulate):
    """Products large enough for 256 x 256 tiles: whole tiles, ends of every kind, result rows that allow no wide stores. fp32 sums
    of exact products, in another order than the reference's: 1e-4 at most at these depths; a bf16 result is rounded once more,
    2^-9 / sqrt 3 = 0.0011 of it in the mean."""
    from tesseract_b200.ops.gemm import gemm_bf16
    g = torch.Generator(device=dev).manual_seed(M + N + K)
    a = torch.randn(*((K, M) if a_mn else (M, K)), device=dev, generator=g).bfloat16()
    b = torch.randn(*((K, N) if b_mn else (N, K)), device=dev, generator=g).bfloat16()
    rows = torch.randn(M, N + pad, device=dev, generator=g).to(out)
    beside, c = rows[:, N:].clone(), rows[:, :N]
    ref = (a.t() if a_mn else a).double() @ (b if b_mn else b.t()).double() + (c.double() if accumulate else 0)
    gemm_bf16(a, b, a_mn=a_mn, b_mn=b_mn, out=c, accumulate=accumulate)
    torch.cuda.synchronize()
    _status_ok()
    assert float((c.double() - ref).norm() / ref.norm()) < (3e-3 if out == torch.bfloat16 else 1e-4)
    assert torch.equal(rows[:, N:], beside)


@pytest.mark.parametrize("M,N,K,pad,cut", [(3000, 4104, 6152, 0, (256, 2, 74, 142)), (3000, 4104, 6152, 3, (256, 2, 74, 142)),     # whole tiles, then halves, some beyond N
                                           (1800, 6392, 6152, 0, (256, 2, 74, 134)), (3000, 5384, 6152, 0, (256, 2, 132, 132)),
                                           (3000, 6392, 6152, 0, (192, 2, 204, 204)), (3000, 6392, 6152, 3, (192, 2, 204, 204)),
                                           (2600, 2048, 8200, 0, (192, 2, 66, 66)),                                                # whole tiles only
                                           (3000, 2048, 2056, 0, (192, 1, 132, 132)), (1072, 1152, 3264, 0, (128, 1, 45, 45)),     # halves only
                                           (2600, 12104, 72, 0, (256, 1, 528, 528))])                                              # two blocks of K
@pytest.mark.parametrize("a_mn", [False, True])
@pytest.mark.parametrize("b_mn", [False, True])
@pytest.mark.parametrize("out,accumulate", [(torch.bfloat16, False), (torch.bfloat16, True), (torch.float32, False)])
def test_gemm_kinds_of_tiles(dev, M, N, K, pad, cut, a_mn, b_mn, out, accumulate):
    """Every kind of tile of two SMs that the rule chooses (``cut``, on 148 SMs) at its edges, stored by TMA or (rows off 16 bytes) directly. Bounds as
    above; a wrong column or row of a tile would stand out by the size of the result."""
    from tesseract_b200.ops.gemm import gemm_bf16, gemm_plan
    if torch.cuda.get_device_properties(dev).multi_processor_count == 148:
        assert gemm_plan(M, N, K) == cut
    g = torch.Generator(device=dev).manual_seed(M + N + K)
    a = torch.randn(*((K, M) if a_mn else (M, K)), device=dev, generator=g).bfloat16()
    b = torch.randn(*((K, N) if b_mn else (N, K)), device=dev, generator=g).bfloat16()
    rows = torch.randn(M, N + pad, device=dev, generator=g).to(out)
    beside, c = rows[:, N:].clone(), rows[:, :N]
    ref = (a.t() if a_mn else a).double() @ (b if b_mn else b.t()).double() + (c.double() if accumulate else 0)
    gemm_bf16(a, b, a_mn=a_mn, b_mn=b_mn, out=c, accumulate=accumulate)
    torch.cuda.synchronize()
    _status_ok()
    assert float((c.double() - ref).norm() / ref.norm()) < (3e-3 if out == torch.bfloat16 else 1e-4)
    # a value's error: half a step of bf16, 2^-9 of the largest, or what fp32 sums of this depth leave
    assert float((c.double() - ref).abs().max()) <= float(ref.abs().max()) * (2.0 ** -8 if out == torch.bfloat16 else 1e-4)
    assert torch.equal(rows[:, N:], beside)


@pytest.mark.parametrize("M,N,K", [(32000, 4096, 4096), (4096, 14336, 4096), (1024, 14336, 4096), (2048, 8192, 4096), (8192, 6144, 4096)])
def test_gemm_products_that_halves_suit(dev, M, N, K):
    """At this depth halves of 256 columns are 6 - 20 % faster than whole tiles of either width where both need as many rounds (times beside the rule)."""
    from tesseract_b200.ops.gemm import gemm_plan
    if torch.cuda.get_device_properties(dev).multi_processor_count == 148:
        assert gemm_plan(M, N, K)[:2] == (256, 1)


def _gemm_layouts(dev, M, N, K, pad, run, pairs_of=((torch.bfloat16, False), (torch.bfloat16, True), (torch.float32, False), (torch.float32, True))):
    """All layouts of the operands and forms of the result of one size, by ``run(a, b, c, a_mn, b_mn, accumulate)``; bounds as above."""
    g = torch.Generator(device=dev).manual_seed(M + N + K)
    a, b = torch.randn(M, K, device=dev, generator=g).bfloat16(), torch.randn(N, K, device=dev, generator=g).bfloat16()
    product = a.double() @ b.double().t()
    for out, accumulate in pairs_of:
        rows = torch.randn(M, N + pad, device=dev, generator=g).to(out)
        ref = product + (rows[:, :N].double() if accumulate else 0)
        for a_mn in (False, True):
            for b_mn in (False, True):
                got = rows.clone()
                run(a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b, got[:, :N], a_mn, b_mn, accumulate)
                torch.cuda.synchronize()
                _status_ok()
                what = (out, accumulate, a_mn, b_mn)
                c = got[:, :N].double()
                assert float((c - ref).norm() / ref.norm()) < (3e-3 if out == torch.bfloat16 else 1e-4), what
                assert float((c - ref).abs().max()) <= float(ref.abs().max()) * (2.0 ** -8 if out == torch.bfloat16 else 1e-4), what
                assert torch.equal(got[:, N:], rows[:, N:]), what


@pytest.mark.parametrize("n,per", [(256, 2), (192, 2), (256, 1), (192, 1), (128, 1)])
@pytest.mark.parametrize("M,wide,K,pad", [(2248, 9, 264, 0), (2248, 9, 264, 3), (5000, 8, 8, 0), (5000, 8, 72, 0), (5000, 8, 584, 0)])
def test_gemm_each_kind_of_tiles(dev, n, per, M, wide, K, pad):
    """Each kind by itself, at sizes that have all of it: a last column of tiles with one half (so that the next one starts on the other accumulator),
    several tiles per pair, the rest of a round as halves, some beyond N, and one to ten blocks of K in rings of four and of six."""
    from tesseract_b200 import _native
    N = (wide - 1) * per * n + n - 56
    pairs, tiles = torch.cuda.get_device_properties(dev).multi_processor_count // 2, -(-M // 256) * wide
    assert pairs != 74 or (tiles > pairs and 0 < 2 * (tiles % pairs) <= pairs)

    def run(a, b, c, a_mn, b_mn, accumulate):
        _native.check(_native.lib().tsb_gemm_bf16_pairs(a.data_ptr(), b.data_ptr(), c.data_ptr(), M, N, K, a.stride(0), b.stride(0), c.stride(0), int(a_mn),
                                                        int(b_mn), int(c.dtype == torch.float32), int(accumulate), n, per,
                                                        _native.stream_ptr(a.device)), "tsb_gemm_bf16_pairs")
    _gemm_layouts(dev, M, N, K, pad, run)


def test_gemm_kinds_that_there_are_not(dev):
    from tesseract_b200 import _native
    a = torch.zeros(512, 64, device=dev, dtype=torch.bfloat16)
    c = torch.zeros(512, 512, device=dev, dtype=torch.bfloat16)
    call = lambda M, N, n, per: _native.lib().tsb_gemm_bf16_pairs(a.data_ptr(), a.data_ptr(), c.data_ptr(), M, N, 64, 64, 64, 512, 0, 0, 0, 0, n, per,
                                                                  _native.stream_ptr(a.device))
    assert all(call(*w) == -2 for w in ((512, 512, 128, 2), (512, 512, 64, 1), (512, 512, 256, 3), (512, 512, 256, 0), (128, 512, 256, 1), (512, 184, 256, 1)))
    assert call(512, 512, 256, 2) == 0
    torch.cuda.synchronize()
    _status_ok()


@pytest.mark.parametrize("bn", [64, 128, 256])
@pytest.mark.parametrize("ctas", [0, 37])
@pytest.mark.parametrize("K", [72, 1000])
def test_gemm_tiles_of_one_sm_many_per_cta(dev, bn, ctas, K):
    """Three and twelve tiles per CTA (the phases of ring and accumulators flip), ragged ends of all three sizes."""
    from tesseract_b200.ops.gemm import gemm_bf16
    M, N = 2616, 20 * bn + 40
    _gemm_layouts(dev, M, N, K, 0, lambda a, b, c, a_mn, b_mn, accumulate: gemm_bf16(a, b, a_mn=a_mn, b_mn=b_mn, out=c, accumulate=accumulate, block_n=bn,
                                                                                    max_ctas=ctas),
                  ((torch.bfloat16, False), (torch.float32, True)))


def _block_model(dev, width, heads, kv, ffn, seed=0):
    from tesseract_b200.models import LlamaConfig, LlamaModel
    from tesseract_b200.optim import ParamArena
    cfg = LlamaConfig(vocab_size=96, hidden_size=width, num_hidden_layers=2, num_attention_heads=heads, num_key_value_heads=kv,
                      intermediate_size=ffn, max_position_embeddings=512, dtype=torch.bfloat16)
    model = LlamaModel(cfg, device=dev, init_std=0.05, seed=seed)
    return model, ParamArena.from_module(model)


@pytest.mark.parametrize("width,heads,kv,ffn,B,S", [(128, 2, 1, 256, 1, 1), (128, 2, 2, 264, 2, 129), (256, 2, 1, 688, 3, 77), (512, 4, 4, 1032, 1, 300),
                                                    (512, 8, 2, 1024, 2, 128)])
def test_block_in_one_call_gives_what_its_modules_give(dev, width, heads, kv, ffn, B, S):
    """The same launches, so the same bits, but for the gradient that leaves the first block: it is a sum of two, which the block rounds once (2^-9 of it) and
    autograd twice; and beyond 256 keys for dQ, whose parts add up in any order, and what depends on it (a last bit of bf16 here and there)."""
    model, arena = _block_model(dev, width, heads, kv, ffn)
    g = torch.Generator(device=dev).manual_seed(S)
    tok, tgt = (torch.randint(0, 96, (B, S), device=dev, generator=g) for _ in range(2))
    results = []
    for hooked in (False, True):
        handles = [blk.norm_1.register_forward_hook(lambda *a: None) for blk in model.layers] if hooked else []
        x = model.embed_tokens(tok)
        assert (model.layers[0]._whole(x, None) is None) is hooked
        arena.zero_grad()
        for _ in range(2):                                     # gradients add up
            loss = model.loss(tok, tgt)
            loss.backward()
        results.append((float(loss.detach()), {n: p.main_grad.clone() for n, p in model.named_parameters()}))
        for h in handles:
            h.remove()
    _status_ok()
    assert results[0][0] == results[1][0]
    for n, a in results[0][1].items():
        if S <= 256 and n != "embed_tokens.weight":
            assert torch.equal(a, results[1][1][n]), n
        else:
            assert _rel_err(a, results[1][1][n].float()) < 5e-3, n


def _run_block(blk, arena, x, res, dout, dres, around=contextlib.nullcontext()):
    """(out, residual stream, gradients of x, of res and of the weights by name), everything cloned."""
    arena.zero_grad()
    x, res = (None if t is None else t.detach().clone().requires_grad_() for t in (x, res))
    with around:
        out, stream = blk.forward_fused(x, res)
    ins = [x] if res is None else [x, res]
    dx = torch.autograd.grad([out, stream], ins, [dout, dres])
    return ([out.detach().clone(), stream.detach().clone()], list(dx),
            {n: p.main_grad.clone() for n, p in blk.named_parameters()})


def _block_inputs(dev, B, S, width, seed=0):
    g = torch.Generator(device=dev).manual_seed(seed + S)
    return [torch.randn(B, S, width, device=dev, generator=g).bfloat16() for _ in range(4)]


BEHIND_DQ = ("norm_1.weight", "attn.q_proj.weight")      # gradients that depend on dQ


def _same_blocks(a, b, exact):
    """Of up to 256 keys the parts of dQ are two per value, whose sum is the same in either order; of more, only what does not depend on dQ is."""
    assert all(torch.equal(s, t) for s, t in zip(a[0], b[0]))
    for n in a[2]:
        if exact or n not in BEHIND_DQ:
            assert torch.equal(a[2][n], b[2][n]), n
        else:
            assert _rel_err(a[2][n], b[2][n].float()) < 2e-3, n
    for s, t in zip(a[1], b[1]):
        assert torch.equal(s, t) if exact else _rel_err(s, t.float()) < 2e-3


@pytest.mark.parametrize("kind", ["copy", "host", "pinned", "off"])
@pytest.mark.parametrize("has_res", [True, False])
def test_block_under_hooks_on_saved_tensors(dev, kind, has_res):
    """What is saved may come back somewhere else (activations kept on the host), at any address; the weights' rows are all there."""
    model, arena = _block_model(dev, 256, 2, 1, 688)
    blk = model.layers[1]
    x, res, dout, dres = _block_inputs(dev, 2, 150, 256)
    res = res if has_res else None
    assert blk._whole(x.requires_grad_(), res) is not None
    want = _run_block(blk, arena, x, res, dout, dres)
    moved = lambda t: torch.empty(t.numel() + 1, device=t.device, dtype=t.dtype)[1:].view(t.shape).copy_(t)
    around = {"copy": lambda: torch.autograd.graph.saved_tensors_hooks(lambda t: t.detach().clone(), lambda t: t),
              "off": lambda: torch.autograd.graph.saved_tensors_hooks(lambda t: t.detach(), moved),
              "host": lambda: torch.autograd.graph.save_on_cpu(), "pinned": lambda: torch.autograd.graph.save_on_cpu(pin_memory=True)}[kind]()
    got = _run_block(blk, arena, x, res, dout, dres, around)
    _status_ok()
    _same_blocks(got, want, exact=True)


@pytest.mark.parametrize("width,heads,kv,ffn", [(512, 4, 1, 1792), (512, 4, 4, 1024), (512, 8, 8, 1408), (1024, 8, 1, 2048)])
def test_block_holds_no_more_memory_than_its_modules(dev, width, heads, kv, ffn):
    """The most that is held during a forward and backward pass over two blocks (32 MB a piece of the stream and more, so that what a
    few small buffers differ by, or their rounding to 512 bytes, does not count: 1 MB)."""
    model, arena = _block_model(dev, width, heads, kv, ffn)
    x, _, dout, dres = _block_inputs(dev, 64, 512, width)
    x.requires_grad_()
    most = []
    for hooked in (False, True):
        handles = [blk.norm_1.register_forward_hook(lambda *a: None) for blk in model.layers] if hooked else []
        assert (model.layers[0]._whole(x, None) is None) is hooked
        for _ in range(2):
            torch.cuda.synchronize()
            before = torch.cuda.memory_allocated()
            torch.cuda.reset_peak_memory_stats()
            a, r = model.layers[0].forward_fused(x, None)
            a, r = model.layers[1].forward_fused(a, r)
            y = model.norm(a, r)[0]
            del a, r
            g, = torch.autograd.grad(y, x, dout)
            torch.cuda.synchronize()
            peak = torch.cuda.max_memory_allocated() - before
            del y, g
        most.append(peak)
        for h in handles:
            h.remove()
    _status_ok()
    assert most[0] <= most[1] + (1 << 20), most


def test_block_counts_the_launches_of_its_modules(dev):
    from tesseract_b200 import _native
    model, arena = _block_model(dev, 256, 2, 1, 688)
    blk = model.layers[1]
    x, res, dout, dres = _block_inputs(dev, 2, 40, 256)
    counts = []
    for hooked in (False, True):
        h = blk.norm_1.register_forward_hook(lambda *a: None) if hooked else None
        arena.zero_grad()
        x, res = (t.detach().requires_grad_() for t in (x, res))
        at = [_native.launch_count()]
        out, stream = blk.forward_fused(x, res)
        at.append(_native.launch_count())
        torch.autograd.grad([out, stream], [x, res], [dout, dres])
        at.append(_native.launch_count())
        counts.append([b - a for a, b in zip(at[:-1], at[1:])])
        if h:
            h.remove()
    assert counts[0] == counts[1] == [9, 17]


@pytest.mark.parametrize("width,heads,kv,ffn,B,S", [(128, 2, 1, 264, 2, 1), (256, 2, 2, 688, 1, 129), (512, 4, 1, 1032, 2, 256), (512, 8, 2, 1024, 1, 400)])
@pytest.mark.parametrize("has_res", [True, False])
def test_block_against_its_modules_bit_by_bit(dev, width, heads, kv, ffn, B, S, has_res):
    """As above, with every gradient of one block; what leaves a block without a residual stream behind it is rounded once or twice, 2^-8 at most."""
    model, arena = _block_model(dev, width, heads, kv, ffn)
    blk = model.layers[0]
    x, res, dout, dres = _block_inputs(dev, B, S, width)
    res = res if has_res else None
    got = _run_block(blk, arena, x, res, dout, dres)
    h = blk.norm_1.register_forward_hook(lambda *a: None)
    want = _run_block(blk, arena, x, res, dout, dres)
    h.remove()
    _status_ok()
    if not has_res:
        assert _rel_err(got[1].pop(), want[1].pop().float()) < 2 ** -8
    _same_blocks(got, want, exact=S <= 256)


@pytest.mark.parametrize("kind", ["again", "reentrant", "checkpoint", "side", "marker"])
def test_block_where_autograd_is_used_otherwise(dev, kind):
    """A graph kept for a second pass, recomputation of either kind, a stream of the program's own, and the marker by which data parallelism hears that a
    block's gradients are complete: the bits of a plain pass."""
    from torch.utils.checkpoint import checkpoint
    from tesseract_b200.parallel.data_parallel import _BucketMarker
    model, arena = _block_model(dev, 256, 2, 1, 688)
    blk = model.layers[1]
    x, res, dout, dres = _block_inputs(dev, 2, 200, 256)
    want = _run_block(blk, arena, x, res, dout, dres)
    arena.zero_grad()
    torch.cuda.synchronize()
    side = torch.cuda.Stream() if kind == "side" else torch.cuda.current_stream()
    fired = []

    class Reducer:
        def _bucket_ready(self, bid):
            fired.append((bid, {n: p.main_grad.clone() for n, p in blk.named_parameters()}))

    with torch.cuda.stream(side):
        x, res = (t.detach().clone().requires_grad_() for t in (x, res))
        ins = [_BucketMarker.apply(t, Reducer(), 3) for t in (x, res)] if kind == "marker" else [x, res]
        if kind in ("reentrant", "checkpoint"):
            out, stream = checkpoint(blk.forward_fused, *ins, use_reentrant=kind == "reentrant")
        else:
            out, stream = blk.forward_fused(*ins)
        torch.autograd.backward([out, stream], [dout, dres], retain_graph=kind == "again")
        if kind == "again":
            arena.zero_grad()
            x.grad = res.grad = None
            torch.autograd.backward([out, stream], [dout, dres])
    torch.cuda.synchronize()
    _status_ok()
    got = ([out.detach(), stream.detach()], [x.grad, res.grad], {n: p.main_grad.clone() for n, p in blk.named_parameters()})
    _same_blocks(got, want, exact=True)
    if kind == "marker":
        assert [bid for bid, _ in fired] == [3, 3] and all(torch.equal(t, got[2][n]) for n, t in fired[0][1].items())
    if kind == "again":
        with pytest.raises(RuntimeError):
            torch.autograd.backward([out, stream], [dout, dres])          # (the graph was given back)


def test_block_runs_its_modules_where_they_are_not_plain(dev):
    from tesseract_b200.nn.modules import Linear
    model, arena = _block_model(dev, 128, 2, 1, 256)
    blk = model.layers[1]
    x = torch.randn(2, 8, 128, device=dev, dtype=torch.bfloat16, requires_grad=True)
    whole = lambda: blk._whole(x, None) is not None
    assert whole()
    for m in (blk.norm_1, blk.attn, blk.attn.v_proj, blk.norm_2, blk.ffn, blk.ffn.down_proj):
        h = m.register_forward_pre_hook(lambda *a: None)
        assert not whole()
        h.remove()
        h = m.register_full_backward_hook(lambda *a: None)
        assert not whole()
        h.remove()
    blk.ffn.up_proj.weight.requires_grad_(False)
    assert not whole()
    blk.ffn.up_proj.weight.requires_grad_(True)
    kept = blk.attn.k_proj
    blk.attn.k_proj = torch.nn.Linear(128, 64, bias=False, device=dev, dtype=torch.bfloat16)
    assert not whole()                                          # another class
    blk.attn.k_proj = Linear(128, 64, bias=False, device=dev, dtype=torch.bfloat16)
    assert not whole()                                          # no main_grad, apart from its neighbours
    blk.attn.k_proj = kept
    assert whole()
    with torch.no_grad():
        assert not whole()
    assert blk._whole(x.detach(), None) is None and blk._whole(x.float(), None) is None and blk._whole(x[0], None) is None


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,F,shift", [(1, 16, 0), (3, 2048, 0), (5, 2064, 0), (700, 4112, 0), (66000, 16, 0), (7, 2056, 0), (9, 2048, 8)])
def test_swiglu_in_pieces_of_32_bytes(dev, dtype, rows, F, shift):
    """Edges of the wide kernels (last CTA of a row, second row of a thread, more rows than the grid), and what keeps the others: F off 16, rows off 32
    bytes. Values of a few units: one rounding of the type's precision each, plus fp32 exponentials (2^-20)."""
    from tesseract_b200 import _native
    g = torch.Generator(device=dev).manual_seed(F)
    def t(n):
        return torch.randn(n + shift, device=dev, generator=g).to(dtype)[shift:]
    gu, do = t(rows * 2 * F).view(rows, 2 * F), t(rows * F).view(rows, F)
    out, dgu = t(rows * F).view(rows, F), t(rows * 2 * F).view(rows, 2 * F)
    code, s = _native.dtype_code(dtype), _native.stream_ptr(dev)
    _native.check(_native.lib().tsb_swiglu_fwd(gu.data_ptr(), out.data_ptr(), rows, F, code, s), "fwd")
    _native.check(_native.lib().tsb_swiglu_bwd(do.data_ptr(), gu.data_ptr(), dgu.data_ptr(), rows, F, code, s), "bwd")
    x = gu.double().requires_grad_()
    ref = torch.nn.functional.silu(x[:, :F]) * x[:, F:]
    ref.backward(do.double())
    eps = torch.finfo(dtype).eps / 2 + 2.0 ** -18
    assert bool(((out.double() - ref).abs() <= ref.abs() * eps + 1e-6).all())
    assert bool(((dgu.double() - x.grad).abs() <= x.grad.abs() * eps + 2e-6).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens,H,Hkv,D,bs", [(1, 4, 2, 64, 8), (77, 3, 3, 128, 16), (2051, 32, 8, 128, 16), (700, 5, 1, 64, 12)])
def test_prompt_rotation_and_append_in_one_pass(dev, dtype, tokens, H, Hkv, D, bs):
    """Against the two kernels that it stands for, the same bits; a token without a slot is not stored."""
    from tesseract_b200 import _native, ops
    g = torch.Generator(device=dev).manual_seed(tokens)
    nb = tokens // bs + 2
    qkv = torch.randn(tokens, (H + 2 * Hkv) * D, device=dev, generator=g).to(dtype)
    pools = [torch.randn(nb, Hkv, bs, D, device=dev, generator=g).to(dtype) for _ in range(2)]
    cos, sin = ops.rope_tables(4096, D, 1e4, dev)
    pos = torch.randint(0, 4096, (tokens,), device=dev, generator=g, dtype=torch.int32)
    slots = torch.randperm(nb * bs, generator=torch.Generator().manual_seed(2))[:tokens].int().to(dev)
    slots[tokens // 2] = -1
    a, b, (k1, v1), (k2, v2) = qkv.clone(), qkv.clone(), [p.clone() for p in pools], [p.clone() for p in pools]
    lib, code, s = _native.lib(), _native.dtype_code(dtype), _native.stream_ptr(qkv.device)
    _native.check(lib.tsb_rope_append_paged(a.data_ptr(), cos.data_ptr(), sin.data_ptr(), pos.data_ptr(), slots.data_ptr(), k1.data_ptr(), v1.data_ptr(),
                                            tokens, H, Hkv, D, bs, code, s), "one")
    b = ops.rope_qkv(b, cos, sin, num_heads=H, num_kv_heads=Hkv, head_dim=D, seq_len=1, positions=pos)
    _native.check(lib.tsb_kv_append_paged(b.data_ptr(), cos.data_ptr(), sin.data_ptr(), pos.data_ptr(), slots.data_ptr(), k2.data_ptr(), v2.data_ptr(),
                                          None, None, None, tokens, H, Hkv, D, bs, code, 0, s), "two")
    assert torch.equal(a, b) and torch.equal(k1, k2) and torch.equal(v1, v2)
    kept = torch.zeros(nb * bs, dtype=torch.bool, device=dev)
    kept[slots[slots >= 0].long()] = True
    rest = ~kept.view(nb, 1, bs, 1).expand_as(k1)
    assert torch.equal(k1[rest], pools[0][rest])
    assert lib.tsb_rope_append_paged(a.data_ptr() + 2, cos.data_ptr(), sin.data_ptr(), pos.data_ptr(), slots.data_ptr(), k1.data_ptr(), v1.data_ptr(),
                                     tokens, H, Hkv, D, bs, code, s) == -2


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("D", [64, 72, 128])
def test_rotation_rounds_the_same_products(dev, dtype, D):
    """The rotation of rows to the last bit: of each sum one product is rounded by itself and the other fused, which of them is part of the result (a
    16-bit value moves in about one of 50 thousand). Fused sums from 64 bits: a product of 24 bits each is exact there."""
    from tesseract_b200 import _native, ops
    g = torch.Generator(device=dev).manual_seed(D)
    T, n = 20000, 4
    cos, sin = ops.rope_tables(4096, D, 1e4, dev)
    pos = torch.randint(0, 4096, (T,), device=dev, generator=g, dtype=torch.int32)
    x = torch.randn(T, n * D, device=dev, generator=g).to(dtype)
    got = ops.rope_qkv(x.clone(), cos, sin, num_heads=n - 2, num_kv_heads=1, head_dim=D, seq_len=1, positions=pos).view(T, n, -1, 4, 2)[:, :n - 1]
    a, b = x.view(T, n, -1, 4, 2)[:, :n - 1].float().unbind(-1)
    c, s = (t[pos.long()].view(T, 1, -1, 4) for t in (cos, sin))
    fma = lambda p, q, r: (p.double() * q.double() + r.double()).float().to(dtype)
    second = fma(b, c, a * s)
    assert torch.equal(got[..., 0], fma(a, c, -(b * s)))
    if dtype != torch.float32:
        second[..., 1:] = fma(a, s, b * c)[..., 1:]
    assert torch.equal(got[..., 1], second)
    if dtype != torch.float32 and D != 72:                       # the append of a decode step: each pair like the first one there
        y, k = x.clone(), torch.zeros(T, 1, 1, D, device=dev, dtype=dtype)
        v, slots = torch.zeros_like(k), torch.arange(T, device=dev, dtype=torch.int32)
        _native.check(_native.lib().tsb_kv_append_paged(y.data_ptr(), cos.data_ptr(), sin.data_ptr(), pos.data_ptr(), slots.data_ptr(), k.data_ptr(),
                                                        v.data_ptr(), None, None, None, T, n - 2, 1, D, 1, _native.dtype_code(dtype), 1,
                                                        _native.stream_ptr(x.device)), "append")
        pairs = torch.cat([y.view(T, n, D)[:, :n - 2], k.view(T, 1, D)], 1).view(T, n - 1, -1, 4, 2)
        assert torch.equal(pairs[..., 0], fma(a, c, -(b * s))) and torch.equal(pairs[..., 1], fma(b, c, a * s))


@pytest.mark.parametrize("size", [32, 4096, 148 * 32 * 256 * 32 + 32, 1 << 30])
def test_zeroes(dev, size):
    from tesseract_b200 import _native
    x = torch.full((size + 64,), 7, dtype=torch.uint8, device=dev)
    _native.check(_native.lib().tsb_zero(x[32:].data_ptr(), size, _native.stream_ptr(x.device)), "tsb_zero")
    assert int(x[:32].min()) == 7 and int(x[32 + size:].min()) == 7 and int(x[32:32 + size].max()) == 0
    assert _native.lib().tsb_zero(x[16:].data_ptr(), 32, 0) == -2 and _native.lib().tsb_zero(x.data_ptr(), 33, 0) == -2


@pytest.mark.parametrize("H,Hkv", [(4, 2), (3, 3), (6, 2)])       # two heads of a group per CTA; two tiles of a head
@pytest.mark.parametrize("Sq,Sk", [(1, 1), (1, 300), (127, 127), (128, 128), (129, 640), (257, 257), (300, 200)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B", [2, 80])                            # a tile per CTA while that fills one round of them; pairs of tiles
def test_flash_forward_tile_pairs(dev, H, Hkv, Sq, Sk, D, B):
    """Ends of tiles and of pairs of tiles, rows without a visible key. P and the output are rounded to bf16 (each 2^-9 / sqrt 3
    of a value in the mean), so the error of a row is about 0.0017 of it; 0.005 leaves three times that."""
    from tesseract_b200 import ops
    g = torch.Generator(device=dev).manual_seed(Sq + Sk + D)
    q = torch.randn(B, Sq, H, D, device=dev, generator=g).bfloat16()
    k, v = (torch.randn(B, Sk, Hkv, D, device=dev, generator=g).bfloat16() for _ in range(2))
    for causal in (True, False):
        with torch.no_grad():
            o = ops.flash_attention(q, k, v, causal=causal)
        torch.cuda.synchronize()
        _status_ok()
        ref = ops.attention_ref(q.transpose(1, 2).float(), k.transpose(1, 2).float(), v.transpose(1, 2).float(),
                                causal=causal).transpose(1, 2)
        assert _rel_err(o, ref) < 5e-3, causal
        if causal and Sq > Sk:
            assert not o[:, :Sq - Sk].any()


@pytest.mark.parametrize("B,H,Hkv,S,D", [(1, 2, 2, 128, 128), (2, 4, 2, 256, 128), (1, 4, 1, 384, 64),
                                          (2, 8, 2, 1000, 128), (1, 2, 1, 77, 64)])
@pytest.mark.parametrize("causal", [True, False])
def test_flash_attention_forward(dev, B, H, Hkv, S, D, causal):
    from tesseract_b200 import ops
    g = torch.Generator(device=dev).manual_seed(S + D)
    qkv = torch.randn(B, S, H + 2 * Hkv, D, device=dev, generator=g).bfloat16()
    q, k, v = qkv[:, :, :H], qkv[:, :, H:H + Hkv], qkv[:, :, H + Hkv:]
    o = ops.flash_attention(q, k, v, causal=causal)
    torch.cuda.synchronize()
    _status_ok()
    ref = ops.attention_ref(q.transpose(1, 2).float(), k.transpose(1, 2).float(), v.transpose(1, 2).float(),
                            causal=causal).transpose(1, 2)
    assert _rel_err(o, ref) < 1.5e-2, _rel_err(o, ref)


def test_flash_attention_rectangular_causal(dev):
    """Chunked prefill: 128 new queries against 384 keys, last query sees every key."""
    from tesseract_b200 import ops
    q = torch.randn(1, 128, 4, 128, device=dev).bfloat16()
    k = torch.randn(1, 384, 2, 128, device=dev).bfloat16()
    v = torch.randn(1, 384, 2, 128, device=dev).bfloat16()
    o = ops.flash_attention(q, k, v, causal=True)
    ref = ops.attention_ref(q.transpose(1, 2).float(), k.transpose(1, 2).float(), v.transpose(1, 2).float(),
                            causal=True).transpose(1, 2)
    _status_ok()
    assert _rel_err(o, ref) < 1.5e-2


@pytest.mark.parametrize("B,H,Hkv,S,D", [(1, 2, 2, 128, 128), (2, 4, 2, 256, 128), (1, 4, 1, 384, 64),
                                          (1, 8, 2, 600, 128)])
@pytest.mark.parametrize("causal", [True, False])
def test_flash_attention_backward(dev, B, H, Hkv, S, D, causal):
    from tesseract_b200 import ops
    g = torch.Generator(device=dev).manual_seed(S * 3 + D)
    qkv = (torch.randn(B, S, H + 2 * Hkv, D, device=dev, generator=g)).bfloat16().requires_grad_()
    o = ops.flash_attention_packed(qkv, H, Hkv, causal=causal)
    do = torch.randn(o.shape, device=dev, generator=g).bfloat16()
    o.backward(do)
    torch.cuda.synchronize()
    _status_ok()
    ref_in = qkv.detach().float().requires_grad_()
    q, k, v = ref_in[:, :, :H], ref_in[:, :, H:H + Hkv], ref_in[:, :, H + Hkv:]
    ref = ops.attention_ref(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), causal=causal).transpose(1, 2)
    ref.backward(do.float())
    assert _rel_err(o, ref) < 1.5e-2
    gq, gk, gv = qkv.grad[:, :, :H], qkv.grad[:, :, H:H + Hkv], qkv.grad[:, :, H + Hkv:]
    rq, rk, rv = ref_in.grad[:, :, :H], ref_in.grad[:, :, H:H + Hkv], ref_in.grad[:, :, H + Hkv:]
    assert _rel_err(gv, rv) < 2e-2, ("dv", _rel_err(gv, rv))
    assert _rel_err(gk, rk) < 2e-2, ("dk", _rel_err(gk, rk))
    assert _rel_err(gq, rq) < 2e-2, ("dq", _rel_err(gq, rq))


@pytest.mark.parametrize("H,Hkv", [(4, 2), (3, 3), (8, 1)])
@pytest.mark.parametrize("Sq,Sk", [(31, 31), (129, 129), (100, 300), (257, 640), (300, 200), (129, 1)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("width", [1.0, 3.0])
def test_flash_backward_tile_edges(dev, H, Hkv, Sq, Sk, D, width):
    """Parts of tiles, more keys than queries, rows without a visible key, scores of unit width and as wide as in trained models. P, dS
    and a gradient are rounded to bf16 (each 2^-9 / sqrt 3 of a value in the mean): about 0.002 of a row; 0.006 leaves three times that."""
    from tesseract_b200 import ops
    g = torch.Generator(device=dev).manual_seed(Sq + Sk + D)
    q = (torch.randn(2, Sq, H, D, device=dev, generator=g) * width).bfloat16().requires_grad_()
    k, v = (torch.randn(2, Sk, Hkv, D, device=dev, generator=g).bfloat16().requires_grad_() for _ in range(2))
    do = torch.randn(2, Sq, H, D, device=dev, generator=g).bfloat16()
    for causal in (True, False):
        blind = max(0, Sq - Sk) if causal else 0                   # rows that see no key
        got = torch.autograd.grad(ops.flash_attention(q, k, v, causal=causal), (q, k, v), do)
        torch.cuda.synchronize()
        _status_ok()
        rq, rk, rv = (t.detach().float().requires_grad_() for t in (q[:, blind:], k, v))
        ref = ops.attention_ref(rq.transpose(1, 2), rk.transpose(1, 2), rv.transpose(1, 2), causal=causal).transpose(1, 2)
        want = torch.autograd.grad(ref, (rq, rk, rv), do[:, blind:].float())
        assert not got[0][:, :blind].any()
        for name, a, b in zip("qkv", (got[0][:, blind:], *got[1:]), want):
            if Sk > 1 or name == "v":                              # (a single key: dQ and dK are 0 but for rounding)
                assert _rel_err(a, b) < 6e-3, (name, causal)


@pytest.mark.parametrize("H,Hkv,Sq", [(2, 1, 65535 * 128 + 20), (1, 1, 65535 * 256 + 20)])
def test_flash_forward_more_tiles_than_a_short_grid_axis(dev, H, Hkv, Sq):
    """More query tiles than the y axis of a grid takes. Rows at both ends: 0.0017 of a row, as for the tiles' edges below."""
    from tesseract_b200 import ops
    g = torch.Generator(device=dev).manual_seed(3)
    q = torch.randn(1, Sq, H, 64, device=dev, generator=g, dtype=torch.bfloat16)
    k, v = (torch.randn(1, 48, Hkv, 64, device=dev, generator=g, dtype=torch.bfloat16) for _ in range(2))
    with torch.no_grad():
        o = ops.flash_attention(q, k, v, causal=False)
    torch.cuda.synchronize()
    _status_ok()
    for rows in (slice(0, 300), slice(Sq - 300, Sq)):
        ref = ops.attention_ref(q[:, rows].transpose(1, 2).float(), k.transpose(1, 2).float(), v.transpose(1, 2).float(), causal=False)
        assert _rel_err(o[:, rows], ref.transpose(1, 2)) < 5e-3


def test_flash_backward_more_tiles_than_a_short_grid_axis(dev):
    """More key tiles than the y axis of a grid takes, a tile's part of queries. Gradients as above: about 0.002 of a row."""
    from tesseract_b200 import ops
    Sq, Sk = 16, 65535 * 128 + 20
    g = torch.Generator(device=dev).manual_seed(4)
    q = torch.randn(1, Sq, 1, 64, device=dev, generator=g, dtype=torch.bfloat16).requires_grad_()
    k, v = (torch.randn(1, Sk, 1, 64, device=dev, generator=g, dtype=torch.bfloat16).requires_grad_() for _ in range(2))
    do = torch.randn(1, Sq, 1, 64, device=dev, generator=g, dtype=torch.bfloat16)
    got = torch.autograd.grad(ops.flash_attention(q, k, v, causal=False), (q, k, v), do)
    torch.cuda.synchronize()
    _status_ok()
    qf, kf, vf, df = (t.detach()[0, :, 0].float() for t in (q, k, v, do))
    p = torch.softmax(qf @ kf.t() / 8.0, -1)
    dp = df @ vf.t()
    ds = p * (dp - (p * dp).sum(1, keepdim=True)) / 8.0
    for name, a, b in zip("qkv", got, (ds @ kf, ds.t() @ qf, p.t() @ df)):
        for rows in (slice(0, 300), slice(-300, None)):
            assert _rel_err(a[0, rows, 0], b[rows]) < 6e-3, name


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("shift", [1, 2, 4])
def test_flash_backward_takes_an_output_at_any_address(dev, D, shift):
    """A saved output that a hook brings back somewhere else, not aligned to 16 bytes: the same dK and dV to the last bit."""
    from tesseract_b200 import ops
    g = torch.Generator(device=dev).manual_seed(D)
    q, k, v, do = (torch.randn(2, 200, 4, D, device=dev, generator=g).bfloat16() for _ in range(4))
    q, k, v = (t.requires_grad_() for t in (q, k, v))
    want = torch.autograd.grad(ops.flash_attention(q, k, v, causal=True), (q, k, v), do)
    moved = []

    def elsewhere(t):
        if t.data_ptr() != o.data_ptr():
            return t
        moved.append(torch.empty(t.numel() + shift, device=dev, dtype=t.dtype)[shift:].view_as(t).copy_(t))
        return moved[-1]

    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.detach(), elsewhere):
        o = ops.flash_attention(q, k, v, causal=True)
    got = torch.autograd.grad(o, (q, k, v), do)
    torch.cuda.synchronize()
    _status_ok()
    assert len(moved) == 1 and moved[0].data_ptr() % 16
    assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
    assert _rel_err(got[0], want[0].float()) < 1e-3                # (dQ is summed by atomics: a last bit of bf16 here and there)


def _make_paged(dev, A, Hkv, D, bs, lens, dtype, int8):
    from tesseract_b200.nn.kv_cache import quantize_kv_per_token
    nb = sum((l + bs - 1) // bs for l in lens) + 3
    perm = torch.randperm(nb)
    k_pool = torch.zeros(nb, Hkv, bs, D, device=dev, dtype=dtype)
    v_pool = torch.zeros_like(k_pool)
    max_blocks = max((l + bs - 1) // bs for l in lens)
    tables = torch.zeros(A, max_blocks, dtype=torch.int32)
    nxt = 0
    for a, l in enumerate(lens):
        n = (l + bs - 1) // bs
        tables[a, :n] = perm[nxt:nxt + n].to(torch.int32)
        nxt += n
        k = torch.randn(Hkv, n * bs, D, device=dev).to(dtype)
        v = torch.randn(Hkv, n * bs, D, device=dev).to(dtype)
        for i in range(n):
            k_pool[tables[a, i]] = k[:, i * bs:(i + 1) * bs]
            v_pool[tables[a, i]] = v[:, i * bs:(i + 1) * bs]
    ks = vs = None
    if int8:
        k_pool, ks = quantize_kv_per_token(k_pool)
        v_pool, vs = quantize_kv_per_token(v_pool)
    return k_pool, v_pool, ks, vs, tables.to(dev), torch.tensor(lens, dtype=torch.int32, device=dev)


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("A,H,Hkv,D,bs,lens", [(3, 8, 2, 128, 16, [37, 500, 1]), (2, 4, 4, 64, 16, [100, 33]),
                                                 (5, 4, 1, 128, 16, [2000, 17, 256, 1024, 999]),
                                                 (1, 16, 2, 128, 32, [4096])])
def test_paged_decode_attention(dev, A, H, Hkv, D, bs, lens, int8):
    from tesseract_b200 import ops
    k_pool, v_pool, ks, vs, tables, lens_t = _make_paged(dev, A, Hkv, D, bs, lens, torch.bfloat16, int8)
    q = torch.randn(A, H, D, device=dev).bfloat16()
    got = ops.paged_decode_attention(q, k_pool, v_pool, tables, lens_t, None, ks, vs)
    torch.cuda.synchronize()
    _status_ok()
    ref = ops.paged_attention_ref(q.float().unsqueeze(1), k_pool, v_pool, tables, lens_t, None, ks, vs).squeeze(1)
    assert (got.float() - ref).abs().max() < 3e-3 * max(1.0, ref.abs().max().item()) + 2e-2, (got.float() - ref).abs().max()


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("A,S,H,Hkv,D,lens", [(3, 24, 8, 2, 128, [37, 500, 24]), (2, 7, 4, 4, 64, [100, 33]),
                                                (1, 200, 8, 1, 128, [1000]), (2, 16, 4, 2, 128, [40, 9])])
def test_paged_prefill_attention_reads_the_pool_in_place(dev, A, S, H, Hkv, D, lens, int8):
    """Chunked prefill over paged keys (the S new tokens already appended): every new token runs as a decode query
    with its own causal length, on the kernel that reads the pool (INT8 included) in place. The last case has a
    request shorter than the chunk: its leading rows see no key and return zeros, as in the reference formulation."""
    from tesseract_b200 import _native, ops
    k_pool, v_pool, ks, vs, tables, lens_t = _make_paged(dev, A, Hkv, D, 16, lens, torch.bfloat16, int8)
    q = torch.randn(A, S, H, D, device=dev).bfloat16()
    before = _native.launch_count()
    got = ops.paged_prefill_attention(q, k_pool, v_pool, tables, lens_t, None, ks, vs)
    torch.cuda.synchronize()
    _status_ok()
    assert _native.launch_count() > before                         # the native kernel ran, not the gathered fallback
    ref = ops.paged_attention_ref(q.float(), k_pool, v_pool, tables, lens_t, None, ks, vs)
    assert got.shape == ref.shape
    assert (got.float() - ref).abs().max() < 3e-3 * max(1.0, ref.abs().max().item()) + 2e-2, (got.float() - ref).abs().max()


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("A,H,Hkv,D,lens", [(3, 8, 2, 128, [37, 500, 1]), (5, 4, 1, 128, [2000, 17, 256, 1024, 999]),
                                              (2, 4, 4, 64, [100, 33]), (130, 8, 2, 128, [300] * 130)])
def test_paged_decode_attention_mx_operand(dev, A, H, Hkv, D, lens, int8):
    """The attention output leaving as the quantised operand of the output projection (the split merge writes E4M3
    bytes and scale words itself) is bit-identical to the stand-alone quantiser applied to the bf16 attention output."""
    from tesseract_b200 import ops
    from tesseract_b200.ops import fp8
    k_pool, v_pool, ks, vs, tables, lens_t = _make_paged(dev, A, Hkv, D, 16, lens, torch.bfloat16, int8)
    q = torch.randn(A, H, D, device=dev).bfloat16()
    o = ops.paged_decode_attention(q, k_pool, v_pool, tables, lens_t, None, ks, vs)
    want_q, want_sf = fp8.quantize_act_mx(o.view(A, H * D))
    got_q, got_sf = ops.paged_decode_attention_mx(q, k_pool, v_pool, tables, lens_t, None, ks, vs)
    torch.cuda.synchronize()
    _status_ok()
    assert torch.equal(got_q, want_q)
    assert torch.equal(got_sf[:, :A], want_sf[:, :A])


@pytest.mark.parametrize("world,V,rows", [(2, 2048, 5), (8, 128256, 33), (4, 1000, 1)])
def test_vocab_parallel_argmax_candidates(dev, world, V, rows):
    """The two kernels of the vocabulary-parallel arg-max with the ranks emulated on one GPU: every rank packs the
    candidate of its shard, the packed rows are summed in bf16 (what the all-reduce does), the unpack kernel returns
    the global arg-max -- ties included (lowest index wins)."""
    from tesseract_b200.serving.engine import argmax_rows, argmax_rows_pack, argmax_rows_unpack, vocab_shard_rows
    shard = vocab_shard_rows(V, world)
    assert shard % 128 == 0 and (world - 1) * shard < V <= world * shard
    logits = torch.randn(rows, V, device=dev).bfloat16()
    logits[0, 7] = logits[0, V - 3] = 50.0                      # a tie across the first and the last shard
    if rows > 2:
        logits[2, V - 1] = 60.0                                 # the winner is the very last column
    total = torch.zeros(rows, 4 * world, device=dev, dtype=torch.float32)
    for r in range(world):
        local = logits[:, r * shard:min(V, (r + 1) * shard)].contiguous()
        packed = torch.full((rows, 4 * world), 7.0, device=dev, dtype=torch.bfloat16)
        argmax_rows_pack(local, packed, r, world)
        total += packed.float()
    got = argmax_rows_unpack(total.bfloat16(), world, shard)
    torch.cuda.synchronize()
    want = argmax_rows(logits)
    assert torch.equal(got, want) and got[0].item() == 7
    assert torch.equal(logits.gather(1, got.long()[:, None])[:, 0], logits.max(dim=-1).values)


def test_out_of_range_indices_are_redirected_and_reported(dev):
    """Data-dependent indices are checked in the kernels: a token id outside the vocabulary reads row 0, a block-table
    entry outside the pool reads block 0 (never memory outside the tensor), the rows that had valid indices are
    unaffected, and the status word tells the host (code 4)."""
    from tesseract_b200 import _native, ops
    stream = torch.cuda.current_stream().cuda_stream
    assert _native.read_status(stream) == 0
    V, D = 64, 128
    table = torch.randn(V, D, device=dev).bfloat16()
    ids = torch.tensor([[3, V + 5, 7, -2]], device=dev)
    out = ops.embedding(ids, table)
    torch.cuda.synchronize()
    assert torch.equal(out[0, 0], table[3]) and torch.equal(out[0, 2], table[7])
    assert torch.equal(out[0, 1], table[0]) and torch.equal(out[0, 3], table[0])
    assert _native.read_status(stream) == 4                              # reading clears it
    assert _native.read_status(stream) == 0
    A, H, Hkv, Dh, bs = 3, 8, 2, 128, 16
    lens = [40, 100, 17]
    k_pool, v_pool, _, _, tables, lens_t = _make_paged(dev, A, Hkv, Dh, bs, lens, torch.bfloat16, False)
    q = torch.randn(A, H, Dh, device=dev).bfloat16()
    good = ops.paged_decode_attention(q, k_pool, v_pool, tables, lens_t)
    bad_tables = tables.clone()
    bad_tables[1, 2] = k_pool.shape[0] + 7                                # a block that does not exist
    got = ops.paged_decode_attention(q, k_pool, v_pool, bad_tables, lens_t)
    torch.cuda.synchronize()
    assert _native.read_status(stream) == 4
    assert torch.isfinite(got.float()).all() and torch.equal(got[0], good[0]) and torch.equal(got[2], good[2])
    again = ops.paged_decode_attention(q, k_pool, v_pool, tables, lens_t)  # the context is intact
    torch.cuda.synchronize()
    assert torch.equal(again, good) and _native.read_status(stream) == 0


@pytest.mark.parametrize("int8", [False, True])
def test_kv_append_paged_rope_and_quant(dev, int8):
    from tesseract_b200 import _native, ops
    from tesseract_b200.nn.kv_cache import quantize_kv_per_token
    T, H, Hkv, D, bs, nb = 37, 4, 2, 128, 16, 8
    cos, sin = ops.rope_tables(256, D, 10000.0, dev)
    qkv = torch.randn(T, (H + 2 * Hkv) * D, device=dev).bfloat16()
    positions = torch.randint(0, 200, (T,), device=dev, dtype=torch.int32)
    slots = torch.randperm(nb * bs, device=dev)[:T].to(torch.int32)
    if int8:
        k_pool = torch.zeros(nb, Hkv, bs, D, device=dev, dtype=torch.int8)
        k_scale = torch.ones(nb, Hkv, bs, device=dev)
        v_scale = torch.ones_like(k_scale)
    else:
        k_pool = torch.zeros(nb, Hkv, bs, D, device=dev, dtype=torch.bfloat16)
        k_scale = v_scale = None
    v_pool = torch.zeros_like(k_pool)
    q_out = torch.empty(T, H, D, device=dev, dtype=torch.bfloat16)
    work = qkv.clone()
    _native.check(_native.lib().tsb_kv_append_paged(
        work.data_ptr(), cos.data_ptr(), sin.data_ptr(), positions.data_ptr(), slots.data_ptr(), k_pool.data_ptr(),
        v_pool.data_ptr(), k_scale.data_ptr() if int8 else None, v_scale.data_ptr() if int8 else None, q_out.data_ptr(),
        T, H, Hkv, D, bs, 1, 1, _native.stream_ptr(dev)), "tsb_kv_append_paged")
    torch.cuda.synchronize()
    x = qkv.float().view(T, H + 2 * Hkv, D)
    rot = ops.rope_ref(x[:, :H + Hkv], cos, sin, positions.long())
    assert _rel_err(q_out, rot[:, :H]) < 1e-2
    k_ref = rot[:, H:].bfloat16().float()
    v_ref = x[:, H + Hkv:]
    blk, off = (slots // bs).long(), (slots % bs).long()
    if int8:
        kq, ksr = quantize_kv_per_token(k_ref)
        got_k = k_pool[blk, :, off].float() * k_scale[blk, :, off][..., None]
        got_v = v_pool[blk, :, off].float() * v_scale[blk, :, off][..., None]
        assert (got_k - k_ref).abs().max() <= ksr.max() * 1.01 + 1e-3
        assert (got_v - v_ref).abs().max() <= v_scale.max() * 1.01 + 1e-3
    else:
        assert _rel_err(k_pool[blk, :, off], k_ref) < 1e-2
        assert torch.equal(v_pool[blk, :, off], qkv.view(T, H + 2 * Hkv, D)[:, H + Hkv:])


def test_device_sampling_kernels(dev):
    from tesseract_b200.serving import argmax_rows, sample_top_p_rows
    logits = torch.randn(37, 5000, device=dev).bfloat16()
    logits[3, 100] = logits[3, 4000] = 50.0
    got = argmax_rows(logits)
    ref = logits.float().argmax(-1)
    assert int(got[3]) == 100
    assert torch.equal(got.long(), ref) or (got.long() != ref).sum() <= 1
    for V in (5003, 128256, 7):                    # scalar tail / unaligned rows, the Llama-3 vocabulary, tiny
        lg = torch.randn(9, V, device=dev).bfloat16()
        lg[2, V - 1] = 60.0                         # the maximum sits in the tail
        lg[4, 0] = lg[4, V // 2] = 55.0             # ties resolve to the lowest index
        got2 = argmax_rows(lg)
        assert int(got2[2]) == V - 1 and int(got2[4]) == 0
        vals = lg.float().gather(1, got2.long().view(-1, 1)).view(-1)
        assert torch.equal(vals, lg.float().max(-1).values)
    peaked = torch.full((8, 1000), -10.0, device=dev).bfloat16()
    peaked[:, 7] = 5.0
    peaked[:, 9] = 4.5
    picks = torch.stack([sample_top_p_rows(peaked, 1.0, 0.9, 123, s) for s in range(40)])
    assert set(picks.unique().tolist()) <= {7, 9} and (picks == 7).float().mean() > 0.4
    a = sample_top_p_rows(logits, 0.8, 0.95, 5, 1)
    b = sample_top_p_rows(logits, 0.8, 0.95, 5, 1)
    assert torch.equal(a, b) and int(a.min()) >= 0 and int(a.max()) < 5000
    # every draw lies inside the smallest nucleus of the fp32 reference (sorted cumulative mass), on a vocabulary of
    # Llama-3 size with a spread of logits that puts thousands of tokens into the nucleus
    big = (torch.randn(12, 128256, device=dev) * 2.0).bfloat16()
    probs = torch.softmax(big.float() / 0.9, dim=-1)
    sp, _ = probs.sort(dim=-1, descending=True)
    first = (sp.cumsum(-1) >= 0.5).float().argmax(-1)                  # index of the element that completes the nucleus
    thr = sp.gather(1, first.view(-1, 1)).view(-1)
    sizes = (probs >= thr.view(-1, 1)).sum(-1)
    assert int(sizes.min()) > 100
    seen = set()
    for s in range(8):
        pick = sample_top_p_rows(big, 0.9, 0.5, 77, s).long()
        p_pick = probs.gather(1, pick.view(-1, 1)).view(-1)
        assert (p_pick >= thr * (1 - 1e-3)).all()
        seen |= set(pick.tolist())
    assert len(seen) > 40                                              # and the draws do move around inside it


def test_device_sampler_top_k_penalty_and_step_counter(dev):
    """Top-k keeps exactly the k largest logits (ties at the k-th value survive), the repetition penalty follows the
    host sampler's per-occurrence rule, and the graph-safe step counter gives the draw of the same explicit step."""
    from tesseract_b200.serving.engine import repetition_penalty_rows_, sample_rows
    g = torch.Generator(device=dev).manual_seed(3)
    V, rows = 4096, 16
    logits = torch.randn(rows, V, device=dev, generator=g).bfloat16()
    # every token whose logit reaches the 5th largest VALUE survives (bf16 logits tie often)
    kth = torch.topk(logits.float(), 5, dim=-1).values[:, -1]
    topk_sets = [set(torch.nonzero(logits[r].float() >= kth[r]).flatten().tolist()) for r in range(rows)]
    assert all(5 <= len(sset) <= 12 for sset in topk_sets)
    for step in range(6):
        out = sample_rows(logits, 1.0, 5, 1.0, seed=11, step=step).tolist()
        assert all(t in topk_sets[r] for r, t in enumerate(out))
    assert sample_rows(logits, 1.0, 1, 1.0, seed=1, step=0).tolist() == logits.float().argmax(-1).tolist()
    tied = torch.zeros(1, 64, device=dev, dtype=torch.float32)
    tied[0, [3, 9, 20]] = 5.0                                           # three-way tie at the top, k = 2: all three stay
    seen = {int(sample_rows(tied, 1.0, 2, 1.0, seed=5, step=s)[0]) for s in range(64)}
    assert seen == {3, 9, 20}
    counter = torch.tensor([4], dtype=torch.int64, device=dev)
    a = sample_rows(logits, 0.8, 0, 0.9, seed=2, step=4)
    b = sample_rows(logits, 0.8, 0, 0.9, seed=2, step=0, step_counter=counter)
    assert torch.equal(a, b)
    x = torch.tensor([[2.0, -1.0, 0.5, 4.0]], device=dev)
    hist = torch.tensor([[0, 1, 0, 3, 7]], dtype=torch.int32, device=dev)   # token 0 twice; 7 is out of range
    repetition_penalty_rows_(x, hist, torch.tensor([4], dtype=torch.int32, device=dev), 2.0)
    assert torch.allclose(x, torch.tensor([[0.5, -2.0, 0.5, 2.0]], device=dev))
    _status_ok()


@pytest.mark.parametrize("kv_int8", [False, True])
def test_serving_engine_graph_vs_eager_and_generate(dev, kv_int8):
    from tesseract_b200.models import GenerateConfig, LlamaConfig, LlamaModel
    from tesseract_b200.models.scheduler import EngineConfig
    from tesseract_b200.serving import ServingEngine
    cfg = LlamaConfig(vocab_size=512, hidden_size=512, num_hidden_layers=2, num_attention_heads=4,
                      num_key_value_heads=2, intermediate_size=1024, max_position_embeddings=256, dtype=torch.bfloat16)
    model = LlamaModel(cfg, device=dev, init_std=0.3, seed=2)
    g = torch.Generator().manual_seed(1)
    prompts = [torch.randint(0, 512, (n,), generator=g).tolist() for n in (5, 37, 64, 9, 130, 17)]
    outs = {}
    for graph in (True, False):
        eng = ServingEngine(model, EngineConfig(block_size=16, num_blocks=64, max_seq_len=256, max_batch_size=4,
                                                kv_int8=kv_int8), use_cuda_graph=graph)
        # every bucket (1, 2, 4) captured up front on padding rows; nothing is captured while requests run
        assert eng.warm_graphs() == (3 if graph else 0)
        ids = [eng.add_request(p, GenerateConfig(max_new_tokens=12)) for p in prompts]
        eng.run()
        assert eng.free_blocks() == 64 and eng.warm_graphs() == 0
        outs[graph] = [eng.result(i) for i in ids]
        m = eng.metrics()
        assert m["requests"] == len(prompts) and m["decode_tok_s"] > 0
    assert outs[True] == outs[False]
    # admitting at most 40 prompt tokens per step changes the schedule, not a request's tokens (bf16 KV: batch
    # composition does not enter a request's arithmetic)
    eng = ServingEngine(model, EngineConfig(block_size=16, num_blocks=64, max_seq_len=256, max_batch_size=4,
                                            kv_int8=kv_int8), use_cuda_graph=False, max_prefill_tokens=40)
    ids = [eng.add_request(p, GenerateConfig(max_new_tokens=12)) for p in prompts]
    eng.run()
    chunked = [eng.result(i) for i in ids]
    assert eng.steps > m["steps"] and all(len(a) == len(b) for a, b in zip(chunked, outs[False]))
    same = sum(int(a == b) for x, y in zip(chunked, outs[False]) for a, b in zip(x, y))
    assert same >= 0.9 * sum(len(x) for x in chunked)
    _status_ok()
    if not kv_int8:
        agree = 0
        for p, got in zip(prompts, outs[True]):
            ref = model.generate(p, GenerateConfig(max_new_tokens=12))
            assert len(got) == len(ref) and got[:len(p)] == p
            agree += sum(int(a == b) for a, b in zip(got[len(p):], ref[len(p):]))
        assert agree >= 0.7 * 12 * len(prompts), agree


def test_serving_engine_fp8_prefill_weights(dev):
    """Opt-in E4M3 weight copies for prefill-sized GEMMs: the projection agrees with bf16 within fp8 error, decode
    sized batches keep the bf16 path, and a run over prompts longer than 512 tokens finishes every request."""
    from tesseract_b200.models import GenerateConfig, LlamaConfig, LlamaModel
    from tesseract_b200.models.scheduler import EngineConfig
    from tesseract_b200.serving import ServingEngine
    cfg = LlamaConfig(vocab_size=512, hidden_size=512, num_hidden_layers=2, num_attention_heads=4,
                      num_key_value_heads=2, intermediate_size=1024, max_position_embeddings=1024, dtype=torch.bfloat16)
    model = LlamaModel(cfg, device=dev, init_std=0.05, seed=2)
    ecfg = EngineConfig(block_size=16, num_blocks=256, max_seq_len=1024, max_batch_size=4)
    eng = ServingEngine(model, ecfg, use_cuda_graph=False, fp8_prefill=True)
    assert len(eng._w8) == 4 * cfg.num_hidden_layers
    x = (torch.randn(1024, 512, device=dev, generator=torch.Generator(device=dev).manual_seed(0))).bfloat16()
    for w in (eng.wqkv[0], eng.wgu[1]):
        got, ref = eng._mm(x, w).float(), x.float() @ w.w.float().t()
        assert _rel_err(got, ref) < 0.06
        small = eng._mm(x[:64], w).float()                       # decode-sized: bf16 path, tight agreement
        assert _rel_err(small, ref[:64]) < 1e-2
    g = torch.Generator().manual_seed(1)
    prompts = [torch.randint(0, 512, (n,), generator=g).tolist() for n in (700, 40, 300)]
    ids = [eng.add_request(p, GenerateConfig(max_new_tokens=8)) for p in prompts]
    eng.run()
    outs = [eng.result(i) for i in ids]
    assert [len(o) for o in outs] == [len(p) + 8 for p in prompts] and eng.free_blocks() == 256
    assert all(0 <= t < 512 for o in outs for t in o)
    _status_ok()


@pytest.mark.parametrize("kv_int8", [False, True])
def test_serving_engine_fp8_block_scaled_weights(dev, kv_int8):
    """weights="fp8": every projection and the LM head are held as E4M3 with 128 x 128 block scales. The engine's
    products agree with the dequantised weights (decode-sized batches quantise the activations to E4M3 with one
    power-of-two scale per 32 columns and run on the tensor core's block scaling, prompt-sized ones quantise them
    1 x 128), greedy decoding mostly agrees with the bf16 engine, top-p sampling runs inside the CUDA
    graph and is reproducible from the seed."""
    from tesseract_b200.models import GenerateConfig, LlamaConfig, LlamaModel
    from tesseract_b200.models.scheduler import EngineConfig
    from tesseract_b200.ops.gemm import _dequant_block128
    from tesseract_b200.serving import ServingEngine
    cfg = LlamaConfig(vocab_size=512, hidden_size=512, num_hidden_layers=2, num_attention_heads=4,
                      num_key_value_heads=2, intermediate_size=1024, max_position_embeddings=512, dtype=torch.bfloat16)
    ecfg = EngineConfig(block_size=16, num_blocks=256, max_seq_len=512, max_batch_size=8, kv_int8=kv_int8)
    prompts = [[(11 * i + j) % 512 for j in range(30 + 7 * i)] for i in range(5)]

    def run(weights, **kw):
        eng = ServingEngine(LlamaModel(cfg, device=dev, init_std=0.05, seed=4), ecfg, weights=weights, **kw)
        ids = [eng.add_request(p, GenerateConfig(max_new_tokens=10)) for p in prompts]
        eng.run()
        return eng, [eng.result(i)[len(p):] for i, p in zip(ids, prompts)]

    ref_model = LlamaModel(cfg, device=dev, init_std=0.05, seed=4)
    eng8, out8 = run("fp8")
    assert eng8.wqkv[0].q is not None and eng8.w_head.q is not None and eng8.wqkv[0].w is None
    assert eng8.weight_bytes() < 0.56 * sum(p.numel() * 2 for n, p in ref_model.named_parameters()
                                            if "proj" in n or "lm_head" in n)
    x = torch.randn(600, 512, device=dev, generator=torch.Generator(device=dev).manual_seed(0)).bfloat16()
    W = eng8.wgu[1]
    ref = x.float() @ _dequant_block128(W.q, W.s).t()
    assert _rel_err(eng8._mm(x[:48], W).float(), ref[:48]) < 0.05           # fp8 x fp8 block-scaled GEMM (1 x 128 scales)
    assert _rel_err(eng8._mm(x, W).float(), ref) < 0.05
    Wd = eng8.wdown[1]
    assert Wd.pow2                                                           # decode-sized: E4M3 activations, MX scales
    xd = torch.randn(48, Wd.shape[1], device=dev, generator=torch.Generator(device=dev).manual_seed(1)).bfloat16()
    refd = xd.float() @ _dequant_block128(Wd.q, Wd.s).t()
    assert _rel_err(eng8._mm(xd, Wd).float(), refd) < 0.04
    eng8.decode_gemm = "stream"                                              # A/B switch: bf16 activations, weights widened
    assert _rel_err(eng8._mm(xd, Wd).float(), refd) < 1.2e-2
    eng8.decode_gemm = "auto"
    _, out16 = run("bf16")
    same = sum(a == b for x8, x16 in zip(out8, out16) for a, b in zip(x8, x16))
    assert all(len(o) == 10 for o in out8)
    # a random-weight model has near-tied logits, so greedy paths drift apart once one token differs: most first
    # tokens agree, and a fair share of the rest
    assert sum(a[0] == b[0] for a, b in zip(out8, out16)) >= 3 and same / 50 > 0.2
    # sampled decoding inside the captured graph: same seed, same tokens; another seed, other tokens
    _, s1 = run("fp8", temperature=1.0, top_p=0.9, seed=7)
    _, s2 = run("fp8", temperature=1.0, top_p=0.9, seed=7)
    _, s3 = run("fp8", temperature=1.0, top_p=0.9, top_k=40, seed=8)
    assert s1 == s2 and s1 != s3
    assert all(0 <= t < 512 for o in s3 for t in o)
    _status_ok()


@pytest.mark.parametrize("M,N,K", [(1, 4096, 4096), (64, 6144, 4096), (256, 4096, 14336), (37, 1000, 520)])
def test_decode_linear_split_k(dev, M, N, K):
    from tesseract_b200 import ops
    x = torch.randn(M, K, device=dev).bfloat16()
    w = (torch.randn(N, K, device=dev) * 0.05).bfloat16()
    got = ops.decode_linear(x, w)
    torch.cuda.synchronize()
    _status_ok()
    assert _rel_err(got, x.float() @ w.float().t()) < 8e-3


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("M,N,K,bn,split", [(1, 4096, 4096, 0, 0), (64, 6144, 4096, 0, 0), (128, 4096, 14336, 0, 0),
                                            (141, 1536, 4096, 0, 0), (37, 1000, 576, 48, 2), (256, 768, 4096, 0, 0),
                                            (16, 300, 128, 112, 1), (96, 28672, 4096, 0, 0), (8, 520, 1024, 256, 8)])
def test_stream_linear_bf16_and_fp8_block_scaled(dev, M, N, K, bn, split, fp8):
    """The weight-streaming decode GEMM against an fp32 product of the same (dequantised) operands; ragged N, M
    beyond one row block, every cluster split, and the programmatic-launch flag."""
    from tesseract_b200 import ops
    from tesseract_b200.ops import fp8 as f8
    from tesseract_b200.ops.gemm import _dequant_block128, stream_linear
    g = torch.Generator(device=dev).manual_seed(M * 7 + N)
    x = torch.randn(M, K, device=dev, generator=g).bfloat16()
    w = (torch.randn(N, K, device=dev, generator=g) * 0.05).bfloat16()
    if fp8:
        if K % 128:
            pytest.skip("block scales need K % 128 == 0")
        q, sc = f8.quantize_weight(w)
        want = x.float() @ _dequant_block128(q, sc).t()
        got = stream_linear(x, q, sc, bn=bn, split=split)
        got_pdl = stream_linear(x, q, sc, bn=bn, split=split, pdl=True)
        # the same weights packed tile-major (every tile one contiguous run): bit-identical result
        from tesseract_b200.ops.gemm import pack_fp8_weight, stream_linear_plan
        pbn = bn if bn else stream_linear_plan(M, N, K, True)[0]
        got_packed = stream_linear(x, pack_fp8_weight(q, pbn), sc, bn=pbn, split=split, packed_n=N)
        assert torch.equal(got_packed, stream_linear(x, q, sc, bn=pbn, split=split))
        # and the quantisation itself is the usual E4M3 error against the bf16 weights
        full = x.float() @ w.float().t()
        assert ((want - full).norm() / full.norm()).item() < 0.05
    else:
        want = x.float() @ w.float().t()
        got = stream_linear(x, w, bn=bn, split=split)
        got_pdl = stream_linear(x, w, bn=bn, split=split, pdl=True)
    torch.cuda.synchronize()
    assert got.shape == (M, N)
    err = ((got.float() - want).norm() / want.norm()).item()
    assert err < (1.2e-2 if fp8 else 6e-3), err
    assert (got.float() - want).abs().max().item() < 0.05 * want.abs().max().item() + 0.05
    assert torch.equal(got, got_pdl)
    # the result lands in a caller's (strided) buffer as well
    buf = torch.zeros(M, N + 8, device=dev, dtype=torch.bfloat16)
    stream_linear(x, q if fp8 else w, sc if fp8 else None, out=buf[:, :N], bn=bn, split=split)
    assert torch.equal(buf[:, :N], got) and float(buf[:, N:].abs().max()) == 0.0
    from tesseract_b200 import _native
    assert _native.read_status(torch.cuda.current_stream().cuda_stream) == 0


@pytest.mark.parametrize("M,K", [(5, 256), (130, 4096), (256, 1024)])
def test_quantize_act_mx_matches_the_torch_restatement(dev, M, K):
    """The activation quantiser of the MX path: E4M3 payload and UE8M0 exponent words equal to the torch restatement
    (powers of two make the scaling exact, so the bytes must agree), and the round trip stays within E4M3 precision."""
    from tesseract_b200.ops import fp8 as f8
    g = torch.Generator(device=dev).manual_seed(M + K)
    x = (torch.randn(M, K, device=dev, generator=g) * torch.exp(torch.randn(M, 1, device=dev, generator=g) * 2)).bfloat16()
    x[0, :64] = 0                                                          # two all-zero blocks
    q, sf = f8.quantize_act_mx(x)
    q_ref, sf_ref = f8.quantize_act_mx_ref(x)
    assert torch.equal(sf, sf_ref)
    assert torch.equal(q, q_ref)
    q_a, sf_a = f8.quantize_act_mx(x, atoms=True)                         # the same words laid out as 512-byte atoms
    assert torch.equal(q_a, q) and torch.equal(f8._atoms_to_words(sf_a), sf) and torch.equal(sf_a, f8._words_to_atoms(sf))
    back = f8.dequantize_act_mx(q, sf)
    # three mantissa bits for normal values; values far below their block's maximum land on the subnormal grid
    amax = x.float().abs().view(M, K // 32, 32).amax(dim=2, keepdim=True).expand(M, K // 32, 32).reshape(M, K)
    assert ((back - x.float()).abs() <= x.float().abs() * 2 ** -4 + amax * 2 ** -16).all()


@pytest.mark.parametrize("M,N,K,bn,split", [(16, 4096, 4096, 0, 0), (141, 6144, 4096, 0, 0), (64, 28672, 4096, 0, 0),
                                            (128, 4096, 14336, 0, 0), (8, 200, 256, 0, 0), (300, 1024, 1024, 0, 0),
                                            (37, 1000, 512, 48, 2), (256, 768, 4096, 0, 0), (24, 520, 1024, 240, 8),
                                            (200, 4096, 4096, 208, 4), (1, 4096, 4096, 128, 1),
                                            (1000, 1000, 512, 0, 0), (4096, 4096, 4096, 0, 0), (257, 96, 256, 0, 0),
                                            (2048, 14336, 1024, 0, 0), (640, 200, 384, 0, 0)])
def test_mx_linear_block_scaled_fp8_on_the_tensor_core(dev, M, N, K, bn, split):
    """tcgen05.mma kind::mxf8f6f4.block_scale GEMMs (the weight-streaming kernel up to 256 rows, the persistent
    tiled kernel above) against an fp32 product of the same dequantised operands.
    The operands are drawn directly in their quantised form with a different exponent for every (row, 32-column) block
    of the activations and every 128 x 128 block of the weights, so that a scale that reaches the wrong row, column
    block or byte shows up as an error of a factor of two or more."""
    from tesseract_b200 import _native
    from tesseract_b200.ops import fp8 as f8
    g = torch.Generator(device=dev).manual_seed(M * 11 + N + K)

    def payload(rows, cols):
        b = torch.randint(0, 256, (rows, cols), device=dev, generator=g, dtype=torch.int32)
        b = torch.where((b & 0x7F) == 0x7F, b & 0x80 | 0x30, b)           # no NaN encodings
        return b.to(torch.uint8)

    q = payload(M, K)
    ea = torch.randint(120, 131, (M, K // 32), device=dev, generator=g, dtype=torch.int64).view(M, K // 128, 4)
    words = ea[:, :, 0] | (ea[:, :, 1] << 8) | (ea[:, :, 2] << 16) | (ea[:, :, 3] << 24)
    sf = torch.full((K // 128, (M + 127) // 128 * 128), 0x7F7F7F7F, dtype=torch.int64, device=dev)
    sf[:, :M] = words.t()
    sf = sf.to(torch.int32)
    wq = payload(N, K)
    ws = torch.exp2(torch.randint(-12, -4, ((N + 127) // 128, K // 128), device=dev, generator=g).float())
    want = f8.dequantize_act_mx(q, sf) @ f8.dequantize_weight(wq, ws).t()
    if M > 256:                                                          # the persistent tiled kernel takes scale atoms
        sf = f8._words_to_atoms(sf)
    got = f8.mx_linear(q, sf, wq, ws, bn=bn, split=split)
    got_pdl = f8.mx_linear(q, sf, wq, ws, bn=bn, split=split, pdl=True)
    torch.cuda.synchronize()
    assert got.shape == (M, N)
    err = ((got.float() - want).norm() / want.norm()).item()
    assert err < 4e-3, err                                                 # bf16 rounding of the result only
    assert (got.float() - want).abs().max().item() < 0.01 * want.abs().max().item()
    assert torch.equal(got, got_pdl)
    buf = torch.zeros(M, N + 8, device=dev, dtype=torch.bfloat16)
    f8.mx_linear(q, sf, wq, ws, out=buf[:, :N], bn=bn, split=split)
    assert torch.equal(buf[:, :N], got) and float(buf[:, N:].abs().max()) == 0.0
    assert _native.read_status(torch.cuda.current_stream().cuda_stream) == 0


def test_mx_fused_producers_match_their_two_kernel_forms(dev):
    """RMSNorm (+ residual) and SwiGLU that write the quantised GEMM operand directly: the dequantised result equals
    that of the stand-alone kernel followed by the quantiser (up to a bf16 rounding that falls the other way in a
    handful of places: the row sum is added up in a different order), the residual output is the same."""
    from tesseract_b200 import ops
    from tesseract_b200.ops import fp8 as f8
    g = torch.Generator(device=dev).manual_seed(9)
    for M, D in [(7, 4096), (130, 4096), (33, 1024)]:
        x = torch.randn(M, D, device=dev, generator=g).bfloat16()
        r = torch.randn(M, D, device=dev, generator=g).bfloat16()
        w = (1 + 0.1 * torch.randn(D, device=dev, generator=g)).bfloat16()
        for res in (None, r):
            q, sf, h = f8.rms_norm_quant_mx(x, w, 1e-5, residual=res)
            if res is None:
                y, h_ref = ops.rms_norm(x, w, 1e-5), x
            else:
                y, h_ref = ops.rms_norm(x, w, 1e-5, residual=res)
            q2, sf2 = f8.quantize_act_mx(y)
            assert torch.equal(h, h_ref)
            a, b = f8.dequantize_act_mx(q, sf), f8.dequantize_act_mx(q2, sf2)
            assert ((a - b).abs() > 0).float().mean().item() < 2e-3 and _rel_err(a, b) < 2e-3
            assert _rel_err(a, y.float()) < 0.04
    for M, F in [(5, 14336), (200, 1792)]:
        gu = torch.randn(M, 2 * F, device=dev, generator=g).bfloat16()
        q, sf = f8.swiglu_quant_mx(gu)
        q2, sf2 = f8.quantize_act_mx(ops.swiglu(gu))
        assert torch.equal(q, q2) and torch.equal(sf[:, :M], sf2[:, :M])
    _status_ok()


def test_mx_linear_from_bf16_operands(dev):
    """Quantise-then-multiply against the bf16 product: the error is that of rounding both operands to E4M3."""
    from tesseract_b200.ops import fp8 as f8
    g = torch.Generator(device=dev).manual_seed(5)
    for M, N, K in [(32, 4096, 4096), (160, 14336, 4096), (3000, 6144, 4096)]:
        x = torch.randn(M, K, device=dev, generator=g).bfloat16()
        w = (torch.randn(N, K, device=dev, generator=g) * 0.05).bfloat16()
        wq, ws = f8.quantize_weight(w, pow2=True)
        assert f8.scales_are_pow2(ws)
        q, sf = f8.quantize_act_mx(x, atoms=M > 256)
        got = f8.mx_linear(q, sf, wq, ws)
        full = x.float() @ w.float().t()
        assert ((got.float() - full).norm() / full.norm()).item() < 0.06


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,L,d,N", [(2, 1, 64, 16), (1, 50, 96, 8), (2, 300, 128, 16), (1, 1000, 64, 32),
                                      (2, 300, 1024, 16), (1, 333, 2080, 8), (3, 65, 704, 16)])   # single-pass kernel
def test_selective_scan_and_conv1d(dev, dtype, B, L, d, N):
    from tesseract_b200.ops import ssm
    g = torch.Generator(device=dev).manual_seed(L + N)
    u = torch.randn(B, L, d, device=dev, generator=g).to(dtype)
    delta = torch.nn.functional.softplus(torch.randn(B, L, d, device=dev, generator=g)).to(dtype) * 0.1
    A = -torch.exp(torch.randn(d, N, device=dev, generator=g) * 0.3)
    Bm = torch.randn(B, L, N, device=dev, generator=g).to(dtype)
    Cm = torch.randn(B, L, N, device=dev, generator=g).to(dtype)
    D = torch.randn(d, device=dev, generator=g)
    st = torch.randn(B, d, N, device=dev, generator=g)
    y, s_out = ssm.selective_scan(u, delta, A, Bm, Cm, D, st)
    yr, sr = ssm.selective_scan_ref(u.float(), delta.float(), A, Bm.float(), Cm.float(), D, st)
    tol = 3e-2 if dtype == torch.bfloat16 else 2e-4
    assert _rel_err(y, yr) < tol and _rel_err(s_out, sr) < tol
    w = torch.randn(d, 4, device=dev, generator=g)
    bias = torch.randn(d, device=dev, generator=g)
    for silu in (False, True):
        got = ssm.causal_conv1d(u, w, bias, silu=silu)
        ref = ssm.causal_conv1d_ref(u.float(), w, bias, silu=silu)
        assert _rel_err(got, ref) < (2e-2 if dtype == torch.bfloat16 else 1e-5)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M", [1, 3, 16])
def test_quantized_gemv(dev, dtype, M):
    from tesseract_b200.nn import Linear
    from tesseract_b200.quant import QuantizedLinear, QuantizedLinearInt4G, unpack_int4_group
    lin = Linear(1024, 768, bias=True)
    x = torch.randn(M, 1024)
    q8 = QuantizedLinear.from_linear(lin).to(dev)
    q4 = QuantizedLinearInt4G.from_linear(lin, 128).to(dev)
    if dtype != torch.float32:
        q8.bias.data, q4.bias.data = q8.bias.data.to(dtype), q4.bias.data.to(dtype)
    xd = x.to(dev).to(dtype)
    w8 = q8.q_weight.float() * q8.weight_scale[:, None]
    w4 = unpack_int4_group(q4.q_weight.cpu(), q4.weight_scale.cpu(), 128).to(dev)
    tol = 1.5e-2 if dtype == torch.bfloat16 else 1e-4
    assert _rel_err(q8(xd), xd.float() @ w8.t() + q8.bias.float()) < tol
    assert _rel_err(q4(xd), xd.float() @ w4.t() + q4.bias.float()) < tol


@pytest.mark.parametrize("M", [17, 200, 1024])
def test_quantized_linear_large_batch_runs_on_the_native_gemm(dev, M):
    """More rows than the GEMV kernels take: the packed weights are widened to bf16 by the native kernel (bit-identical
    to the reference dequantisation) and multiplied on the tcgen05 GEMM."""
    from tesseract_b200 import _native, quant
    from tesseract_b200.quant import unpack_int4_group
    g = torch.Generator().manual_seed(M)
    w = torch.randn(768, 1024, generator=g)
    q8, s8 = (t.to(dev) for t in quant.pack_int8_symmetric(w))
    q4, s4 = (t.to(dev) for t in quant.pack_int4_group(w, 128))
    x = torch.randn(M, 1024, generator=g).to(dev).bfloat16()
    w8 = torch.empty(768, 1024, device=dev, dtype=torch.bfloat16)
    _native.check(_native.lib().tsb_dequant_w8_bf16(q8.data_ptr(), s8.data_ptr(), w8.data_ptr(), 768, 1024,
                                                    _native.stream_ptr(x.device)), "tsb_dequant_w8_bf16")
    assert torch.equal(w8, (q8.float() * s8[:, None].float()).bfloat16())
    w4 = torch.empty(768, 1024, device=dev, dtype=torch.bfloat16)
    _native.check(_native.lib().tsb_dequant_w4g_bf16(q4.data_ptr(), s4.data_ptr(), w4.data_ptr(), 768, 1024, 128,
                                                     _native.stream_ptr(x.device)), "tsb_dequant_w4g_bf16")
    assert torch.equal(w4, unpack_int4_group(q4.cpu(), s4.cpu(), 128).to(dev).bfloat16())
    before = _native.launch_count()
    with torch.no_grad():
        y8 = quant.dequantize_matmul_int8(x, q8, s8)
        y4 = quant.dequantize_matmul_int4_group(x, q4, s4, 128)
    torch.cuda.synchronize()
    _status_ok()
    assert _native.launch_count() >= before + 4                 # two dequantisers, two GEMMs
    assert _rel_err(y8, x.float() @ w8.float().t()) < 1e-2
    assert _rel_err(y4, x.float() @ w4.float().t()) < 1e-2



def test_moe_router_and_sort(dev):
    from tesseract_b200.nn.moe import route_topk
    from tesseract_b200.ops import moe
    T, E, k = 777, 8, 2
    logits = torch.randn(T, E, device=dev)
    logits[5, 3] = logits[5, 6] = 4.0          # tie: lower index first
    probs, idx, gates, counts = moe.route_native(logits, k)
    with torch.enable_grad():
        pr, ir, gr = route_topk(logits.requires_grad_(), k)
    assert torch.allclose(probs, pr, atol=1e-6) and torch.equal(idx, ir) and torch.allclose(gates, gr, atol=1e-6)
    assert idx[5].tolist() == [3, 6]
    assert torch.equal(counts.long(), torch.bincount(idx.reshape(-1), minlength=E))
    offsets, pos, tok = moe.sort_by_expert(idx, counts)
    assert offsets.tolist() == [0] + torch.cumsum(counts, 0).tolist()
    flat_e = idx.reshape(-1)
    assert sorted(pos.tolist()) == list(range(T * k))
    assert torch.equal(tok[pos.long()].long(), torch.arange(T * k, device=dev) // k)
    for e in range(E):
        rows = pos[flat_e == e]
        assert int(rows.min()) >= offsets[e] and int(rows.max()) < offsets[e + 1]


@pytest.mark.parametrize("E,N,K,counts", [(4, 256, 192, [130, 0, 257, 1]), (8, 512, 256, [100] * 8),
                                          (3, 1024, 1024, [1000, 300, 5])])
def test_grouped_gemm_rows_and_wgrad(dev, E, N, K, counts):
    """Row-grouped (forward, input gradient) and reduction-grouped (weight gradient) tcgen05 GEMMs against per-group
    fp32 matmuls; offsets are padded to 128 rows and live on the device."""
    from tesseract_b200.ops import moe
    g = torch.Generator(device=dev).manual_seed(E * 31 + N)
    padded = [(c + 127) // 128 * 128 for c in counts]
    starts = [sum(padded[:e]) for e in range(E)]
    rows_cap = sum(padded) + 256                                  # some unused tail blocks
    offsets = torch.tensor(starts + [sum(padded)], dtype=torch.int32, device=dev)
    a = torch.zeros(rows_cap, K, device=dev, dtype=torch.bfloat16)
    for e in range(E):
        a[starts[e]:starts[e] + counts[e]] = torch.randn(counts[e], K, device=dev, generator=g).bfloat16()
    w = (torch.randn(E, N, K, device=dev, generator=g) * 0.1).bfloat16()
    out = moe.grouped_gemm_rows(a, w[0], N * K, offsets, E)
    dy = torch.zeros(rows_cap, N, device=dev, dtype=torch.bfloat16)
    for e in range(E):
        lo, hi = starts[e], starts[e] + counts[e]
        ref = a[lo:hi].float() @ w[e].float().t()
        if counts[e]:
            assert _rel_err(out[lo:hi], ref) < 1e-2
        dy[lo:hi] = torch.randn(counts[e], N, device=dev, generator=g).bfloat16()
    dx = moe.grouped_gemm_rows(dy, w[0], N * K, offsets, E, b_mn=True)
    dw = torch.full((E, N, K), 7.0, device=dev, dtype=torch.float32)
    moe.grouped_gemm_wgrad(dy, a, offsets, E, dw, N * K, K, accumulate=False)
    dw_acc = dw.clone()
    moe.grouped_gemm_wgrad(dy, a, offsets, E, dw_acc, N * K, K, accumulate=True)
    torch.cuda.synchronize()
    for e in range(E):
        lo, hi = starts[e], starts[e] + counts[e]
        if counts[e]:
            assert _rel_err(dx[lo:hi], dy[lo:hi].float() @ w[e].float()) < 1e-2
        ref_w = dy[lo:hi].float().t() @ a[lo:hi].float()
        if counts[e]:
            assert _rel_err(dw[e], ref_w) < 1e-2
            assert _rel_err(dw_acc[e], 2 * ref_w) < 1e-2
        else:
            assert float(dw[e].abs().max()) == 0.0
    from tesseract_b200 import _native
    assert _native.read_status(torch.cuda.current_stream().cuda_stream) == 0


def test_moe_grouped_layer_forward_backward(dev):
    """The grouped-GEMM expert path against the per-expert reference path of the same module: output, input
    gradient, router-gate gradient and every expert weight gradient."""
    from tesseract_b200.nn.moe import MoEFeedForward, route_topk
    from tesseract_b200.ops import moe as moe_ops
    torch.manual_seed(1)
    layer = MoEFeedForward(256, 384, num_experts=4, num_experts_per_tok=2, dtype=torch.bfloat16, device=dev)
    x = torch.randn(300, 256, device=dev).bfloat16().requires_grad_(True)
    probs, idx, gates = route_topk(layer.gate(x.detach()), 2)
    gates = gates.detach().to(torch.bfloat16).requires_grad_(True)
    dout = torch.randn(300, 256, device=dev).bfloat16()

    out = moe_ops.moe_ffn_grouped(x, idx, gates, layer)
    out.backward(dout)
    got = [x.grad.clone(), gates.grad.clone()] + [p.grad.clone() for p in layer.experts.parameters()]
    x.grad = None
    gates.grad = None
    for p in layer.experts.parameters():
        p.grad = None
    ref = layer._sparse_reference(x, idx, gates)
    ref.backward(dout)
    want = [x.grad, gates.grad] + [p.grad for p in layer.experts.parameters()]
    assert _rel_err(out, ref) < 2e-2
    for g_, w_ in zip(got, want):
        assert _rel_err(g_, w_) < 3e-2


def test_moe_layer_gpu_matches_dense_reference(dev):
    from tesseract_b200.nn.moe import MoEFeedForward
    torch.manual_seed(0)
    moe_l = MoEFeedForward(256, 512, num_experts=4, num_experts_per_tok=2, dtype=torch.bfloat16, device=dev)
    x = torch.randn(3, 40, 256, device=dev).bfloat16()
    with torch.no_grad():
        out = moe_l(x)
        ref = moe_l.forward_dense_reference(x)
    assert _rel_err(out, ref) < 3e-2


def test_graph_train_step_replays_as_one_cuda_graph(dev):
    """Graph-mode training on the GPU: forward + backward recorded once and replayed as a CUDA graph gives the
    eager tape's loss and gradients on fresh batches."""
    import torch.nn.functional as F
    from tesseract_b200.graph import GraphTrainStep
    torch.manual_seed(0)
    model = torch.nn.Sequential(torch.nn.Flatten(), torch.nn.Linear(64, 48), torch.nn.ReLU(), torch.nn.Linear(48, 10)).to(dev)
    x, y = torch.randn(32, 1, 8, 8, device=dev), torch.randint(0, 10, (32,), device=dev)
    step = GraphTrainStep(model, F.cross_entropy, x, y)
    assert step.executor.cuda_graph
    for _ in range(3):
        x, y = torch.randn(32, 1, 8, 8, device=dev), torch.randint(0, 10, (32,), device=dev)
        loss = step(x, y).clone()
        got = [p.grad.clone() for p in model.parameters()]
        for p in model.parameters():
            p.grad = None
        ref = F.cross_entropy(model(x), y)
        ref.backward()
        assert abs(float(loss) - float(ref)) < 1e-4
        for g_, p in zip(got, model.parameters()):
            assert _rel_err(g_, p.grad) < 1e-3
        with torch.no_grad():
            for p in model.parameters():
                p.sub_(0.1 * p.grad)            # in-place update: the next replay must see it

"""Kernels that large products and many rows take, at the sizes where their tiles and chunks end."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _ops():
    from openagents_b200.ops import cuda_ops
    return cuda_ops


def _randn(*shape, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(*shape, generator=g, device=DEV)


def _bound(A, B):
    """Sums of exact products in 32 bits, in any order and with truncated partial sums: far below 2^-17 of the sum of magnitudes."""
    return 2.0 ** -17 * (A.float().abs() @ B.float().abs().t()) + 1e-6


# one tile and its remainders; a split of every length down to one K block; columns that end inside a 32-column chunk
@pytest.mark.parametrize("tile_n", [256, 128])
@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (300, 520, 200), (129, 44, 72), (1000, 800, 768), (5000, 640, 136), (65, 4096, 1024)])
def test_gemm_pair(M, N, K, tile_n):
    ops = _ops()
    A, B = _randn(M, K, seed=1).bfloat16(), _randn(N, K, seed=2).bfloat16()
    bias, x0 = _randn(N, seed=3), _randn(M, N, seed=4)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    ref, tol = A.float() @ B.float().t(), _bound(A, B)
    guard = torch.full((M + 8, N + 4), 7.0, device=DEV)            # what lies beyond the result stays
    out = guard[:M, :N]
    ops.gemm_pair(A, B, M, N, K, out, bias=bias, alpha=0.5, tile_n=tile_n, status=status)
    assert ((out - (0.5 * ref + bias)).abs() <= tol).all()
    assert (guard[M:] == 7.0).all() and (guard[:, N:] == 7.0).all()
    for splits in (1, 2, 5):
        out = x0.clone()
        ops.gemm_pair(A, B, M, N, K, out, add=True, bias=bias, splits=splits, tile_n=tile_n, status=status)
        assert ((out - (x0 + ref + bias)).abs() <= tol + 1e-5).all(), splits
    if N % 8 == 0:
        r = _randn(M, N, seed=5).bfloat16()
        for act, f in ((ops.ACT_NONE, lambda v: v), (ops.ACT_GELU, lambda v: torch.nn.functional.gelu(v, approximate="tanh")), (ops.ACT_RELU2, lambda v: v.relu() ** 2)):
            want = f(ref + bias) + r.float()
            for dt, eps in ((torch.bfloat16, 2.0 ** -8), (torch.float16, 2.0 ** -10)):
                if dt == torch.float16 and act == ops.ACT_RELU2:
                    continue                                       # squares leave the range
                out = torch.empty((M, N), dtype=dt, device=DEV)
                ops.gemm_pair(A, B, M, N, K, out, bias=bias, resid_bf16=r, act=act, tile_n=tile_n, status=status)
                slope = 1.0 if act != ops.ACT_RELU2 else 2.0 * (ref + bias).abs().max().item()
                # the hardware's tanh is good to 2^-11
                assert ((out.float() - want).abs() <= slope * tol + (eps + 2.0 ** -10) * (f(ref + bias).abs() + want.abs()) + 2e-3).all(), (act, dt)
    if N % 32 == 0:
        out = torch.empty((M, N // 2), dtype=torch.bfloat16, device=DEV)
        ops.gemm_pair(A, B, M, N, K, out, swiglu=True, tile_n=tile_n, status=status)
        want = torch.nn.functional.silu(ref[:, 0::2]) * ref[:, 1::2]
        assert torch.allclose(out.float(), want, rtol=2.0 ** -7, atol=1e-3 * float(want.abs().max()))
    if M % 8 == 0 and N % 8 == 0:
        out = x0.clone()
        ops.gemm_pair(A.t().contiguous(), B.t().contiguous(), M, N, K, out, add=True, splits=2, mn_major=True, tile_n=tile_n, status=status)
        assert ((out - (x0 + ref)).abs() <= tol + 1e-5).all()
    torch.cuda.synchronize()
    assert int(status) == 0


def test_gemm_pair_refuses_what_it_cannot_store():
    ops = _ops()
    A, B = _randn(256, 64, seed=6).bfloat16(), _randn(256, 64, seed=7).bfloat16()
    with pytest.raises(RuntimeError):                              # rows of the result that do not start on 16 bytes
        ops.gemm_pair(A, B, 256, 256, 64, torch.empty((256, 257), device=DEV)[:, :256])
    with pytest.raises(RuntimeError):                              # splits add up: they need something to add to
        ops.gemm_pair(A, B, 256, 256, 64, torch.empty((256, 256), device=DEV), splits=2)
    for splits in (1, 2):                                          # 16-bit results are stored, never added to
        with pytest.raises(RuntimeError):
            ops.gemm_pair(A, B, 256, 256, 64, torch.empty((256, 256), dtype=torch.bfloat16, device=DEV), add=True, splits=splits)


@pytest.mark.parametrize("mn_major", [False, True])
@pytest.mark.parametrize("M,N,K", [(256, 512, 4096), (2048, 4096, 512)])      # one that would split K, and one of many tiles
def test_products_in_16_bits_are_whole_with_accumulate_set(M, N, K, mn_major):
    """``accumulate`` adds to fp32 results; a 16-bit result is stored whole, flag or not."""
    ops = _ops()
    A, B = _randn(M, K, seed=50).bfloat16(), _randn(N, K, seed=51).bfloat16()
    a, b = (A.t().contiguous(), B.t().contiguous()) if mn_major else (A, B)
    out, status = torch.full((M, N), 3.0, dtype=torch.bfloat16, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.gemm_bf16(a, b, M, N, K, lda=a.stride(0), ldb=b.stride(0), out_bf16=out, accumulate=True, mn_major=mn_major, status=status)
    ref = A.float() @ B.float().t()
    assert ((out.float() - ref).abs() <= _bound(A, B) + 2.0 ** -8 * ref.abs()).all() and int(status) == 0


@pytest.mark.parametrize("T", [127, 128, 200])                     # either side of the row count where the kernel changes
@pytest.mark.parametrize("D", [32, 2880, 4096, 8192, 8224])        # 8192: the longest row of the many-row kernel
def test_rmsnorm_many_rows(T, D):
    ops = _ops()
    x, g = _randn(T, D, seed=8) * 3, _randn(D, seed=9)
    hf, hb = torch.empty((T, D), device=DEV), torch.empty((T, D), dtype=torch.bfloat16, device=DEV)
    for gain in (g, None):
        ops.rmsnorm(x, gain, 1e-5, hb=hb, hf=hf)
        ref = x.double() * torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True) + 1e-5) * (1 if gain is None else gain.double())
        assert ((hf - ref).abs() <= 2.0 ** -20 * ref.abs() + 1e-12).all()
        assert torch.equal(hb, hf.bfloat16())


@pytest.mark.parametrize("style", ["pairs", "half"])
@pytest.mark.parametrize("hd,Hq,Hkv", [(64, 5, 2), (128, 4, 1), (16, 3, 3)])
def test_rope_kv_many_tokens(style, hd, Hq, Hkv):
    """The kernel for many tokens against the one for few, over the same tokens a hundred at a time."""
    ops = _ops()
    T, st = 300, 0 if style == "pairs" else 1
    qkv = _randn(T, (Hq + 2 * Hkv) * hd, seed=10)
    g = torch.Generator().manual_seed(11)
    pos = torch.randint(0, 9000, (T,), generator=g).int().to(DEV)  # some beyond the table
    slot = torch.randperm(320, generator=g)[:T].int().to(DEV)
    slot[5] = -1
    tab = ops.rope_table(8192, hd, 500000.0, DEV)
    outs = []
    for step in (T, 100):
        kc = torch.zeros((20, Hkv, 16, hd), dtype=torch.float16, device=DEV)
        vc = torch.zeros_like(kc)
        q32, q16 = torch.empty((T, Hq * hd), device=DEV), torch.empty((T, Hq * hd), dtype=torch.float16, device=DEV)
        for lo in range(0, T, step):
            s = slice(lo, lo + step)
            ops.rope_kv(qkv[s], pos[s], slot[s], q32[s], q16[s], kc, vc, Hq, Hkv, hd, 16, 500000.0, st, 0.125, table=tab)
        outs.append((q32, q16, kc, vc))
    for a, b in zip(*outs):                                        # a contracted multiply-add may round differently
        assert torch.allclose(a.float(), b.float(), rtol=2.0 ** -10 if a.dtype == torch.float16 else 2.0 ** -21, atol=1e-6)
    assert torch.equal(outs[0][3], outs[1][3])


# experts without rows, with a few (an operand of 16, 32 and 64 rows each) and with more than one block of 64; K that ends inside a stage of 256
@pytest.mark.parametrize("E,d,f,cap,T,top_k", [(8, 256, 256, 256, 3, 2), (3, 352, 96, 128, 50, 2), (16, 416, 160, 128, 100, 1), (40, 96, 64, 128, 77, 4),
                                               (2, 512, 320, 256, 150, 2), (4, 2880, 2880, 256, 200, 2)])
def test_moe_gemm_on_packed_weights(E, d, f, cap, T, top_k):
    """The expert GEMMs on MXFP4 blocks against the same on their exact bf16 expansion: equal products, sums in another order."""
    from openagents_b200.gguf import GgmlType
    from openagents_b200.gguf import torch_codecs as tc
    ops = _ops()
    raw13, raw2 = (tc.quantize(_randn(*s, seed=20 + i) * 0.02, GgmlType.MXFP4) for i, s in enumerate(((E * 2 * f, d), (E * d, f))))
    w13, w2 = tc.dequantize(raw13, GgmlType.MXFP4, (E, 2 * f, d)), tc.dequantize(raw2, GgmlType.MXFP4, (E, d, f))
    q13, q2 = tc.pack_mxfp4_wide(raw13, E * 2 * f), tc.pack_mxfp4_wide(raw2, E * d)
    g = torch.Generator(device=DEV).manual_seed(22)
    chosen = torch.rand(T, E, device=DEV, generator=g).topk(top_k, 1).indices
    x = _randn(T, d, seed=23).bfloat16()
    recv = torch.full((E * cap, d), float("nan"), dtype=torch.bfloat16, device=DEV)         # what no token wrote is never used
    meta, gate = torch.zeros((E * cap, 2), dtype=torch.int32, device=DEV), torch.rand(E * cap, device=DEV, generator=g)
    counts = torch.zeros(E, dtype=torch.int32, device=DEV)
    for e in range(E):
        rows = (chosen == e).any(1).nonzero().flatten()
        counts[e] = len(rows)
        recv[e * cap: e * cap + len(rows)], meta[e * cap: e * cap + len(rows), 1] = x[rows], rows.int()
    mid = torch.full((E * cap, f), 7.0, dtype=torch.bfloat16, device=DEV)
    y0 = _randn(T, d, seed=24)
    y = y0.clone()
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.moe_qgemm(*q13, recv, E, cap, 2 * f, d, counts, T * top_k, out_bf16=mid, ldo=f, status=status)
    ops.moe_qgemm(*q2, mid, E, cap, d, f, counts, T * top_k, y=y, ldo=d, meta=meta, gate_w=gate, status=status)
    torch.cuda.synchronize()
    assert int(status) == 0
    ref, scale = y0.double(), y0.double().abs()
    for e in range(E):
        n = int(counts[e])
        s = slice(e * cap, e * cap + n)
        gu, mag = recv[s].float() @ w13[e].t(), recv[s].float().abs() @ w13[e].t().abs()
        want = torch.nn.functional.silu(gu[:, 0::2]) * gu[:, 1::2]
        tol = 2.0 ** -17 * (mag[:, 0::2] * gu[:, 1::2].abs() + mag[:, 1::2] * gu[:, 0::2].abs()) * 1.1 + 2.0 ** -8 * want.abs() + 1e-6     # |d silu| < 1.1
        assert ((mid[s].float() - want).abs() <= tol).all()
        assert (mid[e * cap + n: (e + 1) * cap] == 7.0).all()
        rows = meta[s, 1].long()
        ref.index_add_(0, rows, gate[s, None].double() * (mid[s].double() @ w2[e].double().t()))
        scale.index_add_(0, rows, gate[s, None].double() * (mid[s].double().abs() @ w2[e].double().t().abs()))
    assert ((y - ref).abs() <= 2.0 ** -17 * scale).all()


def test_packed_weights_hold_every_code_and_refuse_large_scales():
    """All sixteen codes at all places of a block, by the layout's own rules, on the host."""
    from openagents_b200.gguf import torch_codecs as tc
    blocks = torch.zeros((1, 16, 17), dtype=torch.uint8)
    for b in range(16):
        blocks[0, b, 0] = 100 + b
        codes = (torch.arange(32) + b) % 16
        blocks[0, b, 1:] = (codes[:16] | (codes[16:] << 4)).to(torch.uint8)
    words, scales = tc.pack_mxfp4_wide(blocks.reshape(-1), 1)
    values = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6], dtype=torch.float64)
    h = words.reshape(16, 4, 2, 2).to(torch.int64)
    h = h[..., 0] | (h[..., 1] << 8)                               # [block, word, half]
    bits = lambda at, n: (h >> at) & ((1 << n) - 1)
    parts = [(bits(15, 1), bits(6, 3)), (bits(12, 1), bits(3, 3)), (bits(9, 1), bits(0, 3)), (bits(13, 1), bits(10, 2) | (bits(14, 1) << 2))]
    got = torch.stack([values[m] * (1 - 2 * s) for s, m in parts], 2).reshape(16, 32)
    for b in range(16):
        codes = (torch.arange(32) + b) % 16
        assert torch.equal(got[b], values[codes & 7] * (1 - 2 * (codes >> 3)))
    assert scales.shape == (2, 1, 8) and scales.flatten().tolist() == [226 + b for b in range(16)]
    blocks[0, 3, 0] = 129
    assert tc.pack_mxfp4_wide(blocks.reshape(-1), 1) is None


@pytest.mark.parametrize("kind", ["Q4_K", "Q6_K"])
@pytest.mark.parametrize("T,N,K", [(65, 300, 512), (128, 128, 256), (129, 384, 1024), (300, 200, 2048)])
def test_fused_dequant_gemm_of_short_prompts(kind, T, N, K):
    """Tiles of 128 tokens: as near to the exact product as the bf16 expansion of the weights is."""
    from openagents_b200.gguf import GgmlType
    from openagents_b200.gguf import torch_codecs as tc
    from openagents_b200.models.qweight import QWeight, RawTensor
    ops, t = _ops(), GgmlType[kind]
    raw = tc.quantize(_randn(N, K, seed=30) * 0.05, t)
    w, exact = QWeight.from_raw(RawTensor(t, (N, K), raw)), tc.dequantize(raw, t, (N, K)).double()
    x, r = _randn(T, K, seed=31).bfloat16(), _randn(T, N, seed=32)
    ref = x.double() @ exact.t()
    dense = x.double() @ w.dequant_into(torch.empty((N, K), dtype=torch.bfloat16, device=DEV)).double().t()
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    y = r.clone()
    ops.qgemm(w, x, T, out_f32=y, epi=ops.QEPI_ADD, status=status)
    got = y.double() - r.double()
    # Errors of K independent roundings: the ratio of two such norms over T * N results scatters by well under a tenth; 32-bit sums add 2^-22.
    assert (got - ref).norm() <= 1.1 * (dense - ref).norm() + 2.0 ** -22 * (ref.norm() + r.double().norm())
    if N % 32 == 0:
        out = torch.empty((T, N // 2), dtype=torch.bfloat16, device=DEV)
        ops.qgemm(w, x, T, out_bf16=out, ldo=N // 2, epi=ops.QEPI_SWIGLU, status=status)
        want = torch.nn.functional.silu(got[:, 0::2]) * got[:, 1::2]
        assert torch.allclose(out.double(), want, rtol=2.0 ** -7, atol=1e-3 * float(want.abs().max()))
    assert int(status) == 0


@pytest.mark.parametrize("kind", ["Q4_K", "Q6_K"])
@pytest.mark.parametrize("spread", [1.0, 30.0])                    # weights of one size, and heavy tails inside every block
def test_fused_dequant_gemm_of_short_prompts_rounds_weights_once(kind, spread):
    """One-hot rows give the weights themselves: the very ones of the bf16 expansion, in every row and superblock."""
    from openagents_b200.gguf import GgmlType
    from openagents_b200.gguf import torch_codecs as tc
    from openagents_b200.models.qweight import QWeight, RawTensor
    ops, t, N, K = _ops(), GgmlType[kind], 392, 1280
    weights = _randn(N, K, seed=33) * 0.02 * spread ** _randn(N, K, seed=34).clamp(-2, 2)
    weights[5] = 0.0
    weights[6, :512] = weights[6, :512].abs() + 0.5
    w = QWeight.from_raw(RawTensor(t, (N, K), tc.quantize(weights, t)))
    y, status = torch.empty((K, N), device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.qgemm(w, torch.eye(K, device=DEV).bfloat16(), K, out_f32=y, epi=ops.QEPI_STORE, status=status)
    assert torch.equal(y.t(), w.dequant_into(torch.empty((N, K), dtype=torch.bfloat16, device=DEV)).float()) and int(status) == 0


@pytest.mark.parametrize("D", [64, 256, 264, 512, 768, 776, 1024, 1032])      # either side of every width that a row in registers is built for
@pytest.mark.parametrize("rows,add", [(5, False), (3000, True)])
def test_layernorm_backward_widths(D, rows, add):
    from openagents_b200.ops import train_ops as tops
    x, dy, dx0 = (_randn(rows, D, seed=40 + i).bfloat16() for i in range(3))
    g, b = _randn(D, seed=43), _randn(D, seed=44)
    y, mean, rstd = torch.empty_like(x), torch.empty(rows, device=DEV), torch.empty(rows, device=DEV)
    tops.layernorm_fwd(x, g, b, 1e-5, y, mean, rstd)
    dx, dg, db = dx0.clone(), torch.zeros(D, device=DEV), torch.zeros(D, device=DEV)
    tops.layernorm_bwd(dy, x, g, mean, rstd, dx, add, dg, db)
    xr, gr, br = (t.double().requires_grad_(True) for t in (x, g, b))
    torch.nn.functional.layer_norm(xr, (D,), gr, br, 1e-5).backward(dy.double())
    want = xr.grad + (dx0.double() if add else 0)
    # one rounding to bf16 of the result (and the terms' 32-bit errors, which a difference of terms of size one can show)
    assert ((dx.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all()
    for got, ref in ((dg, gr.grad), (db, br.grad)):      # sums of `rows` terms of size about one to ten in 32 bits
        assert ((got.double() - ref).abs() <= 2.0 ** -18 * rows + 1e-4).all()


def _pair_sizes_inplace(ops, M, N, K, how):
    A, B, x0, bias = _randn(M, K, seed=60).bfloat16(), _randn(N, K, seed=61).bfloat16(), _randn(M, N, seed=62), _randn(N, seed=63)
    x, status = x0.clone(), torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.gemm_bf16(A, B, M, N, K, out_f32=x, bias=bias, resid_f32=x if how == "resid" else None, accumulate=how == "accumulate", status=status)
    return (x - (x0 + A.float() @ B.float().t() + bias)).abs() <= _bound(A, B) + 1e-5, int(status)


@pytest.mark.parametrize("how", ["resid", "accumulate"])
@pytest.mark.parametrize("M,N,K", [(2048, 4096, 512), (300, 2048, 4096), (1000, 4100, 776)])      # many tiles; few, with K split; tiles that end inside
def test_large_products_added_in_place(M, N, K, how):
    ok, status = _pair_sizes_inplace(_ops(), M, N, K, how)
    assert ok.all() and status == 0


# more than 128 rows an expert on average; a group of an odd number of 128-row tiles, so that a pair's tile ends in the next one's rows; experts
# without rows, with one, with all; several stages of K with a remainder; columns that end inside a tile
@pytest.mark.parametrize("counts,K,f,d", [((0, 1, 129, 257, 384, 384), 200, 160, 328), ((384,), 712, 144, 64), ((256, 131, 384), 64, 512, 768)])
def test_expert_products_of_many_rows(counts, K, f, d):
    ops, E, cap = _ops(), len(counts), 384
    x, w13 = _randn(E * cap, K, seed=64).bfloat16(), _randn(E * 2 * f, K, seed=65).bfloat16() * 0.1
    cnt, rows = torch.tensor(counts, dtype=torch.int32, device=DEV), sum(counts)
    assert rows > 128 * E
    gate, status = torch.rand(E * cap, device=DEV) + 0.5, torch.zeros(1, dtype=torch.int32, device=DEV)
    live = torch.cat([torch.arange(c, device=DEV) + e * cap for e, c in enumerate(counts)])
    for w in (None, gate):                                         # a weight multiplies the expert's input
        mid = torch.full((E * cap, f), 7.0, dtype=torch.bfloat16, device=DEV)
        ops.moe_gemm(x, w13, E, cap, 2 * f, K, cnt, 1, out_bf16=mid, ldc=f, gate_w=w, live_rows=rows, status=status)
        for e, c in enumerate(counts):
            s = slice(e * cap, e * cap + c)
            scale = 1.0 if w is None else w[s, None]
            gu, mag = scale * (x[s].float() @ w13[e * 2 * f:(e + 1) * 2 * f].float().t()), scale * (x[s].float().abs() @ w13[e * 2 * f:(e + 1) * 2 * f].float().abs().t())
            want = torch.nn.functional.silu(gu[:, 0::2]) * gu[:, 1::2]
            tol = 2.0 ** -17 * 1.1 * (mag[:, 0::2] * (gu[:, 1::2].abs() + 1) + mag[:, 1::2] * gu[:, 0::2].abs()) + (2.0 ** -8 + 2.0 ** -10) * want.abs() + 1e-5
            assert ((mid[s].float() - want).abs() <= tol).all(), e
            assert (mid[e * cap + -(-c // 32) * 32:(e + 1) * cap] == 7.0).all(), e        # the patch of 32 rows that holds the last one, and no further
    h, w2 = _randn(E * cap, K, seed=66).bfloat16(), _randn(E * d, K, seed=67).bfloat16()
    tokens = torch.randperm(E * cap, generator=torch.Generator().manual_seed(68)).to(DEV) % 500
    meta = torch.stack((torch.zeros_like(tokens), tokens), 1).int().contiguous()
    for w in (None, gate):
        y0 = _randn(500, d, seed=69)
        y = y0.clone()
        ops.moe_gemm(h, w2, E, cap, d, K, cnt, 2, ldc=d, meta=meta, gate_w=w, sym_off=y.data_ptr(), live_rows=rows, status=status)
        ref, scale = y0.double(), y0.double().abs()
        per_row = torch.cat([h[e * cap:e * cap + c].double() @ w2[e * d:(e + 1) * d].double().t() for e, c in enumerate(counts)])
        mags = torch.cat([h[e * cap:e * cap + c].double().abs() @ w2[e * d:(e + 1) * d].double().t().abs() for e, c in enumerate(counts)])
        g = torch.ones(rows, 1, device=DEV).double() if w is None else w[live, None].double()
        ref.index_add_(0, tokens[live], g * per_row)
        scale.index_add_(0, tokens[live], g * mags)
        assert ((y - ref).abs() <= 2.0 ** -17 * scale).all()
    assert int(status) == 0


@pytest.mark.parametrize("T", [295, 296, 297, 298, 592, 593, 4096])      # from 297 tokens on a CTA takes two of them, the last one what is left
@pytest.mark.parametrize("E,d,top_k", [(32, 2880, 4), (5, 72, 2)])
def test_routing_of_many_tokens(T, E, d, top_k):
    ops = _ops()
    h32, wr, br = _randn(T, d, seed=70), _randn(E, d, seed=71) / d ** 0.5, _randn(E, seed=72)
    h = h32.bfloat16()
    recv, meta = torch.full((E * T, d), 9.0, dtype=torch.bfloat16, device=DEV), torch.full((E * T, 2), -1, dtype=torch.int32, device=DEV)
    weight, counts = torch.zeros(E * T, device=DEV), torch.zeros(E, dtype=torch.int32, device=DEV)
    ids, w = torch.empty((T, top_k), dtype=torch.int32, device=DEV), torch.empty((T, top_k), device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.moe_route_dispatch(h, h32, wr, br, top_k, E, T, *(t.data_ptr() for t in (recv, meta, weight, counts)), None, topk_ids=ids, topk_w=w, status=status)
    one_i, one_w = torch.empty_like(ids), torch.empty_like(w)
    for lo in range(0, T, 250):                                    # the form of one token a CTA
        s = slice(lo, min(T, lo + 250))
        ops.moe_route_dispatch(None, h32[s], wr, br, top_k, E, 0, 0, 0, 0, 0, None, topk_ids=one_i[s], topk_w=one_w[s])
    logits = h32.double() @ wr.double().t() + br.double()
    tol = 2.0 ** -20 * (h32.double().abs() @ wr.double().abs().t() + br.double().abs()).max()
    # the chosen are the largest but for ties within the sums' error, in either form
    for i, v in ((ids, w), (one_i, one_w)):
        chosen = logits.gather(1, i.long())
        assert (logits.topk(top_k, 1).values - chosen).abs().max() <= 2 * tol
        assert torch.allclose(v.double(), torch.softmax(chosen, 1), atol=1e-5)
    assert (ids == one_i).float().mean() > 0.999
    assert torch.equal(counts.long(), torch.bincount(ids.flatten().long(), minlength=E)) and int(status) == 0
    for e in range(E):
        n = int(counts[e])
        s = slice(e * T, e * T + n)
        t = meta[s, 1].long()
        assert (meta[s, 0] == 0).all() and torch.equal(t.sort().values, (ids == e).any(1).nonzero().flatten())
        assert torch.equal(recv[s], h[t]) and torch.equal(weight[s], w[t][ids[t] == e])
        assert (recv[s.stop:(e + 1) * T] == 9.0).all()


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("window,use_sinks", [(0, True), (1024, True), (1056, False), (0, False)])
def test_prefill_attention_of_head_size_64(window, use_sinks, exact):
    """Head size 64 on tcgen05, with the long windows and sinks it takes there: cold prompts, chunks behind a context, one token, ends inside a block."""
    from test_gpu_kernels import _paged_kv

    from openagents_b200.oracle import nn
    ops, hd, Hq, Hkv = _ops(), 64, 8, 2
    ctx, qlen = [1500, 1217, 129, 2050], [1500, 64, 1, 257]
    kc, vc, table, Ks, Vs = _paged_kv(4, Hkv, hd, ctx, seed=73)
    starts = [sum(qlen[:b]) for b in range(4)]
    q = (_randn(sum(qlen), Hq * hd, seed=74) * (3.0 / hd ** 0.5)).half()
    sinks = _randn(Hq, seed=75) if use_sinks else None
    out, status = torch.zeros((sum(qlen), Hq * hd), dtype=torch.bfloat16, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    ops.attn_prefill_tc05(q, kc, vc, table, i32(starts), i32(qlen), i32(ctx), 4, max(qlen), Hq, Hkv, window=window, sinks=sinks, out_bf16=out,
                          status=status, dk=hd, dv=hd, exact_max=exact)
    assert int(status) == 0
    for b in range(4):
        s, n = starts[b], qlen[b]
        ref = nn.attention(q[s:s + n].float().cpu().view(n, Hq, hd), Ks[b], Vs[b], torch.arange(ctx[b] - n, ctx[b]), torch.arange(ctx[b]),
                           window=window, sinks=None if sinks is None else sinks.cpu(), scale=1.0).reshape(n, -1)
        # probabilities in 16 bits (2^-11 of values of size about one, averaged) and the result in bf16
        assert ((out[s:s + n].float().cpu() - ref).abs() <= 2.0 ** -8 * ref.abs() + 4e-3).all(), b


@pytest.mark.parametrize("gain", [0.3, 1.0, 3.0])                  # deviation of the scores: flat to peaked rows
@pytest.mark.parametrize("T", [400, 1500])
def test_prefill_attention_of_head_size_64_is_as_near_as_mma_sync(T, gain):
    """The two kernels that serve head size 64, against 64 bits, on the same 16-bit inputs."""
    from test_gpu_kernels import _paged_kv
    ops, hd, Hq, Hkv = _ops(), 64, 8, 2
    kc, vc, table, Ks, Vs = _paged_kv(1, Hkv, hd, [T], seed=91)
    q = (_randn(T, Hq * hd, seed=92) * (gain / hd ** 0.5)).half()
    i32 = lambda v: torch.tensor([v], dtype=torch.int32, device=DEV)
    a, b, status = torch.empty((T, Hq * hd), device=DEV), torch.empty((T, Hq * hd), device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.attn_prefill_tc05(q, kc, vc, table, i32(0), i32(T), i32(T), 1, T, Hq, Hkv, out_f32=a, status=status, dk=hd, dv=hd, exact_max=True)
    ops.attn_prefill(q, kc, vc, table, table.shape[1], i32(0), i32(T), i32(T), 1, T, Hq, Hkv, hd, out_f32=b)
    K, V = (t[0].double().to(DEV).repeat_interleave(Hq // Hkv, 1) for t in (Ks, Vs))
    s = torch.einsum("thd,shd->hts", q.double().view(T, Hq, hd), K).masked_fill(torch.ones(T, T, device=DEV).triu(1).bool(), float("-inf"))
    ref = torch.einsum("hts,shd->thd", s.softmax(-1), V).reshape(T, -1)
    # norms of T * 512 errors scatter by far less than 2 %
    assert (a - ref).norm() <= 1.02 * (b - ref).norm() and int(status) == 0
    with pytest.raises(RuntimeError):
        ops.attn_prefill_tc05(q.view(-1, 128).repeat(1, 8), kc, vc, table, i32(0), i32(T), i32(T), 1, T, Hq, Hkv, out_f32=a, exact_max=True)


# K of one K block, of a two-block stage and a half, of a ring that just fits, wraps, and wraps with a remainder; columns for tiles of 64, 128 and 256
@pytest.mark.parametrize("M", [1, 7, 33, 64])
@pytest.mark.parametrize("K", [64, 72, 192, 768, 1032, 4104])
@pytest.mark.parametrize("N,add", [(192, False), (192, True), (2304, True), (14848, False), (28672, False)])
def test_few_row_products_with_weights_loaded_ahead(M, K, N, add):
    """``b_ready`` moves loads of B ahead of the wait for the kernel before; A is written by that very kernel."""
    ops = _ops()
    src, B, x0 = _randn(M, K, seed=76), _randn(N, K, seed=77).bfloat16(), _randn(M, N, seed=78)
    gain, status = torch.ones(K, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    if K % 32:                                                     # the norm takes rows of whole 32s: the same values by a plain copy
        write = lambda A: A.copy_(src)
    else:
        write = lambda A: ops.rmsnorm(src, gain, 1e-5, hb=A)
    outs = []
    for ready in (True, False):
        A = torch.full((M, K), float("nan"), dtype=torch.bfloat16, device=DEV)      # what a load ahead of the wait would bring
        out = x0.clone() if add else torch.empty((M, N), device=DEV)
        torch.cuda.synchronize()
        write(A)
        ops.gemm_bf16(A, B, M, N, K, out_f32=out, accumulate=add, b_ready=ready, status=status)
        outs.append(out)
    tol = _bound(A, B) + 1e-5
    assert ((outs[0] - outs[1]).abs() <= 2 * tol).all()
    assert ((outs[0] - A.float() @ B.float().t() - (x0 if add else 0)).abs() <= tol).all() and int(status) == 0


@pytest.mark.parametrize("hd,Hq,Hkv", [(64, 8, 2), (128, 4, 4), (64, 6, 2), (128, 16, 1)])
@pytest.mark.parametrize("S", [1, 2, 31, 33, 65, 300])             # splits of one lane's first and second, of more than 64, and of more than one chunk of factors
@pytest.mark.parametrize("use_sinks", [False, True])
def test_decode_attention_merges_any_number_of_splits(hd, Hq, Hkv, S, use_sinks):
    """Splits without a page among them, and every form of the output."""
    from test_gpu_kernels import _paged_kv

    from openagents_b200.oracle import nn
    ops, lens = _ops(), [1, 700, 333]
    kc, vc, table, Ks, Vs = _paged_kv(3, Hkv, hd, lens, seed=80)
    q = _randn(3, Hq * hd, seed=81) * (2.0 / hd ** 0.5)
    sinks = _randn(Hq, seed=82) if use_sinks else None
    scratch, counters = torch.full((ops.attn_decode_scratch_floats(3, Hq, Hkv, hd, S) + 1,), float("nan"), device=DEV), torch.zeros(3 * Hq, dtype=torch.int32, device=DEV)
    out, outb, status = torch.empty((3, Hq * hd), device=DEV), torch.empty((3, Hq * hd), dtype=torch.bfloat16, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    for _ in range(2):                                             # the counters are left as they were
        ops.attn_decode(q, kc, vc, table, torch.tensor(lens, dtype=torch.int32, device=DEV), 3, Hq, Hkv, hd, S=S, sinks=sinks, out_f32=out, out_bf16=outb,
                        scratch=scratch[1:], counters=counters, status=status)       # scratch that starts on four bytes only
        for b in range(3):
            ref = nn.attention(q[b:b + 1].cpu().view(1, Hq, hd), Ks[b], Vs[b], torch.tensor([lens[b] - 1]), torch.arange(lens[b]),
                               sinks=sinks.cpu() if use_sinks else None, scale=1.0).reshape(-1)
            assert torch.allclose(out[b].cpu(), ref, atol=3e-3, rtol=3e-3), (b, (out[b].cpu() - ref).abs().max())
        assert torch.equal(outb, out.bfloat16()) and int(counters.abs().sum()) == 0 and int(status) == 0


@pytest.mark.parametrize("rows,D", [(12287, 768), (12288, 768), (12288, 64), (2400, 1024), (2400, 1032)])      # either side of where two CTAs an SM take over
def test_layernorm_backward_grids(rows, D):
    from openagents_b200.ops import train_ops as tops
    x, dy = _randn(rows, D, seed=83).bfloat16(), _randn(rows, D, seed=84).bfloat16()
    g, b = _randn(D, seed=85), _randn(D, seed=86)
    y, mean, rstd = torch.empty_like(x), torch.empty(rows, device=DEV), torch.empty(rows, device=DEV)
    tops.layernorm_fwd(x, g, b, 1e-5, y, mean, rstd)
    dx, dg, db = torch.zeros_like(x), torch.zeros(D, device=DEV), torch.zeros(D, device=DEV)
    tops.layernorm_bwd(dy, x, g, mean, rstd, dx, False, dg, db)
    xr, gr, br = (t.double().requires_grad_(True) for t in (x, g, b))
    torch.nn.functional.layer_norm(xr, (D,), gr, br, 1e-5).backward(dy.double())
    assert ((dx.double() - xr.grad).abs() <= 2.0 ** -8 * xr.grad.abs() + 1e-4).all()
    for got, ref in ((dg, gr.grad), (db, br.grad)):
        assert ((got.double() - ref).abs() <= 2.0 ** -18 * rows + 1e-4).all()


@pytest.mark.parametrize("kind", ["Q4_K", "Q6_K"])
@pytest.mark.parametrize("N,K", [(1, 256), (3, 1280), (5461, 768), (16384, 256), (4100, 1024)])      # 1, 15, 16383, 16384 and 16400 superblocks
def test_expansion_of_any_number_of_superblocks(kind, N, K):
    from openagents_b200.gguf import GgmlType
    from openagents_b200.gguf import torch_codecs as tc
    from openagents_b200.models.qweight import QWeight, RawTensor
    t = GgmlType[kind]
    raw = tc.quantize(_randn(N, K, seed=87), t)
    out = torch.full((N + 1, K), 7.0, dtype=torch.bfloat16, device=DEV)
    QWeight.from_raw(RawTensor(t, (N, K), raw)).dequant_into(out[:N])
    want = tc.dequantize(raw, t, (N, K))
    # one rounding to bf16, of a multiply-add in 32 bits whose terms are of the block's size
    assert ((out[:N].float() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -20 * want.abs().max()).all() and (out[N] == 7.0).all()


@pytest.mark.parametrize("T,Hq,Hkv", [(128, 16, 8), (128, 15, 8), (146, 13, 7), (147, 13, 7), (127, 64, 8)])      # 2^18 values, below and above; 128 tokens
@pytest.mark.parametrize("style", ["pairs", "half"])
def test_rope_kv_either_side_of_the_wide_kernel(T, Hq, Hkv, style):
    """Against the same tokens a few at a time."""
    ops, hd, st = _ops(), 64, 0 if style == "pairs" else 1
    qkv, pos = _randn(T, (Hq + 2 * Hkv) * hd, seed=88), torch.arange(T, device=DEV).int()
    tab = ops.rope_table(256, hd, 10000.0, DEV)
    outs = []
    for step in (T, 50):
        kc = torch.zeros((T // 16 + 1, Hkv, 16, hd), dtype=torch.float16, device=DEV)
        vc, q16 = torch.zeros_like(kc), torch.empty((T, Hq * hd), dtype=torch.float16, device=DEV)
        for lo in range(0, T, step):
            s = slice(lo, lo + step)
            ops.rope_kv(qkv[s], pos[s], pos[s], None, q16[s], kc, vc, Hq, Hkv, hd, 16, 10000.0, st, 0.125, table=tab)
        outs.append((q16, kc, vc))
    for a, b in zip(*outs):                                        # a contracted multiply-add may round differently
        assert torch.allclose(a.float(), b.float(), rtol=2.0 ** -10, atol=1e-6)


@pytest.mark.parametrize("T,D", [(148, 8192), (149, 8192), (148, 4128), (149, 4128), (128, 4096), (127, 4096)])
def test_rmsnorm_either_side_of_the_many_row_kernel(T, D):
    ops = _ops()
    x, g = _randn(T, D, seed=89), _randn(D, seed=90)
    hf, hb = torch.empty((T, D), device=DEV), torch.empty((T, D), dtype=torch.bfloat16, device=DEV)
    ops.rmsnorm(x, g, 1e-5, hb=hb, hf=hf)
    ref = x.double() * torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True) + 1e-5) * g.double()
    assert ((hf - ref).abs() <= 2.0 ** -20 * ref.abs() + 1e-12).all() and torch.equal(hb, hf.bfloat16())

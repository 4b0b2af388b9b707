"""GPU numerics of the kernels that share one result between several CTAs, at the sizes where they
can go wrong: edges of tiles, reductions shorter than the split, ranks that fill several 64-column
groups, odd head groups."""

import pytest
import torch

from lorafusion_b200.utils.testing import assert_close_two_rounds

pytestmark = pytest.mark.gpu


def _rand(*shape, scale=1.0, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32) * scale).to(torch.bfloat16)


def _f32mm(a, b):
    torch.backends.cuda.matmul.allow_tf32 = False
    return a.float() @ b.float()


@pytest.mark.parametrize("split", [1, 2, 4, 8])
@pytest.mark.parametrize("R,K", [(64, 200), (128, 520), (192, 1032), (256, 4096)])
def test_rank_wide_products(split, R, K, monkeypatch):
    """S', dS, dB and dA for every split, down to slices without a single block (K = 200 has four
    blocks); ragged last tile, three segments of different lengths, one tile without an adapter.
    Twice the same bits: the partial sums are added in a fixed order."""
    from lorafusion_b200.ops import lora_kernels as lk
    from lorafusion_b200.ops.philox import dropout_threshold, keep_mask

    n, M, p = 3, 128 * 5 + 72, [0.1, 0.0, 0.5]
    segs = [(1, 0, 128), (-1, 128, 256), (2, 256, 640), (0, 640, M)]
    tile_adapter = torch.tensor([1, -1, 2, 2, 2, 0], dtype=torch.int32, device="cuda")
    x, s, a, b = _rand(M, K, seed=1), _rand(M, R, scale=0.1, seed=2), _rand(n, R, K, scale=0.05, seed=3), \
        _rand(n, K, R, scale=0.05, seed=4)
    alpha = torch.tensor([2.0, 0.5, 1.0], device="cuda")
    drop = lk.DropoutSpec(seed=(5 << 32) | 77, stream_id=9, row_offset=3, col_offset=16,
                          adapter_thresh16=torch.tensor([dropout_threshold(v) for v in p], dtype=torch.int32, device="cuda"),
                          adapter_inv_keep=torch.tensor([1 / (1 - v) for v in p], device="cuda"))
    monkeypatch.setattr(lk, "reduction_split", lambda *_: split)
    table = lk.SegmentTable(segs, torch.device("cuda"), total_rows=M)
    out = []
    for _ in range(2):
        da, db = torch.ones(n, R, K, device="cuda"), torch.ones(n, K, R, device="cuda")
        lk.lora_da(x, s, table, da, dropout=drop)
        lk.lora_db(x, s, table, db)
        out.append((lk.lora_down(x, a, tile_adapter=tile_adapter, adapter_scale=alpha, dropout=drop),
                    lk.lora_ds(x, b, tile_adapter=tile_adapter, adapter_scale=alpha), da, db))
    assert all(torch.equal(u, v) for u, v in zip(*out))
    down, ds, da, db = out[0]
    assert not down[128:256].any() and not ds[128:256].any()
    for ad, r0, r1 in segs:
        if ad < 0:
            continue
        keep = keep_mask(r1 - r0, K, p[ad], (5 << 32) | 77, 9, row_offset=3 + r0, col_offset=16).cuda()
        xh = torch.where(keep, x[r0:r1].float() / (1 - p[ad]), torch.zeros((), device="cuda")).to(torch.bfloat16)
        assert_close_two_rounds(down[r0:r1], alpha[ad] * _f32mm(xh, a[ad].t()), msg=f"S' {ad}")
        assert_close_two_rounds(ds[r0:r1], alpha[ad] * _f32mm(x[r0:r1], b[ad]), msg=f"dS {ad}")
        # fp32 sums of at most 384 products of magnitude 0.1 in another order
        assert_close_two_rounds(db[ad], 1 + _f32mm(x[r0:r1].t(), s[r0:r1]), rtol=1e-4, atol=1e-4, msg=f"dB {ad}")
        assert_close_two_rounds(da[ad], 1 + _f32mm(s[r0:r1].t(), xh), rtol=1e-4, atol=1e-4, msg=f"dA {ad}")


def test_philox_with_row_and_column_parts_taken_out_drops_everything_at_p_near_one():
    """A threshold of 65536 (p above 1 - 2^-17) does not fit the packed comparison: all is dropped."""
    from lorafusion_b200.ops import lora_kernels as lk

    x, a = _rand(130, 128), _rand(1, 64, 128)
    s = lk.lora_down(x, a, tile_adapter=None, adapter_scale=None, dropout=lk.DropoutSpec(p=1 - 2.0 ** -18))
    assert not s.any()


@pytest.mark.parametrize("M,N,K,ctas", [(600, 1104, 16392, 8), (1000, 2816, 6000, 20), (513, 256, 5000, 0)])
@pytest.mark.parametrize("p", [None, 0.0, 0.1])
def test_pair_products_with_the_last_wave_cut(M, N, K, ctas, p):
    """Forward (``p`` None, with bias) and dX products of the CTA-pair kernels whose last wave is cut
    along the reduction: same results as fp32 math, twice the same bits."""
    from lorafusion_b200.ops import _native as nv
    from lorafusion_b200.ops.gemm import _pair_scratch_bytes, launch_gemm
    from lorafusion_b200.ops.philox import dropout_threshold, keep_mask

    assert _pair_scratch_bytes(M, N, K, ctas, 0) > 0, "the case is meant to be cut"
    R = 64
    x, s = _rand(M, K, seed=1), _rand(M, R, scale=0.2, seed=2)
    w = _rand(N, K, scale=0.03, seed=3) if p is None else _rand(K, N, scale=0.03, seed=3)
    b2 = _rand(N, R, scale=0.2, seed=4) if p is None else _rand(R, N, scale=0.2, seed=4)
    bias = _rand(N, seed=5) if p is None else None
    kw = dict(a=x, b=w, M=M, N=N, K=K, bn=256, a2=s, b2=b2, K2=R, max_ctas=ctas, pair=True)
    if p is None:
        kw.update(bias=bias, b2_adapter_rows=N)
        ref = _f32mm(x, w.t()) + _f32mm(s, b2.t()) + bias.float()
    else:
        kw.update(b_mn=True, b2_mn=True, b2_adapter_rows=R)
        slab = _f32mm(s, b2)
        if p > 0:
            kw.update(nacc=2, epi=nv.EPI_BF16_DROPMIX, thresh16=dropout_threshold(p), inv_keep=1 / (1 - p), seed=7,
                      stream_id=2)
            slab = torch.where(keep_mask(M, N, p, 7, 2).cuda(), slab / (1 - p), torch.zeros((), device="cuda"))
        ref = _f32mm(x, w) + slab
    outs = []
    for _ in range(2):
        out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
        launch_gemm(out=out, **kw)
        outs.append(out)
    assert torch.equal(*outs)
    assert_close_two_rounds(outs[0], ref, msg=f"pair product {M} x {N} x {K}")


@pytest.mark.parametrize("lens,Hq,Hkv", [([1], 1, 1), ([129, 3, 128], 3, 1), ([300, 257], 10, 2), ([700, 31, 513], 8, 1),
                                         ([128] * 150, 5, 1), ([65], 2, 2), ([200, 7], 17, 1), ([130], 4, 4),
                                         ([700, 31, 513], 4, 4), ([128, 1, 2000], 2, 2), ([600] * 50, 5, 5)])
def test_attention_head_groups(lens, Hq, Hkv):
    """Odd groups (the last pair of heads has one), groups split over CTAs (few tiles) and whole
    (150 tiles), sequences around the tile size; forward, and backward with its row deltas (warps on 2, 4, 8
    or 16 heads, 17 leave one to a group of its own).  Groups of one head have a kernel of their own, in either order
    of launch (fifty sequences of five heads: more than eight waves)."""
    from lorafusion_b200.ops import attention as att

    D, M = 128, sum(lens)
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    qkv = _rand(M, (Hq + 2 * Hkv) * D, scale=0.7, seed=5).requires_grad_(True)
    dout = _rand(M, Hq * D, seed=6)
    out = att.packed_attention(qkv, att.build_attn_tiles(cu, "cuda"), Hq, Hkv)
    grad, = torch.autograd.grad(out, [qkv], dout)
    ref_in = qkv.detach().float().requires_grad_(True)
    parts = ref_in.split([Hq * D, Hkv * D, Hkv * D], dim=1)
    ref = att.attention_reference(parts[0].reshape(M, Hq, D), parts[1].reshape(M, Hkv, D), parts[2].reshape(M, Hkv, D),
                                  cu).reshape(M, Hq * D)
    ref_grad, = torch.autograd.grad(ref, [ref_in], dout.float())
    # bf16 probabilities and outputs: 2^-8 of values around one
    assert_close_two_rounds(out, ref, atol=2e-2, msg="attention fwd")
    assert_close_two_rounds(grad, ref_grad, atol=5e-2, scale_atol_by_rms=True, msg="attention bwd")


def test_nf4_codes_at_the_midpoints():
    """Codes next to every midpoint, blocks of zeros, and a block count that leaves the last CTA
    nearly empty: the same codes as the CPU quantiser; a NaN weight encodes as the CPU's 0th code."""
    from lorafusion_b200.ops import nf4

    mids = (nf4.NF4_CODE[:-1] + nf4.NF4_CODE[1:]) / 2
    vals = torch.cat([mids, -mids, torch.tensor([0.0, 1.0, -1.0])]).to(torch.bfloat16)
    grid = torch.cat([vals, (vals.float() * 1.004).to(torch.bfloat16), (vals.float() * 0.996).to(torch.bfloat16)])
    w = torch.zeros(33, 64 * 9, dtype=torch.bfloat16)
    w.view(-1)[64:64 + 64 * 4] = torch.nn.functional.pad(grid, (0, 256 - grid.numel()))
    w.view(-1)[128::64] = 1.0   # absmax of the blocks that follow
    w[20:] = torch.randn(13, 64 * 9).to(torch.bfloat16)
    q_gpu, q_cpu = nf4.quantize_nf4(w.cuda()), nf4.quantize_nf4(w)
    assert torch.equal(q_gpu.packed.cpu(), q_cpu.packed)
    assert (q_gpu.absmax_q.cpu().int() - q_cpu.absmax_q.int()).abs().max() <= 1
    assert abs(q_gpu.offset - q_cpu.offset) < 1e-6 and torch.allclose(q_gpu.nested.cpu(), q_cpu.nested, rtol=1e-5)
    ref = nf4.dequantize_nf4_reference(q_gpu)
    assert torch.allclose(nf4.dequantize_nf4(q_gpu).float(), ref.float(), rtol=1e-2, atol=1e-6)
    w[0, 5] = float("nan")
    assert int(nf4.quantize_nf4(w.cuda()).packed[0, 2]) & 15 == 0


@pytest.mark.parametrize("n", [1, 17])
def test_adapters_are_packed_and_gradients_unpacked(n):
    """Rank 4 to 40, a missing adapter, an unaligned and a strided and an fp32 source; more adapters than
    one launch takes."""
    from lorafusion_b200.ops import lora_kernels as lk
    from lorafusion_b200.ops.lora import _adapter_entry

    K, N, R = 200, 72, 64
    dev = torch.device("cuda", torch.cuda.current_device())
    ab = []
    for i in range(n):
        r = (4, 40, 9)[i % 3]
        a, b = _rand(r, K, seed=i), _rand(N, r, seed=100 + i)
        if i % 4 == 1:
            a = _rand(r, K + 1, seed=i)[:, 1:]
        if i % 4 == 2:
            a, b = a.float(), _rand(r, N, seed=100 + i).t()
        ab.append((None, None) if i == 3 else (a, b))
    entries = [_adapter_entry(a, b, K, N, dev) for a, b in ab]
    a_all, b_all = lk.pack_stacks(entries, K, N, R, dev)
    da, db = torch.randn(n, R, K, device=dev), torch.randn(n, N, R, device=dev)
    grads = [(None, None, 0) if a is None else (torch.empty(a.shape, dtype=torch.bfloat16, device=dev),
                                                None if i == 0 else torch.empty(b.shape, dtype=torch.bfloat16, device=dev),
                                                a.shape[0]) for i, (a, b) in enumerate(ab)]
    lk.unpack_grads(grads, da, db, K, N, R)
    for i, (a, b) in enumerate(ab):
        ra, rb = torch.zeros(R, K, device=dev), torch.zeros(N, R, device=dev)
        if a is not None:
            r = a.shape[0]
            ra[:r], rb[:, :r] = a.float(), b.float()
            assert torch.equal(grads[i][0], da[i, :r].to(torch.bfloat16))
            assert grads[i][1] is None or torch.equal(grads[i][1], db[i, :, :r].to(torch.bfloat16))
        assert torch.equal(a_all[i].float(), ra.to(torch.bfloat16).float())
        assert torch.equal(b_all[i].float(), rb.to(torch.bfloat16).float())


@pytest.mark.parametrize("M", [1, 100, 640])
@pytest.mark.parametrize("p", [0.0, 0.1])
def test_one_call_layer_equals_its_building_blocks(M, p):
    """``linear_fwd`` / ``linear_bwd`` against the separate launches, and a single adapter without tables
    against the same batch with them: the same bits, bias and precomputed S' included; no dX wanted."""
    from lorafusion_b200.ops import lora_kernels as lk
    from lorafusion_b200.ops.batch_info import single_adapter_batch_info

    K, N, R = 264, 520, 64
    x, dy, w, bias = _rand(M, K, seed=1), _rand(M, N, seed=2), _rand(N, K, scale=0.05, seed=3), _rand(N, seed=4)
    a, b = _rand(1, R, K, scale=0.05, seed=5), _rand(1, N, R, scale=0.05, seed=6)
    one = lk.OneAdapter(M, 2.0, p, 11)
    table = single_adapter_batch_info(M, 16, 2.0, p, device="cuda", seed=11)
    drop = one.dropout_spec(5)
    assert drop == table.dropout_spec(5) or p == 0
    s = lk.lora_down(x, a, tile_adapter=None, adapter_scale=None, scale=2.0, dropout=drop)
    y = lk.base_lora_fwd(x, w, s, b, tile_adapter=None, bias=bias)
    ds = lk.lora_ds(dy, b, tile_adapter=None, adapter_scale=None, scale=2.0)
    dx = lk.base_lora_dx(dy, w, ds, a, tile_adapter=None, dropout=drop)
    da, db = torch.zeros(1, R, K, device="cuda"), torch.zeros(1, N, R, device="cuda")
    segs = lk.SegmentTable([(0, 0, M)], torch.device("cuda"), total_rows=M)
    lk.lora_db(dy, s, segs, db)
    lk.lora_da(x, ds, segs, da, dropout=drop)
    for info in (one, table):
        got_y, got_s = lk.linear_fwd(x, w, a, b, info, drop, bias=bias)
        assert torch.equal(got_y, y) and torch.equal(got_s, s)
        assert torch.equal(lk.linear_fwd(x, w, a, b, info, drop, bias=bias, s=s)[0], y)
        got_da, got_db = torch.zeros_like(da), torch.zeros_like(db)
        assert torch.equal(lk.linear_bwd(dy, x, s, w, a, b, info, drop, got_da, got_db, True), dx)
        assert torch.equal(got_da, da) and torch.equal(got_db, db)
        assert lk.linear_bwd(dy, x, s, None, a, b, info, drop, None, None, False) is None


@pytest.mark.parametrize("K,N", [(264, 520), (5000, 256), (256, 5000)])
@pytest.mark.parametrize("ps", [(0.0, 0.0, 0.0), (0.1, 0.1, 0.1), (0.1, 0.0, 0.5)])
def test_one_call_layer_of_several_adapters_equals_its_building_blocks(K, N, ps):
    """Three adapters and a tile without one, stacks cut out of longer and wider ones, a pitched ``S'``, a mask of a
    shard (row and column offset); with 5000 features the last wave of the forward's or of dX's big product is cut:
    the same bits as the separate launches."""
    from dataclasses import replace

    from lorafusion_b200.ops import lora_kernels as lk
    from lorafusion_b200.ops.batch_info import prepare_multi_lora_batch_info
    from lorafusion_b200.ops.gemm import _pair_scratch_bytes

    R, n, M = 64, 3, 640
    info = prepare_multi_lora_batch_info([100, 128, 128, 200], [1, -1, 0, 2], [16, 0, 16, 16],
                                         [ps[1], 0.0, ps[0], ps[2]], [2.0, 0.0, 0.5, 1.0], device="cuda",
                                         seed=(3 << 32) | 5)
    assert info.total_padded_tokens == M
    assert (_pair_scratch_bytes(M, N, K, 0, 0) > 0) == (K == 5000)
    assert (_pair_scratch_bytes(M, K, N, 0, 0) > 0) == (N == 5000)
    drop = replace(info.dropout_spec(5), row_offset=256, col_offset=512)
    x, dy, w = _rand(M, K, seed=1), _rand(M, N, seed=2), _rand(N, K, scale=0.05, seed=3)
    a, b = _rand(n, 2 * R, K, scale=0.05, seed=5)[:, R:], _rand(n, N, R + 64, scale=0.05, seed=6)[:, :, 64:]
    ta, sc, segs = info.tile_adapter, info.adapter_scale, info.segment_table
    s = lk.lora_down(x, a, tile_adapter=ta, adapter_scale=sc, dropout=drop)
    y = lk.base_lora_fwd(x, w, s, b, tile_adapter=ta)
    ds = lk.lora_ds(dy, b, tile_adapter=ta, adapter_scale=sc)
    dx = lk.base_lora_dx(dy, w, ds, a, tile_adapter=ta, dropout=drop)
    da, db = torch.zeros(n, R, K, device="cuda"), torch.zeros(n, N, R, device="cuda")
    lk.lora_db(dy, s, segs, db)
    lk.lora_da(x, ds, segs, da, dropout=drop)
    got_y, got_s = lk.linear_fwd(x, w, a, b, info, drop)
    assert torch.equal(got_y, y) and torch.equal(got_s, s)
    pitched = torch.full((M, R + 8), float("nan"), dtype=torch.bfloat16, device="cuda")[:, 8:]
    pitched.copy_(s)
    assert torch.equal(lk.linear_fwd(x, w, None, b, info, drop, s=pitched)[0], y)
    got_da, got_db = torch.zeros_like(da), torch.zeros_like(db)
    assert torch.equal(lk.linear_bwd(dy, x, pitched, w, a, b, info, drop, got_da, got_db, True), dx)
    assert torch.equal(got_da, da) and torch.equal(got_db, db)


def test_fused_multi_lora_gradients_of_a_partly_missing_adapter():
    """``A`` missing while ``B`` is given: that adapter contributes nothing and its ``B`` gets no gradient; the
    other one's gradients are those of a layer that holds it alone.  Wrong shapes and types are refused."""
    from lorafusion_b200.ops import fused_linear_lora, fused_linear_multi_lora

    x, w = _rand(256, 128, seed=1).requires_grad_(True), _rand(264, 128, scale=0.05, seed=2)
    a, b, b2 = (_rand(*s, scale=0.1, seed=i).requires_grad_(True) for i, s in enumerate([(8, 128), (264, 8), (264, 4)], 3))
    y = fused_linear_multi_lora(x, w, lora_a_list=[a, None], lora_b_list=[b, b2], seq_len_list=[256], lora_idx_list=[0],
                                alpha_list=[2.0])
    dy = _rand(256, 264, seed=9)
    dx, da, db, none = torch.autograd.grad(y, [x, a, b, b2], dy, allow_unused=True)
    alone = fused_linear_lora(x, w, a, b, 2.0)
    assert none is None and torch.equal(y, alone)
    for got, want in zip((dx, da, db), torch.autograd.grad(alone, [x, a, b], dy)):
        assert torch.equal(got, want)
    with pytest.raises(ValueError):
        fused_linear_lora(x.float(), w, a, b, 2.0)
    with pytest.raises(ValueError):
        fused_linear_lora(x, w, a[:, :64], b, 2.0)


@pytest.mark.parametrize("V", [1, 64, 1000, 4096, 4097, 50257])
def test_cross_entropy_stays_inside_its_row(V):
    """Labels in the first and last column, ignored ones and ones of V or more (up to the next row and past the last):
    rows with a valid label get exactly what they get alone, columns past V and the memory behind stay as they were,
    and a row whose label has no column gets softmax * grad_scale."""
    from lorafusion_b200.ops import elementwise as ew

    ld, scale = V // 8 * 8 + 16, 0.25
    labels = [0, V, V - 1, V + 7, -1, ld + 3, V // 2, 5 * V]
    buf = _rand(len(labels) + 2, ld, seed=1)
    before = buf.clone()
    lab = torch.tensor(labels, dtype=torch.int32, device="cuda")
    loss = ew.cross_entropy_inplace(buf[:len(labels), :V], lab, scale)
    assert torch.equal(buf[:, V:], before[:, V:]) and torch.equal(buf[len(labels):], before[len(labels):])
    for i, label in enumerate(labels):
        logits = before[i, :V].float()
        want = logits.softmax(0)
        if 0 <= label < V:
            want[label] -= 1
        elif label < 0:
            want.zero_()
        # bf16 results (2^-9 of the value) of fp32 exponentials
        assert torch.allclose(buf[i, :V].float(), want * scale, rtol=6e-3, atol=1e-6), label
        ref = 0.0 if label < 0 else float(logits.logsumexp(0) - logits[min(label, V - 1)])
        assert abs(float(loss[i]) - ref) < 1e-3
        alone = before[i:i + 1].clone()
        if label < V:
            ew.cross_entropy_inplace(alone[:, :V], lab[i:i + 1], scale)
            assert torch.equal(alone[0], buf[i]), label


@pytest.mark.parametrize("M,heads,D", [(1, 1, 128), (19001, 1, 16), (4777, 1, 128), (1201, 5, 128), (33, 40, 128),
                                       (599, 2, 64), (7, 3, 256), (65, 2, 64)])
def test_rope_with_several_tokens_a_block(M, heads, D):
    """Token counts that leave the last block ragged; the heads behind the rotated ones and the rows behind the batch
    stay as they were."""
    from lorafusion_b200.ops import elementwise as ew

    qkv = _rand(M + 70, (heads + 1) * D, seed=3)
    before = qkv.clone()
    pos = torch.randint(0, 50, (M,), device="cuda", dtype=torch.int32)
    ang = torch.rand(50, D // 2, device="cuda") * 6
    ew.rope_inplace(qkv[:M], pos, ang.cos(), ang.sin(), heads, D)
    c, s = ang.cos()[pos.long()][:, None], ang.sin()[pos.long()][:, None]
    lo, hi = before[:M, :heads * D].float().view(M, heads, 2, D // 2).unbind(2)
    ref = torch.stack([lo * c - hi * s, hi * c + lo * s], dim=2).reshape(M, heads * D)
    # fp32 arithmetic rounded to bf16 once: half an ulp is 2^-9 of the value, plus cancellation of fp32 products
    assert torch.allclose(qkv[:M, :heads * D].float(), ref, rtol=4e-3, atol=1e-5)
    assert torch.equal(qkv[:M, heads * D:], before[:M, heads * D:]) and torch.equal(qkv[M:], before[M:])


@pytest.mark.parametrize("M,I", [(1, 8), (300, 8), (19001, 8), (9001, 24), (2501, 64), (1187, 1000), (33, 2056),
                                 (3, 4104), (5, 8200)])
def test_swiglu_backward_of_short_and_long_rows(M, I):
    """Several rows a CTA (long batches of short rows), one row a CTA and rows in pieces; ragged last CTAs and odd
    vector counts."""
    from lorafusion_b200.ops import elementwise as ew

    gu, d = _rand(M, 2 * I, seed=1), _rand(M, I, seed=2)
    leaf = gu.float().requires_grad_(True)
    g, u = leaf.split(I, dim=1)
    ref, = torch.autograd.grad(torch.nn.functional.silu(g) * u, [leaf], d.float())
    # fp32 arithmetic with an approximate exponential (2^-22), rounded to bf16 once
    assert torch.allclose(ew.swiglu_bwd(d, gu).float(), ref, rtol=5e-3, atol=1e-5)


@pytest.mark.parametrize("rows,ld,col0,cols", [(700, 30, 3, 24), (1, 12289, 0, 12289), (333, 7, 0, 7),
                                               (300, 64, 16, 16)])
def test_adam_regions_of_any_size(rows, ld, col0, cols):
    """One update of regions with odd sizes (the last one vectorisable), longer than what the CTAs of a work item take
    in one go: weights, moments, bf16 copy and cleared gradient; memory around the region untouched."""
    from lorafusion_b200.ops import elementwise as ew

    n, off, st = rows * ld, 12, 8
    g0 = torch.Generator(device="cuda").manual_seed(7)
    grad, mas, m, v = (torch.rand(k, generator=g0, device="cuda") + 0.1 for k in [n + 40] + [rows * cols + 20] * 3)
    work = torch.full((n + 40,), 3.0, dtype=torch.bfloat16, device="cuda")
    want = [t[st:st + rows * cols].clone() for t in (mas, m, v)]
    before = [t.clone() for t in (grad, mas, m, v)]
    table = torch.tensor([[off, rows, ld, col0, cols, st]], dtype=torch.int64, device="cuda")
    ew.adam_chunks(table, grad, mas, m, v, work, lr=0.01, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=1,
                   grad_scale=0.5)
    g = 0.5 * before[0][off:off + n].view(rows, ld)[:, col0:col0 + cols].reshape(-1)
    want[1] = 0.9 * want[1] + 0.1 * g
    want[2] = 0.95 * want[2] + 0.05 * g * g
    want[0] = want[0] * (1 - 0.01 * 0.1) - 0.01 * (want[1] / (1 - 0.9)) / ((want[2] / (1 - 0.95)).sqrt() + 1e-8)
    # fp32 with approximate divisions and roots (2^-22) of values around one
    for got, ref, old in zip((mas, m, v), want, before[1:]):
        assert torch.allclose(got[st:st + rows * cols], ref, rtol=1e-5, atol=1e-6)
        assert torch.equal(got[:st], old[:st]) and torch.equal(got[st + rows * cols:], old[st + rows * cols:])
    copy = torch.full((rows, ld), 3.0, dtype=torch.bfloat16, device="cuda")
    copy[:, col0:col0 + cols] = mas[st:st + rows * cols].to(torch.bfloat16).view(rows, cols)
    assert torch.equal(work[off:off + n], copy.view(-1)) and (work[:off] == 3).all() and (work[off + n:] == 3).all()
    assert not grad[off:off + n].any() and torch.equal(grad[off + n:], before[0][off + n:])


@pytest.mark.parametrize("blocks", [1, 127, 128, 129, 300, 7104 * 16 + 5])
@pytest.mark.parametrize("double_quant", [True, False])
def test_nf4_expansion_around_the_work_of_a_cta(blocks, double_quant):
    """A CTA expands 128 blocks of 64 codes at a time; 888 persistent ones (second-level scales) or one a piece."""
    from lorafusion_b200.ops import nf4

    q = nf4.quantize_nf4(_rand(blocks, 64, seed=2), double_quant)
    out = torch.full((blocks + 2, 64), 7.0, dtype=torch.bfloat16, device="cuda")
    nf4.dequantize_nf4(q, out=out[:blocks])
    # the product of two fp32 values, rounded to bf16; the scale may be fused (2^-24)
    assert torch.allclose(out[:blocks].float(), nf4.dequantize_nf4_reference(q).float(), rtol=8e-3, atol=1e-6)
    assert (out[blocks:] == 7).all()


@pytest.mark.parametrize("H", [8, 64, 2048, 2056, 8200, 16384])
@pytest.mark.parametrize("with_residual", [False, True])
def test_rmsnorm_backward_of_short_and_long_rows(H, with_residual):
    """Every number of vectors a thread keeps (1, 2, 5 to 8), few columns and the widest rows."""
    from lorafusion_b200.ops import elementwise as ew

    M = 37
    x, w, dy, dres = _rand(M, H, seed=1), _rand(H, seed=2), _rand(M, H, seed=3), _rand(M, H, seed=4)
    _, h, rstd = ew.rmsnorm_fwd(x, w, 1e-5)
    leaf = x.float().requires_grad_(True)
    y = leaf * torch.rsqrt(leaf.pow(2).mean(1, keepdim=True) + 1e-5) * w.float()
    ref, = torch.autograd.grad(y, [leaf], dy.float())
    if with_residual:
        ref = ref + dres.float()
    got = ew.rmsnorm_bwd(dy, h, w, rstd, dres if with_residual else None)
    # fp32 sums in another order, rounded to bf16 once (2^-9 of values around one)
    assert torch.allclose(got.float(), ref, rtol=6e-3, atol=2e-3)


@pytest.mark.parametrize("p", [0.0, 0.1])
def test_multi_lora_of_an_adapter_with_several_segments(p):
    """Three segments of adapter 0 around one of adapter 1: gradients are those of all its tokens.  Frozen adapters may
    have short ones, too."""
    from lorafusion_b200.ops import fused_linear_multi_lora
    from lorafusion_b200.ops.philox import keep_mask

    K, N, lens, ids, alpha = 256, 384, [2100, 128, 300, 100], [0, 1, 0, 0], {0: 2.0, 1: 0.5}
    kw = dict(seq_len_list=lens, lora_idx_list=ids, alpha_list=[alpha[i] for i in ids], dropout_p_list=[p] * 4, seed=9,
              stream_id=2)
    starts = [0, 2176, 2304, 2688]
    M = 2816
    x, w = _rand(M, K, seed=1).requires_grad_(True), _rand(N, K, scale=0.05, seed=2)
    ab = [(_rand(8, K, scale=0.1, seed=3 + i).requires_grad_(True),
           _rand(N, 8, scale=0.1, seed=5 + i).requires_grad_(True)) for i in range(2)]
    for i, n in zip(starts, lens):   # (the rows between segments are padding)
        with torch.no_grad():
            x[i + n:(i + n + 127) // 128 * 128] = 0
    dy = _rand(M, N, seed=9)
    y = fused_linear_multi_lora(x, w, lora_a_list=[v[0] for v in ab], lora_b_list=[v[1] for v in ab], **kw)
    got = torch.autograd.grad(y, [x] + [t for v in ab for t in v], dy)
    leaves = [t.detach().float().requires_grad_(True) for t in [x] + [t for v in ab for t in v]]
    keep = keep_mask(M, K, p, 9, 2).cuda() if p > 0 else torch.ones(M, K, dtype=torch.bool, device="cuda")
    xh = torch.where(keep, leaves[0] / (1 - p), torch.zeros((), device="cuda"))
    ref = leaves[0] @ w.float().t()
    delta = torch.zeros_like(ref)
    for i, n, ad in zip(starts, lens, ids):
        rows = slice(i, (i + n + 127) // 128 * 128)
        delta[rows] = alpha[ad] * (xh[rows] @ leaves[1 + 2 * ad].t()) @ leaves[2 + 2 * ad].t()
    want = torch.autograd.grad(ref + delta, leaves, dy.float())
    assert_close_two_rounds(y, ref + delta, msg="y")
    for g, r, name in zip(got, want, ("dx", "dA0", "dB0", "dA1", "dB1")):
        # S' and dS are rounded to bf16 (2^-9) on the way into sums of up to 2500 terms
        assert_close_two_rounds(g, r, rtol=2e-2, atol=2e-2, scale_atol_by_rms=True, msg=name)
    frozen = [t.detach() for v in ab for t in v]
    short = dict(kw, seq_len_list=[128] * 4)
    xs = x.detach()[:512].requires_grad_(True)
    y = fused_linear_multi_lora(xs, w, lora_a_list=frozen[::2], lora_b_list=frozen[1::2], **short)
    assert torch.autograd.grad(y, [xs], dy[:512])[0].shape == (512, K)
    y = fused_linear_multi_lora(xs, w, lora_a_list=[v[0] for v in ab], lora_b_list=frozen[1::2], **short)
    with pytest.raises(ValueError):
        torch.autograd.grad(y, [ab[0][0]], dy[:512])


@pytest.mark.parametrize("split", [1, 2, 8])
@pytest.mark.parametrize("shift", [1, 2, 4])
def test_db_into_a_buffer_of_any_alignment(split, shift, monkeypatch):
    """fp32 accumulators that start on any float: the same bits as in an aligned buffer, nothing beside them written."""
    from lorafusion_b200.ops import lora_kernels as lk

    M, N, R, n = 700, 136, 64, 2
    monkeypatch.setattr(lk, "reduction_split", lambda *_: split)
    table = lk.SegmentTable([(1, 0, 384), (0, 384, 700)], torch.device("cuda"), total_rows=M)
    dy, s = _rand(M, N, seed=1), _rand(M, R, scale=0.1, seed=2)
    buf = torch.ones(n * N * R + 8, device="cuda")
    db = buf[shift:shift + n * N * R].view(n, N, R)
    lk.lora_db(dy, s, table, db)
    ref = torch.ones(n, N, R, device="cuda")
    lk.lora_db(dy, s, table, ref)
    assert torch.equal(db, ref) and (buf[:shift] == 1).all() and (buf[shift + n * N * R:] == 1).all()


def test_nf4_weights_share_no_code_table():
    """Writing into the table of one weight leaves the others, and those quantised later, as they are."""
    from lorafusion_b200.ops import nf4

    w = _rand(64, 512, seed=1)
    first, second = nf4.quantize_nf4(w), nf4.quantize_nf4(w)
    want = nf4.dequantize_nf4(second).clone()
    first.code256.zero_()
    with torch.inference_mode():
        third = nf4.quantize_nf4(w)
    for q in (second, third, nf4.quantize_nf4(w)):
        assert torch.equal(q.code256.cpu(), nf4.dynamic_code_8bit()) and torch.equal(nf4.dequantize_nf4(q), want)
    assert not nf4.quantize_nf4(w).code256.is_inference()


@pytest.mark.parametrize("V", [9, 1000, 4096, 4100, 32000, 50257])
@pytest.mark.parametrize("masked", [0.3, 0.97])
def test_cross_entropy_of_masked_logits(V, masked):
    """Logits of minus infinity, whole vectors of them in front of the finite ones too, and of the lowest finite value:
    they have no weight, and no NaN comes of them."""
    from lorafusion_b200.ops import elementwise as ew

    M, ld = 40, (V + 7) // 8 * 8
    buf = _rand(M, ld, seed=1, scale=3.0)
    g = torch.Generator(device="cuda").manual_seed(5)
    hide = torch.rand(M, ld, generator=g, device="cuda") < masked
    hide[:, 8:V // 2] = True          # the first vectors of most threads
    hide[:, 0] = False
    buf[hide] = float("-inf")
    buf[M // 2:] = torch.nan_to_num(buf[M // 2:], neginf=torch.finfo(torch.bfloat16).min)
    lab = torch.zeros(M, dtype=torch.int32, device="cuda")
    logits = buf[:, :V].float()
    loss = ew.cross_entropy_inplace(buf[:, :V], lab, 0.5)
    want = logits.softmax(1)
    want[:, 0] -= 1
    # fp32 sums with an approximate exponential (2^-22), gradients rounded to bf16 once
    assert torch.allclose(loss, logits.logsumexp(1) - logits[:, 0], rtol=1e-5, atol=1e-4)
    assert torch.allclose(buf[:, :V].float(), want * 0.5, rtol=6e-3, atol=1e-6)


def test_cross_entropy_of_a_single_nan_in_a_thread():
    """A thread that sees nothing but a NaN logit adds nothing to the row's sum, as ever: only its own column is NaN."""
    from lorafusion_b200.ops import elementwise as ew

    buf = _rand(3, 8, seed=2)
    buf[1, 4] = float("nan")
    loss = ew.cross_entropy_inplace(buf[:, :7], torch.zeros(3, dtype=torch.int32, device="cuda"), 1.0)
    assert loss.isfinite().all() and buf.isnan().nonzero().tolist() == [[1, 4]]

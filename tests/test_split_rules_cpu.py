"""The rules that decide how a result is shared between CTAs, on the CPU."""

import pytest
import torch


@pytest.mark.parametrize("tiles", [1, 3, 37, 64, 74, 128, 148, 149, 1000])
@pytest.mark.parametrize("k_blocks", [1, 3, 4, 16, 17, 128])
def test_reduction_split_keeps_all_pieces_resident(tiles, k_blocks):
    from lorafusion_b200.ops.lora_kernels import reduction_split

    c = reduction_split(tiles, k_blocks)
    assert c in (1, 2, 4, 8)
    assert c == 1 or (tiles * c <= 296 and k_blocks >= 2 * c)
    assert c == 8 or tiles * c * 2 > 296 or k_blocks < 4 * c   # or the next larger one would have been taken


def test_segment_rows_are_the_owned_segments_longest_first():
    from lorafusion_b200.ops.lora_kernels import SegmentTable, segment_rows

    segs = [(2, 0, 128), (-1, 128, 512), (0, 512, 512), (1, 512, 1024), (3, 1024, 1152)]
    assert segment_rows(segs) == [(1, 512, 1024, 0), (2, 0, 128, 0), (3, 1024, 1152, 0)]
    table = SegmentTable(segs, torch.device("cpu"))
    assert table.device_rows().tolist() == [list(r) for r in segment_rows(segs)]
    with pytest.raises(ValueError):
        SegmentTable([(0, 0, 128), (0, 128, 256)], torch.device("cpu")).device_rows()
    with pytest.raises(ValueError):
        SegmentTable([(0, 0, 100), (1, 100, 256)], torch.device("cpu")).device_rows()


def test_last_wave_is_cut_only_where_it_pays():
    """Scratch in bytes of 148 SMs (74 pairs): none for whole waves, short reductions and slices that would not
    fill the idle pairs; counters and partial tiles otherwise."""
    from lorafusion_b200.ops import _native as nv

    scratch = nv.cuda_lib().lf_gemm_pair_scratch
    tile = 256 * 256 * 4
    assert scratch(256 * 74, 256, 8192, 0) == 0          # one whole wave
    assert scratch(2048, 2048, 2048, 0) == 0             # 64 tiles of 32 blocks
    assert scratch(1000, 8192, 8192, 0) == 0             # 54 of 74 pairs busy: 216 slices would cost more
    assert scratch(2048, 4096, 128256, 0) == 54 * 4 * tile + 3584     # 128 tiles of 2004 blocks
    assert scratch(0, 256, 256, 0) == 0


def test_adapters_with_several_segments():
    """Accepted where the tokens of a segment used to be summed in chunks (fewer than 96 pieces of segment x 128
    features, a segment of 2048 tokens): the n-th segments of all adapters form the n-th launch.  Refused otherwise."""
    from lorafusion_b200.ops.lora_kernels import SegmentTable, segment_rows

    segs = [(0, 0, 128), (1, 128, 384), (0, 384, 2560), (-1, 2560, 2688), (1, 2688, 2816), (0, 2816, 2944)]
    assert segment_rows(segs) == [(1, 128, 384, 0), (0, 0, 128, 0), (0, 384, 2560, 0), (1, 2688, 2816, 0),
                                  (0, 2816, 2944, 0)]
    staged = torch.tensor([9] * 4 + [v for r in segment_rows(segs) for v in r], dtype=torch.int32)
    for table in (SegmentTable(segs, torch.device("cpu")),
                  SegmentTable(segs, torch.device("cpu"), staged=(staged, 4, 24))):
        assert table.repeats
        got = [[tuple(r) for r in rows.tolist()] for rows in table.passes(128 * 19)]
        assert got == [segment_rows(segs)[:2], segment_rows(segs)[2:4], segment_rows(segs)[4:]]
        with pytest.raises(ValueError):
            table.passes(128 * 19 + 1)      # 5 segments x 20 tiles
    with pytest.raises(ValueError):
        SegmentTable([(0, 0, 2047), (0, 2048, 2176)], torch.device("cpu")).passes(128)
    with pytest.raises(ValueError):
        SegmentTable([(0, 0, 1920), (0, 1920, 2176)], torch.device("cpu")).passes(128)
    assert len(SegmentTable([(0, 0, 2048), (0, 2048, 2176)], torch.device("cpu")).passes(128)) == 2
    one = SegmentTable([(0, 0, 128), (1, 128, 256)], torch.device("cpu"))
    assert not one.repeats and torch.equal(one.passes(10 ** 6)[0], one.device_rows()) and len(one.passes(64)) == 1


def test_frozen_adapters_may_have_several_segments(monkeypatch):
    """The input's gradient alone needs no work list: such a batch is not refused, and does not take the one-call
    path."""
    from lorafusion_b200.ops import lora as L
    from lorafusion_b200.ops import lora_kernels as lk
    from lorafusion_b200.ops.batch_info import prepare_multi_lora_batch_info

    seen = []
    for name in ("lora_ds", "lora_db", "lora_da", "base_lora_dx", "linear_bwd"):
        monkeypatch.setattr(lk, name, lambda *a, _n=name, **k: seen.append(_n))
    info = prepare_multi_lora_batch_info([128, 128], [0, 0], [8, 8], [0.0] * 2, [1.0] * 2, device="cpu")
    z = lambda *s: torch.zeros(*s, dtype=torch.bfloat16)  # noqa: E731
    stack = L.LoRAStack(z(1, 64, 128), z(1, 128, 64))
    L.lora_linear_backward(z(256, 128), z(256, 128), z(256, 64), z(128, 128), stack, info)
    assert seen == ["lora_ds", "base_lora_dx"]


@pytest.mark.parametrize("M,N,K,pairs", [
    # measured, alone against in pairs: 43 / 58, 48 / 63, 72 / 86, 61 / 74, 165 / 185, 24.2 / 25.9, 8.5 / 9.9 us
    (128, 19456, 4096, False), (100, 21504, 5120, False), (100, 22016, 8192, False), (384, 10240, 8192, False),
    (128, 57344, 8192, False), (128, 4096, 4096, False), (257, 512, 512, False),
    # 36.4 / 32.4, 57 / 48, 194 / 175, 62 / 50, 78 / 55 (cut), 85 / 71 us
    (128, 14336, 4096, True), (257, 8192, 8192, True), (511, 8192, 28672, True), (128, 10240, 8192, True),
    (300, 4096, 14336, True), (511, 19456, 4096, True),
])
def test_which_kernel_takes_a_product_of_few_rows(M, N, K, pairs):
    from lorafusion_b200.ops import gemm

    assert gemm._pair_is_faster(M, N, K, 0, 0) == pairs


def test_blocks_of_a_pair_count_waves_and_the_cut():
    from lorafusion_b200.ops import _native as nv

    blocks = nv.cuda_lib().lf_gemm_pair_blocks
    assert blocks(256 * 74, 256, 8192, 0) == 128 and blocks(256 * 75, 256, 640, 0) == 20    # one and two waves
    # 54 of 74 pairs busy with 2004 blocks in the second wave, cut in four: 3 / 4 of it, 30 + 0.27 * 54 * 4 on top
    assert blocks(2048, 4096, 128256, 0) == pytest.approx(2004 + 2004 * 0.75 + 30 + 0.27 * 216)
    assert blocks(0, 256, 256, 0) == 0

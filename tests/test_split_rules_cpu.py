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

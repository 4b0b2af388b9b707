"""What the one-call LoRA layer (``linear_fwd`` / ``linear_bwd``) hands to native code, on CPU tensors with the
library's entry points replaced: operands of a wrong type, shape or length are refused, strided ones are described
as they lie in memory."""

import ctypes as C

import pytest
import torch

from lorafusion_b200.ops import _native as nv
from lorafusion_b200.ops import lora_kernels as lk

M, K, N, R, n = 192, 264, 136, 64, 3


@pytest.fixture
def calls(monkeypatch):
    """The argument blocks of the native calls made, copied."""
    seen = []

    class Lib:
        def __getattr__(self, name):
            if name in ("lf_lora_linear_fwd", "lf_lora_linear_bwd"):
                def call(ref):
                    seen.append(nv.LfLoraLinearArgs.from_buffer_copy(ref._obj))
                    return 0
                return call
            return getattr(real, name)

    real = nv.cuda_lib()
    monkeypatch.setattr(nv, "cuda_lib", lambda: Lib())
    monkeypatch.setattr(nv, "err_word", lambda device: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(nv, "current_stream_ptr", lambda: 0)
    return seen


def _bf(*shape):
    return torch.zeros(*shape, dtype=torch.bfloat16)


def _operands(**change):
    """Valid operands of both directions, some of them replaced."""
    ops = dict(x=_bf(M, K), w=_bf(N, K), a=_bf(n, R, K), b=_bf(n, N, R), s=_bf(M, R), dy=_bf(M, N),
               da=torch.zeros(n, R, K), db=torch.zeros(n, N, R), drop=lk.NO_DROPOUT)
    ops.update(change)
    return ops


def _fwd(o, s=True):
    return lk.linear_fwd(o["x"], o["w"], o["a"], o["b"], lk.OneAdapter(M, 1.0, 0.0, 0), o["drop"],
                         s=o["s"] if s else None)


def _bwd(o, need_dx=True):
    return lk.linear_bwd(o["dy"], o["x"], o["s"], o["w"], o["a"], o["b"], lk.OneAdapter(M, 1.0, 0.0, 0), o["drop"],
                         o["da"], o["db"], need_dx)


FORWARD = {
    "A of another type": dict(a=torch.zeros(n, R, K)),
    "B of another type": dict(b=torch.zeros(n, N, R)),
    "S' of another type": dict(s=torch.zeros(M, R)),
    "A with a strided last dimension": dict(a=_bf(n, R, 2 * K)[:, :, ::2]),
    "S' with too few rows": dict(s=_bf(M - 1, R)),
    "S' of another rank": dict(s=_bf(M, 2 * R)),
}
BACKWARD = {
    "dy with fewer rows than x": dict(dy=_bf(M - 128, N)),
    "dy of another width": dict(dy=_bf(M, N + 8)),
    "S' with too few rows": dict(s=_bf(M - 1, R)),
    "S' of another type": dict(s=torch.zeros(M, R)),
    "dA of another type": dict(da=torch.zeros(n, R, K, dtype=torch.float64)),
    "dB of another type": dict(db=_bf(n, N, R)),
    "dA of another shape": dict(da=torch.zeros(n, R, K - 8)),
    "dB of another shape": dict(db=torch.zeros(n, N - 8, R)),
    "dA that is not contiguous": dict(da=torch.zeros(n, R, 2 * K)[:, :, :K]),
    "dB that is not contiguous": dict(db=torch.zeros(n, 2 * N, R)[:, ::2]),
    "A of another type": dict(a=torch.zeros(n, R, K)),
    "B of another type": dict(b=torch.zeros(n, N, R)),
}


@pytest.mark.parametrize("change", FORWARD, ids=str)
def test_forward_refuses(calls, change):
    with pytest.raises(ValueError):
        _fwd(_operands(**FORWARD[change]), s="S'" in change)
    assert not calls


@pytest.mark.parametrize("change", BACKWARD, ids=str)
def test_backward_refuses(calls, change):
    with pytest.raises(ValueError):
        _bwd(_operands(**BACKWARD[change]))
    assert not calls


def _read2d(ptr, rows, cols, ld):
    """The bf16 matrix that native code would read."""
    raw = (C.c_uint16 * ((rows - 1) * ld + cols)).from_address(ptr)
    flat = torch.frombuffer(raw, dtype=torch.int16).view(torch.bfloat16)
    return flat.as_strided((rows, cols), (ld, 1))


def test_strided_operands_are_described_as_they_lie(calls, monkeypatch):
    """Stacks cut out of wider or longer ones, and a pitched ``S'``: what the native call would read equals the
    operands, in both directions."""
    wide = lambda *s: torch.arange(int(torch.tensor(s).prod())).remainder(251).to(torch.bfloat16).view(*s)  # noqa: E731
    layouts = [dict(a=wide(n, 2 * R, K)[:, :R], b=wide(n, N + 8, R)[:, :N]),          # rows of longer stacks: copied
               dict(a=wide(n, R, K + 16)[:, :, 8:8 + K], b=wide(n, N, R + 64)[:, :, 64:]),   # pitched: read in place
               dict(s=wide(M, R + 64)[:, 64:])]
    seen = []
    lib = nv.cuda_lib()
    for entry in ("lf_lora_linear_fwd", "lf_lora_linear_bwd"):
        def call(ref):
            p = ref._obj
            seen.append([(name, _read2d(ptr, rows, cols, ld).clone()) for name, ptr, rows, cols, ld in (
                ("a", p.a_all, n * R, K, p.a_ld), ("b", p.b_all, n * N, R, p.b_ld), ("s", p.s, M, R, p.s_ld)) if ptr])
            return 0
        monkeypatch.setattr(type(lib), entry, staticmethod(call), raising=False)
    for change in layouts:
        o = _operands(**change)
        _fwd(o)              # with S': A is not read
        _fwd(o, s=False)     # S' is an output: whatever its memory holds
        _bwd(o)
        for i, names in ((-3, "bs"), (-2, "ab"), (-1, "abs")):
            got = dict(seen[i])
            for name in names:
                assert torch.equal(got[name], o[name].reshape(got[name].shape)), name
            assert i != -3 or "a" not in got
    assert len(seen) == 3 * len(layouts)


def test_what_a_direction_does_not_read_is_not_looked_at(calls):
    """A given ``S'`` makes ``A`` unused in the forward; without ``dA`` / ``dB`` / ``dX`` the backward reads neither
    ``x`` nor ``S'`` nor ``A`` nor ``w``."""
    _fwd(_operands(a=None))
    _bwd(_operands(x=None, da=None))
    _bwd(_operands(s=torch.zeros(1), db=None))
    _bwd(_operands(w=None, a=None), need_dx=False)
    assert len(calls) == 4


def test_offsets_of_a_sharded_mask_reach_the_kernels(calls):
    drop = lk.DropoutSpec(seed=1, stream_id=2, p=0.1, row_offset=384, col_offset=4096)
    _fwd(_operands(drop=drop), s=False)
    _bwd(_operands(drop=drop))
    assert [(c.row_offset, c.col_offset) for c in calls] == [(384, 4096)] * 2


def test_batches_put_together_by_hand(calls):
    """Without a tile table every token belongs to adapter 0, whose scale and segments count all the same; without scales
    they are one."""
    from dataclasses import replace

    from lorafusion_b200.ops.batch_info import prepare_multi_lora_batch_info

    info = prepare_multi_lora_batch_info([M], [0], [16], [0.0], [2.0], device="cpu")
    o = _operands()
    for batch in (replace(info, tile_adapter=None), replace(info, adapter_scale=None)):
        lk.linear_fwd(o["x"], o["w"], o["a"], o["b"], batch, o["drop"])
        lk.linear_bwd(o["dy"], o["x"], o["s"], o["w"], o["a"], o["b"], batch, o["drop"], o["da"], o["db"], True)
    ptr = lambda t: t.data_ptr()  # noqa: E731
    for c in calls[:2]:
        assert c.tile_adapter is None and c.adapter_scale == ptr(info.adapter_scale)
    for c in calls[2:]:
        assert c.tile_adapter == ptr(info.tile_adapter) and c.adapter_scale is None and c.scale == 1.0
    for c in calls[1::2]:
        assert c.seg_rows == ptr(info.segment_table.device_rows()) and c.num_segs == 1

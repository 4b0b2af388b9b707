"""Adapter ids and rows of a batch are checked against the adapters and rows given, before anything is launched."""

from dataclasses import replace

import pytest
import torch

from lorafusion_b200.ops import lora_kernels as lk
from lorafusion_b200.ops import lora as L
from lorafusion_b200.ops.batch_info import prepare_multi_lora_batch_info

K, N, R = 64, 128, 64


def _batch(ids=(0, 2), lens=(100, 200)):
    z = [16] * len(ids)
    return prepare_multi_lora_batch_info(list(lens), list(ids), z, [0.0] * len(ids), [1.0] * len(ids), device="cpu",
                                         num_adapters=max(ids) + 1)


def _call(info, n, rows, **kw):
    stack = L.LoRAStack(torch.zeros(n, R, K, dtype=torch.bfloat16), torch.zeros(n, N, R, dtype=torch.bfloat16), **kw)
    x, dy = torch.zeros(rows, K, dtype=torch.bfloat16), torch.zeros(rows, N, dtype=torch.bfloat16)
    w, s = torch.zeros(N, K, dtype=torch.bfloat16), torch.zeros(rows, R, dtype=torch.bfloat16)
    L.lora_linear_forward(x, w, stack, info)
    L.lora_linear_backward(dy, x, s, w, stack, info)


@pytest.fixture
def launched(monkeypatch):
    seen = []
    monkeypatch.setattr(lk, "linear_fwd", lambda *a, **k: seen.append("fwd") or (None, None))
    monkeypatch.setattr(lk, "linear_bwd", lambda *a, **k: seen.append("bwd"))
    return seen


@pytest.mark.parametrize("rows", [1, 128, 256, 300, 384])
def test_batches_that_fit_pass(launched, rows):
    """Fewer rows than the batch, a ragged last tile and adapters beyond those of the batch are all fine."""
    _call(_batch(), 3, rows)
    _call(_batch(), 5, rows)
    _call(_batch(ids=(-1, 0)), 1, rows)
    _call(replace(_batch(), total_padded_tokens=0), 3, rows)   # a batch put together by hand: the table counts
    assert launched == ["fwd", "bwd"] * 4


def test_an_adapter_that_is_not_given_is_refused(launched):
    for direction in (L.lora_linear_forward, L.lora_linear_backward):
        with pytest.raises(ValueError, match="adapter"):
            _call(_batch(), 2, 384)
    with pytest.raises(ValueError, match="adapter"):
        _call(_batch(), 3, 384, da=torch.zeros(2, R, K))
    with pytest.raises(ValueError, match="adapter"):   # no tile table: the work list of the gradients names it
        _call(replace(_batch(), tile_adapter=None), 2, 384)
    # its segment holds no tokens: no kernel meets the id
    _call(_batch(ids=(0, 2), lens=(100, 0)), 1, 128)
    assert launched == ["fwd"] + ["fwd", "bwd"]


def test_more_rows_than_the_batch_are_refused(launched):
    with pytest.raises(ValueError, match="rows"):
        _call(_batch(), 3, 385)
    assert not launched


def test_backward_alone_is_checked_too(launched):
    stack = L.LoRAStack(torch.zeros(2, R, K, dtype=torch.bfloat16), torch.zeros(2, N, R, dtype=torch.bfloat16))
    z = lambda *s: torch.zeros(*s, dtype=torch.bfloat16)  # noqa: E731
    with pytest.raises(ValueError, match="adapter"):
        L.lora_linear_backward(z(384, N), z(384, K), z(384, R), z(N, K), stack, _batch())
    with pytest.raises(ValueError, match="rows"):
        L.lora_linear_backward(z(512, N), z(512, K), z(512, R), z(N, K), stack, _batch(ids=(0, 1)))
    assert not launched


@pytest.mark.gpu
def test_fused_multi_lora_refuses_before_it_launches():
    z = lambda *s: torch.zeros(*s, dtype=torch.bfloat16, device="cuda")  # noqa: E731
    info = prepare_multi_lora_batch_info([100, 200], [0, 2], [8, 8], [0.0, 0.0], [1.0, 1.0], device="cuda",
                                         num_adapters=3)
    ab = dict(lora_a_list=[z(8, K)] * 3, lora_b_list=[z(N, 8)] * 3, batch_info=info)
    with pytest.raises(ValueError, match="adapter"):
        L.fused_linear_multi_lora(z(384, K), z(N, K), **dict(ab, lora_b_list=[z(N, 8)] * 2))
    with pytest.raises(ValueError, match="rows"):
        L.fused_linear_multi_lora(z(512, K), z(N, K), **ab)
    assert not L.fused_linear_multi_lora(z(384, K), z(N, K), **ab).any()

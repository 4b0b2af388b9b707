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

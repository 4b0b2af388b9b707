"""Calls of the C entry points that have nothing to do return without a launch, also on a machine without a GPU."""

import subprocess
import sys

CALLS = [
    "lf_rope_inplace(None, None, None, None, 4, 2, 0, 8, 0, None)",      # heads of no width
    "lf_rope_inplace(None, None, None, None, 4, 0, 128, 8, 0, None)",    # no heads to rotate
    "lf_rope_inplace(None, None, None, None, 0, 2, 128, 8, 0, None)",
    "lf_swiglu_fwd(None, None, 4, 0, None)",
    "lf_swiglu_bwd(None, None, None, 4, 0, None)",
    "lf_cross_entropy(None, None, None, 0, 8, 8, 1.0, None)",
    "lf_nf4_quantize(None, None, None, 0, None)",
    "lf_nf4_double_quantize(None, 0, None, None, None, None, None, None, None, None)",
    "lf_nf4_dequantize(None, None, None, None, None, 0.0, None, 0, None)",
]


def test_nothing_to_do():
    """In a process of its own: a division by zero in native code ends it."""
    lines = ["from lorafusion_b200.ops import _native as nv", "lib = nv.cuda_lib()"]
    lines += [f"print({i}, lib.{c}, flush=True)" for i, c in enumerate(CALLS)]
    done = subprocess.run([sys.executable, "-c", "\n".join(lines)], capture_output=True, text=True, timeout=300)
    assert done.stdout.split("\n")[:-1] == [f"{i} 0" for i in range(len(CALLS))], (done.returncode, done.stderr[-500:])

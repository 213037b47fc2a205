"""CPU: the rules that pick a form for a call, and what they take into account besides sizes."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def in_a_process_of_its_own(code):
    """Settings of torch that cannot be taken back stay out of the other tests."""
    done = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]


@pytest.mark.parametrize("setting,tf32", [
    ("m.fp32_precision = 'tf32'", True), ("m.allow_tf32 = True", True), ("torch.backends.fp32_precision = 'tf32'", True), ("m.allow_tf32 = True; m.fp32_precision = 'ieee'", False)])
def test_tf32_is_read_through_either_interface(setting, tf32):
    """The rule for f32 products reads the precision however a program has set it; torch's older getter raises after some of these."""
    in_a_process_of_its_own(f"import torch; from lit_llama_b200 import mixers; m = torch.backends.cuda.matmul\n{setting}\nassert mixers._tf32_products() is {tf32}")


def test_f32_products_of_no_entries_or_too_many_rows_stay_with_the_library():
    """Products that the tensor-core kernel refuses: a sum over nothing is zeros, and rows past its grid (16 * 65535) are products like others."""
    import torch
    from lit_llama_b200 import mixers

    w, rows = torch.empty(1024, 8), 16 * 65535
    assert mixers._f32_sizes(torch.empty(1024, 8), w) and mixers._f32_sizes(torch.empty(rows, 8), w)
    assert not mixers._f32_sizes(torch.empty(1024, 0), torch.empty(1024, 0)) and not mixers._f32_sizes(torch.empty(rows + 1, 8), w)
    assert not mixers._f32_sizes(torch.empty(1024, 16), w)


def test_calls_that_torch_follows_stay_with_torch():
    """Forward-mode derivatives, function transforms, tracing and modes see a product only where it is torch's; a default device does not count."""
    import torch
    from lit_llama_b200 import mixers
    from torch.utils.flop_counter import FlopCounterMode

    x, seen = torch.zeros(2, 2), []

    def look(t):
        seen.append(mixers._followed())
        return t + 1

    look(x)
    with torch.device("cpu"):
        look(x)
    assert seen == [False, False]
    with torch.autograd.forward_ad.dual_level():
        look(x)
    torch.vmap(look)(x)
    torch.jit.trace(look, x, check_trace=False)
    with FlopCounterMode(display=False):
        look(x)
    assert seen[2:] and all(seen[2:])

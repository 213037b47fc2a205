"""GPU: infinities and NaN in the operands of the prompt kernels reach the tokens that see them and no others."""
import ctypes as C
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF = torch.bfloat16
INF, NAN = math.inf, math.nan


@pytest.mark.parametrize("what,bad", [("v", INF), ("v", NAN), ("k", INF), ("k", NAN), ("q", -INF), ("beta", NAN)])
@pytest.mark.parametrize("delta", [0, 1])
def test_scan_outputs_before_a_bad_token_are_untouched(delta, what, bad):
    """A chunk of 16 tokens is computed at once; a token's operands must still reach no earlier token of its chunk: the same bits as without it."""
    from lit_llama_b200 import _seqlib as S

    T, H, K, V, at = 45, 3, 64, 32, 20
    g = torch.Generator(device=DEV).manual_seed(7)
    ops = {"q": torch.randn(T, H, K, generator=g, device=DEV), "k": torch.randn(T, H, K, generator=g, device=DEV) / 8,
           "v": torch.randn(T, H, V, generator=g, device=DEV), "beta": torch.randn(T, H, generator=g, device=DEV)}
    decay = torch.rand(T, H, K, generator=g, device=DEV) * 0.5 + 0.5
    state0 = torch.randn(1, H, V, K, generator=g, device=DEV)
    meta, lib = torch.zeros(2, dtype=torch.int32, device=DEV), S.lib()
    work = torch.empty(lib.b2l_seq_scan_work_floats(T, H), device=DEV)

    def run():
        out, state = torch.empty(T, H, V, device=DEV), state0.clone()
        a = S.ScanArgs(q=ops["q"].data_ptr(), ldq=H * K, k=ops["k"].data_ptr(), ldk=H * K, v=ops["v"].data_ptr(), ldv=H * V, q_mult=1.0, decay=decay.data_ptr(), ldd=H * K,
                       decay_per_channel=1, beta=ops["beta"].data_ptr() if delta else None, ldb=H, delta=delta, state=state.data_ptr(), meta=meta.data_ptr(),
                       out=out.data_ptr(), ldo=H * V, T=T, heads=H, qk_heads=H, K=K, V=V, act_dtype=S.act_code(torch.float32), work_state=work.data_ptr(), n_chunks=1)
        S.check(lib.b2l_seq_scan(C.byref(a), S.stream_ptr()), "scan")
        return out, state

    clean, _ = run()
    ops[what][at, 1, *([5] if what != "beta" else [])] = bad
    got, _ = run()
    assert bool(clean.isfinite().all()) and torch.equal(got[:at], clean[:at])
    assert torch.equal(got[:, [0, 2]], clean[:, [0, 2]])                # the other heads see nothing of it
    assert what == "beta" and not delta or not bool(got[at, 1].isfinite().all())
    if what == "v":                                                    # one value column only
        assert torch.equal(got[:, :, :5], clean[:, :, :5]) and torch.equal(got[:, :, 6:], clean[:, :, 6:])

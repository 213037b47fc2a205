"""GPU: a CTA whose waits run out (marked so after its work, nothing is delayed) leaves NaN and never a finite sum without its part."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,splits", [(17, 256, 4096, 8), (33, 4096, 4096, 4), (70, 5120, 13824, 3), (257, 128, 512, 1)])
def test_int4_prompt_gemm_with_k_split_over_a_cluster(M, N, K, splits):
    from gpu_util import rand_q4, tile
    from lit_llama_b200 import _lib as L

    _, qw, sc, z = rand_q4(N, K, "cuda", seed=M)
    qt, x, y = tile(L, qw, N, K), torch.randn(M, K, device="cuda").bfloat16(), torch.empty(M, N, device="cuda", dtype=torch.bfloat16)

    def run(flags):
        y.zero_()
        a = L.Q4LinearArgs(x=x.data_ptr(), ldx=K, qw_tiled=qt.data_ptr(), scales=sc.data_ptr(), zeros=z.data_ptr(), sz_dtype=L.sz_dtype_of(sc), y=y.data_ptr(), ldy=N,
                           M=M, N=N, K=K, flags=flags)
        L.check(L.lib().b2l_q4_gemm(C.byref(a), L.stream_ptr()), "b2l_q4_gemm")
        return y

    clean = run(0).clone()
    assert bool(clean.isfinite().all())
    for rank in range(splits):
        assert bool(run((1 + rank) << 8).isnan().all())
    assert torch.equal(run((1 + splits) << 8), clean)         # no such rank: the number of parts is what is written above

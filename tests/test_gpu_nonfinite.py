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


def same(got, want, tol):
    """Infinities and NaN in the same places, the rest within tol of rms + value (the rows next to a bad one take another summation order)."""
    got, want = got.double(), want.double()
    fin = want.isfinite()
    assert torch.equal(got[~fin].nan_to_num(7.0, 8.0, 9.0), want[~fin].nan_to_num(7.0, 8.0, 9.0))
    assert bool(((got[fin] - want[fin]).abs() < tol * (want[fin].pow(2).mean().sqrt() + want[fin].abs())).all())


def attend_seen(q, k, v, scale, seen):
    """Row by row over the keys it sees only, float64: q [T, H, K], k [S, H, K], v [S, H, V], seen [T, S]."""
    out = torch.empty(*q.shape[:2], v.shape[2], dtype=torch.float64, device=q.device)
    for t in range(q.shape[0]):
        j = seen[t].nonzero()[:, 0]
        s = torch.einsum("hk,shk->hs", q[t].double(), k[j].double()) * scale
        w = torch.exp(s - s.amax(1, keepdim=True))
        out[t] = torch.einsum("hs,shv->hv", w, v[j].double()) / w.sum(1, keepdim=True)
    return out


@pytest.mark.parametrize("T,pos0,window,K,V", [(200, 0, 64, 64, 32), (131, 90, 150, 128, 128)])
@pytest.mark.parametrize("what,bad", [("v", INF), ("v", -INF), ("v", NAN), ("k", -INF), ("k", NAN)])
def test_local_attention(what, bad, T, pos0, window, K, V):
    """f32 outputs: 1e-5 as for finite operands (sums of a few hundred f32 products), here of the largest single difference: 1e-4."""
    from lit_llama_b200 import _seqlib as S

    H, G, n = 4, 2, pos0 + T
    g = torch.Generator(device=DEV).manual_seed(T)
    q = torch.randn(T, H, K, generator=g, device=DEV)
    k, v = torch.randn(n, G, K, generator=g, device=DEV).to(BF), torch.randn(n, G, V, generator=g, device=DEV).to(BF)
    for at in (70, n - 9):                                              # in the first and in the last row tile
        (k if what == "k" else v)[at, 1, 3] = bad
    ring_k, ring_v = torch.zeros(1, 256, G, K, dtype=BF, device=DEV), torch.zeros(1, 256, G, V, dtype=BF, device=DEV)
    ring_k[0, :pos0], ring_v[0, :pos0] = k[:pos0], v[:pos0]
    meta, out = torch.tensor([0, pos0], dtype=torch.int32, device=DEV), torch.empty(T, H, V, device=DEV)
    kn, vn = k[pos0:].contiguous(), v[pos0:].contiguous()
    a = S.AttnArgs(q=q.data_ptr(), k_new=kn.data_ptr(), v_new=vn.data_ptr(), ldv=G * V, cache_k=ring_k.data_ptr(), cache_v=ring_v.data_ptr(), meta=meta.data_ptr(),
                   out=out.data_ptr(), ldo=H * V, scale=K ** -0.5, out_mult=1.0, block=256, T=T, heads=H, kv_heads=G, K=K, V=V, act_dtype=S.act_code(BF), window=window, out_f32=1)
    S.check(S.lib().b2l_seq_block_attention(C.byref(a), S.stream_ptr()), "attention")
    i, j = torch.arange(pos0, n, device=DEV)[:, None], torch.arange(n, device=DEV)[None]
    same(out, attend_seen(q, k.repeat_interleave(2, 1), v.repeat_interleave(2, 1), K ** -0.5, (j <= i) & (i - j < window)), 1e-4)


@pytest.mark.parametrize("splits", [1, 3])
@pytest.mark.parametrize("what,bad", [("v", INF), ("k", -INF), ("k", NAN)])
def test_expanded_latent_attention(what, bad, splits):
    """bf16 outputs: half an ulp, 2^-8 of the value with room for the splits' f32 sums."""
    from lit_llama_b200 import _seqlib as S

    T, H, dn, dr, V, pos0 = 140, 2, 64, 64, 64, 30
    n = pos0 + T
    g = torch.Generator(device=DEV).manual_seed(splits)
    kv, shared = torch.randn(n, H, V + dn, generator=g, device=DEV).to(BF), torch.randn(n, dr, generator=g, device=DEV).to(BF)
    kv[100, 1, 5 if what == "v" else V + 5] = bad
    q = torch.randn(T, H, dn + dr, generator=g, device=DEV)
    meta, out = torch.tensor([0, pos0], dtype=torch.int32, device=DEV), torch.empty(T, H, V, dtype=BF, device=DEV)
    work, scale = torch.empty(splits, T * H, V + 2, device=DEV), (dn + dr) ** -0.5
    a = S.LatentAttnArgs(q_a=q.data_ptr(), ldqa_t=H * (dn + dr), ldqa_h=dn + dr, q_b=q.data_ptr() + 4 * dn, ldqb_t=H * (dn + dr), ldqb_h=dn + dr, key_a=kv.data_ptr(),
                         ldka=H * (V + dn), hska=V + dn, slot_stride_a=0, key_b=shared.data_ptr(), ldkb=dr, slot_stride_b=n * dr, meta=meta.data_ptr(), out=out.data_ptr(),
                         ldo=H * V, work=work.data_ptr(), scale=scale, T=T, heads=H, heads_per_group=1, n_a=V + dn, n_b=dr, vdim=V, score_off=V, splits=splits,
                         act_dtype=S.act_code(BF), window=0)
    S.check(S.lib().b2l_seq_latent_attention(C.byref(a), S.stream_ptr()), "latent attention")
    keys = torch.cat([kv[..., V:], shared[:, None].expand(n, H, dr)], dim=2)
    seen = torch.arange(n, device=DEV)[None] <= torch.arange(pos0, n, device=DEV)[:, None]
    same(out, attend_seen(q, keys, kv[..., :V], scale, seen), 2.0 ** -8)


@pytest.mark.parametrize("bad", [INF, NAN])
def test_llama_prompt_attention(bad):
    """Angle 0 everywhere (q and k stay as they are); an infinite value reaches the rows from its token on, in its own column."""
    from lit_llama_b200 import _lib as L

    lib, T, nh, hs, S = L.lib(), 150, 2, 128, 256
    g = torch.Generator(device=DEV).manual_seed(3)
    qkv = torch.randn(1, T, 3, nh, hs, generator=g, device=DEV).to(BF)
    qkv[0, 100, 2, 1, 9] = bad
    q, k, v = qkv[0].unbind(1)
    rope = torch.stack([torch.ones(S, hs // 2), torch.zeros(S, hs // 2)], -1).to(DEV)
    pos, ring = torch.arange(T, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    ck, cv = torch.zeros(1, nh, S, hs, dtype=BF, device=DEV), torch.zeros(1, nh, S, hs, dtype=BF, device=DEV)
    y, work = torch.empty(T, nh, hs, dtype=BF, device=DEV), torch.zeros(lib.b2l_attn_workspace_bytes(1, nh, hs, T, S) // 4 + 1, device=DEV)
    mine = qkv.clone()
    L.check(lib.b2l_attention(mine.data_ptr(), ck.data_ptr(), cv.data_ptr(), rope.data_ptr(), pos.data_ptr(), ring.data_ptr(), y.data_ptr(), work.data_ptr(), 1, T, nh, hs, S, S, 0,
                              L.stream_ptr()), "attention")
    same(y, attend_seen(q, k, v, hs ** -0.5, pos[None] <= pos[:, None]), 2.0 ** -8)


def _delta_layer(W, h, D, H, K):
    from lit_llama_b200 import mixers as X
    from lit_llama_b200.state import SequenceStatePool

    m = X.ChannelDeltaMixer("a", W, "a.", heads=H, kv_heads=H, dim=K, vdim=K, conv=4, eps=1e-6)
    pool = SequenceStatePool(m.state_specs(), 1, torch.device(DEV))

    def run():
        slot = pool.acquire("r")
        y = m.forward(h, X.StepContext(h.shape[0], torch.zeros(2, dtype=torch.int32, device=DEV), pool.tensors, BF, pos_hint=0, slot_hint=slot))
        pool.release("r")
        return y, {n: t.clone() for n, t in pool.tensors.items()}

    return run


def _delta_weights(g, D, H, K, rank_a, rank_g):
    def lin(o, i):
        return (torch.randn(o, i, generator=g, device=DEV) * i ** -0.5).to(BF)

    W = {"a." + n: lin(o, i) for n, o, i in (("q", H * K, D), ("k", H * K, D), ("v", H * K, D), ("b", H, D), ("a1", rank_a, D), ("a2", H * K, rank_a), ("g1", rank_g, D),
                                             ("g2", H * K, rank_g), ("o", D, H * K))}
    for n in "qkv":
        W[f"a.{n}.conv"] = lin(H * K, 4)
    W["a.A_log"], W["a.dt_bias"], W["a.norm"] = lin(H, 4)[:, 0].contiguous(), lin(H * K, 4)[:, 0].contiguous(), lin(K, 4)[:, 0] + 1
    return W


@pytest.mark.parametrize("path,ranks", [("g1", (64, 64)), ("a1", (64, 64)), ("g1", (20, 36)), ("a1", (36, 20)), ("a1", (160, 136))])
def test_delta_layer_keeps_decay_and_gate_apart(path, ranks):
    """An infinite entry of the gate's inner projection reaches that token's gate only: the state and every other token keep their bits.  One of the decays'
    makes decays of 0 and 1, and no gate NaN."""
    D, H, K, T, at = 256, 2, 64, 90, 40
    g = torch.Generator(device=DEV).manual_seed(ranks[0])
    W, h = _delta_weights(g, D, H, K, *ranks), torch.randn(T, D, generator=g, device=DEV).to(BF)
    for n in ("q", "k", "v", "b", "a1", "g1"):
        W["a." + n][:, 0] = 0                                           # channel 0 feeds the bad entry alone
    for n in ("a2", "g2"):
        W["a." + n][W["a." + n] == 0] = 0.5                             # infinity times zero would be NaN by right
    h[:, 0] = 0
    h[at, 0] = 1e4
    clean, state = _delta_layer(W, h, D, H, K)()
    W["a." + path][3, 0] = 3e38                                         # the product's only infinite entry: token `at`, number 3
    got, st = _delta_layer(W, h, D, H, K)()
    assert bool(clean.isfinite().all()) and bool(got.isfinite().all()) and bool(st["a.S"].isfinite().all())
    assert torch.equal(got[:at], clean[:at]) and not torch.equal(got[at], clean[at])
    if path == "g1":
        assert torch.equal(got[at + 1:], clean[at + 1:]) and all(torch.equal(st[n], state[n]) for n in st)


def test_delta_layer_follows_its_second_factors():
    """a2 and g2 are read where the caller keeps them: changed in place, the next call sees them."""
    D, H, K = 256, 2, 64
    g = torch.Generator(device=DEV).manual_seed(5)
    W, h = _delta_weights(g, D, H, K, 64, 64), torch.randn(20, D, generator=g, device=DEV).to(BF)
    run = _delta_layer(W, h, D, H, K)
    before, _ = run()
    for n in ("a2", "g2"):
        W["a." + n].mul_(-2)
    (got, st), (want, st_want) = run(), _delta_layer(W, h, D, H, K)()
    assert torch.equal(got, want) and torch.equal(st["a.S"], st_want["a.S"]) and not torch.equal(got, before)

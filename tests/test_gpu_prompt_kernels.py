"""GPU: the kernels of long prompts at the edges of their tiles, each through the C ABI against a float64 restatement on the same operands:
tensor-core attention (local, expanded latent, LLaMA cache), the scans in chunks of 16 tokens, the four-tap convolution, the int4 GEMM's
tile heights and K splits.

Tolerances: f32 sums of exact products, relative to the result's norm.  A score is a sum of at most 192 products and a row sums at most some
hundred weighted values, so errors of about sqrt(192 + keys) 2^-24 of the summed magnitudes reach the result: 2e-6 with weights that
multiply the score's error by its size (scores up to ~10), 1e-5 allowed.  bf16 outputs add their own rounding, 2^-9 per value: 2.5e-3."""
import ctypes as C
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF = torch.bfloat16


def rel(got, want):
    return float((got.double() - want.double()).norm() / (want.double().norm() + 1e-30))


def attend(q, k, v, scale, seen, sink=None, cap=0.0):
    """q [T, H, K], k [S, H, K], v [S, H, V] in float64, seen [T, S]; sink [H] scores."""
    s = torch.einsum("thk,shk->hts", q, k) * scale
    if cap:
        s = cap * torch.tanh(s / cap)
    s = s.masked_fill(~seen[None], -math.inf)
    if sink is not None:
        s = torch.cat([s, sink[:, None, None].expand(-1, s.shape[1], 1)], dim=2)
    return torch.einsum("hts,shv->thv", torch.softmax(s, -1)[..., :k.shape[0]], v)


@pytest.mark.parametrize("T,H,G,K,V,pos0,window,block,sink,cap", [
    (64, 8, 2, 128, 128, 0, 0, 512, 1, 0.0),        # half a row tile
    (127, 6, 2, 192, 16, 0, 33, 40, 0, 0.0),        # one part of the query in shared memory, the narrowest values, a window below a key tile
    (129, 8, 4, 64, 96, 100, 0, 128, 1, 30.0),      # block-local with history across a block border, score cap, values over one and a half atoms
    (200, 4, 4, 16, 64, 333, 150, 160, 0, 0.0),     # one MMA step per product, history wraps in the ring
    (300, 4, 1, 48, 80, 50, 1000, 1024, 1, 0.0),    # key size between atoms
    (1, 320, 320, 128, 128, 0, 0, 64, 0, 0.0),      # one token of many heads stays on the other kernels
])
def test_local_attention_tiles(T, H, G, K, V, pos0, window, block, sink, cap):
    from lit_llama_b200 import _seqlib as S

    g = torch.Generator(device=DEV).manual_seed(T + K)
    n = pos0 + T
    q = torch.randn(T, H, K, generator=g, device=DEV) * 2
    k = torch.randn(n, G, K, generator=g, device=DEV).to(BF)
    v = torch.randn(n, G, V, generator=g, device=DEV).to(BF)
    ring_k, ring_v = torch.zeros(2, block, G, K, dtype=BF, device=DEV), torch.zeros(2, block, G, V, dtype=BF, device=DEV)
    for j in range(max(0, pos0 - block), pos0):
        ring_k[1, j % block], ring_v[1, j % block] = k[j], v[j]
    meta = torch.tensor([1, pos0], dtype=torch.int32, device=DEV)
    out = torch.empty(T, H * V, device=DEV)
    kn, vn = k[pos0:].contiguous(), v[pos0:].contiguous()
    a = S.AttnArgs(q=q.data_ptr(), k_new=kn.data_ptr(), v_new=vn.data_ptr(), ldv=G * V, cache_k=ring_k.data_ptr(), cache_v=ring_v.data_ptr(), meta=meta.data_ptr(),
                   out=out.data_ptr(), ldo=H * V, scale=K ** -0.5, softcap=cap, out_mult=0.5, has_sink=sink, block=block, T=T, heads=H, kv_heads=G, K=K, V=V,
                   act_dtype=S.act_code(BF), window=window, out_f32=1)
    S.check(S.lib().b2l_seq_block_attention(C.byref(a), S.stream_ptr()), "attention")
    i, j = torch.arange(pos0, n, device=DEV)[:, None], torch.arange(n, device=DEV)[None]
    seen = (j <= i) & ((i - j < window) if window else (i // block == j // block))
    rep = H // G
    want = 0.5 * attend(q.double(), k.double().repeat_interleave(rep, 1), v.double().repeat_interleave(rep, 1), K ** -0.5, seen,
                        torch.zeros(H, dtype=torch.float64, device=DEV) if sink else None, cap)
    assert rel(out.view(T, H, V), want) < 1e-5
    last = n - 1                                        # the ring afterwards: the last token's block or the last `block` tokens
    for p in range(max(pos0, last - block + 1 if window else last // block * block), n):
        assert torch.equal(ring_k[1, p % block], k[p]) and torch.equal(ring_v[1, p % block], v[p])


@pytest.mark.parametrize("T,H,dn,dr,V,pos0,window,sink,splits", [(32, 3, 128, 64, 128, 0, 0, True, 1), (70, 2, 64, 64, 16, 59, 0, False, 5), (129, 4, 32, 16, 48, 300, 100, True, 3),
                                                                 (65, 2, 128, 0, 128, 1000, 0, True, 30), (257, 2, 128, 64, 128, 7, 64, False, 2)])
def test_expanded_latent_attention_tiles(T, H, dn, dr, V, pos0, window, sink, splits):
    """Key splits (also empty ones), windows, a key part shared by the heads or none; sizes whose columns are not whole 64-column steps."""
    from lit_llama_b200 import _seqlib as S

    g = torch.Generator(device=DEV).manual_seed(T + dn)
    n = pos0 + T
    kv = torch.randn(n, H, V + dn, generator=g, device=DEV).to(BF)
    shared = torch.randn(2, n, 24 + dr, generator=g, device=DEV).to(BF)
    q = torch.randn(T, H, dn + dr, generator=g, device=DEV)
    sk = torch.randn(H, generator=g, device=DEV)
    meta = torch.tensor([1, pos0], dtype=torch.int32, device=DEV)
    out = torch.empty(T, H * V, dtype=BF, device=DEV)
    work = torch.full((splits, T * H, V + 2), float("nan"), device=DEV)
    scale = (dn + dr) ** -0.5
    a = S.LatentAttnArgs(q_a=q.data_ptr(), ldqa_t=H * (dn + dr), ldqa_h=dn + dr, q_b=q.data_ptr() + 4 * dn, ldqb_t=H * (dn + dr), ldqb_h=dn + dr,
                         key_a=kv.data_ptr(), ldka=H * (V + dn), hska=V + dn, slot_stride_a=0, key_b=shared.data_ptr() + 48, ldkb=24 + dr,
                         slot_stride_b=n * (24 + dr), sink=sk.data_ptr() if sink else None, meta=meta.data_ptr(), out=out.data_ptr(), ldo=H * V, work=work.data_ptr(),
                         scale=scale, T=T, heads=H, heads_per_group=1, n_a=V + dn, n_b=dr, vdim=V, score_off=V, splits=splits, act_dtype=S.act_code(BF), window=window)
    S.check(S.lib().b2l_seq_latent_attention(C.byref(a), S.stream_ptr()), "latent attention")
    keys = torch.cat([kv[..., V:].double(), shared[1, :, None, 24:].double().expand(n, H, dr)], dim=2)
    i, j = torch.arange(pos0, n, device=DEV)[:, None], torch.arange(n, device=DEV)[None]
    seen = (j <= i) & ((i - j < window) if window else (j >= 0))
    want = attend(q.double(), keys, kv[..., :V].double(), scale, seen, sk.double() if sink else None)
    assert rel(out.view(T, H, V), want) < 2.5e-3


@pytest.mark.parametrize("B,T,nh,S,ring,start", [(1, 64, 3, 128, 0, 0), (2, 129, 2, 200, 37, 0), (1, 130, 2, 300, 290, 100), (2, 300, 1, None, 0, 0)])
def test_llama_prompt_attention_tiles(B, T, nh, S, ring, start):
    """64 rows and more at head size 128: cache with and without a turned ring, a second portion behind earlier slots, no cache."""
    from lit_llama_b200 import _lib as L

    lib, hs, C_ = L.lib(), 128, nh * 128
    g = torch.Generator(device=DEV).manual_seed(T)
    qkv = torch.randn(B, T, 3 * C_, generator=g, device=DEV).to(BF)
    block = 512
    theta = 1.0 / (10000.0 ** (torch.arange(0, hs, 2, device=DEV).float() / hs))
    ang = torch.outer(torch.arange(block, device=DEV).float(), theta)
    rope = torch.stack([ang.cos(), ang.sin()], -1).contiguous()
    pos = torch.arange(start, start + T, device=DEV)

    def turn(x):
        r = rope[pos][None, :, None]
        u, w = x.float()[..., 0::2], x.float()[..., 1::2]
        return torch.stack([u * r[..., 0] - w * r[..., 1], w * r[..., 0] + u * r[..., 1]], -1).flatten(-2).to(BF)

    q, k, v = qkv.view(B, T, 3, nh, hs).unbind(2)
    q, k = turn(q), turn(k)
    y = torch.empty(B, T, C_, dtype=BF, device=DEV)
    work = torch.zeros(lib.b2l_attn_workspace_bytes(B, nh, hs, T, S or T) // 4 + 1, device=DEV)
    mine = qkv.clone()
    if S is None:
        L.check(lib.b2l_attention_nocache(mine.data_ptr(), rope.data_ptr(), y.data_ptr(), work.data_ptr(), B, T, nh, hs, block, L.stream_ptr()), "attention")
        kk, vv, seen = k, v, torch.ones(T, T, dtype=torch.bool, device=DEV).tril()
    else:
        kk, vv = (torch.randn(B, S, nh, hs, generator=g, device=DEV).to(BF) for _ in range(2))
        kk[:, start:start + T], vv[:, start:start + T] = k, v
        slot = (torch.arange(S, device=DEV) + ring) % S
        ck, cv = torch.empty(B, nh, S, hs, dtype=BF, device=DEV), torch.empty(B, nh, S, hs, dtype=BF, device=DEV)
        ck[:, :, slot], cv[:, :, slot] = kk.transpose(1, 2), vv.transpose(1, 2)
        ck[:, :, slot[start:start + T]] = 0
        cv[:, :, slot[start:start + T]] = 0
        ring_start = torch.tensor([ring], dtype=torch.int32, device=DEV)
        L.check(lib.b2l_attention(mine.data_ptr(), ck.data_ptr(), cv.data_ptr(), rope.data_ptr(), pos.data_ptr(), ring_start.data_ptr(), y.data_ptr(), work.data_ptr(),
                                  B, T, nh, hs, S, block, 0, L.stream_ptr()), "attention")
        assert torch.equal(ck[:, :, slot[start:start + T]], k.transpose(1, 2)) and torch.equal(cv[:, :, slot[start:start + T]], v.transpose(1, 2))
        seen = torch.arange(S, device=DEV)[None] <= pos[:, None]
    for b in range(B):
        want = attend(q[b].double(), kk[b].double(), vv[b].double(), hs ** -0.5, seen)
        assert rel(y[b].view(T, nh, hs), want) < 2.5e-3


@pytest.mark.parametrize("T,K,V,H,G,form", [(32, 64, 16, 2, 2, "delta"), (47, 128, 48, 4, 2, "delta"), (100, 128, 32, 3, 1, "channel"), (33, 64, 64, 2, 2, "scalar"), (400, 128, 64, 4, 1, "scalar")])
def test_scans_sixteen_tokens_at_a_time(T, K, V, H, G, form):
    """Whole chunks and a remainder, from a state that is not zero; strong and weak decays side by side (a factor of e^-6 per step underflows
    nothing and overflows no quotient); against the token-by-token recurrence in float64.  Same tolerance as the other recurrence tests."""
    from lit_llama_b200 import _seqlib as S

    g = torch.Generator(device=DEV).manual_seed(T + K + V)
    q, k = torch.randn(T, G, K, generator=g, device=DEV), torch.randn(T, G, K, generator=g, device=DEV)
    k = k / k.norm(dim=-1, keepdim=True)
    v = torch.randn(T, H, V, generator=g, device=DEV)
    a = torch.exp(-6 * torch.rand(T, H, 1 if form == "scalar" else K, generator=g, device=DEV) ** 3)
    beta = torch.randn(T, H, generator=g, device=DEV)
    vs, skip = torch.rand(T, H, generator=g, device=DEV) + 0.1, torch.randn(H, generator=g, device=DEV)
    state = torch.randn(2, H, V, K, generator=g, device=DEV) * 0.1
    s64, want = state[1].double().clone(), torch.empty(T, H, V, dtype=torch.float64, device=DEV)
    rep = H // G
    for t in range(T):
        kt, qt = k[t].double().repeat_interleave(rep, 0), q[t].double().repeat_interleave(rep, 0)
        s64 = s64 * a[t].double()[:, None, :]
        if form == "delta":
            u = torch.sigmoid(beta[t].double())[:, None] * (v[t].double() - torch.einsum("hvk,hk->hv", s64, kt))
        else:
            u = v[t].double() * (vs[t].double()[:, None] if form == "scalar" else 1.0)
        s64 = s64 + u[:, :, None] * kt[:, None, :]
        want[t] = 0.5 * torch.einsum("hvk,hk->hv", s64, qt) + (skip.double()[:, None] * v[t].double() if form == "scalar" else 0)
    lib, out = S.lib(), torch.empty(T, H * V, device=DEV)
    meta = torch.tensor([1, 0], dtype=torch.int32, device=DEV)
    n = lib.b2l_seq_scan_work_floats(T, H)
    assert n > 0 and lib.b2l_seq_scan_work_floats(31, H) == 0
    other = state[0].clone()
    work = torch.empty(n, device=DEV)
    args = S.ScanArgs(q=q.data_ptr(), ldq=G * K, k=k.data_ptr(), ldk=G * K, v=v.data_ptr(), ldv=H * V, q_mult=0.5, decay=a.data_ptr(), ldd=a.shape[1] * a.shape[2],
                      decay_per_channel=int(form != "scalar"), beta=beta.data_ptr() if form == "delta" else None, ldb=H, delta=int(form == "delta"),
                      vscale=vs.data_ptr() if form == "scalar" else None, ldvs=H, skip=skip.data_ptr() if form == "scalar" else None, state=state.data_ptr(),
                      meta=meta.data_ptr(), out=out.data_ptr(), ldo=H * V, T=T, heads=H, qk_heads=G, K=K, V=V, act_dtype=S.act_code(torch.float32), work_state=work.data_ptr(),
                      n_chunks=1)
    S.check(lib.b2l_seq_scan(C.byref(args), S.stream_ptr()), "scan")
    assert rel(out.view(T, H, V), want) < 2e-5 and rel(state[1], s64) < 2e-5
    assert torch.equal(state[0], other)


@pytest.mark.parametrize("T,K,V,H,G,form", [(64, 128, 128, 9, 3, "delta"), (79, 128, 16, 65, 13, "delta"), (144, 128, 48, 2, 1, "delta"), (161, 128, 128, 5, 5, "channel"),
                                            (65, 128, 64, 18, 1, "scalar"), (175, 128, 16, 1, 1, "scalar"), (512, 64, 16, 4, 2, "channel"), (527, 64, 128, 2, 2, "scalar"),
                                            (208, 128, 16, 160, 160, "delta"), (145, 128, 32, 256, 2, "scalar")])
def test_scans_on_the_tensor_cores(T, K, V, H, G, form):
    """The least portions by either side of the rule, last chunks of 1, 15 and 16 tokens, one tile of value columns and all eight, heads that share q and k, and
    portions in two and more segments (2048 chunks times heads each)."""
    test_scans_sixteen_tokens_at_a_time(T, K, V, H, G, form)


@pytest.mark.parametrize("T,K,V,H,G", [(300, 128, 48, 13, 1), (512, 128, 64, 32, 1), (576, 128, 64, 13, 1), (700, 128, 128, 11, 1), (1040, 128, 48, 13, 1), (1041, 128, 16, 11, 1),
                                       (1047, 64, 80, 15, 1), (1056, 128, 32, 28, 2)])
def test_scans_of_heads_that_share_a_cta(T, K, V, H, G):
    """One decay per head: two, four and eight heads a CTA (148 SMs), last groups of 1, 3, 5, 6 and 7 heads whose warps take value columns in turn or nothing."""
    test_scans_sixteen_tokens_at_a_time(T, K, V, H, G, "scalar")


@pytest.mark.parametrize("delta", [0, 1])
@pytest.mark.parametrize("T", [144, 777])
def test_scan_on_the_tensor_cores_is_as_near_as_token_by_token(T, delta):
    """Rows apart by 3 entries (no 16-byte copies), one head, against float64 and against the form that walks token by token: 16-token sums of three bf16 parts are no
    further off than twice its error (measured: 0.6 to 1.0 of it)."""
    from lit_llama_b200 import _seqlib as S

    H, K, V, ld = 3, 128, 32, 3 * 128 + 3
    lib, g = S.lib(), torch.Generator(device=DEV).manual_seed(T + delta)
    q, k, v = (torch.randn(T, ld, generator=g, device=DEV) for _ in range(3))
    k[:, :H * K] = torch.nn.functional.normalize(k[:, :H * K].view(T, H, K), dim=-1).view(T, H * K)
    a, beta, state0 = torch.rand(T, H, K, generator=g, device=DEV) * 0.5 + 0.5, torch.randn(T, H, generator=g, device=DEV), torch.randn(1, H, V, K, generator=g, device=DEV)
    meta = torch.zeros(2, dtype=torch.int32, device=DEV)
    s64, want = state0[0].double(), torch.empty(T, H, V, dtype=torch.float64, device=DEV)
    for t in range(T):
        kt, qt, vt = (x[t, :H * n].double().view(H, n) for x, n in ((k, K), (q, K), (v, V)))
        s64 = s64 * a[t].double()[:, None, :]
        u = torch.sigmoid(beta[t].double())[:, None] * (vt - torch.einsum("hvk,hk->hv", s64, kt)) if delta else vt
        s64 = s64 + u[:, :, None] * kt[:, None, :]
        want[t] = torch.einsum("hvk,hk->hv", s64, qt)
    errs = []
    for work in (torch.empty(lib.b2l_seq_scan_work_floats(T, H), device=DEV), None):
        out, state = torch.empty(T, H, V, device=DEV), state0.clone()
        args = S.ScanArgs(q=q.data_ptr(), ldq=ld, k=k.data_ptr(), ldk=ld, v=v.data_ptr(), ldv=ld, q_mult=1.0, decay=a.data_ptr(), ldd=H * K, decay_per_channel=1,
                          beta=beta.data_ptr() if delta else None, ldb=H, delta=delta, state=state.data_ptr(), meta=meta.data_ptr(), out=out.data_ptr(), ldo=H * V, T=T, heads=H,
                          qk_heads=H, K=K, V=V, act_dtype=S.act_code(torch.float32), work_state=work.data_ptr() if work is not None else None, n_chunks=1)
        S.check(lib.b2l_seq_scan(C.byref(args), S.stream_ptr()), "scan")
        errs.append((rel(out, want), rel(state[0], s64)))
    assert errs[0][0] < 2 * errs[1][0] and errs[0][1] < 2 * errs[1][1] and max(errs[0]) < 1e-6


@pytest.mark.parametrize("v_mean,least,norm,shared", [(0.0, 0.5, 1.0, 0.0), (2.0, 0.99, 1.0, 0.0), (2.0, 0.9, 1.0, 2.0), (2.0, 0.5, 1.0, 2.0), (0.0, 0.9, 2.0, 0.0), (2.0, 0.9, 3.0, 0.0)])
@pytest.mark.parametrize("form,G", [("delta", 4), ("channel", 4), ("scalar", 1)])
def test_scan_on_the_tensor_cores_keeps_what_the_f32_form_keeps(form, G, v_mean, least, norm, shared):
    """Against float64 with values of a mean, decays near 1, keys of other lengths and keys with a part in common (whose sums truncation would bias): no further off than
    the walk in f32.  Both errors are sums of some 1e6 roundings, equal to a few percent from seed to seed: an eighth more at most, measured 0.5 to 1.06."""
    from lit_llama_b200 import _seqlib as S

    T, H, K, V = 1536, 4, 128, 128
    lib, g = S.lib(), torch.Generator(device=DEV).manual_seed(3)
    delta, per = int(form == "delta"), int(form != "scalar")
    q, k = (torch.randn(T, G, K, generator=g, device=DEV) for _ in range(2))
    k = norm * torch.nn.functional.normalize(k + shared * torch.randn(1, G, K, generator=g, device=DEV), dim=-1)
    q, v = q * K ** -0.5 + 0.25 * shared * k, torch.randn(T, H, V, generator=g, device=DEV) + v_mean
    a, beta = torch.rand(T, H, K if per else 1, generator=g, device=DEV) * (1 - least) + least, torch.randn(T, H, generator=g, device=DEV)
    s64, want = torch.zeros(H, V, K, dtype=torch.float64, device=DEV), torch.empty(T, H, V, dtype=torch.float64, device=DEV)
    for t in range(T):
        kt, qt = k[t].double().repeat_interleave(H // G, 0), q[t].double().repeat_interleave(H // G, 0)
        s64 = s64 * a[t].double()[:, None, :]
        u = torch.sigmoid(beta[t].double())[:, None] * (v[t].double() - torch.einsum("hvk,hk->hv", s64, kt)) if delta else v[t].double()
        s64 = s64 + u[:, :, None] * kt[:, None, :]
        want[t] = torch.einsum("hvk,hk->hv", s64, qt)
    fast = lib.b2l_seq_scan_work_floats(T, H)
    meta, work, errs = torch.zeros(2, dtype=torch.int32, device=DEV), torch.empty(fast, device=DEV), []
    for floats in (fast, T // 16 * H * 512):                            # the second holds the walk's matrices only
        out, state = torch.empty(T, H, V, device=DEV), torch.zeros(1, H, V, K, device=DEV)
        args = S.ScanArgs(q=q.data_ptr(), ldq=G * K, k=k.data_ptr(), ldk=G * K, v=v.data_ptr(), ldv=H * V, q_mult=1.0, decay=a.data_ptr(), ldd=a.shape[1] * a.shape[2],
                          decay_per_channel=per, beta=beta.data_ptr() if delta else None, ldb=H, delta=delta, state=state.data_ptr(), meta=meta.data_ptr(), out=out.data_ptr(),
                          ldo=H * V, T=T, heads=H, qk_heads=G, K=K, V=V, act_dtype=S.act_code(torch.float32), work_state=work.data_ptr(), n_chunks=1)
        S.check(lib.b2l_seq_scan_within(C.byref(args), floats, S.stream_ptr()), "scan")
        errs.append((rel(out, want), rel(state[0], s64)))
    assert errs[0] != errs[1] and all(x < 1.125 * y for x, y in zip(*errs)), errs


@pytest.mark.parametrize("what,bad", [("v", math.inf), ("k", math.nan), ("k", -math.inf), ("q", math.inf), ("decay", math.nan), ("beta", math.nan), ("state", math.inf), ("state", math.nan)])
@pytest.mark.parametrize("delta", [0, 1])
def test_scan_on_the_tensor_cores_with_infinities(delta, what, bad):
    """Tokens before a bad one, other heads and (values) other columns keep their bits; the rest is what the form that walks token by token gives: infinities and NaN in
    the same places, finite results to 1e-5 of their row (f32 sums in two orders)."""
    from lit_llama_b200 import _seqlib as S

    T, H, K, V, at = 161, 2, 128, 32, 70
    g = torch.Generator(device=DEV).manual_seed(11)
    ops = {"q": torch.randn(T, H, K, generator=g, device=DEV), "k": torch.randn(T, H, K, generator=g, device=DEV) / 12, "v": torch.randn(T, H, V, generator=g, device=DEV),
           "beta": torch.randn(T, H, generator=g, device=DEV), "decay": torch.rand(T, H, K, generator=g, device=DEV) * 0.5 + 0.5, "state": torch.randn(1, H, V, K, generator=g, device=DEV)}
    meta, lib = torch.zeros(2, dtype=torch.int32, device=DEV), S.lib()
    work = torch.empty(lib.b2l_seq_scan_work_floats(T, H), device=DEV)

    def run(space):
        out, state = torch.empty(T, H, V, device=DEV), ops["state"].clone()
        a = S.ScanArgs(q=ops["q"].data_ptr(), ldq=H * K, k=ops["k"].data_ptr(), ldk=H * K, v=ops["v"].data_ptr(), ldv=H * V, q_mult=1.0, decay=ops["decay"].data_ptr(), ldd=H * K,
                       decay_per_channel=1, beta=ops["beta"].data_ptr() if delta else None, ldb=H, delta=delta, state=state.data_ptr(), meta=meta.data_ptr(),
                       out=out.data_ptr(), ldo=H * V, T=T, heads=H, qk_heads=H, K=K, V=V, act_dtype=S.act_code(torch.float32), work_state=space, n_chunks=1)
        S.check(lib.b2l_seq_scan(C.byref(a), S.stream_ptr()), "scan")
        return out, state

    clean, clean_state = run(work.data_ptr())
    if what == "state":
        ops["state"][0, 1, 3, 5] = bad
    else:
        ops[what][at, 1, *([5] if what != "beta" else [])] = bad
    (got, st), (want, st_want) = run(work.data_ptr()), run(None)
    assert torch.equal(got[:, 0], clean[:, 0]) and torch.equal(st[0, 0], clean_state[0, 0])
    if what != "state":
        assert torch.equal(got[:at], clean[:at])
    if what in ("v", "state"):
        c = 5 if what == "v" else 3
        assert torch.equal(got[:, :, :c], clean[:, :, :c]) and torch.equal(got[:, :, c + 1:], clean[:, :, c + 1:]) and torch.equal(st[0, 1, c + 1:], clean_state[0, 1, c + 1:])
    for x, y in ((got, want), (st, st_want)):
        fin = y.isfinite()
        assert torch.equal(x.isnan(), y.isnan()) and torch.equal(x[~fin & ~y.isnan()], y[~fin & ~y.isnan()])
        x, y = x.double().where(fin, 0.0), y.double().where(fin, 0.0)
        assert bool(((x - y).abs() <= 1e-5 * y.norm(dim=-1, keepdim=True)).all())


@pytest.mark.parametrize("what,bad", [("v", math.inf), ("v", math.nan), ("vscale", math.inf), ("vscale", math.nan), ("decay", math.inf), ("decay", math.nan), ("k", -math.inf), ("k", math.nan),
                                      ("q", math.inf), ("state", -math.inf), ("state", math.nan)])
@pytest.mark.parametrize("T,H", [(700, 11), (200, 5)])
def test_scan_of_heads_that_share_a_cta_with_infinities(T, H, what, bad):
    """The same for one decay per head and q and k shared by all heads: earlier tokens and (but for q and k) other heads keep their bits, the rest has its infinities and NaN
    where the form that walks token by token has them, and is within 1e-5 of the row elsewhere (f32 sums in two orders)."""
    from lit_llama_b200 import _seqlib as S

    K, V, at, head = 128, 32, 70, 3
    g = torch.Generator(device=DEV).manual_seed(T)
    ops = {"q": torch.randn(T, 1, K, generator=g, device=DEV), "k": torch.randn(T, 1, K, generator=g, device=DEV) / 12, "v": torch.randn(T, H, V, generator=g, device=DEV),
           "vscale": torch.rand(T, H, generator=g, device=DEV) + 0.5, "decay": torch.rand(T, H, generator=g, device=DEV) * 0.5 + 0.5,
           "state": torch.randn(1, H, V, K, generator=g, device=DEV)}
    meta, lib = torch.zeros(2, dtype=torch.int32, device=DEV), S.lib()
    work = torch.empty(lib.b2l_seq_scan_work_floats(T, H), device=DEV)

    def run(space):
        out, state = torch.empty(T, H, V, device=DEV), ops["state"].clone()
        a = S.ScanArgs(q=ops["q"].data_ptr(), ldq=K, k=ops["k"].data_ptr(), ldk=K, v=ops["v"].data_ptr(), ldv=H * V, q_mult=1.0, decay=ops["decay"].data_ptr(), ldd=H,
                       decay_per_channel=0, vscale=ops["vscale"].data_ptr(), ldvs=H, delta=0, state=state.data_ptr(), meta=meta.data_ptr(), out=out.data_ptr(), ldo=H * V, T=T,
                       heads=H, qk_heads=1, K=K, V=V, act_dtype=S.act_code(torch.float32), work_state=space, n_chunks=1)
        S.check(lib.b2l_seq_scan(C.byref(a), S.stream_ptr()), "scan")
        return out, state

    clean, clean_state = run(work.data_ptr())
    ops[what][(0, head, 4, 5) if what == "state" else (at, 0, 5) if what in "qk" else (at, head, 5) if what == "v" else (at, head)] = bad
    (got, st), (want, st_want) = run(work.data_ptr()), run(None)
    others = [h for h in range(H) if h != head]
    if what not in "qk":
        assert torch.equal(got[:, others], clean[:, others]) and torch.equal(st[0, others], clean_state[0, others])
    if what != "state":
        assert torch.equal(got[:at], clean[:at])
    assert not bool(got.isfinite().all())
    for x, y in ((got, want), (st, st_want)):
        fin = y.isfinite()
        assert torch.equal(x.isnan(), y.isnan()) and torch.equal(x[~fin & ~y.isnan()], y[~fin & ~y.isnan()])
        x, y = x.double().where(fin, 0.0), y.double().where(fin, 0.0)
        assert bool(((x - y).abs() <= 1e-5 * y.norm(dim=-1, keepdim=True)).all())


@pytest.mark.parametrize("T,Ch,bias", [(33, 8, True), (48, 1032, False), (100, 2304, True)])
def test_four_tap_convolution_of_long_portions(T, Ch, bias):
    from lit_llama_b200 import _seqlib as S

    g = torch.Generator(device=DEV).manual_seed(T)
    x, w = torch.randn(T, Ch + 8, generator=g, device=DEV).to(BF), torch.randn(Ch, 4, generator=g, device=DEV).to(BF)
    b, state = torch.randn(Ch, generator=g, device=DEV).to(BF), torch.randn(2, 3, Ch, generator=g, device=DEV).to(BF)
    full = torch.cat([state[1], x[:, :Ch]]).double()
    want = sum(full[j:j + T] * w[:, j].double() for j in range(4)) + (b.double() if bias else 0)
    want = want * torch.sigmoid(want)
    out, meta = torch.empty(T, Ch, device=DEV), torch.tensor([1, 5], dtype=torch.int32, device=DEV)
    S.check(S.lib().b2l_seq_conv_silu(x.data_ptr(), Ch + 8, w.data_ptr(), b.data_ptr() if bias else None, state.data_ptr(), meta.data_ptr(), out.data_ptr(), Ch, T, Ch, 4,
                                      S.act_code(BF), S.stream_ptr()), "convolution")
    assert rel(out, want) < 1e-6 and torch.equal(state[1], x[-3:, :Ch])


@pytest.mark.parametrize("M,N,K", [(17, 130, 11008), (33, 4096, 4096), (203, 11008, 4096), (257, 128, 512), (513, 384, 64)])
def test_q4_gemm_tile_heights_and_splits(M, N, K):
    """Token tiles of 16, 48, 208, 64 and 96 and K split over clusters of 8, 4 and 1 CTAs (148 SMs): f32 sums of exact bf16 products, one bf16
    rounding."""
    from gpu_util import rand_q4, relerr, tile
    from lit_llama_b200 import _lib as L

    lv, qw, sc, z = rand_q4(N, K, DEV, seed=M + N + K)
    qt = tile(L, qw, N, K)
    x = torch.randn(M, K, device=DEV).bfloat16()
    y = torch.full((M + 1, N), 7.0, device=DEV, dtype=BF)
    a = L.Q4LinearArgs(x=x.data_ptr(), ldx=K, qw_tiled=qt.data_ptr(), scales=sc.data_ptr(), zeros=z.data_ptr(), sz_dtype=L.sz_dtype_of(sc), y=y.data_ptr(), ldy=N, M=M, N=N, K=K)
    assert L.lib().b2l_q4_gemm(C.byref(a), L.stream_ptr()) == 0, L.lib().b2l_last_error()
    want = x.double() @ ((lv.to(BF) - z.to(BF)) * sc.to(BF)).double().t()
    assert relerr(y[:M], want) < 2.0 ** -9 and bool((y[M] == 7).all())


def test_expanded_latent_attention_with_heads_apart():
    """Keys and values head by head ([heads][positions][entries], rows of one head next to each other): the same result as position by position."""
    from lit_llama_b200 import _seqlib as S

    T, H, dn, V, pos0 = 150, 3, 64, 64, 90
    n, g = pos0 + T, torch.Generator(device=DEV).manual_seed(5)
    kv, q = torch.randn(n, H, V + dn, generator=g, device=DEV).to(BF), torch.randn(T, H, dn, generator=g, device=DEV)
    apart, meta = kv.transpose(0, 1).contiguous(), torch.tensor([0, pos0], dtype=torch.int32, device=DEV)
    res = []
    for rows, ldka, hska in ((kv, H * (V + dn), V + dn), (apart, V + dn, n * (V + dn))):
        out = torch.empty(T, H * V, dtype=BF, device=DEV)
        a = S.LatentAttnArgs(q_a=q.data_ptr(), ldqa_t=H * dn, ldqa_h=dn, key_a=rows.data_ptr(), ldka=ldka, hska=hska, slot_stride_a=0, meta=meta.data_ptr(), out=out.data_ptr(),
                             ldo=H * V, scale=dn ** -0.5, T=T, heads=H, heads_per_group=1, n_a=V + dn, n_b=0, vdim=V, score_off=V, splits=1, act_dtype=S.act_code(BF))
        S.check(S.lib().b2l_seq_latent_attention(C.byref(a), S.stream_ptr()), "latent attention")
        res.append(out)
    seen = torch.arange(n, device=DEV)[None] <= torch.arange(pos0, n, device=DEV)[:, None]
    assert rel(res[0].view(T, H, V), attend(q.double(), kv[..., V:].double(), kv[..., :V].double(), dn ** -0.5, seen)) < 2.5e-3
    assert torch.equal(res[0], res[1])


@pytest.mark.parametrize("rot", [8192, 8208])
def test_attention_operands_of_very_wide_heads(rot):
    """The angles of a token wait in shared memory up to 8192 rotated entries; beyond that every head forms its own.  cos and sin of f32 angles
    up to 40 are good to 40 * 2^-24, products and sums add a few 2^-24: 1e-5 of the largest entries."""
    from lit_llama_b200 import _seqlib as S

    T, g = 3, torch.Generator(device=DEV).manual_seed(rot)
    x, freq = torch.randn(T, 2 * rot, generator=g, device=DEV), torch.rand(rot // 2, generator=g, device=DEV)
    q, k, meta = torch.empty(T, rot, device=DEV), torch.empty(T, rot, device=DEV), torch.tensor([0, 30], dtype=torch.int32, device=DEV)
    a = S.QkvPrepArgs(proj=x.data_ptr(), ld=2 * rot, q_off=0, k_off=rot, v_off=0, eps=1e-6, freq=freq.data_ptr(), rot_dims=rot, rot_mult=1.0, meta=meta.data_ptr(),
                      q_out=q.data_ptr(), k_out=k.data_ptr(), T=T, heads=1, kv_heads=1, K=rot, V=16, act_dtype=S.act_code(torch.float32))
    S.check(S.lib().b2l_seq_qkv_prep(C.byref(a), S.stream_ptr()), "operands")
    ang = (torch.arange(30, 30 + T, device=DEV).double()[:, None] * freq.double())
    for got, src in ((q, x[:, :rot]), (k, x[:, rot:])):
        u, v = src.double()[:, :rot // 2], src.double()[:, rot // 2:]
        want = torch.cat([u * ang.cos() - v * ang.sin(), v * ang.cos() + u * ang.sin()], 1)
        assert float((got - want).abs().max()) < 1e-5 * float(want.abs().max())


@pytest.mark.parametrize("T,H,G,K,norms,mix", [(1, 16, 4, 128, "qk", True), (1187, 2, 1, 16, "qk", False), (700, 16, 4, 128, "", True), (900, 3, 2, 24, "k", True), (5, 130, 6, 128, "qk", False),
                                               (9, 40, 8, 128, "q", True), (3, 300, 20, 128, "qk", True), (300, 130, 6, 128, "k", False), (150, 126, 4, 128, "", True), (4, 256, 10, 128, "", False)])
def test_attention_operands_by_quads_of_pairs(T, H, G, K, norms, mix):
    """One to eight units per thread, one to four tokens per CTA with a remainder, rows too long for that, either row's norm, the query temperature, mixed values.  Angles up to 40 are good to
    40 * 2^-24, products and sums add a few 2^-24: 1e-5 of the largest entry; k and v are rounded to bf16 on top (2^-9 of an entry)."""
    from lit_llama_b200 import _seqlib as S

    V, pos0, g = 40, 30, torch.Generator(device=DEV).manual_seed(T + H)
    n = (H + G) * K + G * V + 12
    x = torch.randn(T, n, generator=g, device=DEV).to(BF)
    o_k, o_v = H * K + 4, (H + G) * K + 4
    w = {c: (torch.randn(m * K, generator=g, device=DEV) * 0.1 + 1).to(BF) for c, m in (("q", H), ("k", G))}
    freq, vf, lam = torch.rand(K // 2, generator=g, device=DEV) * 40 / (pos0 + T), torch.randn(T, G * V, generator=g, device=DEV).to(BF), torch.tensor([0.3], device=DEV).to(BF)
    meta, q, k, v = torch.tensor([0, pos0], dtype=torch.int32, device=DEV), torch.full((T + 1, H * K), 7.0, device=DEV), torch.full((T + 1, G * K), 7.0, device=DEV).to(BF), torch.empty(T, G * V, device=DEV).to(BF)
    a = S.QkvPrepArgs(proj=x.data_ptr(), ld=n, q_off=0, k_off=o_k, v_off=o_v, q_norm=w["q"].data_ptr() if "q" in norms else None, k_norm=w["k"].data_ptr() if "k" in norms else None,
                      whole_row=int(bool(norms)), eps=1e-6, freq=freq.data_ptr(), rot_dims=K, rot_mult=1.1, meta=meta.data_ptr(), q_out=q.data_ptr(), k_out=k.data_ptr(),
                      v_first=vf.data_ptr() if mix else None, ldvf=G * V, lambda_=lam.data_ptr() if mix else None, v_out=v.data_ptr() if mix else None, T=T, heads=H, kv_heads=G, K=K, V=V,
                      act_dtype=S.act_code(BF), temp_coef=0.2, temp_every=64)
    assert n % 4 == 0
    S.check(S.lib().b2l_seq_qkv_prep(C.byref(a), S.stream_ptr()), "operands")
    pos = torch.arange(pos0, pos0 + T, device=DEV).double()
    ang = pos[:, None] * freq.double()
    temp = 1 + 0.2 * torch.log(torch.floor((pos + 1) / 64) + 1)
    for got, at, m, c in ((q, 0, H, "q"), (k, o_k, G, "k")):
        r = x[:, at:at + m * K].double()
        if c in norms:
            r = r / torch.sqrt((r * r).mean(-1, keepdim=True) + 1e-6) * w[c].double()
        r = r.view(T, m, K)
        u, z, co, si = r[..., :K // 2], r[..., K // 2:], ang.cos()[:, None] * 1.1, ang.sin()[:, None] * 1.1
        want = torch.cat([u * co - z * si, z * co + u * si], -1).view(T, m * K) * (temp[:, None] if c == "q" else 1.0)
        err, top = (got[:T].double() - want).abs(), float(want.abs().max())
        assert bool((err <= 1e-5 * top + (2.0 ** -8 * want.abs() if c == "k" else 0)).all()) and bool((got[T] == 7).all())
    if mix:
        want = (1 - lam.double()) * x[:, o_v:o_v + G * V].double() + lam.double() * vf.double()
        assert bool(((v.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all())


@pytest.mark.parametrize("T,H,G,K,norms,mix", [(1, 16, 4, 128, "qk", True), (1187, 2, 1, 16, "qk", False), (777, 8, 2, 128, "qk", True), (900, 3, 2, 24, "k", True), (700, 16, 4, 128, "", True),
                                               (9, 40, 8, 128, "q", True), (5, 130, 6, 128, "qk", False)])
def test_attention_operands_by_quads_of_pairs_in_f32(T, H, G, K, norms, mix, monkeypatch):
    """The same in float32: one and two units per thread, rows too long for that; the queries hold the tolerance above without a bf16 rounding."""
    import sys

    monkeypatch.setattr(sys.modules[__name__], "BF", torch.float32)
    test_attention_operands_by_quads_of_pairs(T, H, G, K, norms, mix)


@pytest.mark.parametrize("T,H,K,V,want", [(2048, 4, 128, 128, "chunks"), (2048, 8, 64, 64, "chunks"), (300, 1, 128, 16, "walk"), (2048, 16, 128, 128, "walk"), (257, 64, 128, 64, "walk"),
                                          (47, 2, 64, 32, "steps"), (48, 2, 64, 32, "walk"), (63, 64, 64, 64, "steps"), (64, 64, 64, 64, "walk")])
def test_scan_plan_and_its_neighbours(T, H, K, V, want):
    """The planned form of a scan without the delta rule (148 SMs) and the forms it was chosen over: the same outputs and state up to the order
    of f32 sums (2048 decayed terms, 1e-6 of the norm)."""
    from lit_llama_b200 import _seqlib as S

    lib, g = S.lib(), torch.Generator(device=DEV).manual_seed(T + H)
    q, k, v = (torch.randn(T, H, n, generator=g, device=DEV) for n in (K, K, V))
    a, state0 = torch.rand(T, H, K, generator=g, device=DEV) * 0.3 + 0.7, torch.randn(1, H, V, K, generator=g, device=DEV)
    meta, n_chunks = torch.zeros(2, dtype=torch.int32, device=DEV), C.c_int(0)
    n = lib.b2l_seq_scan_plan(T, H, K, V, 1, 0, 0, 0, C.byref(n_chunks))
    assert want == ("chunks" if n_chunks.value > 1 else "walk" if n else "steps")
    assert want != "walk" or n == lib.b2l_seq_scan_work_floats(T, H)
    assert lib.b2l_seq_scan_plan(T, H, K, V, 0, 1, 0, 0, C.byref(n_chunks)) == 0 and n_chunks.value == 1      # delta rule, one decay per head: step by step

    def run(chunks, floats):
        out, state, ws = torch.empty(T, H, V, device=DEV), state0.clone(), torch.full((max(floats, 1) + 64,), 3.0, device=DEV)
        wd = torch.empty(chunks * H * K, device=DEV)
        args = S.ScanArgs(q=q.data_ptr(), ldq=H * K, k=k.data_ptr(), ldk=H * K, v=v.data_ptr(), ldv=H * V, q_mult=1.0, decay=a.data_ptr(), ldd=H * K, decay_per_channel=1,
                          state=state.data_ptr(), meta=meta.data_ptr(), out=out.data_ptr(), ldo=H * V, T=T, heads=H, qk_heads=H, K=K, V=V, act_dtype=S.act_code(torch.float32),
                          work_state=ws.data_ptr() if floats else None, work_decay=wd.data_ptr(), n_chunks=chunks)
        S.check(lib.b2l_seq_scan(C.byref(args), S.stream_ptr()), "scan")
        assert bool((ws[floats:] == 3).all()) or not floats
        return out, state

    out, state = run(1, 0)
    lib.b2l_seq_scan_plan(T, H, K, V, 1, 0, 0, 0, C.byref(n_chunks))
    for got, st in (run(n_chunks.value, n), run(1, lib.b2l_seq_scan_work_floats(T, H))):
        assert rel(got, out) < 1e-6 and rel(st, state) < 1e-6


@pytest.mark.parametrize("T,K,V,H,G,form", [(2048, 128, 128, 16, 16, "delta"), (70, 128, 128, 9, 3, "delta"), (401, 128, 16, 160, 160, "delta"), (512, 128, 64, 32, 1, "scalar"),
                                            (2100, 128, 48, 18, 3, "scalar"), (530, 64, 112, 6, 2, "channel"), (48, 64, 32, 3, 3, "delta")])
def test_scan_in_the_space_it_has(T, K, V, H, G, form):
    """The space counted exactly for the sizes (nothing behind it is written), the fewer floats of the form in f32, and one less, which goes token by token with the
    bits of a call without space.  Sums in another order: 1e-6 of the norm."""
    from lit_llama_b200 import _seqlib as S

    lib, g = S.lib(), torch.Generator(device=DEV).manual_seed(T + V)
    delta, per = int(form == "delta"), int(form != "scalar")
    q, k, v = torch.randn(T, G, K, generator=g, device=DEV), torch.randn(T, G, K, generator=g, device=DEV), torch.randn(T, H, V, generator=g, device=DEV)
    k = k / k.norm(dim=-1, keepdim=True)
    a, beta = torch.rand(T, H, K if per else 1, generator=g, device=DEV) * 0.3 + 0.7, torch.randn(T, H, generator=g, device=DEV)
    state0, meta = torch.randn(1, H, V, K, generator=g, device=DEV), torch.zeros(2, dtype=torch.int32, device=DEV)
    n_chunks, least = C.c_int(0), C.c_longlong(0)
    fast = lib.b2l_seq_scan_space(T, H, G, K, V, per, delta, 0, 0, C.byref(n_chunks), C.byref(least))
    assert n_chunks.value == 1 and 0 < fast <= lib.b2l_seq_scan_work_floats(T, H)

    def run(floats):
        out, state, ws = torch.empty(T, H, V, device=DEV), state0.clone(), torch.full((floats + 4096,), 3.0, device=DEV)
        args = S.ScanArgs(q=q.data_ptr(), ldq=G * K, k=k.data_ptr(), ldk=G * K, v=v.data_ptr(), ldv=H * V, q_mult=1.0, decay=a.data_ptr(), ldd=a.shape[1] * a.shape[2],
                          decay_per_channel=per, beta=beta.data_ptr() if delta else None, ldb=H, delta=delta, state=state.data_ptr(), meta=meta.data_ptr(), out=out.data_ptr(),
                          ldo=H * V, T=T, heads=H, qk_heads=G, K=K, V=V, act_dtype=S.act_code(torch.float32), work_state=ws.data_ptr() if floats else None, n_chunks=1)
        S.check(lib.b2l_seq_scan_within(C.byref(args), floats, S.stream_ptr()), "scan")
        assert bool((ws[floats:] == 3).all())
        return out, state, bool((ws != 3).any())

    out, state, _ = run(0)
    got, st, used = run(fast)
    assert used and rel(got, out) < 1e-6 and rel(st, state) < 1e-6
    if least.value:
        slow, st_slow, used = run(fast - 1)
        assert used and rel(slow, out) < 1e-6 and rel(st_slow, state) < 1e-6 and not torch.equal(slow, got)
        small, st_small, used = run(least.value)
        assert used and torch.equal(small, slow) and torch.equal(st_small, st_slow)
    none, st_none, used = run((least.value or fast) - 1)
    assert not used and torch.equal(none, out) and torch.equal(st_none, state)


@pytest.mark.parametrize("T,K,V,H,G,form", [(47, 128, 48, 24, 2, "delta"), (47, 128, 48, 25, 5, "delta"), (70, 64, 64, 18, 3, "scalar"), (70, 64, 64, 20, 4, "scalar"),
                                            (33, 128, 128, 9, 9, "channel"), (33, 128, 128, 10, 5, "channel")])
def test_scans_by_columns_per_cta(T, K, V, H, G, form):
    """Eight value columns per CTA up to 148 CTAs and sixteen beyond: both sides of the rule."""
    test_scans_sixteen_tokens_at_a_time(T, K, V, H, G, form)


@pytest.mark.parametrize("T,pos0,q_scale,v_mean", [(130, 1900, 1.0, 0.0), (130, 1900, 1.0, 2.0), (200, 900, 4.0, 0.0), (64, 4000, 0.1, 2.0)])
def test_local_attention_rounds_like_f32_over_many_keys(T, pos0, q_scale, v_mean):
    """Sums over thousands of keys carry no bias of the tensor core's truncating adds: relative error below 8e-7 = 13 * 2^-24 (rounded adds of 32
    tile products err by some 3 * 2^-24, scores up to 16 add as much again; truncating accumulators gave 7e-6 to 2.4e-5 here, the f32 kernel
    4e-7 to 1.2e-6), and the mean error towards zero below 4e-7."""
    from lit_llama_b200 import _seqlib as S

    H, G, K, V, n = 8, 2, 128, 64, pos0 + T
    g = torch.Generator(device=DEV).manual_seed(T)
    q, k = torch.randn(T, H, K, generator=g, device=DEV) * q_scale, torch.randn(n, G, K, generator=g, device=DEV).to(BF)
    v = (torch.randn(n, G, V, generator=g, device=DEV) + v_mean).to(BF)
    ring_k, ring_v = k.new_zeros(1, n, G, K), v.new_zeros(1, n, G, V)
    ring_k[0, :pos0], ring_v[0, :pos0] = k[:pos0], v[:pos0]
    kn, vn, out = k[pos0:].contiguous(), v[pos0:].contiguous(), torch.empty(T, H, V, device=DEV)
    meta = torch.tensor([0, pos0], dtype=torch.int32, device=DEV)
    a = S.AttnArgs(q=q.data_ptr(), k_new=kn.data_ptr(), v_new=vn.data_ptr(), ldv=G * V, cache_k=ring_k.data_ptr(), cache_v=ring_v.data_ptr(), meta=meta.data_ptr(),
                   out=out.data_ptr(), ldo=H * V, scale=K ** -0.5, out_mult=1.0, block=n, T=T, heads=H, kv_heads=G, K=K, V=V, act_dtype=S.act_code(BF), window=n, out_f32=1)
    S.check(S.lib().b2l_seq_block_attention(C.byref(a), S.stream_ptr()), "attention")
    seen = torch.arange(n, device=DEV)[None] <= torch.arange(pos0, n, device=DEV)[:, None]
    want = attend(q.double(), k.double().repeat_interleave(H // G, 1), v.double().repeat_interleave(H // G, 1), K ** -0.5, seen)
    assert rel(out, want) < 8e-7
    assert abs(float(((out.double() - want) * want.sign()).sum() / want.abs().sum())) < 4e-7


@pytest.mark.parametrize("M,N,K", [(70, 5120, 13824), (208, 5120, 5120), (350, 4096, 11008), (256, 16384, 1024)])
def test_q4_gemm_other_plans(M, N, K):
    """On 148 SMs: splits of three with five token groups and, uneven, with thirteen (some warps sum a second one), of two with eleven,
    the full tile of 256 tokens."""
    test_q4_gemm_tile_heights_and_splits(M, N, K)


@pytest.mark.parametrize("M,N,K", [(40, 19300, 192), (300, 9700, 320), (20, 38000, 64), (600, 9600, 128)])
def test_q4_gemm_several_tiles_per_cta(M, N, K):
    """More tiles than the 148 SMs: one and two accumulators, k counts that end in half a unit, the second token group without a block; rows whose
    zero point or scale is outside the range in which levels are taken as subnormals, beside ordinary ones.  Products are exact, sums f32."""
    from gpu_util import rand_q4, tile
    from lit_llama_b200 import _lib as L

    lv, qw, sc, z = rand_q4(N, K, DEV, seed=M + N + K)
    sc, z = sc.to(BF), z.to(BF)
    z[64:128:5], z[200:230:3], z[300] = 2.0 ** -120, 0.0, -0.0
    sc[130:160:7], sc[260:270], sc[N - 3] = 2.0 ** 104, 2.0 ** -128, -(2.0 ** 101)
    qt = tile(L, qw, N, K)
    x = torch.randn(M, K, device=DEV).bfloat16()
    y = torch.full((M + 1, N), 7.0, device=DEV, dtype=BF)
    a = L.Q4LinearArgs(x=x.data_ptr(), ldx=K, qw_tiled=qt.data_ptr(), scales=sc.data_ptr(), zeros=z.data_ptr(), sz_dtype=L.sz_dtype_of(sc), y=y.data_ptr(), ldy=N, M=M, N=N, K=K)
    assert L.lib().b2l_q4_gemm(C.byref(a), L.stream_ptr()) == 0, L.lib().b2l_last_error()
    want = x.double() @ ((lv.to(BF) - z) * sc).double().t()
    err = (y[:M].double() - want).norm(dim=0) / want.norm(dim=0)          # per feature: one bf16 rounding
    assert float(err.max()) < 2.0 ** -8 and bool((y[M] == 7).all())


@pytest.mark.parametrize("T,K,V,per_channel", [(65, 128, 48, True), (130, 192, 112, True), (129, 64, 16, False), (200, 80, 128, False)])
def test_local_attention_gates_along_the_rows(T, K, V, per_channel):
    """Outputs stored several rows at a time (2, 1, 8 and 1 of them), gates through shared memory or one per row, rows that end within a turn."""
    from lit_llama_b200 import _seqlib as S

    H, G, win = 4, 2, 96
    g = torch.Generator(device=DEV).manual_seed(T + K)
    q, k, v = torch.randn(T, H, K, generator=g, device=DEV), torch.randn(T, G, K, generator=g, device=DEV).to(BF), torch.randn(T, G, V, generator=g, device=DEV).to(BF)
    n_gate = H * V if per_channel else 8
    gate = (torch.randn(T, n_gate, generator=g, device=DEV) * 3).to(BF)
    gate[1, 0], gate[2, 1] = 100.0, -100.0
    ring_k, ring_v = k.new_zeros(1, win, G, K), v.new_zeros(1, win, G, V)
    out, meta = torch.full((T + 1, H * V), 7.0, device=DEV, dtype=BF), torch.zeros(2, dtype=torch.int32, device=DEV)
    a = S.AttnArgs(q=q.data_ptr(), k_new=k.data_ptr(), v_new=v.data_ptr(), ldv=G * V, cache_k=ring_k.data_ptr(), cache_v=ring_v.data_ptr(), meta=meta.data_ptr(),
                   gate=gate.data_ptr(), ldg=n_gate, gate_per_channel=int(per_channel), out=out.data_ptr(), ldo=H * V, scale=K ** -0.5, out_mult=0.5, block=win, T=T,
                   heads=H, kv_heads=G, K=K, V=V, act_dtype=S.act_code(BF), window=win)
    S.check(S.lib().b2l_seq_block_attention(C.byref(a), S.stream_ptr()), "attention")
    i, j = torch.arange(T, device=DEV)[None], torch.arange(T, device=DEV)[:, None]
    want = attend(q.double(), k.double().repeat_interleave(H // G, 1), v.double().repeat_interleave(H // G, 1), K ** -0.5, (i <= j) & (j - i < win))
    gd = torch.sigmoid(gate.double()).view(T, H, V) if per_channel else torch.sigmoid(gate.double())[:, :H, None]
    assert rel(out[:T].view(T, H, V), want * gd * 0.5) < 2.5e-3 and bool((out[T] == 7).all())


def test_expanded_latent_attention_with_unaligned_queries():
    """Queries whose rows start on 4-byte boundaries only are read entry by entry: the same bits as aligned ones."""
    from lit_llama_b200 import _seqlib as S

    T, H, dn, V = 140, 3, 64, 64
    g = torch.Generator(device=DEV).manual_seed(9)
    kv, q = torch.randn(T, H, V + dn, generator=g, device=DEV).to(BF), torch.randn(T, H, dn, generator=g, device=DEV)
    odd = torch.zeros(T, H * dn + 1, device=DEV)
    odd[:, 1:] = q.view(T, H * dn)
    meta, outs = torch.zeros(2, dtype=torch.int32, device=DEV), []
    for at, ld in ((q.data_ptr(), H * dn), (odd.data_ptr() + 4, H * dn + 1)):
        out = torch.empty(T, H * V, device=DEV, dtype=BF)
        a = S.LatentAttnArgs(q_a=at, ldqa_t=ld, ldqa_h=dn, key_a=kv.data_ptr(), ldka=H * (V + dn), hska=V + dn, meta=meta.data_ptr(), out=out.data_ptr(), ldo=H * V,
                             scale=dn ** -0.5, T=T, heads=H, heads_per_group=1, n_a=V + dn, n_b=0, vdim=V, score_off=V, splits=1, act_dtype=S.act_code(BF))
        S.check(S.lib().b2l_seq_latent_attention(C.byref(a), S.stream_ptr()), "latent attention")
        outs.append(out)
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("act", ["sigmoid", "silu"])
def test_gates_are_within_rounding_of_float64(act):
    """Logistic gates in f32 from -120 to 120, infinities and NaN: expf within its documented 2 ulp (4 * 2^-24 of its value), one addition and one quotient
    (2^-24 each)."""
    from lit_llama_b200 import _seqlib as S

    x = torch.cat([torch.linspace(-120, 120, 40001, device=DEV), torch.tensor([math.inf, -math.inf, math.nan, 0.0, -0.0], device=DEV)])
    y = torch.empty_like(x)
    S.check(S.lib().b2l_seq_unary_act(x.data_ptr(), x.numel(), y.data_ptr(), x.numel(), 1, x.numel(), S.ACT_SIGMOID if act == "sigmoid" else S.ACT_SILU, None,
                                      S.act_code(torch.float32), S.stream_ptr()), "b2l_seq_unary_act")
    xd = x.double()
    want = torch.sigmoid(xd) * (1 if act == "sigmoid" else xd)
    big = want.isfinite() & (want.abs() > 2.0 ** -100)
    assert float(((y.double() - want).abs() / want.abs())[big].max()) < 4 * 2.0 ** -24 * 1.5
    assert bool((y[want.isfinite() & ~big].abs() < 2.0 ** -99).all()) and float(y[-5]) == (1.0 if act == "sigmoid" else math.inf) and math.isnan(float(y[-3]))
    assert float(y[-4]) == 0.0 if act == "sigmoid" else math.isnan(float(y[-4]))


@pytest.mark.parametrize("act", ["sigmoid", "silu"])
def test_small_gates_are_not_lost(act):
    """Down to where 1 + e^-x leaves f32 (x = -88.72) a gate keeps its value: the bound above while the result is normal, and one subnormal step (2^-149) more
    below."""
    from lit_llama_b200 import _seqlib as S

    x = torch.linspace(-88.7, -40, 20001, device=DEV)
    y = torch.empty_like(x)
    S.check(S.lib().b2l_seq_unary_act(x.data_ptr(), x.numel(), y.data_ptr(), x.numel(), 1, x.numel(), S.ACT_SIGMOID if act == "sigmoid" else S.ACT_SILU, None,
                                      S.act_code(torch.float32), S.stream_ptr()), "b2l_seq_unary_act")
    want = torch.sigmoid(x.double()) * (1 if act == "sigmoid" else x.double())
    assert bool(((y.double() - want).abs() <= 6 * 2.0 ** -24 * want.abs() + 2.0 ** -149).all())


@pytest.mark.parametrize("T,H,G,K,V,pos0,window,block,sink,cap", [
    (64, 8, 2, 128, 128, 0, 512, 512, 0, 0.0), (130, 4, 1, 192, 16, 300, 96, 100, 1, 0.0), (257, 4, 2, 64, 112, 90, 0, 128, 0, 30.0), (200, 8, 8, 16, 64, 1000, 333, 333, 1, 0.0), (777, 4, 2, 64, 64, 1300, 1250, 1250, 0, 0.0)])
def test_f32_local_attention_in_three_parts(T, H, G, K, V, pos0, window, block, sink, cap):
    """f32 keys and values as three bf16 parts each: older keys from the ring (entries nobody sees are NaN), windows and blocks, room that nothing has
    written yet, more rows than a CTA's one, and the f32 tiles without room.  Products above 2^-24 are kept and every tile's sum is rounded: the bound of f32 sums at the top."""
    from lit_llama_b200 import _seqlib as S

    n, g, f32 = pos0 + T, torch.Generator(device=DEV).manual_seed(T + K), torch.float32
    q, k, v = torch.randn(T, H, K, generator=g, device=DEV), torch.randn(n, G, K, generator=g, device=DEV), torch.randn(n, G, V, generator=g, device=DEV)
    ring_k, ring_v = k.new_full((1, block, G, K), math.nan), v.new_full((1, block, G, V), math.nan)
    old = torch.arange(max(0, pos0 - window + 1) if window else pos0 // block * block, pos0, device=DEV)
    ring_k[0, old % block], ring_v[0, old % block] = k[old], v[old]
    kn, vn, meta = k[pos0:].contiguous(), v[pos0:].contiguous(), torch.tensor([0, pos0], dtype=torch.int32, device=DEV)
    gate = torch.randn(T, H * V, generator=g, device=DEV)
    i, j = torch.arange(n, device=DEV)[None], torch.arange(pos0, n, device=DEV)[:, None]
    seen = (i <= j) & ((j - i < window) if window else (i // block == j // block))
    want = attend(q.double(), k.double().repeat_interleave(H // G, 1), v.double().repeat_interleave(H // G, 1), K ** -0.5, seen,
                  torch.zeros(H, device=DEV, dtype=torch.float64) if sink else None, cap) * torch.sigmoid(gate.double()).view(T, H, V)
    for room in (True, False):
        out = torch.full((T + 1, H * V), 7.0, device=DEV)
        a = S.AttnArgs(q=q.data_ptr(), k_new=kn.data_ptr(), v_new=vn.data_ptr(), ldv=G * V, cache_k=ring_k.data_ptr(), cache_v=ring_v.data_ptr(), meta=meta.data_ptr(),
                       gate=gate.data_ptr(), ldg=H * V, gate_per_channel=1, out=out.data_ptr(), ldo=H * V, scale=K ** -0.5, softcap=cap, has_sink=sink, out_mult=1.0,
                       block=block, T=T, heads=H, kv_heads=G, K=K, V=V, act_dtype=S.act_code(f32), window=window, no_append=1)
        floats = S.lib().b2l_seq_block_attention_work_floats(C.byref(a))
        work = torch.full((floats,), math.nan, device=DEV)
        if room:
            assert floats > 0
            a.work, a.work_floats = work.data_ptr(), floats
        S.check(S.lib().b2l_seq_block_attention(C.byref(a), S.stream_ptr()), "attention")
        assert rel(out[:T].view(T, H, V), want) < 2e-6 and bool((out[T] == 7).all())


@pytest.mark.parametrize("T,n,group,gate_first,act", [(3, 2048, 2048, 1, "silu"), (2, 1032, 1032, 0, "sigmoid"), (5, 8192, 4096, 1, None), (2, 6400, 6400, 0, "silu"), (3, 1544, 772, 1, "silu")])
def test_gated_norm_of_wide_groups(T, n, group, gate_first, act):
    """One, two and four steps of 2048 channels, a last step that ends within the CTA, groups that do not start on 16 bytes (the form for those); one bf16 rounding of f32 sums."""
    from lit_llama_b200 import _seqlib as S

    g = torch.Generator(device=DEV).manual_seed(n)
    o, w = torch.randn(T, n + 4, generator=g, device=DEV), torch.randn(group, generator=g, device=DEV).to(BF)
    gate, out = torch.randn(T, n + 8, generator=g, device=DEV).to(BF), torch.full((T, n + 8), 7.0, device=DEV, dtype=BF)
    S.check(S.lib().b2l_seq_group_norm_gate(o.data_ptr(), n + 4, w.data_ptr(), 1, gate.data_ptr() if act else None, n + 8, S.ACT_SILU if act == "silu" else S.ACT_SIGMOID, gate_first,
                                            1e-6, 1.5, out.data_ptr(), n + 8, T, n, group, S.act_code(BF), S.stream_ptr()), "norm")
    x, z = o[:, :n].double().view(T, -1, group), gate[:, :n].double().view(T, -1, group)
    z = torch.sigmoid(z) * (z if act == "silu" else 1.0) if act else torch.ones_like(z)
    x = x * z if gate_first else x
    want = 1.5 * x / (x.pow(2).mean(-1, keepdim=True) + 1e-6).sqrt() * w.double() * (1.0 if gate_first else z)
    got = out[:, :n].double().view(T, -1, group)
    assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all()) and bool((out[:, n:] == 7).all())


@pytest.mark.parametrize("T,n,gate_first,act", [(2100, 512, 1, "silu"), (1037, 1024, 0, "sigmoid"), (700, 2048, 1, None), (1500, 768, 0, "silu")])
def test_gated_norm_of_four_groups_a_warp(T, n, gate_first, act):
    """Four, eight and sixteen groups of 128 a token, the last CTA's fewer warps; six groups (the form of one a warp); the tolerance of the wide groups."""
    test_gated_norm_of_wide_groups(T, n, 128, gate_first, act)


@pytest.mark.parametrize("D,off", [(4, 0), (1020, 0), (1024, 4), (1028, 0), (2052, 0), (4096, 0), (4100, 0), (1022, 0), (1024, 1)])
@pytest.mark.parametrize("dt", [BF, torch.float32])
def test_rows_by_fours(D, off, dt):
    """Embedding, norms and cast: fours at the end of each width, widths and starts (`off` elements in) that have none (the other forms).  One rounding of f32
    sums of D squares: 2^-8 of a bf16 output, D 2^-24 at most of an f32 one (4e-6 for the rounding of its square root and products below that)."""
    from lit_llama_b200 import _seqlib as S

    g = torch.Generator(device=DEV).manual_seed(D + off)
    T, V, code, st, lib = 5, 11, S.act_code(dt), S.stream_ptr(), S.lib()

    def rows(n, t=dt):
        return torch.randn(n * D + off, generator=g, device=DEV).to(t)[off:].view(n, D)

    def near(got, want, mag=None):
        tol = (2.0 ** -8 if got.dtype == BF else max(4e-6, D * 2.0 ** -24)) * (want.abs() if mag is None else mag)
        return bool(((got.double() - want).abs() <= tol + 1e-6).all())

    def norm(t):
        return t * (t.pow(2).mean(-1, keepdim=True) + 1e-6).rsqrt()

    table, tok = rows(V), torch.tensor([3, 0, 10, 7, 3], device=DEV)
    x, h = rows(T, torch.float32), rows(T)
    S.check(lib.b2l_seq_embed(tok.data_ptr(), 1, table.data_ptr(), code, 1.5, x.data_ptr(), h.data_ptr(), T, D, V, st), "embed")
    want = table[tok].float() * 1.5
    assert torch.equal(x, want) and torch.equal(h, want.to(dt))
    w, wn, y, pick = rows(1)[0], rows(1)[0], rows(T), torch.tensor([4, 1], dtype=torch.int32, device=DEV)
    S.check(lib.b2l_seq_rmsnorm(x.data_ptr(), w.data_ptr(), 1e-6, h.data_ptr(), pick.data_ptr(), 2, D, code, st), "rmsnorm")
    assert near(h[:2], norm(x[pick.long()].double()) * w.double())
    x0, add = x.double(), 0.7 * norm(y.double()) * w.double()
    S.check(lib.b2l_seq_norm_add_norm(y.data_ptr(), w.data_ptr(), 1e-6, 0.7, x.data_ptr(), wn.data_ptr(), h.data_ptr(), T, D, code, st), "norm_add_norm")
    assert near(x, x0 + add, x0.abs() + add.abs()) and near(h, norm(x0 + add) * wn.double(), (norm(x0.abs() + add.abs()) * wn.double()).abs() * 1.5)
    out = torch.full((T, D + 4), 7.0, device=DEV)
    S.check(lib.b2l_seq_cast_f32(y.data_ptr(), D, out.data_ptr(), D + 4, T, D, code, st), "cast")
    assert torch.equal(out[:, :D], y.float()) and bool((out[:, D:] == 7).all())


@pytest.mark.parametrize("C_,off", [(8, 0), (2040, 0), (2048, 8), (4104, 0), (12288, 0), (2044, 0), (13, 0), (4096, 1)])
@pytest.mark.parametrize("wide", [torch.int64, torch.int32])
def test_embedding_rows_are_copied(C_, off, wide):
    """Rows of one and several 16-byte rounds a thread, rows and starts that have none; tokens outside the table read row 0."""
    from lit_llama_b200 import _lib as L

    V, idx = 9, torch.tensor([3, 8, 0, -1, 9, 3], device=DEV, dtype=wide)
    table = torch.randn(V * C_ + off, device=DEV).to(BF)[off:].view(V, C_)
    out = torch.full((7 * C_ + off,), 7.0, device=DEV, dtype=BF)[off:].view(7, C_)
    L.check(L.lib().b2l_embedding(idx.data_ptr(), int(wide is torch.int64), table.data_ptr(), out.data_ptr(), 6, C_, V, L.stream_ptr()), "embedding")
    assert torch.equal(out[:6], table[[3, 8, 0, 0, 0, 3]]) and bool((out[6] == 7).all())


@pytest.mark.parametrize("rq,rk,dr,rot,inter,off", [(4, 512, 0, 0, 0, 0), (516, 20, 8, 4, 1, 0), (1028, 512, 64, 64, 0, 0), (2048, 2048, 4, 2, 1, 0), (2052, 4, 4, 4, 0, 0), (768, 510, 64, 64, 1, 0), (768, 512, 64, 64, 1, 1)])
@pytest.mark.parametrize("dt", [BF, torch.float32])
def test_latent_rows_by_fours(rq, rk, dr, rot, inter, off, dt):
    """Each number of fours a thread, ranks and starts that have none (the other form), positions past the cache left alone.  Tolerances as for the norms
    above; a rotated entry is two products of angles below 400, themselves 2^-15 off as f32 (256 <= angle < 512): 4e-5 of the pair."""
    from lit_llama_b200 import _seqlib as S

    g = torch.Generator(device=DEV).manual_seed(rq + rk)
    T, pos0, max_pos, ld = 6, 300, 304, rq + rk + dr + 4
    proj = torch.randn(T * ld + off, generator=g, device=DEV)[off:].view(T, ld)
    wq, wk = torch.randn(rq, generator=g, device=DEV).to(dt), torch.randn(rk, generator=g, device=DEV).to(dt)
    freq, meta = torch.rand(max(rot // 2, 1), generator=g, device=DEV), torch.tensor([1, pos0], dtype=torch.int32, device=DEV)
    cq, cache = torch.full((T, rq), 7.0, device=DEV, dtype=dt), torch.full((3, max_pos, rk + dr), 7.0, device=DEV, dtype=dt)
    S.check(S.lib().b2l_seq_latent_prep(proj.data_ptr(), ld, 0, rq, wq.data_ptr(), cq.data_ptr(), rq, rk, wk.data_ptr(), dr, freq.data_ptr(), rot, inter, 1.25, 1e-6,
                                        meta.data_ptr(), cache.data_ptr(), max_pos, T, S.act_code(dt), S.stream_ptr()), "latent_prep")
    p, n = proj.double(), max_pos - pos0

    def near(got, want, mag, eps):
        return bool(((got.double() - want).abs() <= (2.0 ** -8 if dt == BF else 0.0) * want.abs() + eps * mag + 1e-6).all())

    def norm(t):
        return t * (t.pow(2).mean(-1, keepdim=True) + 1e-6).rsqrt()

    want = norm(p[:, :rq]) * wq.double()
    assert near(cq, want, want.abs(), max(4e-6, rq * 2.0 ** -24))
    want = (norm(p[:, rq:rq + rk]) * wk.double())[:n]
    assert near(cache[1, pos0:, :rk], want, want.abs(), max(4e-6, rk * 2.0 ** -24))
    k = p[:n, rq + rk:rq + rk + dr].clone()
    if rot:
        a, b = (slice(0, rot, 2), slice(1, rot, 2)) if inter else (slice(0, rot // 2), slice(rot // 2, rot))
        ang = torch.arange(pos0, max_pos, device=DEV, dtype=torch.float64)[:, None] * freq[:rot // 2].double()
        u, v = k[:, a].clone(), k[:, b].clone()
        k[:, a], k[:, b] = 1.25 * (u * ang.cos() - v * ang.sin()), 1.25 * (v * ang.cos() + u * ang.sin())
    assert near(cache[1, pos0:, rk:], k, 8.0, 4e-5)
    assert bool((cache[0] == 7).all() and (cache[2] == 7).all() and (cache[1, :pos0] == 7).all())


@pytest.mark.parametrize("T,H,size,off,rot,inter,apart", [(1200, 5, 192, 128, 64, 0, 0), (1000, 7, 132, 4, 128, 1, 4), (6000, 1, 64, 0, 60, 0, 0), (1500, 4, 72, 64, 4, 1, 8), (900, 8, 136, 0, 132, 0, 0),
                                                          (1500, 4, 72, 2, 64, 0, 0), (30, 4, 192, 128, 64, 1, 0)])
@pytest.mark.parametrize("src,dst", [(BF, torch.float32), (torch.float32, torch.float32), (BF, BF)])
def test_rotation_of_four_heads_a_warp(T, H, size, off, rot, inter, apart, src, dst):
    """One and two pairs a lane, entries before and after the turned ones, the last warp's fewer heads; more pairs, odd offsets and few tokens (the other form).
    Angles below 0.1 (T + 10) rounded to 2^-24 of themselves, products and sums 2^-22: 1e-5 and T 2^-27 of the largest entry, and a bf16 output's rounding."""
    from lit_llama_b200 import _seqlib as S

    g = torch.Generator(device=DEV).manual_seed(T + size)
    hs = size + apart
    x, freq = torch.randn(T, H * hs, generator=g, device=DEV).to(src), torch.rand(rot // 2, generator=g, device=DEV) * 0.1
    meta, out = torch.tensor([0, 10], dtype=torch.int32, device=DEV), torch.full((T, H * hs), 7.0, device=DEV, dtype=dst)
    S.check(S.lib().b2l_seq_rope(x.data_ptr(), H * hs, int(src is torch.float32), freq.data_ptr(), rot, inter, off, 0.5, 1.1, meta.data_ptr(), out.data_ptr(), H * hs,
                                 int(dst is torch.float32), T, H, size, hs, hs, S.act_code(BF), S.stream_ptr()), "rope")
    want = x.double().view(T, H, hs)[..., :size].clone()
    a, b = (slice(off, off + rot, 2), slice(off + 1, off + rot, 2)) if inter else (slice(off, off + rot // 2), slice(off + rot // 2, off + rot))
    ang = torch.arange(10, T + 10, device=DEV).double()[:, None, None] * freq.double()
    u, v = want[..., a].clone(), want[..., b].clone()
    want[..., a], want[..., b] = 1.1 * (u * ang.cos() - v * ang.sin()), 1.1 * (v * ang.cos() + u * ang.sin())
    want *= 0.5
    got = out.view(T, H, hs)
    tol = (1e-5 + T * 2.0 ** -27) * float(want.abs().max()) + (2.0 ** -8 * want.abs() if dst is BF else 0.0)
    assert bool(((got[..., :size].double() - want).abs() <= tol).all()) and bool((got[..., size:] == 7).all())


@pytest.mark.parametrize("n", [14, 12, 3, 1])
def test_slots_are_zeroed_at_once(n):
    """18, 16, 7 and 5 ranges of whole words (a launch takes 16, so two, one and part of one), odd sizes and empty ones; the neighbouring slots stay."""
    from lit_llama_b200 import _seqlib as S

    sizes = [16, 48, 33, 0, 4096 * 16, 2, 1 << 20] + [32 * (i + 1) for i in range(n)]
    pools = [torch.full((3, n), 5, dtype=torch.uint8, device=DEV) for n in sizes]
    for some in (range(len(sizes)), [3, len(sizes) - 1], [5]):           # all of them, one word range beside an empty one, one odd size
        picked, n = [pools[i] for i in some], len(some)
        for t in picked:
            t.fill_(5)
        S.check(S.lib().b2l_seq_zero_slots((C.c_void_p * n)(*[t.data_ptr() or None for t in picked]), (C.c_size_t * n)(*[sizes[i] for i in some]), n, 1, S.stream_ptr()), "zero")
        for t in picked:
            assert bool((t[1] == 0).all()) and bool((t[0] == 5).all()) and bool((t[2] == 5).all())


@pytest.mark.parametrize("M,N,K", [(1, 128, 8), (17, 130, 72), (113, 300, 64), (70, 2200, 1000), (300, 1025, 200)])
def test_f32_linear_in_three_parts(M, N, K):
    """Token tiles of 16 to 112, ragged features, k that ends within a stage, rows apart; infinite and NaN operands come out as FMAs give them.
    Sums of 64 products of 2^-24 relative error each, rounded once per 64 k: far below sqrt(K) 2^-24."""
    from lit_llama_b200 import _seqlib as S

    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    x, w = torch.randn(M, K + 4, generator=g, device=DEV)[:, :K], torch.randn(N, K + 8, generator=g, device=DEV)[:, :K]
    y = torch.full((M + 1, N + 1), 7.0, device=DEV)

    def run():
        S.check(S.lib().b2l_seq_linear_f32(x.data_ptr(), x.stride(0), w.data_ptr(), w.stride(0), y.data_ptr(), N + 1, M, N, K, S.stream_ptr()), "b2l_seq_linear_f32")
        assert bool((y[M] == 7).all()) and bool((y[:, N] == 7).all())
        return y[:M, :N]

    assert rel(run(), x.double() @ w.double().t()) < 4e-7
    x[0, 1], w[N // 2, 2], w[N - 1] = math.inf, math.nan, w[N - 1] * 1e30
    x[M - 1] *= 1e12
    want, got = torch.nn.functional.linear(x, w), run()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got == math.inf, want == math.inf) and torch.equal(got == -math.inf, want == -math.inf)


@pytest.mark.parametrize("T", [1, 2, 3, 4, 7])
def test_convolution_of_few_tokens_carries_its_inputs(T):
    """Portions of fewer tokens than taps keep some of the inputs carried so far; a portion in two halves gives the same bits as in one."""
    from lit_llama_b200 import _seqlib as S

    Ch, g = 520, torch.Generator(device=DEV).manual_seed(T)
    x, w = torch.randn(2 * T, Ch, generator=g, device=DEV).to(BF), torch.randn(Ch, 4, generator=g, device=DEV).to(BF)
    first, meta = torch.randn(2, 3, Ch, generator=g, device=DEV).to(BF), torch.tensor([1, 0], dtype=torch.int32, device=DEV)

    def run(parts):
        state, outs = first.clone(), []
        for p in parts:
            out = torch.empty(p.shape[0], Ch, device=DEV)
            S.check(S.lib().b2l_seq_conv_silu_unit(p.data_ptr(), Ch, w.data_ptr(), None, state.data_ptr(), meta.data_ptr(), out.data_ptr(), Ch, p.shape[0], Ch, 4, 0, 128, 2, 64, 1e-6,
                                                   0.5, 1.0, S.act_code(BF), S.stream_ptr()), "convolution")
            outs.append(out)
        return torch.cat(outs), state

    whole, state = run([x])
    halves, state2 = run([x[:T], x[T:]])
    assert torch.equal(whole, halves) and torch.equal(state, state2) and torch.equal(state[0], first[0])
    assert torch.equal(state[1], torch.cat([first[1], x])[-3:])
    full = torch.cat([first[1], x]).double()
    want = sum(full[j:j + 2 * T] * w[:, j].double() for j in range(4))
    want = want * torch.sigmoid(want)
    for at, m in ((0, 0.5), (128, 1.0)):
        h = want[:, at:at + 128].view(2 * T, 2, 64)
        want[:, at:at + 128] = (m * h / (h.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt()).view(2 * T, 128)
    assert rel(whole, want) < 1e-6


@pytest.mark.parametrize("T,G,K,bias", [(33, 3, 64, True), (50, 2, 128, False), (20, 2, 128, False), (40, 1, 256, True), (35, 2, 48, False)])
def test_convolution_with_unit_heads(T, G, K, bias):
    """Unit q and k heads out of the convolution's own pass (16, 8 and 32 lanes a head) or after it (short portions, heads of 48): values, gaps between
    the parts, the state.  f32 sums of at most 256 squares."""
    from lit_llama_b200 import _seqlib as S

    k_at = G * K if K != 48 else 104
    v_at, Ch = 2 * k_at, 2 * k_at + 40
    g = torch.Generator(device=DEV).manual_seed(T + K)
    x, w, b = torch.randn(T, Ch + 8, generator=g, device=DEV).to(BF), torch.randn(Ch, 4, generator=g, device=DEV).to(BF), torch.randn(Ch, generator=g, device=DEV).to(BF)
    state = torch.randn(2, 3, Ch, generator=g, device=DEV).to(BF)
    xs = torch.cat([state[1], x[:, :Ch]]).double()
    y = sum(xs[j:j + T] * w[:, j].double() for j in range(4)) + (b.double() if bias else 0.0)
    want = torch.nn.functional.silu(y)
    for at, m in ((0, K ** -0.5), (k_at, 1.0)):
        h = want[:, at:at + G * K].view(T, G, K)
        want[:, at:at + G * K] = (h / torch.sqrt((h * h).sum(-1, keepdim=True) + 1e-6) * m).view(T, G * K)
    out, meta = torch.full((T, Ch), 7.0, device=DEV), torch.tensor([1, 9], dtype=torch.int32, device=DEV)
    S.check(S.lib().b2l_seq_conv_silu_unit(x.data_ptr(), Ch + 8, w.data_ptr(), b.data_ptr() if bias else None, state.data_ptr(), meta.data_ptr(), out.data_ptr(), Ch, T, Ch, 4,
                                           0, k_at, G, K, 1e-6, K ** -0.5, 1.0, S.act_code(BF), S.stream_ptr()), "convolution")
    for lo, hi in ((0, k_at), (k_at, v_at), (v_at, Ch)):
        assert rel(out[:, lo:hi], want[:, lo:hi]) < 1e-6
    assert torch.equal(state[1], xs[-3:].to(BF))


@pytest.mark.parametrize("T,G,K,bias", [(1, 2, 16, True), (2, 3, 64, False), (3, 2, 128, True), (6, 3, 8, True), (9, 5, 4, False), (1597, 16, 64, True), (1602, 12, 128, False), (1599, 8, 256, True),
                                        (3003, 100, 8, False)])
def test_convolution_of_unit_heads_by_fours(T, G, K, bias):
    """Tiles of four and of eight tokens with every remainder, heads of four lanes and more (their roots shared out) and of fewer (token by token)."""
    test_convolution_with_unit_heads(T, G, K, bias)


@pytest.mark.parametrize("size,mode", [(8, 0), (24, 1), (128, 0), (128, 1)])
def test_decays_of_eight_channels(size, mode):
    """exp(-exp(A) softplus(z + b)) and sigmoid(z)^(1/tau) in groups of 8 channels, from -100 to 100 and at infinity.  The exponent e carries the sum's
    rounding, the softplus (3 * 2^-24), the coefficient (2 * 2^-24) and the product, 7 * 2^-24 in all, and e multiplies that; expf adds 2 * 2^-24."""
    from lit_llama_b200 import _seqlib as S

    T, H = 37, 3
    g = torch.Generator(device=DEV).manual_seed(size)
    a, bias, A = (torch.randn(T, H * size, generator=g, device=DEV) * 30).to(BF), torch.randn(H * size, generator=g, device=DEV).to(BF), torch.randn(H, generator=g, device=DEV).to(BF)
    a[0, 0], a[1, 1] = math.inf, -math.inf
    out, dt = torch.empty(T, H * size, device=DEV), torch.empty(T, H * size, device=DEV)
    S.check(S.lib().b2l_seq_decay(a.data_ptr(), H * size, bias.data_ptr(), A.data_ptr(), mode, 16.0 if mode else 0.0, out.data_ptr(), None if mode else dt.data_ptr(), T, H, size,
                                  S.act_code(BF), S.stream_ptr()), "decay")
    z = a.double() + bias.double()
    sp = torch.nn.functional.softplus(-z if mode else z, threshold=1e9)
    e = sp / 16.0 if mode else sp * torch.exp(A.double()).repeat_interleave(size)
    want = torch.exp(-e)
    ok = e < 80
    assert bool((((out.double() - want).abs() / want) < (7 * e + 2) * 2.0 ** -24)[ok].all()) and bool((out[~ok] < 1e-30).all())
    if not mode:
        fin = sp.isfinite() & (sp > 1e-35)
        assert float(((dt.double() - sp).abs() / sp)[fin].max()) < 4e-7 and float(dt[0, 0]) == math.inf and float(dt[1, 1]) == 0.0


@pytest.mark.parametrize("M,N,K,own", [(300, 1024, 1024, True), (9, 32000, 1024, True), (7, 65536, 1024, False), (255, 1024, 1024, False), (600, 1024, 512, True), (700, 1024, 128, True)])
def test_f32_linear_takes_the_form_its_rule_says(M, N, K, own):
    """Through the entry point of the mixers: sizes on both sides of the line, and callers whom only the library's product serves (derivatives, TF32, rows off a
    16-byte boundary).  Which one ran shows in the bits.  f32 sums of K products: 4 sqrt(K) 2^-24 of the norm."""
    from lit_llama_b200 import _seqlib as S
    from lit_llama_b200 import mixers

    g = torch.Generator(device=DEV).manual_seed(M + N)
    wide, w = torch.randn(M, K + 12, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV) * K ** -0.5
    x, library = wide[:, 4:K + 4], torch.nn.functional.linear
    y, here = mixers.linear(x, w), torch.empty(M, N, device=DEV)
    S.check(S.lib().b2l_seq_linear_f32(x.data_ptr(), x.stride(0), w.data_ptr(), K, here.data_ptr(), N, M, N, K, S.stream_ptr()), "b2l_seq_linear_f32")
    assert torch.equal(y, here if own else library(x, w)) and not torch.equal(here, library(x, w))
    assert rel(y, x.double() @ w.double().t()) < 4 * K ** 0.5 * 2.0 ** -24
    off = wide[:, 3:K + 3]
    assert torch.equal(mixers.linear(off, w), library(off, w))
    wg = w.clone().requires_grad_()
    mixers.linear(x, wg).sum().backward()
    assert wg.grad is not None
    with torch.autograd.forward_ad.dual_level():
        out = mixers.linear(torch.autograd.forward_ad.make_dual(x, torch.ones_like(x)), w)
        assert torch.autograd.forward_ad.unpack_dual(out).tangent is not None
    torch.backends.cuda.matmul.allow_tf32 = True
    try:
        assert torch.equal(mixers.linear(x, w), library(x, w))
    finally:
        torch.backends.cuda.matmul.allow_tf32 = False

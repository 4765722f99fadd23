"""Sizes at which the tiling, the scheduling or the dispatch of a kernel changes, against float64 PyTorch.

Bounds: a bf16 result is one rounding (2^-9 relative, 2^-9 / sqrt(3) = 1.1e-3 in the 2-norm) of fp32 sums whose bf16 inputs are exact;
where a bf16 intermediate (P, dS, an activation) enters a further product its rounding adds about as much again
per factor.  5e-3 covers one such intermediate, 1e-2 a chain of them.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(*shape, scale=1.0, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32) * scale).to(torch.bfloat16)


def _rel(got, want):
    return ((got.double() - want.double()).norm() / want.double().norm().clamp_min(1e-30)).item()


def _status_ok():
    from lightron_b200.ops import native
    assert native.device_status() == {}


# ---- attention -------------------------------------------------------------------------------------


def _attention64(q, k, v, do, causal):
    q, k, v = (t.detach().double().requires_grad_(True) for t in (q, k, v))
    B, Sq, hq, d = q.shape
    Sk, rep = k.shape[1], hq // k.shape[2]
    kk, vv = (t.repeat_interleave(rep, 2).transpose(1, 2) for t in (k, v))
    s = q.transpose(1, 2) @ kk.transpose(-1, -2) * d ** -0.5
    if causal:
        s = s.masked_fill(torch.ones(Sq, Sk, dtype=torch.bool, device="cuda").triu(1 + Sk - Sq), -float("inf"))
    o = (s.softmax(-1) @ vv).transpose(1, 2)
    return (o.detach(), *torch.autograd.grad(o, [q, k, v], do.double()))


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("B,Sq,Sk,hq,hkv,causal,scale", [
    (1, 2, 2, 1, 1, True, 1.0),              # smaller than anything that is tiled
    (1, 128, 128, 2, 1, True, 1.0),          # one key block, the second query tile empty
    (2, 129, 129, 4, 2, True, 1.0),          # one row over
    (1, 255, 640, 2, 2, True, 1.0),          # more keys than queries
    (1, 300, 77, 2, 1, False, 1.0),          # last key block ragged, no mask
    (9, 200, 200, 8, 4, True, 1.0),          # 36 (batch, kv head) pairs: past one of the backward's groups of 32
    (1, 700, 700, 4, 1, True, 8.0),          # large scores: the running maximum moves, exponents underflow
])
def test_attention_tile_edges(B, Sq, Sk, hq, hkv, causal, scale, d):
    from lightron_b200.ops import functional as OF
    q, k, v, do = _rand(B, Sq, hq, d, scale=scale, seed=1), _rand(B, Sk, hkv, d, seed=2), _rand(B, Sk, hkv, d, seed=3), _rand(B, Sq, hq, d, seed=4)
    o, lse = OF.flash_fwd_native(q, k, v, causal, d ** -0.5)
    got = (o, *OF.flash_bwd_native(q, k, v, o, lse, do, causal, d ** -0.5))
    _status_ok()
    for name, g, w in zip(("o", "dq", "dk", "dv"), got, _attention64(q, k, v, do, causal)):
        if w.norm() > 1e-6:                  # (with one visible key dq and dk vanish)
            assert _rel(g, w) < 1e-2, name


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("B,S,hq,hkv", [
    (2, 1100, 20, 4),        # 360 query tiles: more than two per SM, so that CTAs go on with a second one; 8 to 9 key blocks, ragged
    (6, 130, 40, 8),         # 480 tiles of one and two key blocks, the second tile two rows long
])
def test_attention_tiles_taken_over(B, S, hq, hkv, d):
    """Every tile is done once, and what lies behind the outputs' last rows is not written (tiles end inside them)."""
    from lightron_b200.ops import functional as OF, native
    q, k, v, do = _rand(B, S, hq, d, seed=1), _rand(B, S, hkv, d, seed=2), _rand(B, S, hkv, d, seed=3), _rand(B, S, hq, d, seed=4)
    buf = [torch.full((B * S + 128, h, d), 7.0, dtype=torch.bfloat16, device="cuda") for h in (hq, hq, hkv, hkv)]
    o, dq, dk, dv = (t[:B * S].view(B, S, -1, d) for t in buf)
    lse = torch.empty(B, hq, S, dtype=torch.float32, device="cuda")
    native.call("lb_flash_fwd_tc", q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr(), B, S, S, hq, hkv, d,
                q.stride(1), k.stride(1), v.stride(1), o.stride(1), d ** -0.5, 1, native.stream_ptr())
    OF.flash_bwd_native(q, k, v, o, lse, do, True, d ** -0.5, dq, dk, dv)
    _status_ok()
    for name, g, w in zip(("o", "dq", "dk", "dv"), (o, dq, dk, dv), _attention64(q, k, v, do, True)):
        assert _rel(g, w) < 1e-2, name
    assert all(bool((t[B * S:] == 7.0).all()) for t in buf)


def test_attention_forward_second_group_of_heads():
    """Longest tiles first within as many heads as have 48 MB of keys and values: 24 of these 32, the second group smaller."""
    from lightron_b200.ops import functional as OF
    B, Sq, Sk, hq, hkv, d = 2, 300, 8192, 16, 8, 128
    q, k, v = _rand(B, Sq, hq, d, seed=1), _rand(B, Sk, hkv, d, seed=2), _rand(B, Sk, hkv, d, seed=3)
    o, lse = OF.flash_fwd_native(q, k, v, True, d ** -0.5)
    _status_ok()
    for b in range(B):
        for h in range(hq):
            s = (q[b, :, h].double() @ k[b, :, h // 2].double().t()) * d ** -0.5
            s.masked_fill_(torch.ones(Sq, Sk, dtype=torch.bool, device="cuda").triu(1 + Sk - Sq), -float("inf"))
            assert _rel(o[b, :, h], s.softmax(-1) @ v[b, :, h // 2].double()) < 5e-3, (b, h)
            assert torch.allclose(lse[b, h].double(), s.logsumexp(-1), atol=1e-4), (b, h)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("n,Sk,S", [(128, 384, 512), (200, 300, 640)])
def test_attention_over_a_prefix_of_longer_buffers(n, Sk, S, d):
    """Context parallelism: the first Sk keys of every batch of a gather buffer of S rows, each 128-key block behind a counter (which
    has been reached here: one rank waits for nobody), and the backward over the same buffers."""
    from lightron_b200.ops import functional as OF, native
    from lightron_b200.parallel import cp_fused
    B, hq, hkv = 2, 4, 2
    q, do = _rand(B, n, hq, d, seed=1), _rand(B, n, hq, d, seed=4)
    kb, vb = _rand(B, S, hkv, d, seed=2), _rand(B, S, hkv, d, seed=3)
    kb[:, Sk:], vb[:, Sk:] = 100.0, -100.0                               # not yet keys of this prefix
    o, lse = torch.empty_like(q), torch.empty(B, hq, n, device="cuda")
    flags = torch.full((B, S // 128), 5, dtype=torch.int32, device="cuda")
    native.call("lb_flash_fwd_cp", q.data_ptr(), kb.data_ptr(), vb.data_ptr(), o.data_ptr(), lse.data_ptr(), B, n, Sk, S, hq, hkv, d,
                hq * d, hq * d, d ** -0.5, 1, flags.data_ptr(), 5, 0, 0, 0, 0, 0, 1, 0, None, None, None, 0, native.stream_ptr())
    got = (o, *cp_fused._bwd_call(q, kb, vb, Sk, S, o, lse, do, d ** -0.5))
    _status_ok()
    want = _attention64(q, kb[:, :Sk].contiguous(), vb[:, :Sk].contiguous(), do, True)
    for name, g, w in zip(("o", "dq", "dk", "dv"), got, want):
        assert _rel(g, w) < 1e-2, name
    o2, _ = OF.flash_fwd_native(q, kb[:, :Sk].contiguous(), vb[:, :Sk].contiguous(), True, d ** -0.5)
    assert torch.equal(o, o2)


@pytest.mark.parametrize("B,Sq,d,shift", [(1, 2, 64, 0), (2, 129, 128, 1)])
def test_attention_backward_scratch_of_the_caller(B, Sq, d, shift):
    """The form whose caller brings one value per row (4-byte aligned) and the accumulator leaves what lies behind them alone; rows
    that are not on 16 bytes are refused."""
    from lightron_b200.ops import functional as OF, native
    h = 2
    q, k, v, do = (_rand(B, Sq, h, d, seed=i) for i in range(4))
    o, lse = OF.flash_fwd_native(q, k, v, True, d ** -0.5)
    n, n_acc = B * h * Sq, B * h * -(-Sq // 128) * 128 * d
    delta, acc = torch.full((shift + 4 * n + 4096,), 7.0, device="cuda"), torch.zeros(n_acc + 4096, device="cuda")
    out = [torch.empty_like(q) for _ in range(3)]

    def call(o_ptr):
        native.call("lb_flash_bwd_tc", q.data_ptr(), k.data_ptr(), v.data_ptr(), o_ptr, do.data_ptr(), lse.data_ptr(),
                    delta.data_ptr() + 4 * shift, acc.data_ptr(), *(t.data_ptr() for t in out), B, Sq, Sq, h, h, d, *[h * d] * 8, d ** -0.5, 1,
                    native.stream_ptr())
    call(o.data_ptr())
    assert (delta[:shift] == 7).all() and (delta[shift + n:] == 7).all() and (acc[n_acc:] == 0).all()
    for g, w in zip(out, _attention64(q, k, v, do, True)[1:]):
        assert _rel(g, w) < 1e-2
    for g, w in zip(out, OF.flash_bwd_native(q, k, v, o, lse, do, True, d ** -0.5)):
        assert _rel(g, w) < 5e-3
    with pytest.raises(native.NativeError):
        call(o.data_ptr() + 2)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("B,Sq,Sk,hq,hkv,causal,parts", [
    (1, 300, 300, 8, 2, True, True),         # a query block per CTA, ragged last ones
    (2, 1000, 1000, 16, 2, True, True),      # parts that end inside a head, and the last of a key block shorter
    (1, 515, 1290, 16, 1, True, True),       # more keys than queries
    (1, 200, 1100, 16, 2, False, True),
    (1, 1290, 130, 16, 2, False, True),      # few keys, long loops
    (8, 640, 640, 8, 8, True, False),        # enough CTAs
])
def test_attention_backward_in_parts(B, Sq, Sk, hq, hkv, causal, d, parts):
    """Key blocks whose loops are cut, against 64 bits and against the launch with the workspace that leaves them whole; rows behind the last are not
    written.  dK and dV are fp32 sums of the same products in another order, rounded once."""
    from lightron_b200.ops import functional as OF, native
    lib = native.require()
    assert (lib.lb_flash_bwd_chunk(B, Sq, Sk, hq, hkv, int(causal), native.sm_count()) > 0) == parts
    need = lib.lb_flash_bwd_ws_bytes(B, Sq, hq, d)
    assert (lib.lb_flash_bwd_ws_bytes_kv(B, Sq, Sk, hq, hkv, d, int(causal)) > need) == parts
    q, do = _rand(B, Sq, hq, d, seed=1), _rand(B, Sq, hq, d, seed=4)
    k, v = _rand(B, Sk, hkv, d, seed=2), _rand(B, Sk, hkv, d, seed=3)
    o, lse = OF.flash_fwd_native(q, k, v, causal, d ** -0.5)
    buf = [torch.full((B * n + 128, h, d), 7.0, dtype=torch.bfloat16, device="cuda") for n, h in ((Sq, hq), (Sk, hkv), (Sk, hkv))]
    dq, dk, dv = (t[:B * n].view(B, n, -1, d) for t, n in zip(buf, (Sq, Sk, Sk)))
    OF.flash_bwd_native(q, k, v, o, lse, do, causal, d ** -0.5, dq, dk, dv)
    whole = [torch.empty_like(t) for t in (dq, dk, dv)]
    ws = native.flash_bwd_workspace(B, Sq, hq, d, q.device)
    native.call("lb_flash_bwd_tc_ws", q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), do.data_ptr(), lse.data_ptr(), ws.data_ptr(), ws.numel(),
                *(t.data_ptr() for t in whole), B, Sq, Sk, hq, hkv, d, *(t.stride(1) for t in (q, k, v, o, do, *whole)), d ** -0.5, int(causal),
                native.stream_ptr())
    _status_ok()
    for name, g, w, x in zip(("dq", "dk", "dv"), (dq, dk, dv), _attention64(q, k, v, do, causal)[1:], whole):
        assert _rel(g, w) < 1e-2 and _rel(g, x.double()) < 2.0 ** -8, name
    assert all(bool((t[B * n:] == 7.0).all()) for t, n in zip(buf, (Sq, Sk, Sk)))


@pytest.mark.parametrize("B,Sq,Sk,hq,hkv,causal,d", [
    (1, 2000, 2000, 16, 2, True, 64), (2, 300, 300, 8, 2, True, 128), (1, 515, 1290, 16, 1, True, 64), (1, 1290, 130, 16, 2, False, 128),
    (1, 128, 128, 16, 1, True, 128), (1, 2000, 77, 4, 1, False, 64),     # one key block: dQ too
    (1, 640, 4096, 16, 1, True, 64),                                     # many key blocks
])
def test_attention_backward_in_parts_repeats_itself(B, Sq, Sk, hq, hkv, causal, d):
    """dK and dV of key blocks whose loops are cut are the same bits in every run, and dQ too where a key block adds to it alone."""
    from lightron_b200.ops import functional as OF, native
    assert native.require().lb_flash_bwd_chunk(B, Sq, Sk, hq, hkv, int(causal), native.sm_count()) > 0
    q, do = _rand(B, Sq, hq, d, seed=1), _rand(B, Sq, hq, d, seed=4)
    k, v = _rand(B, Sk, hkv, d, seed=2), _rand(B, Sk, hkv, d, seed=3)
    o, lse = OF.flash_fwd_native(q, k, v, causal, d ** -0.5)
    runs = [OF.flash_bwd_native(q, k, v, o, lse, do, causal, d ** -0.5) for _ in range(6)]
    _status_ok()
    for name, g, w in zip(("dq", "dk", "dv"), runs[0], _attention64(q, k, v, do, causal)[1:]):
        assert _rel(g, w) < 1e-2, name
    for r in runs[1:]:
        assert torch.equal(r[1], runs[0][1]) and torch.equal(r[2], runs[0][2])
        assert Sk > 128 or torch.equal(r[0], runs[0][0])


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("B,Sq,Sk,hq,hkv,causal", [
    (1, 1, 1, 1, 1, True),
    (2, 128, 128, 3, 3, True),
    (3, 70, 101, 2, 2, True),
    (40, 129, 128, 8, 4, False),             # two query blocks of two heads in a CTA, the second block of one row
    (2, 33, 127, 4, 4, False),
    (40, 200, 5, 4, 4, False),
])
def test_attention_backward_of_one_key_block(B, Sq, Sk, hq, hkv, causal, d):
    """Up to 128 keys dQ is written by the CTA of its key block: against 64 bits, into rows with a stride, of which nothing else is written."""
    from lightron_b200.ops import functional as OF, native
    assert native.require().lb_flash_bwd_chunk(B, Sq, Sk, hq, hkv, int(causal), native.sm_count()) == 0
    q, do = _rand(B, Sq, hq, d, seed=1), _rand(B, Sq, hq, d, seed=4)
    k, v = _rand(B, Sk, hkv, d, seed=2), _rand(B, Sk, hkv, d, seed=3)
    o, lse = OF.flash_fwd_native(q, k, v, causal, d ** -0.5)
    buf = [torch.full((B * n + 128, h * d + 8), 7.0, dtype=torch.bfloat16, device="cuda") for n, h in ((Sq, hq), (Sk, hkv), (Sk, hkv))]
    out = [t[:B * n, :-8].unflatten(0, (B, n)).unflatten(2, (-1, d)) for t, n in zip(buf, (Sq, Sk, Sk))]
    OF.flash_bwd_native(q, k, v, o, lse, do, causal, d ** -0.5, *out)
    _status_ok()
    want = _attention64(q, k, v, do, causal)[1:]
    if Sk == 1:                              # one key: its weight is one, and dQ and dK are rounding
        want = [torch.zeros_like(want[0]), torch.zeros_like(want[1]), want[2]]
        assert max(float(g.abs().max()) for g in out[:2]) < 1e-3      # (sums of d products of some 1, in fp32)
    for name, g, w in zip(("dq", "dk", "dv"), out, want):
        assert not w.any() or _rel(g, w) < 1e-2, name
    assert all(bool((t[B * n:] == 7.0).all() and (t[:, -8:] == 7.0).all()) for t, n in zip(buf, (Sq, Sk, Sk)))


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("Sq,Sk,hq,hkv,causal", [(1, 1, 1, 1, True), (128, 128, 4, 2, True), (70, 101, 2, 1, True), (65, 128, 2, 2, True), (129, 64, 2, 1, False),
                                                  (300, 65, 4, 4, False), (5, 127, 1, 1, False)])
def test_attention_of_one_key_block(Sq, Sk, hq, hkv, causal, d):
    """Up to 128 keys and few tiles: two threads a row.  The same bits as where tiles are many, for finite scores and others."""
    from lightron_b200.ops import functional as OF, native
    n = 2 * native.sm_count() // (hq * ((Sq + 127) // 128)) + 1      # batches with which the other kernel runs
    q, k, v = _rand(2, Sq, hq, d, seed=1), _rand(2, Sk, hkv, d, seed=2), _rand(2, Sk, hkv, d, seed=3)
    for bad in (None, float("inf"), float("nan"), -float("inf")):
        if bad is not None:
            k[1, Sk // 2, 0, 0] = bad
        o, lse = OF.flash_fwd_native(q, k, v, causal, d ** -0.5)
        many = OF.flash_fwd_native(*(t.repeat((n + 1) // 2 + 1, 1, 1, 1) for t in (q, k, v)), causal, d ** -0.5)
        _status_ok()
        if bad is None:
            assert _rel(o, _attention64(q, k, v, torch.zeros_like(q), causal)[0]) < 1e-2
        for g, w in zip((o, lse), many):
            assert torch.equal(g.nan_to_num(7.0), w[:2].nan_to_num(7.0)) and torch.equal(g.isnan(), w[:2].isnan()), bad


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_attention_bad_scores_stay_in_their_rows(d, bad):
    """A key that is not finite spoils the rows that see it, whichever unit computes its exponentials, and no other."""
    from lightron_b200.ops import functional as OF
    S = 300
    for key in (0, 130, 193, 299):
        q, k, v = _rand(1, S, 1, d, seed=1).abs(), _rand(1, S, 1, d, seed=2), _rand(1, S, 1, d, seed=3)
        k[0, key, 0, 0] = bad
        o, _ = OF.flash_fwd_native(q, k, v, True, d ** -0.5)
        want = torch.arange(S, device="cuda") >= key
        assert torch.equal(o[0, :, 0].isnan().all(-1), want) and torch.equal(o[0, :, 0].isnan().any(-1), want), key


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("S,hq,hkv,causal", [(100, 4, 2, True), (100, 200, 200, False), (300, 4, 4, True), (129, 2, 1, False)])
def test_attention_of_a_sequence_beside_a_bad_one(S, hq, hkv, causal, bad, d):
    """Keys and values that are not finite stay in their sequence, also where the one before it ends inside a tile (with one key block and few
    or many tiles, and with several)."""
    from lightron_b200.ops import functional as OF
    q, k, v = _rand(3, S, hq, d, seed=1), _rand(3, S, hkv, d, seed=2), _rand(3, S, hkv, d, seed=3)
    want = OF.flash_fwd_native(q, k, v, causal, d ** -0.5)
    for t in (k, v):
        keep = t[1, 0].clone()
        t[1, 0] = bad
        for g, w in zip(OF.flash_fwd_native(q, k, v, causal, d ** -0.5), want):
            assert torch.equal(g[::2], w[::2])
        t[1, 0] = keep


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("S,Sk,hq,hkv,causal", [(100, 100, 4, 2, True), (300, 300, 4, 4, True), (129, 129, 2, 1, False), (70, 700, 16, 2, False),
                                                 (40, 50, 200, 200, False)])
def test_attention_gradients_of_a_sequence_beside_a_bad_one(S, Sk, hq, hkv, causal, bad, d):
    """The same for what the backward reads, in whole key blocks, parts and the form of one key block.  dK and dV are the same bits; dQ too
    where one key block adds to it, and else the same fp32 terms in another order, rounded once."""
    from lightron_b200.ops import functional as OF
    q, do = _rand(3, S, hq, d, seed=1), _rand(3, S, hq, d, seed=4)
    k, v = _rand(3, Sk, hkv, d, seed=2), _rand(3, Sk, hkv, d, seed=3)

    def grads():
        o, lse = OF.flash_fwd_native(q, k, v, causal, d ** -0.5)
        for g, w in zip((o, lse), fwd):          # (the forward of these two to the bit: what follows is the backward's alone)
            g[::2] = w[::2]
        return OF.flash_bwd_native(q, k, v, o, lse, do, causal, d ** -0.5)
    fwd = OF.flash_fwd_native(q, k, v, causal, d ** -0.5)
    want = grads()
    for t in (q, k, v, do):
        keep = t[1, 0].clone()
        t[1, 0] = bad
        got = grads()
        t[1, 0] = keep
        for i, (g, w) in enumerate(zip(got, want)):
            assert torch.equal(g[::2], w[::2]) if i or Sk <= 128 else _rel(g[::2], w[::2]) < 2.0 ** -8
    _status_ok()


@pytest.mark.parametrize("d", [64, 128])
def test_attention_over_a_prefix_before_anything_else(d):
    """What lies behind the first Sk keys of a longer buffer does not matter, whatever it is."""
    from lightron_b200.ops import native
    B, n, Sk, S, hq, hkv = 2, 200, 300, 640, 4, 2
    q, kb, vb = _rand(B, n, hq, d, seed=1), _rand(B, S, hkv, d, seed=2), _rand(B, S, hkv, d, seed=3)
    flags, outs = torch.full((B, S // 128), 5, dtype=torch.int32, device="cuda"), []
    for rest in (0.0, float("nan")):
        kb[:, Sk:], vb[:, Sk:] = rest, rest
        o, lse = torch.empty_like(q), torch.empty(B, hq, n, device="cuda")
        native.call("lb_flash_fwd_cp", q.data_ptr(), kb.data_ptr(), vb.data_ptr(), o.data_ptr(), lse.data_ptr(), B, n, Sk, S, hq, hkv, d,
                    hq * d, hq * d, d ** -0.5, 1, flags.data_ptr(), 5, 0, 0, 0, 0, 0, 1, 0, None, None, None, 0, native.stream_ptr())
        outs.append((o, lse))
    _status_ok()
    assert all(torch.equal(a, b) for a, b in zip(*outs)) and bool(outs[1][0].isfinite().all())


# ---- GEMM --------------------------------------------------------------------------------------------


def _form(*problems):
    """(parts, CTAs per tile) of a grouped launch of these (M, N, K) on this device: K in `parts` parts in the split form, or 0 and the
    list form with 1 or 2 CTAs per tile."""
    import ctypes
    from lightron_b200.ops import native
    lib, IA = native.require(), ctypes.c_int * len(problems)
    args = (len(problems), *(IA(*[p[i] for p in problems]) for i in range(3)), native.sm_count())
    parts = lib.lb_gemm_grouped_parts(*args)
    return parts, 0 if parts else lib.lb_gemm_grouped_ctas_per_tile(*args)


@pytest.mark.parametrize("M,N,K,n,form", [
    (9000, 2312, 1032, 1, (0, 2)),           # several tiles per pair, the last ones ragged in rows, columns and depth
    (4225, 4104, 2056, 1, (0, 2)),
    (5000, 2312, 72, 1, (0, 1)), (4096, 2304, 512, 1, (0, 1)), (4225, 4104, 200, 1, (0, 1)),
    # three problems are never split.  One tile each: the second CTA's rows beyond the matrix; then single CTAs
    (130, 520, 4104, 3, (0, 2)), (1, 8, 4096, 3, (0, 2)), (130, 520, 1032, 3, (0, 1)), (1, 8, 8, 3, (0, 1)),
    # the same alone
    (130, 520, 4104, 1, (4, 0)), (1, 8, 4096, 1, (4, 0)), (130, 520, 1032, 1, (4, 0)), (1, 8, 8, 1, (1, 0)),
])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_gemm_forms(M, N, K, n, form, a_mn, b_mn):
    """Pairs of CTAs, single ones and the split form, plain and accumulating; which form ran is part of the test."""
    from lightron_b200.ops import functional as OF
    if a_mn and M % 8:
        M = M // 8 * 8 + 8
    assert _form(*[(M, N, K)] * n) == form
    a, b, c0 = _rand(M, K, seed=1), _rand(N, K, seed=2), _rand(M, N, seed=3)
    ops = (a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b)
    want = a.double() @ b.double().t()
    for acc in (False, True):
        outs = [c0.clone() for _ in range(n)]
        OF.gemm_grouped([(*ops, a_mn, b_mn, out, acc) for out in outs])
        _status_ok()
        for out in outs:
            assert _rel(out, want + c0.double() if acc else want) < 5e-3


@pytest.mark.parametrize("T,n,k,apart", [(16, 16384, 264, 1), (72, 16384, 520, 1), (264, 11264, 2048, 0), (1000, 2304, 768, 0), (72, 768, 768, 0)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_weight_and_data_gradient_launches(T, n, k, apart, accumulate):
    """Both gradients of a linear layer, in one launch or, over few rows, in one each."""
    import ctypes
    from lightron_b200.ops import functional as OF, native
    IA = ctypes.c_int * 2
    assert native.require().lb_gemm_grouped_apart(2, IA(n, T), IA(k, k), IA(T, n), native.sm_count()) == apart
    x, w, dy, old = _rand(T, k, seed=1), _rand(n, k, seed=2), _rand(T, n, seed=3), _rand(n, k, seed=4)
    dw = old.clone()
    _, dx = OF.gemm_grouped([(dy, x, True, True, dw, accumulate), (dy, w, False, True, None, False)])
    _status_ok()
    want = dy.double().t() @ x.double()
    assert _rel(dw, want + old.double() if accumulate else want) < 5e-3 and _rel(dx, dy.double() @ w.double()) < 5e-3


def _gemm_split(ks, a, b, a_mn, b_mn, out, accumulate, epi=0, c2=None, half=0):
    """The split form of a GEMM launch, whatever the rule says about these sizes."""
    import ctypes
    from lightron_b200.ops import native
    P, I, L = (lambda v, t=t: (t * 1)(v) for t in (ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong))
    M, K = (a.shape[1], a.shape[0]) if a_mn else a.shape
    native.call("lb_gemm_split", 1, P(a.data_ptr()), P(b.data_ptr()), P(out.data_ptr()), I(M), I(b.shape[1] if b_mn else b.shape[0]), I(K),
                L(a.stride(0)), L(b.stride(0)), L(out.stride(0)), I(int(a_mn)), I(int(b_mn)), I(int(accumulate)), I(epi),
                P(c2.data_ptr() if epi else 0), L(c2.stride(0) if epi else 0), I(half), ks, native.stream_ptr())


@pytest.mark.parametrize("ks", [1, 2, 4])
@pytest.mark.parametrize("M,N,K", [
    (8, 8, 264),             # one row of tiles of which almost nothing exists, 5 k-blocks: parts of 1 and 2
    (72, 200, 328),          # fewer rows than a tile, loaded without the rest
    (136, 64, 1032),         # a second tile of 8 rows, one column tile, the last k-block ragged
    (1000, 776, 256),        # as many k-blocks as parts
    (133, 72, 261),          # no multiple of 8 in rows or depth (rows of the operands on 16 bytes all the same)
    (1, 8, 193),             # one row, one element in the last k-block
])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
def test_gemm_split_tiles(ks, M, N, K, a_mn, b_mn):
    """Parts of K summed over a cluster; nothing is written behind the last row."""
    if a_mn and M % 8:
        M = M // 8 * 8 + 8
    pad = (K + 7) // 8 * 8
    a, b, c0 = _rand(M, pad, seed=1)[:, :K], _rand(N, pad, seed=2)[:, :K], _rand(M, N, seed=3)
    ops = (a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b)
    want = a.double() @ b.double().t()
    buf = torch.full((M + 8, N), 7.0, dtype=torch.bfloat16, device="cuda")
    _gemm_split(ks, *ops, a_mn, b_mn, buf[:M], False)
    acc = c0.clone()
    _gemm_split(ks, *ops, a_mn, b_mn, acc, True)
    _status_ok()
    assert _rel(buf[:M], want) < 5e-3 and _rel(acc, want + c0.double()) < 5e-3 and bool((buf[M:] == 7.0).all())


@pytest.mark.parametrize("M,N,K", [(8, 8, 513), (72, 200, 1032), (136, 64, 4104), (260, 136, 520)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_gemm_split_in_eight(M, N, K, a_mn, b_mn):
    """Each CTA of a cluster finishes eight columns; eight parts of one and more k-blocks, ragged ones; activations are refused."""
    from lightron_b200.ops import native
    if a_mn and M % 8:
        M = M // 8 * 8 + 8
    pad = (K + 7) // 8 * 8
    a, b, c0 = _rand(M, pad, seed=1)[:, :K], _rand(N, pad, seed=2)[:, :K], _rand(M, N, seed=3)
    ops = (a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b)
    want = a.double() @ b.double().t()
    buf = torch.full((M + 8, N), 7.0, dtype=torch.bfloat16, device="cuda")
    _gemm_split(8, *ops, a_mn, b_mn, buf[:M], False)
    acc = c0.clone()
    _gemm_split(8, *ops, a_mn, b_mn, acc, True)
    _status_ok()
    assert _rel(buf[:M], want) < 5e-3 and _rel(acc, want + c0.double()) < 5e-3 and bool((buf[M:] == 7.0).all())
    with pytest.raises(native.NativeError):
        _gemm_split(8, a, b, False, False, buf[:M], False, 1, acc, N // 16 * 8)


@pytest.mark.parametrize("ks", [1, 2, 4])
@pytest.mark.parametrize("T,K,I", [(8, 264, 8), (130, 328, 72), (300, 768, 264)])
def test_gemm_split_activation(ks, T, K, I):
    """silu(g) u and its gradient in the epilogue of a split tile, half of whose columns are gate and half are up."""
    x, w13, dy, w2 = _rand(T, K, seed=1), _rand(2 * I, K, scale=K ** -0.5, seed=2), _rand(T, K, seed=3), _rand(K, I, scale=K ** -0.5, seed=4)
    gu, h, dgu = (torch.empty(T, n, dtype=torch.bfloat16, device="cuda") for n in (2 * I, I, 2 * I))
    _gemm_split(ks, x, w13, False, False, gu, False, 1, h, I)
    _gemm_split(ks, dy, w2, False, True, dgu, False, 2, gu, I)
    _status_ok()
    want = x.double() @ w13.double().t()
    g64 = gu.double().requires_grad_()
    act = torch.nn.functional.silu(g64[:, :I]) * g64[:, I:]
    act.backward(dy.double() @ w2.double())
    assert _rel(gu, want) < 5e-3 and _rel(h, act.detach()) < 5e-3 and _rel(dgu, g64.grad) < 1e-2


@pytest.mark.parametrize("B,S,hq,hkv,d,K,form", [
    (1, 37, 3, 1, 64, 72, (1, 0)), (2, 65, 4, 2, 128, 2056, (4, 0)), (3, 1000, 32, 8, 64, 264, (0, 1)), (4, 1100, 24, 4, 128, 1032, (0, 2)),
])
@pytest.mark.parametrize("placed", [False, True])
def test_projection_with_rotation(B, S, hq, hkv, d, K, form, placed):
    """The rotation in the epilogue against lb_rope on the projection's output: columns that are rotated and columns that are not, ragged rows,
    positions of the caller's.  One rounding of the same fp32 values (test_rotation_has_the_same_bits_everywhere has their order)."""
    from lightron_b200.ops import functional as OF, native
    N, T = (hq + 2 * hkv) * d, B * S
    assert _form((T, N, K)) == form
    x, w = _rand(T, K, seed=1), _rand(N, K, scale=K ** -0.5, seed=2)
    ang = torch.rand(2 * S, d // 2, device="cuda") * 6.28
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    pos = torch.randperm(2 * S, device="cuda")[:S].int().contiguous() if placed else None
    got, want = torch.empty(T, N, device="cuda", dtype=torch.bfloat16), OF.gemm(x, w)
    native.call("lb_gemm_rope", x.data_ptr(), w.data_ptr(), got.data_ptr(), T, N, K, cos.data_ptr(), sin.data_ptr(), native.ptr(pos), S, d,
                (hq + hkv) * d, native.stream_ptr())
    OF._rope_native_(want, cos, sin, pos, S, hq + hkv, d, False)
    _status_ok()
    assert torch.equal(got[:, (hq + hkv) * d:], want[:, (hq + hkv) * d:])
    # a pair's two products cancel at worst: their fp32 rounding against the pair's size, and one unit in the last place of the result
    size = want.float().view(T, -1, 2).norm(dim=-1, keepdim=True).expand(-1, -1, 2).reshape(T, N)
    assert ((got.float() - want.float()).abs() <= 2.0 ** -7 * want.float().abs() + 2.0 ** -22 * size).all()


@pytest.mark.parametrize("B,S,hq,hkv,d,K,form", [
    (1, 128, 12, 12, 64, 768, (1, 0)), (2, 65, 4, 2, 128, 2056, (4, 0)), (3, 1000, 32, 8, 64, 264, (0, 1)), (4, 1100, 24, 4, 128, 1032, (0, 2)),
])
@pytest.mark.parametrize("placed", [False, True])
def test_rotation_has_the_same_bits_everywhere(B, S, hq, hkv, d, K, form, placed):
    """The rotation in the epilogue, lb_rope there and lb_rope back, against the order of operations that they state: one product of a sum
    rounded to fp32 and the other not, in float64 (whose own rounding, 2^-53, moves none of these values)."""
    from lightron_b200.ops import functional as OF, native
    N, T, heads = (hq + 2 * hkv) * d, B * S, hq + hkv
    assert _form((T, N, K)) == form
    x, w = _rand(T, K, seed=1), _rand(N, K, scale=K ** -0.5, seed=2)
    ang = torch.rand(2 * S, d // 2, device="cuda") * 6.28
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    pos = torch.randperm(2 * S, device="cuda")[:S].int().contiguous() if placed else None
    plain, fused = OF.gemm(x, w), torch.empty(T, N, device="cuda", dtype=torch.bfloat16)
    there, back = plain.clone(), plain.clone()
    native.call("lb_gemm_rope", x.data_ptr(), w.data_ptr(), fused.data_ptr(), T, N, K, cos.data_ptr(), sin.data_ptr(), native.ptr(pos), S, d,
                heads * d, native.stream_ptr())
    OF._rope_native_(there, cos, sin, pos, S, heads, d, False)
    OF._rope_native_(back, cos, sin, pos, S, heads, d, True)
    _status_ok()
    assert torch.equal(fused, there)
    i = slice(0, S) if pos is None else pos.long()
    c, s = (t[i].double().view(1, S, 1, d // 8, 4) for t in (cos, sin))
    a, b = plain[:, :heads * d].double().view(B, S, heads, d // 8, 4, 2).unbind(-1)
    r32, first = lambda t: t.float().double(), torch.tensor([True, False, False, False], device="cuda")
    for got, s, rounds_as in ((there, s, first), (back, -s, torch.ones_like(first))):
        want = torch.stack([a * c - r32(b * s), torch.where(rounds_as, b * c + r32(a * s), a * s + r32(b * c))], -1)
        assert torch.equal(got[:, :heads * d], want.float().bfloat16().reshape(T, -1))
        assert torch.equal(got[:, heads * d:], plain[:, heads * d:])


@pytest.mark.parametrize("T,K,I,form", [(2100, 1032, 2312, (0, 2)), (4000, 256, 1288, (0, 1)), (300, 4096, 264, (4, 0)), (70, 512, 264, (1, 0))])
def test_swiglu_mlp_forms(T, K, I, form):
    """The activation in the epilogue of pairs, whose peer loads the up rows, of single CTAs and of the split form; ragged in every size."""
    from lightron_b200.ops import functional as OF
    assert _form((T, 2 * I, K)) == form
    if form == (0, 2):
        assert _form((K, I, T), (T, I, K)) == form           # down projection: weight gradient and dg | du
    w13 = _rand(2 * I, K, scale=K ** -0.5, seed=2)
    ins = [t.detach().requires_grad_(True) for t in (_rand(T, K, seed=1), w13[:I], w13[I:], _rand(K, I, scale=I ** -0.5, seed=3))]
    dy = _rand(T, K, seed=4)
    y = OF.swiglu_mlp(*ins)
    got = (y, *torch.autograd.grad(y, ins, dy))
    _status_ok()
    x, w1, w3, w2 = (t.detach().double().requires_grad_(True) for t in ins)
    yd = (torch.nn.functional.silu(x @ w1.t()) * (x @ w3.t())) @ w2.t()
    for g, w in zip(got, (yd, *torch.autograd.grad(yd, [x, w1, w3, w2], dy.double()))):
        assert _rel(g, w) < 1e-2


@pytest.mark.parametrize("T,K,I,ctas", [(300, 4096, 264, 2), (70, 512, 264, 1)])
def test_activation_in_small_list_tiles(T, K, I, ctas):
    """Activation epilogues of the list form whose columns are fewer than a tile's: three problems, which are never split."""
    from lightron_b200.ops import functional as OF
    assert _form(*[(T, 2 * I, K)] * 3) == (0, ctas) == _form(*[(T, I, K)] * 3)
    x, w13, dy, w2 = _rand(T, K, seed=1), _rand(2 * I, K, scale=K ** -0.5, seed=2), _rand(T, K, seed=3), _rand(K, I, scale=K ** -0.5, seed=4)
    new = lambda n: [torch.empty(T, n, dtype=torch.bfloat16, device="cuda") for _ in range(3)]
    gus, hs, dgus = new(2 * I), new(I), new(2 * I)
    OF.gemm_grouped([(x, w13, False, False, gu, False, 1, h, I) for gu, h in zip(gus, hs)])
    OF.gemm_grouped([(dy, w2, False, True, dgu, False, 2, gu, I) for dgu, gu in zip(dgus, gus)])
    _status_ok()
    want = x.double() @ w13.double().t()
    for gu, h, dgu in zip(gus, hs, dgus):
        g64 = gu.double().requires_grad_()
        act = torch.nn.functional.silu(g64[:, :I]) * g64[:, I:]
        act.backward(dy.double() @ w2.double())
        assert _rel(gu, want) < 5e-3 and _rel(h, act.detach()) < 5e-3 and _rel(dgu, g64.grad) < 1e-2


# ---- norm ----------------------------------------------------------------------------------


@pytest.mark.parametrize("rows,cols", [(1, 8), (3, 264), (700, 1448), (301, 2056), (130, 4096), (65, 4104), (9, 8192), (5, 8200),
                                       (600, 520), (1187, 256), (301, 2312), (301, 2568), (301, 3336), (301, 3592), (700, 4104), (700, 6152), (700, 8192)])
@pytest.mark.parametrize("residual", [False, True])
def test_rmsnorm_widths(rows, cols, residual):
    from lightron_b200.ops import functional as OF
    x, r, w = _rand(rows, cols, seed=1), _rand(rows, cols, seed=2), (1 + 0.1 * _rand(cols, seed=3).float()).to(torch.bfloat16)
    dh, dy = _rand(rows, cols, seed=4), _rand(rows, cols, seed=5)

    def grads(norm, conv):
        xs = [conv(t).requires_grad_(True) for t in ((x, r, w) if residual else (x, w))]
        outs = norm(*xs)
        return (*outs, *torch.autograd.grad(outs, xs, [conv(t) for t in ((dh, dy) if residual else (dy,))]))

    def norm64(*xs):
        h = xs[0] + xs[1] if residual else xs[0]
        y = h * torch.rsqrt(h.square().mean(-1, keepdim=True) + 1e-5) * xs[-1]
        return (h, y) if residual else (y,)

    def norm_native(*xs):
        return OF.add_rmsnorm(*xs, 1e-5) if residual else (OF.rmsnorm(*xs, 1e-5),)
    for g, want in zip(grads(norm_native, lambda t: t.clone()), grads(norm64, lambda t: t.double())):
        assert _rel(g, want) < 5e-3


# ---- embedding ---------------------------------------------------------------------------------------------


@pytest.mark.parametrize("V,H,T,shift", [(50, 264, 300, 0), (50, 264, 300, 2), (2000, 2048, 700, 0), (40, 8, 1, 4)])
def test_embedding_gradient_alignment(V, H, T, shift):
    """Gradient rows on 16-byte boundaries and ``shift`` elements off them; ids outside [10, V - 10) belong to other ranks.
    An id's sum is rounded to bf16 after every one of its occurrences (about ten here: 4 roundings' worth in the 2-norm)."""
    from lightron_b200.ops import functional as OF
    lo, hi = (10, V - 10)
    tok = torch.randint(0, V, (T,), device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    w = _rand(hi - lo, H, seed=2).requires_grad_(True)
    dy = _rand(T * H + shift, seed=3)[shift:].view(T, H)
    got, = torch.autograd.grad(OF.embedding(tok, w, lo), w, dy)
    mine = (tok >= lo) & (tok < hi)
    want = torch.zeros(hi - lo, H, dtype=torch.float64, device="cuda").index_add_(0, tok[mine] - lo, dy[mine].double())
    assert (got.double() - want).norm() <= 1e-2 * want.norm()


# ---- loss ------------------------------------------------------------------------------------------------


@pytest.mark.parametrize("T,V", [(1, 8), (33, 264), (1025, 1000), (4100, 64), (8192, 8), (8193, 8), (140001, 16)])
def test_cross_entropy_loss_rows(T, V):
    """Fewer rows than threads, more, more than one block takes, ignored ones; the loss is an fp32 sum (1e-6) of fp32 rows over bf16 logits."""
    from lightron_b200.ops import functional as OF
    logits, tgt = _rand(T, V, scale=3.0, seed=1), torch.randint(0, V, (T,), device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    tgt[1::7] = -100
    x = logits.clone().requires_grad_(True)
    loss = OF.cross_entropy(x * 1, tgt)
    got, = torch.autograd.grad(loss, x)
    w = logits.double().requires_grad_(True)
    want = torch.nn.functional.cross_entropy(w, tgt)
    assert abs(loss.item() - want.item()) < 4e-6 * max(1.0, want.item())
    assert _rel(got, torch.autograd.grad(want, w)[0]) < 5e-3


@pytest.mark.parametrize("V", [8, 2040, 2056, 8184, 8200, 32000])
@pytest.mark.parametrize("masked", [None, -float("inf"), torch.finfo(torch.bfloat16).min])
def test_cross_entropy_widths(V, masked):
    """Widths around what a step of the row statistics takes, with masked columns in whole steps and in parts of them."""
    from lightron_b200.ops import functional as OF
    T = 5
    logits, tgt = _rand(T, V, scale=3.0, seed=1), torch.full((T,), V - 1, device="cuda")
    if masked is not None:
        logits[:, :V - 3] = masked
        logits[1, :] = _rand(V, seed=2)
        logits[2, 3:V // 2] = 1.0
    x = logits.clone().requires_grad_(True)
    loss = OF.cross_entropy(x * 1, tgt, n_valid_total=T)
    got, = torch.autograd.grad(loss, x)
    w = logits.double().requires_grad_(True)
    want = torch.nn.functional.cross_entropy(w, tgt)
    assert abs(loss.item() - want.item()) < 4e-6 * max(1.0, want.item())
    assert _rel(got, torch.autograd.grad(want, w)[0]) < 5e-3


# ---- mixture of experts ------------------------------------------------------------------------------------


@pytest.mark.parametrize("T,H,E,k", [(1, 64, 4, 2), (8, 264, 12, 2), (9, 264, 12, 2), (70, 264, 5, 1), (300, 512, 40, 3), (65, 2056, 64, 8),
                                     (8200, 4104, 9, 2)])
def test_moe_router_tiles(T, H, E, k):
    """Ragged last block of tokens, a width that is no multiple of the column tile, one to eight passes over the experts; one token of
    a warp at a time (up to 8 tokens) and four."""
    from lightron_b200.ops import native
    x, wg, dev = _rand(T, H, seed=1), _rand(E, H, scale=H ** -0.5, seed=2), "cuda"
    lib = native.require()
    nblk = lib.lb_moe_router_blocks(T)
    probs, wts = torch.empty(T, E, device=dev), torch.empty(T, k, device=dev)
    idx, within = torch.empty(T, k, dtype=torch.int32, device=dev), torch.zeros(nblk * 32, k, dtype=torch.int32, device=dev)
    hist, psum = torch.empty(nblk, E, dtype=torch.int32, device=dev), torch.empty(nblk, E, device=dev)
    native.call("lb_moe_router", x.data_ptr(), wg.data_ptr(), T, H, E, k, probs.data_ptr(), idx.data_ptr(), wts.data_ptr(),
                within.data_ptr(), hist.data_ptr(), psum.data_ptr(), native.stream_ptr())
    xd, wd = x.double().requires_grad_(True), wg.double().requires_grad_(True)
    want = (xd @ wd.t()).softmax(-1)
    assert torch.allclose(probs.double(), want, atol=1e-6, rtol=1e-4)          # fp32 sums of H exact products
    assert torch.equal(torch.gather(probs, 1, idx.long()), wts) and torch.equal(hist.sum(0), torch.bincount(idx.reshape(-1), minlength=E).int())
    dwts, frac, daux = torch.randn(T, k, device=dev), torch.rand(E, device=dev), torch.tensor([0.7], device=dev)
    dx, dwg = torch.empty_like(x), torch.zeros(E, H, device=dev)
    native.call("lb_moe_router_bwd", x.data_ptr(), wg.data_ptr(), probs.data_ptr(), idx.data_ptr(), dwts.data_ptr(), frac.data_ptr(),
                daux.data_ptr(), dx.data_ptr(), dwg.data_ptr(), T, H, E, k, native.stream_ptr())
    loss = (want.gather(1, idx.long()) * dwts.double()).sum() + 0.7 * E * (frac.double() * want.mean(0)).sum()
    gx, gw = torch.autograd.grad(loss, [xd, wd])
    assert _rel(dx, gx) < 5e-3 and _rel(dwg, gw) < 1e-4


@pytest.mark.parametrize("shift", [0, 1, 2])
def test_moe_router_gradient_alignment(shift):
    """The gate gradient is added to a buffer on 16 bytes or ``shift`` elements off it (fp32 sums: 1e-4 as above)."""
    from lightron_b200.ops import native
    T, H, E, k, dev = 70, 264, 5, 2, "cuda"
    x, wg = _rand(T, H, seed=1), _rand(E, H, scale=H ** -0.5, seed=2)
    probs = torch.rand(T, E, device=dev).softmax(-1)
    idx = torch.stack([torch.randperm(E, device=dev)[:k] for _ in range(T)]).int()
    dwts, frac, dx = torch.randn(T, k, device=dev), torch.zeros(E, device=dev), torch.empty_like(x)
    buf = torch.ones(E * H + 8, device=dev)
    native.call("lb_moe_router_bwd", x.data_ptr(), wg.data_ptr(), probs.data_ptr(), idx.data_ptr(), dwts.data_ptr(), frac.data_ptr(),
                0, dx.data_ptr(), buf.data_ptr() + 4 * shift, T, H, E, k, native.stream_ptr())
    dp = torch.zeros(T, E, dtype=torch.float64, device=dev).scatter_add_(1, idx.long(), dwts.double())
    dl = probs.double() * (dp - (probs.double() * dp).sum(-1, keepdim=True))
    assert _rel(buf[shift:shift + E * H].view(E, H), 1 + dl.t() @ x.double()) < 1e-4 and _rel(dx, dl @ wg.double()) < 5e-3
    assert (buf[:shift] == 1).all() and (buf[shift + E * H:] == 1).all()


def test_moe_expert_without_tokens_gets_zero_gradients():
    """Gradients outside an arena are written, not accumulated, into memory that holds anything."""
    from lightron_b200.config import ModelArgs
    from lightron_b200.models.llama import LightronTransformer, flatten_parameters
    from lightron_b200.models.moe import MoEFeedForward
    H, I, E = 256, 520, 4
    ctx = LightronTransformer(ModelArgs(dim=64, n_layers=0, n_heads=1, vocab_size=64)).ctx
    layer = MoEFeedForward(ModelArgs(dim=H, n_layers=1, n_heads=4, vocab_size=64, intermediate_size=I, moe_num_experts=E, moe_topk=2,
                                     moe_layer_freq=1), ctx, dtype=torch.bfloat16, device="cuda")
    flatten_parameters(layer)
    x = _rand(300, H, seed=1).abs().requires_grad_(True)
    with torch.no_grad():
        for i, p in enumerate(layer.parameters()):
            p.copy_(_rand(*p.shape, scale=p.shape[1] ** -0.5, seed=10 + i))
        layer.gate.weight[2] = -1.0                              # x >= 0: expert 2 is never among the best two
    for p in layer.parameters():
        p.grad = None
    junk = [torch.full((E, 2 * I, H), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(4)]
    del junk
    names, ps = zip(*layer.named_parameters())
    grads = dict(zip(names, torch.autograd.grad(layer(x), ps, _rand(300, H, seed=3))))
    _status_ok()
    for n, g in grads.items():
        assert torch.isfinite(g).all(), n
        assert "experts." not in n or g.untyped_storage().nbytes() <= 2 * 2 * I * H, n        # kept without the other experts' memory
        assert ("experts.2." in n) == (not g.any()), n


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("T,H", [(1, 8), (5, 264), (37, 2056), (9, 4160)])
def test_moe_rows_pushed_and_pulled(T, H, k):
    """Every slot count and row widths around the vectors a warp has in flight, with copies beyond the capacity and infinite row weights of
    those: exact copies out, sums in slot order back."""
    import ctypes
    from lightron_b200.ops import native
    E, cap = 8, T * k + 3
    g = torch.Generator(device="cuda").manual_seed(T + k)
    x = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.rand(T, k, generator=g, device="cuda")
    idx = torch.rand(T, E, generator=g, device="cuda").argsort(1)[:, :k].int().contiguous()
    rows = torch.randperm(T * k, generator=g, device="cuda").int().view(T, k).contiguous()
    rows[-1, -1] = cap                                  # beyond the capacity: neither stored nor read
    seg = torch.zeros(2 * E + 2, dtype=torch.int32, device="cuda")
    buf = torch.zeros(cap, H, device="cuda", dtype=torch.bfloat16)
    words = torch.zeros(64, dtype=torch.int32, device="cuda")
    one = lambda p: (ctypes.c_void_p * 1)(p)
    st = native.stream_ptr()
    live = rows < cap
    for scale in (None, w):
        buf.zero_()
        native.call("lb_moe_push", x.data_ptr(), native.ptr(scale), idx.data_ptr(), 0, 0, 0, rows.data_ptr(), seg.data_ptr(), T, H, E, k, 1, 0,
                    cap, 0, one(buf.data_ptr()), one(words.data_ptr()), st)
        want = torch.zeros(cap, H, device="cuda", dtype=torch.bfloat16)
        src = x[:, None, :].expand(T, k, H) if scale is None else (x[:, None, :].float() * w[..., None]).to(torch.bfloat16)
        want[rows[live].long()] = src[live]
        assert torch.equal(buf, want)
    buf = torch.randn(cap, H, generator=g, device="cuda").to(torch.bfloat16)
    buf[rows[~live].long().clamp(max=cap - 1)] = float("nan")
    w[~live] = float("inf")
    out, dots = torch.empty(T, H, device="cuda", dtype=torch.bfloat16), torch.empty(T, k, device="cuda")
    native.call("lb_moe_pull", out.data_ptr(), w.data_ptr(), idx.data_ptr(), rows.data_ptr(), dots.data_ptr(), x.data_ptr(), T, H, E, k, 1, 0,
                cap, one(buf.data_ptr()), one(words.data_ptr() + 128), 1, st)
    got = torch.where(live[..., None], buf[rows.long().clamp(max=cap - 1)].double(), torch.zeros((), device="cuda", dtype=torch.float64))
    want = (got * torch.where(live, w, 0.0)[..., None].double()).sum(1)
    mass = (got.abs() * torch.where(live, w, 0.0)[..., None].double()).sum(1)
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + (k + 1) * 2.0 ** -23 * mass).all()   # fp32 sums, one rounding to bf16
    terms = got * x[:, None, :].double()
    assert ((dots.double() - terms.sum(-1)).abs() <= (H / 32 + 6) * 2.0 ** -23 * terms.abs().sum(-1)).all()
    native.call("lb_moe_pull", out.data_ptr(), 0, idx.data_ptr(), rows.data_ptr(), 0, 0, T, H, E, k, 1, 0, cap, one(buf.data_ptr()),
                one(words.data_ptr() + 128), 2, st)
    assert ((out.double() - got.sum(1)).abs() <= 2.0 ** -8 * got.sum(1).abs() + k * 2.0 ** -23 * got.abs().sum(1)).all()
    native.device_status()           # the dropped copies were counted: read and cleared


@pytest.mark.parametrize("T,H,k", [(1, 8, 1), (37, 2056, 2), (9, 264, 5)])
def test_moe_rows_pulled_onto_another_row(T, H, k):
    """The k rows and one more, added in fp32 and rounded once."""
    import ctypes
    from lightron_b200.ops import native
    buf, add, out = _rand(T * k, H, seed=1), _rand(T, H, seed=2), torch.empty(T, H, device="cuda", dtype=torch.bfloat16)
    idx = torch.zeros(T, k, dtype=torch.int32, device="cuda")
    rows = torch.randperm(T * k, device="cuda").int().view(T, k).contiguous()
    words = torch.zeros(8, dtype=torch.int32, device="cuda")
    one = lambda p: (ctypes.c_void_p * 1)(p)
    native.call("lb_moe_pull_add", out.data_ptr(), add.data_ptr(), 0, idx.data_ptr(), rows.data_ptr(), 0, 0, T, H, 8, k, 1, 0, T * k,
                one(buf.data_ptr()), one(words.data_ptr()), 1, native.stream_ptr())
    terms = torch.cat([buf[rows.long()].double(), add[:, None].double()], 1)
    assert ((out.double() - terms.sum(1)).abs() <= 2.0 ** -8 * terms.sum(1).abs() + (k + 1) * 2.0 ** -23 * terms.abs().sum(1)).all()
    _status_ok()


@pytest.mark.parametrize("nblk,E", [(1, 1), (31, 9), (33, 8), (129, 64), (300, 5)])
def test_moe_plan_sums_over_blocks(nblk, E):
    """Numbers of blocks and experts around what a step of the plan takes: exact whole numbers, fp32 sums of the probabilities."""
    import ctypes
    from lightron_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(nblk)
    dev, k = "cuda", 1
    hist = torch.randint(0, 9, (nblk, E), generator=g, device=dev, dtype=torch.int32)
    psum = torch.rand(nblk, E, generator=g, device=dev)
    T = int(hist.sum())
    base, row0, seg = (torch.full(s, -1, dtype=torch.int32, device=dev) for s in ((nblk, E), (E,), (2 * E + 2,)))
    frac, aux, words = torch.empty(E, device=dev), torch.empty(1, device=dev), torch.zeros(4096, dtype=torch.int32, device=dev)
    one = lambda p: (ctypes.c_void_p * 1)(p)
    native.call("lb_moe_plan", hist.data_ptr(), psum.data_ptr(), base.data_ptr(), row0.data_ptr(), seg.data_ptr(), frac.data_ptr(), aux.data_ptr(),
                nblk, E, 1, 0, T, k, 1 << 20, one(words.data_ptr() + 4096), one(words.data_ptr()), 1, 1, native.stream_ptr())
    n = hist.sum(0)
    assert torch.equal(base, (hist.cumsum(0) - hist).int())
    start = ((n + 127) // 128 * 128).cumsum(0) - (n + 127) // 128 * 128
    assert torch.equal(row0, start.int()) and torch.equal(seg[:E], start.int()) and torch.equal(seg[E:2 * E], n.int())
    assert int(seg[2 * E + 1]) == T
    want = E * ((n.double() / T) * (psum.double().sum(0) / T)).sum()
    assert abs(float(aux) / float(want) - 1) < (nblk + 8) * 2.0 ** -23
    _status_ok()


@pytest.mark.parametrize("H,I,counts,ctas", [(72, 264, (130, 0, 1, 300), 1), (264, 8, (130, 0, 1, 300), 1), (520, 1032, (130, 0, 1, 300), 1),
                                             (4104, 264, (300, 0, 129, 1290), 2)])
def test_ragged_expert_gemms(H, I, counts, ctas):
    """Activation epilogues and weight gradients in single CTAs and in pairs, whose last tile may end in the next segment: segments of one to several
    tiles, without rows and of one row; widths that end inside a tile and inside a step of 64 columns."""
    from lightron_b200.ops import native
    from lightron_b200.parallel import ep_fused
    LE, cap = len(counts), 1024 if ctas == 1 else 2560
    off, seg = 0, []
    for c in counts:
        seg.append(off)
        off += (c + 127) // 128 * 128
    assert off < cap
    lib, sms = native.require(), native.sm_count()
    assert [lib.lb_gemm_ragged_ctas_per_tile(LE, cap, n, k, sms) for n, k in ((2 * I, H), (I, H), (H, 0))] == [ctas] * 3
    table = torch.tensor([*seg, *counts, off, sum(counts)], dtype=torch.int32, device="cuda")
    x, dy = _rand(cap, H, seed=1), _rand(cap, H, seed=2)
    live = torch.zeros(cap, dtype=torch.bool, device="cuda")
    for o, c in zip(seg, counts):
        live[o:o + c] = True
    x[~live] = 0
    dy[~live] = 0
    up = [_rand(2 * I, H, scale=H ** -0.5, seed=10 + e) for e in range(LE)]
    down = [_rand(H, I, scale=I ** -0.5, seed=20 + e) for e in range(LE)]
    gu, act, dgu = (torch.full((cap, n), 7.0, device="cuda", dtype=torch.bfloat16) for n in (2 * I, I, 2 * I))
    ep_fused._ragged(x, up, gu, table, LE, cap, 2 * I, H, False, epi=1, c2=act, half=I)
    ep_fused._ragged(dy, down, dgu, table, LE, cap, I, H, True, epi=2, c2=gu, half=I)
    old = [_rand(2 * I, H, seed=30 + e) for e in range(LE)]
    dw = [[w.clone() for w in old] for _ in range(2)]
    for accumulate in (0, 1):
        ep_fused._ragged_wgrad(dgu, x, dw[accumulate], table, LE, cap, 2 * I, H, accumulate)
    _status_ok()
    assert (gu[off:] == 7).all() and (act[off:] == 7).all() and (dgu[off:] == 7).all()
    for e, (o, c) in enumerate(zip(seg, counts)):
        r = slice(o, o + c)
        grad = dgu[r].double().t() @ x[r].double()
        for accumulate in (0, 1):
            want = grad + old[e].double() * accumulate
            assert _rel(dw[accumulate][e], want) < 5e-3 if want.any() else not dw[accumulate][e].any()
        if not c:
            continue
        assert _rel(gu[r], x[r].double() @ up[e].double().t()) < 5e-3
        g, u = gu[r].double().split(I, 1)
        sig = torch.sigmoid(g)
        assert _rel(act[r], g * sig * u) < 5e-3
        dh = dy[r].double() @ down[e].double()
        assert _rel(dgu[r], torch.cat([dh * u * sig * (1 + g * (1 - sig)), dh * g * sig], 1)) < 1e-2        # (dh is rounded to bf16 first)


@pytest.mark.parametrize("H,I,counts,ctas", [(72, 264, (130, 0, 1, 300), 1), (4104, 264, (300, 0, 129, 1290), 2)])
def test_ragged_activation_without_gate_and_up(H, I, counts, ctas):
    """The activation alone, with a null C: the same bits, and the output of the call before it is left as it is."""
    from lightron_b200.ops import native
    from lightron_b200.parallel import ep_fused
    LE, cap = len(counts), 1024 if ctas == 1 else 2560
    pad = [(c + 127) // 128 * 128 for c in counts]
    seg = [sum(pad[:e]) for e in range(LE)]
    assert native.require().lb_gemm_ragged_ctas_per_tile(LE, cap, 2 * I, H, native.sm_count()) == ctas
    table = torch.tensor([*seg, *counts, sum(pad), sum(counts)], dtype=torch.int32, device="cuda")
    x, up = _rand(cap, H, seed=1), [_rand(2 * I, H, scale=H ** -0.5, seed=10 + e) for e in range(LE)]
    gu, act, alone = (torch.full((cap, n), 7.0, device="cuda", dtype=torch.bfloat16) for n in (2 * I, I, I))
    ep_fused._ragged(x, up, gu, table, LE, cap, 2 * I, H, False, epi=1, c2=act, half=I)
    gu.fill_(3.0)
    native.call("lb_gemm_ragged_epi", x.data_ptr(), ep_fused._ptr_array(up), 0, table.data_ptr(), LE, cap, 0, 2 * I, H, H, H, 2 * I, 0, 1,
                alone.data_ptr(), I, I, 0, 0, native.stream_ptr())
    _status_ok()
    assert torch.equal(alone, act) and bool((gu == 3.0).all())


@pytest.mark.parametrize("rows,ctas", [(0, 2), (300, 1), (8192, 2)])
def test_expected_rows_choose_the_form_alone(rows, ctas):
    """Fewer or more rows than expected are computed all the same."""
    from lightron_b200.ops import native
    from lightron_b200.parallel import ep_fused
    H, N, counts, seg, cap = 2048, 4104, (500, 0, 129, 1290), (0, 512, 512, 768), 2560
    LE, lib, sms = len(counts), native.require(), native.sm_count()
    held = rows + LE * 128 if rows else cap
    assert [lib.lb_gemm_ragged_ctas_per_tile(LE, held, *a, sms) for a in ((N, H), (H, 0))] == [ctas] * 2
    table = torch.tensor([*seg, *counts, 2176, sum(counts)], dtype=torch.int32, device="cuda")
    x, dy = torch.zeros(cap, H, dtype=torch.bfloat16, device="cuda"), torch.zeros(cap, N, dtype=torch.bfloat16, device="cuda")
    for o, c in zip(seg, counts):
        x[o:o + c], dy[o:o + c] = _rand(c, H, seed=c), _rand(c, N, seed=c + 1)
    w = [_rand(N, H, scale=H ** -0.5, seed=10 + e) for e in range(LE)]
    y = torch.full((cap, N), 7.0, device="cuda", dtype=torch.bfloat16)
    dw = [torch.full((N, H), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(LE)]
    ep_fused._ragged(x, w, y, table, LE, cap, N, H, False, rows=rows)
    ep_fused._ragged_wgrad(dy, x, dw, table, LE, cap, N, H, False, rows)
    _status_ok()
    assert (y[2176:] == 7).all()
    for e, (o, c) in enumerate(zip(seg, counts)):
        r, grad = slice(o, o + c), dy[o:o + c].double().t() @ x[o:o + c].double()
        assert _rel(dw[e], grad) < 5e-3 if c else not dw[e].any()
        assert not c or _rel(y[r], x[r].double() @ w[e].double().t()) < 5e-3


@pytest.mark.parametrize("n", [0, 1, 15, 16, 17, 4095, 4096, 4111, 1 << 20, (1 << 20) + 7])
def test_clear_writes_its_bytes_and_no_others(n):
    from lightron_b200.ops import native
    buf = torch.full((n + 64,), 7, dtype=torch.uint8, device="cuda")
    native.call("lb_clear", buf.data_ptr() + 16, n, native.stream_ptr())
    assert not buf[16:16 + n].any() and (buf[:16] == 7).all() and (buf[16 + n:] == 7).all()
    with pytest.raises(native.NativeError):
        native.call("lb_clear", buf.data_ptr() + 8, n, native.stream_ptr())


# ---- dependent launches --------------------------------------------------------------------------------


@pytest.mark.parametrize("M,N,K", [(128, 768, 2048), (1000, 4096, 768), (40, 64, 64)])      # split over K, list form, one tile
@pytest.mark.parametrize("captured", [False, True])
def test_launches_see_what_the_ones_before_them_wrote(M, N, K, captured):
    """A launch starts under the tail of the one before it (and asks for its second operand ahead of time): weights that have just been
    written, and every step of a chain, are the new ones."""
    from lightron_b200.ops import functional as OF, native
    a, w0, step = _rand(M, K, seed=1), _rand(N, K, seed=2), _rand(N, K, seed=3, scale=0.125)
    norm = torch.ones(N, device="cuda", dtype=torch.bfloat16)
    w, ys = w0.clone(), []

    def chain():
        for _ in range(6):
            native.call("lb_add_inplace", w.data_ptr(), step.data_ptr(), w.numel(), native.stream_ptr())
            y = OF.gemm(a, w)
            ys.append((y, OF.rmsnorm(y, norm, 1e-5)))

    if captured:
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            chain()                                  # (the first launch of a size uploads its schedule)
        torch.cuda.synchronize()
        w.copy_(w0)
        ys.clear()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            chain()
        g.replay()
    else:
        chain()
    torch.cuda.synchronize()
    _status_ok()
    want_w = w0.clone()
    for y, n in ys:
        want_w = (want_w.float() + step.float()).bfloat16()
        want = a.double() @ want_w.double().t()
        # bf16 results: half a unit in the last place is 2^-9 of the value
        assert _rel(y, want) < 5e-3
        assert _rel(n, y.double() * torch.rsqrt(y.double().square().mean(-1, keepdim=True) + 1e-5)) < 5e-3
    assert torch.equal(w, want_w)


@pytest.mark.parametrize("kind", ["plan", "pull", "attention"])
def test_a_wait_for_other_gpus_keeps_no_other_stream_waiting(kind):
    """While a kernel waits for a peer (whose flag nothing sets here: it gives up after half a second and says so), the launch behind it
    holds no SMs: a kernel of another stream that needs half of the chip gets it."""
    import ctypes
    from lightron_b200.ops import functional as OF, native
    a, b = _rand(4096, 2048, seed=1), _rand(4096, 2048, seed=2)
    assert _form((4096, 4096, 2048))[0] == 0                            # a CTA's 200 KB of shared memory on every SM
    q, do = _rand(1, 512, 8, 128, seed=3), _rand(1, 512, 8, 128, seed=4)
    o, lse = OF.flash_fwd_native(q, q, q, False, 128 ** -0.5)
    words, flags = (torch.zeros(4096, dtype=torch.int32, device="cuda") for _ in range(2))
    two = lambda t, at=0: (ctypes.c_void_p * 2)(t.data_ptr() + at, t.data_ptr() + at)
    i32, f32 = (lambda *s, t=t: torch.zeros(*s, dtype=t, device="cuda") for t in (torch.int32, torch.float32))
    buf, out, idx, rows = _rand(128, 64), torch.empty(1, 64, dtype=torch.bfloat16, device="cuda"), i32(1, 1), i32(1, 1)
    hist, psum, base, row0, seg, frac, aux = i32(1, 2), f32(1, 2), i32(1, 2), i32(2), i32(4), f32(2), f32(1)
    kv, q1, l1 = _rand(1, 256, 1, 64, seed=5), _rand(1, 128, 1, 64, seed=6), f32(1, 1, 128)
    o1 = torch.empty_like(q1)

    def waiting(st):
        if kind == "plan":
            native.call("lb_moe_plan", hist.data_ptr(), psum.data_ptr(), base.data_ptr(), row0.data_ptr(), seg.data_ptr(), frac.data_ptr(),
                        aux.data_ptr(), 1, 2, 2, 0, 1, 1, 128, two(words, 4096), two(words), 1, 1, st)
        elif kind == "pull":
            native.call("lb_moe_pull", out.data_ptr(), 0, idx.data_ptr(), rows.data_ptr(), 0, 0, 1, 64, 2, 1, 2, 0, 128, two(buf), two(words), 1, st)
        else:
            native.call("lb_flash_fwd_cp", q1.data_ptr(), kv.data_ptr(), kv.data_ptr(), o1.data_ptr(), l1.data_ptr(), 1, 128, 256, 256, 1, 1, 64,
                        64, 64, 0.125, 0, flags.data_ptr(), 1, 0, 0, 0, 0, 0, 1, 0, None, None, None, 0, st)

    def needs_room():
        OF.flash_bwd_native(q, q, q, o, lse, do, False, 128 ** -0.5)
    side, done = torch.cuda.Stream(), torch.cuda.Event()
    OF.gemm(a, b)                                                       # (the first launch of a size uploads its schedule)
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        needs_room()
    torch.cuda.synchronize()
    native.set_flag_wait_ns(500_000_000)
    try:
        waiting(native.stream_ptr())
        OF.gemm(a, b)
        done.record()
        with torch.cuda.stream(side):
            needs_room()
        side.synchronize()
        early = not done.query()
        torch.cuda.synchronize()
    finally:
        native.set_flag_wait_ns(20_000_000_000)
    assert list(native.device_status()) == ["attention forward" if kind == "attention" else "expert-parallel routing / dispatch / combine"]
    assert early

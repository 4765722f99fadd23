import pytest
import torch

from lightron_b200.config import ModelArgs, PRESETS
from lightron_b200.models import LightronTransformer, init_weights
from lightron_b200.optim import DistributedAdamW
from oracle import oracle_forward, oracle_loss


def _tiny(**kw):
    base = dict(PRESETS["tiny"])
    base.update(max_seq_len=64, n_layers=2)
    base.update(kw)
    return ModelArgs(**base)


def test_state_dict_keys_match_reference_layout():
    m = LightronTransformer(_tiny())
    keys = set(m.state_dict().keys())
    want = {"tok_embeddings.weight", "output.weight", "norm.weight"}
    for i in range(2):
        for n in ("wq", "wk", "wv", "wo"):
            want.add(f"layers.{i}.attention.{n}.weight")
        for n in ("w1", "w2", "w3"):
            want.add(f"layers.{i}.feed_forward.{n}.weight")
        want.add(f"layers.{i}.attention_norm.weight")
        want.add(f"layers.{i}.ffn_norm.weight")
    assert keys == want


def test_forward_matches_oracle_mha_and_gqa():
    for kv in (8, 2):
        a = _tiny(n_kv_heads=kv)
        m = LightronTransformer(a)
        init_weights(m, 1)
        tok = torch.randint(0, a.vocab_size, (2, 48))       # shorter than max_seq_len on purpose
        got = m(tok)
        want = oracle_forward(m.state_dict(), tok, n_layers=2, n_heads=8, n_kv_heads=kv)
        assert torch.allclose(got, want, atol=2e-5, rtol=1e-4), (got - want).abs().max()


def test_loss_and_grads_match_oracle():
    a = _tiny(n_kv_heads=4)
    m = LightronTransformer(a)
    init_weights(m, 2)
    tok = torch.randint(0, a.vocab_size, (2, 64))
    tgt = torch.randint(0, a.vocab_size, (2, 64))
    loss = m.loss(tok, tgt)
    loss.backward()
    sd = {k: v.detach().clone().requires_grad_(True) for k, v in m.state_dict().items()}
    ol = oracle_loss(sd, tok, tgt, n_layers=2, n_heads=8, n_kv_heads=4)
    ol.backward()
    assert abs(loss.item() - ol.item()) < 1e-5
    for name, p in m.named_parameters():
        assert torch.allclose(p.grad, sd[name].grad, atol=1e-6, rtol=1e-3), name


def test_moe_matches_dense_oracle():
    a = _tiny(moe_num_experts=4, moe_topk=2, moe_layer_freq=1, moe_aux_loss_coef=0.0)
    m = LightronTransformer(a)
    init_weights(m, 3)
    tok = torch.randint(0, a.vocab_size, (2, 32))
    got = m(tok)
    want = oracle_forward(m.state_dict(), tok, n_layers=2, n_heads=8, n_kv_heads=8)
    assert torch.allclose(got, want, atol=2e-5, rtol=1e-4)
    assert any("experts.3.w2.weight" in k for k in m.state_dict())


def test_adamw_matches_torch_optim():
    a = _tiny()
    m1 = LightronTransformer(a)
    init_weights(m1, 4)
    m2 = LightronTransformer(a)
    m2.load_state_dict(m1.state_dict())
    o1 = DistributedAdamW(m1, lr=3e-4, weight_decay=0.01)
    o2 = torch.optim.AdamW(m2.parameters(), lr=3e-4, weight_decay=0.01)
    g = torch.Generator().manual_seed(0)
    for _ in range(3):
        tok = torch.randint(0, a.vocab_size, (2, 64), generator=g)
        o1.zero_grad()
        o2.zero_grad()
        m1.loss(tok, tok).backward()
        m2.loss(tok, tok).backward()
        o1.step()
        o2.step()
    for (n, p1), (_, p2) in zip(m1.named_parameters(), m2.named_parameters()):
        assert torch.allclose(p1, p2, atol=1e-6), n


def test_flat_arena_makes_qkv_adjacent():
    from lightron_b200.ops.functional import _rows_adjacent
    a = _tiny(n_kv_heads=2)
    m = LightronTransformer(a)
    init_weights(m, 5)
    DistributedAdamW(m)
    att = m.layers["0"].attention
    assert _rows_adjacent((att.wq.weight, att.wk.weight, att.wv.weight))
    ff = m.layers["0"].feed_forward
    assert _rows_adjacent((ff.w1.weight, ff.w3.weight))


def test_which_layers_run_in_one_call():
    """Only dense blocks of one GPU without hooks or a forward of their own."""
    from lightron_b200.models.llama import _plain_layers
    m = LightronTransformer(_tiny())
    hq, hkv, d, scale, weights = _plain_layers(m.layers)
    assert (hq, hkv, d) == (8, 8, 32) and abs(scale * d ** 0.5 - 1) < 1e-12 and len(weights) == 2
    blk = m.layers["1"]
    assert weights[1][2] is blk.attention.wq.weight and weights[1][10] is blk.feed_forward.w2.weight and weights[0][1] == m.args.norm_eps
    for mod in (blk, blk.attention, blk.feed_forward):
        for register in (mod.register_forward_hook, mod.register_forward_pre_hook, mod.register_full_backward_hook):
            h = register(lambda *a: None)
            assert _plain_layers(m.layers) is None
            h.remove()
        mod.forward = mod.forward
        assert _plain_layers(m.layers) is None
        del mod.forward
    h = torch.nn.modules.module.register_module_forward_hook(lambda *a: None)
    assert _plain_layers(m.layers) is None
    h.remove()
    assert _plain_layers(m.layers) is not None

    class Other(type(blk.attention)):
        pass
    blk.attention.__class__ = Other
    assert _plain_layers(m.layers) is None
    assert _plain_layers(LightronTransformer(_tiny(moe_num_experts=2, moe_topk=1, moe_layer_freq=2)).layers) is None
    assert _plain_layers(torch.nn.ModuleDict()) is None


@pytest.mark.parametrize("switch", ["_FUSED_SWIGLU", "_GROUP_BWD"])
def test_a_fusion_that_is_switched_off_stays_off_in_evaluations(monkeypatch, switch):
    """What compares an evaluation with and without a fusion must not run the same kernels twice."""
    from lightron_b200.models.llama import _plain_layers
    from lightron_b200.ops import functional as OF
    m = LightronTransformer(_tiny())
    assert _plain_layers(m.layers) is not None
    monkeypatch.setattr(OF, switch, False)
    assert _plain_layers(m.layers) is None


def test_a_forward_replaced_for_a_class_is_called(monkeypatch):
    from lightron_b200.models import llama
    m = LightronTransformer(_tiny())
    for cls in (llama.TransformerBlock, llama.Attention, llama.MLP):
        with monkeypatch.context() as p:
            plain = cls.forward
            p.setattr(cls, "forward", lambda self, *a, **kw: plain(self, *a, **kw))
            assert llama._plain_layers(m.layers) is None
        assert llama._plain_layers(m.layers) is not None

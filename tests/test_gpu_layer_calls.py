"""-m gpu: a layer's sublayers as one call into the library (vyomai_b200/block.py) against the same layer launch by launch. Both make the same launches with the same
tilings, so outputs, caches and gradients are the same to the bit."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _config(width, kv_heads, **kw):
    return types.SimpleNamespace(hidden_size=width, num_attention_heads=width // 64, num_key_value_heads=kv_heads, num_hidden_layers=1, max_position_embeddings=300,
                                 hidden_dropout_prob=0.0, layer_norm_eps=1e-5, hidden_act="gelu", **kw)


def _calls(monkeypatch):
    """Names of the entry points called, in order."""
    from vyomai_b200 import _lib
    names, run = [], _lib.run
    monkeypatch.setattr(_lib, "run", lambda fn, st: (names.append(fn), run(fn, st))[1])
    return names


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("cls,seqs,tokens,kv_heads,bias", [("EncoderLayer", 3, 17, 2, True), ("EncoderLayer", 5, 130, 4, True), ("EncoderLayer", 2, 70, 2, False),
                                                           ("VitLayer", 2, 37, 4, True)])
def test_training_layers_in_one_call_per_sublayer(monkeypatch, dtype, cls, seqs, tokens, kv_heads, bias):
    from vyomai_b200 import gemm_tune
    from vyomai_b200.functional import MaskSpec, RopeTables
    from vyomai_b200.layers.attention import VisionAttention
    from vyomai_b200.layers.positional_embeddings import RotaryEmbedding
    from vyomai_b200.models.encoder import EncoderLayer
    torch.manual_seed(tokens)
    cfg = _config(256, kv_heads, attention_bias=bias)
    layer = EncoderLayer(cfg, 0, "gqa" if kv_heads != 4 else None)
    if cls == "VitLayer":
        layer.attention = VisionAttention(cfg, 0)
    layer = layer.to(DEV, dtype).train()
    x = torch.randn(seqs, tokens, 256, device=DEV, dtype=dtype, requires_grad=True)
    pad = torch.ones(seqs, tokens, device=DEV, dtype=torch.long)
    pad[-1, tokens // 2:] = 0
    mask, rope, dy = MaskSpec.from_attention_mask(pad, causal=False), RopeTables(RotaryEmbedding(cfg)(300)) if bias else None, torch.randn_like(x)
    names, params = _calls(monkeypatch), list(layer.parameters())
    gemm_tune.clear()

    def step():
        names.clear()
        y = layer(x, mask, rope)
        return [y] + list(torch.autograd.grad(y, [x] + params, dy))

    by_launch = step()
    assert "vy_attn_block_fwd" not in names and names.count("vy_gemm") >= 12
    whole = step()
    assert [n for n in names if "block" in n] == ["vy_attn_block_fwd", "vy_ffn_block_fwd", "vy_ffn_block_bwd", "vy_attn_block_bwd"] and len(names) == 4
    assert all(torch.equal(a, b) for a, b in zip(by_launch, whole))
    assert [g.shape for g in whole[2:]] == [p.shape for p in params]
    with torch.no_grad():   # the forward pass alone: its products keep no pre-activation and have tilings of their own
        a = layer(x, mask, rope)
        names.clear()
        b = layer(x, mask, rope)
    assert names == ["vy_attn_block_fwd", "vy_ffn_block_fwd"] and torch.equal(a, b)
    layer.feed_forward.dropout.p = 0.5   # dropout: launch by launch
    names.clear()
    layer(x, mask, rope)
    assert "vy_ffn_block_fwd" not in names


@pytest.mark.parametrize("dtype,cache", [(torch.bfloat16, torch.bfloat16), (torch.float32, torch.bfloat16), (torch.float32, torch.float32)])
@pytest.mark.parametrize("seqs,before", [(1, 3), (5, 200), (70, 40)])
def test_cached_layers_in_one_call_per_sublayer(monkeypatch, dtype, cache, seqs, before):
    """A prompt into a cache with more rows than sequences, then a token; an fp32 cache takes prompts launch by launch."""
    from vyomai_b200 import gemm_tune
    from vyomai_b200.functional import MaskSpec, RopeTables
    from vyomai_b200.layers.kv_cache import StaticCacheOne
    from vyomai_b200.layers.positional_embeddings import RotaryEmbedding
    from vyomai_b200.models.decoder import DecoderLayer
    torch.manual_seed(before)
    cfg = _config(256, 2)
    layer, rope = DecoderLayer(cfg, 0, "gqa").to(DEV, dtype).eval(), RopeTables(RotaryEmbedding(cfg)(300))
    prompt, token = torch.randn(seqs, before, 256, device=DEV, dtype=dtype), torch.randn(seqs, 1, 256, device=DEV, dtype=dtype)
    mask, names = MaskSpec.from_attention_mask(torch.ones(seqs, before, device=DEV, dtype=torch.long), causal=True), _calls(monkeypatch)
    gemm_tune.clear()

    def run():
        kv = StaticCacheOne(cfg, max_cache_len=256, batch_size=seqs + 1, dtype=cache, is_gqa=True)
        names.clear()
        with torch.no_grad():
            a, _ = layer(prompt, mask, freqs=rope, use_cache=True, kv_cache=kv, start_pos=0)
            first = list(names)
            b, _ = layer(token, None, freqs=rope, use_cache=True, kv_cache=kv, start_pos=before)
        return [a, b, kv.key_cache[0], kv.value_cache[0]], first, names[len(first):]

    by_launch, _, _ = run()
    whole, first, second = run()
    blocks = ["vy_attn_block_fwd", "vy_ffn_block_fwd"]
    assert second == blocks and (first == blocks if cache == torch.bfloat16 else first[-1] == blocks[1] and "vy_attn_block_fwd" not in first)
    assert all(torch.equal(a, b) for a, b in zip(by_launch, whole))
    bad = StaticCacheOne(cfg, max_cache_len=before, batch_size=seqs, dtype=cache, is_gqa=True)
    with pytest.raises(ValueError), torch.no_grad():
        layer(token, None, freqs=rope, use_cache=True, kv_cache=bad, start_pos=before)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("forget", [False, True])
def test_checkpointed_layers_save_the_same_when_computed_again(dtype, forget):
    """The first layers of a shape go launch by launch, and the last one's backward pass settles the tilings of the others: what a layer saves must not depend on it, or
    torch.utils.checkpoint refuses the recomputation. Nor on whether tilings have been forgotten in between."""
    from torch.utils.checkpoint import checkpoint
    from vyomai_b200 import gemm_tune
    from vyomai_b200.functional import MaskSpec, RopeTables
    from vyomai_b200.layers.positional_embeddings import RotaryEmbedding
    from vyomai_b200.models.encoder import EncoderLayer
    torch.manual_seed(0)
    cfg = _config(256, 2)
    layers, rope, mask = [EncoderLayer(cfg, i, "gqa").to(DEV, dtype).train() for i in range(3)], RopeTables(RotaryEmbedding(cfg)(300)), MaskSpec()
    x, dy = torch.randn(3, 50, 256, device=DEV, dtype=dtype, requires_grad=True), torch.randn(3, 50, 256, device=DEV, dtype=dtype)
    params = [p for m in layers for p in m.parameters()]

    def step(again):
        y = x
        for m in layers:
            y = checkpoint(m, y, mask, rope, use_reentrant=False) if again else m(y, mask, rope)
        if forget and again:
            gemm_tune.LAYERS.clear()
        return [y] + list(torch.autograd.grad(y, [x] + params, dy))

    gemm_tune.clear()
    first, second, plain = step(True), step(True), step(False)
    for got in (first, second):
        assert all(torch.equal(a, b) for a, b in zip(got, plain))


@pytest.mark.parametrize("forward_by_launch", [False, True])
def test_directions_that_go_their_own_ways(monkeypatch, forward_by_launch):
    """One direction as one call, the other launch by launch; weights that lie elsewhere by the time of the backward pass."""
    from vyomai_b200 import gemm_tune
    from vyomai_b200.functional import MaskSpec, RopeTables
    from vyomai_b200.layers.positional_embeddings import RotaryEmbedding
    from vyomai_b200.models.encoder import EncoderLayer
    torch.manual_seed(1)
    cfg = _config(256, 2)
    layer, rope = EncoderLayer(cfg, 0, "gqa").to(DEV, torch.bfloat16).train(), RopeTables(RotaryEmbedding(cfg)(300))
    x, dy = torch.randn(3, 70, 256, device=DEV, dtype=torch.bfloat16, requires_grad=True), torch.randn(3, 70, 256, device=DEV, dtype=torch.bfloat16)
    params, names = list(layer.parameters()), _calls(monkeypatch)

    def step(between=lambda: None):
        y = layer(x, MaskSpec(), rope)
        between()
        return [y] + list(torch.autograd.grad(y, [x] + params, dy))

    gemm_tune.clear()
    want = step()
    step()
    kept = dict(gemm_tune.LAYERS)
    assert len(kept) == 4

    def other_way():
        gemm_tune.LAYERS.clear()
        gemm_tune.LAYERS.update({k: v for k, v in kept.items() if (k[0] == "backward") == forward_by_launch})

    def back():
        gemm_tune.LAYERS.update(kept) if forward_by_launch else other_way()

    if forward_by_launch:
        other_way()
    names.clear()
    got = step(back)
    assert ("vy_attn_block_fwd" in names) != forward_by_launch and ("vy_attn_block_bwd" in names) == forward_by_launch
    assert all(torch.equal(a, b) for a, b in zip(want, got))

    gemm_tune.LAYERS.update(kept)
    spacers = []

    def move():
        for p in params:
            spacers.append(torch.empty(1 << 20, device=DEV))
            p.data = p.data.clone()

    names.clear()
    got = step(move)
    assert "vy_attn_block_bwd" in names and all(torch.equal(a, b) for a, b in zip(want, got))

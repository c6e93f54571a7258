"""The prompt-sized forms of the packed decoders' mixers (csrc/window_attn_tc.cu, window_attn_mma.cu, talk_attn_mma.cu, linear_attn_mma.cu, delta_rule_mma.cu) at
the edges of their tiles and of the rules that choose them, against the float64 oracles and against the form that the same call takes
without the lent workspace. Bound: an fp32 result off by a few units in the last place of its row's largest term per contraction, 16 * 2^-24 of the
output's 2-norm (about 1e-6; the kernels measure 1e-7 to 3e-7)."""
import pytest
import torch

from oracle import hybrid_oracle as OH
from oracle import vazepel_oracle as OV
from oracle import zaparax_oracle as OZ
from tests.hybrid_util import shuffled_batch

pytestmark = pytest.mark.gpu
DEV = "cuda"
BOUND = 16 * 2.0 ** -24


def _err(got, want):
    return float((got.detach().double().cpu() - want.double()).norm() / want.double().norm())


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def _both(monkeypatch, rule, call):
    """call() as it is, and with the rule that lends the workspace saying that this step needs none."""
    from vyomai_b200 import ops
    first = call()
    monkeypatch.setattr(ops._lib.lib(), rule, lambda *a: 0)
    second = call()
    monkeypatch.undo()
    return first, second


@pytest.mark.parametrize("H,G,dk,dv", [(2, 1, 20, 24), (2, 2, 33, 33), (4, 2, 64, 72), (2, 1, 128, 8), (1, 1, 100, 130), (1, 1, 1, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_delta_rule_sixteen_tokens_at_a_time(monkeypatch, H, G, dk, dv, dtype):
    """Sequences that end on, before and after a chunk's edge, one of them carried on from a state; then their continuation. Strided inputs."""
    from vyomai_b200 import ops
    g = torch.Generator().manual_seed(dk)
    lengths, more = [1, 15, 16, 17, 65], [64, 2, 16, 5, 1]
    T = [a + b for a, b in zip(lengths, more)]
    mk = lambda w: [torch.randn(t, w, generator=g).to(dtype) for t in T]  # noqa: E731
    q, k, v, a, b = mk(G * dk), mk(G * dk), mk(H * dv), mk(H * dk), mk(H)
    a_log = torch.randn(H, generator=g) - 1.0
    want = []
    for s, t in enumerate(T):
        unit = lambda x: OH.unit(x.double().view(t, G, dk))  # noqa: E731
        decay = torch.exp(-torch.exp(a_log.double())[None, :, None] * torch.nn.functional.softplus(a[s].double(), threshold=1e9).view(t, H, dk))
        want.append(OH.gated_delta_rule(unit(q[s]) * dk ** -0.5, unit(k[s]), v[s].double().view(t, H, dv), decay, torch.sigmoid(b[s].double())).reshape(t, -1))

    def walk():
        state = torch.full((7, H, dk, dv), float("nan"), device=DEV)
        slots, out = [3, 0, 6, 2, 5], []
        for at, take in (([0] * 5, lengths), (lengths, more)):
            wide = lambda src: torch.cat([torch.cat([src[s][at[s]:at[s] + take[s]] for s in range(5)]).to(DEV), torch.zeros(sum(take), 3, dtype=dtype, device=DEV)], 1)[:, :-3]  # noqa: E731
            batch = ops.PackedBatch(_i32([sum(take[:i]) for i in range(6)]), _i32(at), _i32(slots), max(take))
            out.append(ops.delta_rule(batch, wide(q), wide(k), wide(v), wide(a), wide(b), a_log.to(DEV), state, heads=H, kv_heads=G, dim=dk, vdim=dv, out_dtype=torch.float32).split(take))
        assert bool(torch.isnan(state[[1, 4]]).all())   # other slots untouched
        return [torch.cat([x, y]) for x, y in zip(*out)]

    for form in _both(monkeypatch, "vy_delta_rule_prompt_floats", walk):
        for s in range(5):
            assert _err(form[s], want[s]) < 4 * BOUND, s   # a recurrence: each of the up to 66 steps carries its rounding on


@pytest.mark.parametrize("H,G,dk,dv", [(1, 1, 128, 128), (2, 1, 100, 40), (3, 3, 64, 16), (2, 2, 36, 130), (4, 2, 32, 33), (1, 1, 4, 1)])
@pytest.mark.parametrize("copies", [1, 40])
def test_delta_rule_on_aligned_rows(H, G, dk, dv, copies):
    """Rows that come in quads, few sequences and many (more CTAs than run at once): portions that end on, before and after a chunk's edge, carried on once."""
    from vyomai_b200 import ops
    g = torch.Generator().manual_seed(dk + dv)
    lengths, more = [64, 33, 16, 47], [1, 32, 64, 17]
    T = [a + b for a, b in zip(lengths, more)]
    mk = lambda w: [torch.randn(t, w, generator=g) for t in T]  # noqa: E731
    q, k, v, a, b = mk(G * dk), mk(G * dk), mk(H * dv), mk(H * dk), mk(H)
    a_log = torch.randn(H, generator=g) - 1.0
    want = []
    for s, t in enumerate(T):
        unit = lambda x: OH.unit(x.double().view(t, G, dk))  # noqa: E731
        decay = torch.exp(-torch.exp(a_log.double())[None, :, None] * torch.nn.functional.softplus(a[s].double(), threshold=1e9).view(t, H, dk))
        want.append(OH.gated_delta_rule(unit(q[s]) * dk ** -0.5, unit(k[s]), v[s].double().view(t, H, dv), decay, torch.sigmoid(b[s].double())).reshape(t, -1))
    n = 4 * copies
    state, out = torch.full((n, H, dk, dv), float("nan"), device=DEV), []
    for at, take in (([0] * 4, lengths), (lengths, more)):
        quads = lambda src: torch.nn.functional.pad(torch.cat([src[s][at[s]:at[s] + take[s]] for s in range(4)] * copies), (0, -src[0].shape[1] % 4)).to(DEV)[:, :src[0].shape[1]]  # noqa: E731
        batch = ops.PackedBatch(_i32([sum((take * copies)[:i]) for i in range(n + 1)]), _i32(at * copies), _i32(list(range(n))), max(take))
        out.append(ops.delta_rule(batch, quads(q), quads(k), quads(v), quads(a), quads(b), a_log.to(DEV), state, heads=H, kv_heads=G, dim=dk, vdim=dv, out_dtype=torch.float32).split(take * copies))
    for i in range(n):
        assert _err(torch.cat([out[0][i], out[1][i]]), want[i % 4]) < 4 * BOUND, i   # as above


def test_delta_rule_keeps_a_bad_value_to_its_column_and_later_tokens():
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(1)
    T, H, dk, dv, at, col = 40, 1, 48, 40, 21, 5
    q, k, v, a, b = (torch.randn(T, w, generator=g, device=DEV) for w in (dk, dk, dv, dk, H))
    batch = ops.PackedBatch(_i32([0, T]), _i32([0]), _i32([0]), T)
    run = lambda vv: ops.delta_rule(batch, q, k, vv, a, b, torch.zeros(1, device=DEV), torch.zeros(1, H, dk, dv, device=DEV), heads=H, kv_heads=H, dim=dk, vdim=dv)  # noqa: E731
    clean = run(v)
    for bad in (float("inf"), float("nan")):
        vv = v.clone()
        vv[at, col] = bad
        got = run(vv)
        hit = torch.zeros(T, dv, dtype=torch.bool, device=DEV)
        hit[at:, col] = True
        assert torch.equal(torch.isfinite(got), ~hit)
        assert float((got - clean)[~hit].abs().max()) < 1e-6


@pytest.mark.parametrize("M,N,K", [(33, 256, 1), (64, 257, 7), (65, 512, 16), (129, 514, 17), (300, 1030, 32), (9000, 256, 16)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_thin_products(M, N, K, dtype):
    """Contractions of up to 32 over many rows, two of them in one call, each with its bias, weights with aligned rows and without."""
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(M)
    x = torch.randn(M, 2 * K + 3, generator=g, device=DEV)
    w, b = torch.randn(2, N, K, generator=g, device=DEV).to(dtype), torch.randn(2, N, generator=g, device=DEV).to(dtype)
    wide = (N + 7) // 8 * 8
    out = torch.full((M, 2 * wide), 7.0, device=DEV)
    ops.head_linear(x, w, out, x_head=K + 3, out_head=wide, bias=b)
    want = [x[:, i * (K + 3):i * (K + 3) + K].double() @ w[i].double().T + b[i].double() for i in range(2)]
    for i in range(2):
        assert _err(out[:, i * wide:i * wide + N], want[i].cpu()) < BOUND
        assert bool((out[:, i * wide + N:(i + 1) * wide] == 7.0).all())   # columns behind the products
    one = ops.linear_plain(x[:, :K], w[0], bias=b[0], act="silu", scale=0.5, out_dtype=torch.float32)
    assert _err(one, 0.5 * torch.nn.functional.silu(want[0]).cpu()) < BOUND


@pytest.mark.parametrize("M,N,K,thin", [(500, 512, 24, True), (390, 512, 24, False), (300, 1030, 32, True), (60, 1030, 32, False), (40, 256, 16, True), (40, 256, 12, True), (800, 300, 20, True), (40, 254, 12, False)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_thin_products_on_both_sides_of_the_line(M, N, K, thin, dtype):
    """Weights that come 16 bytes at a time, contractions that fill up a step of eight or four and not."""
    from vyomai_b200 import ops
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        ops.linear_plain(torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV).to(dtype), out_dtype=torch.float32)
        torch.cuda.synchronize()
    assert any("linear_thin_kernel" in e.name for e in prof.events()) == thin
    test_thin_products(M, N, K, dtype)


def _delta_mixer(W=64, H=2, D=32, rank=16, conv=torch.float32):
    """(weights, forward(mixer) on the same 200 tokens) of a delta mixer whose input products are made here."""
    from types import SimpleNamespace
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(1)
    R = lambda *s: torch.randn(*s, generator=g, device=DEV) / s[-1] ** 0.5  # noqa: E731
    n = {"q": H * D, "k": H * D, "v": H * D, "b": H, "a1": rank, "g1": rank}
    w = {**{k: R(v, W) for k, v in n.items()}, "a2": R(H * D, rank), "g2": R(H * D, rank), "dt_bias": R(H * D), "A_log": R(H), "norm": torch.ones(D, device=DEV), "o": R(W, H * D),
         **{k + ".conv": R(H * D, 4) for k in "qkv"}}
    w["k.conv"] = w["k.conv"].to(conv)
    h = R(200, W) * 8
    packed = torch.cat([torch.nn.functional.pad(h @ w[k].T, (0, -v % 8)) for k, v in n.items()], 1)
    parts, at = [], 0
    for v in n.values():
        parts.append(packed[:, at:at + v])
        at += v + -v % 8
    batch = ops.PackedBatch(_i32([0, 130, 200]), _i32([0, 0]), _i32([0, 1]), 130)
    def forward(mixer, parts=parts):
        return mixer.forward(parts, batch, SimpleNamespace(states={"S": torch.zeros(2, H, D, D, device=DEV), **{"conv_" + k: torch.zeros(2, H * D, 3, device=DEV) for k in "qkv"}}))
    return dict(heads=H, kv_heads=H, dim=D, vdim=D, conv=4), w, parts, forward


def test_delta_mixer_reads_its_low_rank_weights_where_they_are():
    """A change of them in place takes effect; blocks of one product and blocks of their own give the same."""
    from vyomai_b200.layers.mixers import GatedDeltaMixer
    cfg, w, parts, forward = _delta_mixer()
    mixer = GatedDeltaMixer(cfg, w, 1e-6, torch.float32, False)
    first = forward(mixer)
    for name in ("a2", "g2", "dt_bias"):
        w[name].mul_(0.25).add_(0.1)
        after = forward(mixer)
        assert torch.equal(after, forward(GatedDeltaMixer(cfg, w, 1e-6, torch.float32, False))) and not torch.equal(after, first)
        first = after
    apart = parts[:4] + [parts[4].clone(), parts[5].clone()]
    for other in (apart, parts[:4] + [parts[4].clone(), parts[5]]):   # the last: rows of another stride, a call each
        assert torch.equal(forward(mixer, other), first)


@pytest.mark.parametrize("M,N,K", [(5, 33, 7), (20, 64, 16), (40, 300, 12), (65, 100, 64), (70, 70, 256)])
def test_two_products_in_one_launch(M, N, K):
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(M)
    x, w, b = torch.randn(2 * M, K, generator=g, device=DEV), torch.randn(2 * N, K, generator=g, device=DEV), torch.randn(2 * N, generator=g, device=DEV)
    halves = lambda t: (t[:t.shape[0] // 2], t[t.shape[0] // 2:])  # noqa: E731
    for order in (1, -1):   # the second operand behind the first one, and before it
        args = [halves(t)[::order] for t in (x, w, b)]
        for i, y in enumerate(ops.linear_pair(*args)):
            assert _err(y, (args[0][i].double() @ args[1][i].double().T + args[2][i].double()).cpu()) < BOUND
    assert ops.linear_pair(halves(x), (w[:N], w[N:].bfloat16()), halves(b)) is None and ops.linear_pair((x[:M], x[:M]), halves(w), (b[:N], b[:N])) is None


@pytest.mark.parametrize("channels", [(64, 64, 128), (5, 64, 33), (260, 512, 4), (128, 384)])
@pytest.mark.parametrize("tokens", [1, 17, 1500])
def test_convolutions_in_one_launch(channels, tokens):
    """The same outputs and states as one call per input, with carried states and without."""
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(tokens)
    batch = ops.PackedBatch(_i32([0, tokens, 2 * tokens, 2 * tokens + 1]), _i32([0, 9, 3]), _i32([2, 0, 1]), tokens)
    p = torch.randn(2 * tokens + 1, sum(channels) + 4, generator=g, device=DEV)
    xs = p[:, :sum(channels)].split(list(channels), 1)
    ws = [torch.randn(c, 4, generator=g, device=DEV).bfloat16() for c in channels]
    states = [torch.randn(3, c, 3, generator=g, device=DEV) for c in channels]
    alone = [s.clone() for s in states]
    got = ops.causal_convs(batch, xs, ws, states).split(list(channels), 1)
    for x, w, s, y, t in zip(xs, ws, alone, got, states):
        want = ops.causal_conv(batch, x, w, s, out_dtype=torch.float32)
        assert _err(y, want.cpu()) < BOUND and torch.equal(s, t)


@pytest.mark.parametrize("last", [4, 5, 6, 7])
def test_convolutions_in_one_launch_keep_rows_on_16_bytes(last):
    """q and k of a delta rule with an odd number of value channels are still read four channels at a time."""
    from vyomai_b200 import ops
    batch = ops.PackedBatch(_i32([0, 40]), _i32([0]), _i32([0]), 40)
    xs, ws = [torch.randn(40, c, device=DEV) for c in (8, 8, last)], [torch.randn(c, 4, device=DEV) for c in (8, 8, last)]
    xs = list(torch.cat(xs, 1).split([8, 8, last], 1))
    got = ops.causal_convs(batch, xs, ws, [torch.zeros(1, w.shape[0], 3, device=DEV) for w in ws])
    assert got.shape == (40, 16 + last) and got.stride(0) % 4 == 0 and got.data_ptr() % 16 == 0
    assert torch.equal(got[:, 16:], ops.causal_conv(batch, xs[2], ws[2], torch.zeros(1, last, 3, device=DEV), out_dtype=torch.float32))


@pytest.mark.parametrize("short", [dict(ld_out=23), dict(ld_out=8), dict(ldx=7)])
def test_convolutions_in_one_launch_check_their_rows(monkeypatch, short):
    """Rows that do not hold what the call writes side by side, or reads, are refused before any launch."""
    from vyomai_b200 import ops
    from vyomai_b200._lib import VyomError
    batch, p = ops.PackedBatch(_i32([0, 40]), _i32([0]), _i32([0]), 40), torch.randn(40, 24, device=DEV)
    ws, states = [torch.randn(8, 4, device=DEV) for _ in range(3)], [torch.zeros(1, 8, 3, device=DEV) for _ in range(3)]
    real = ops._lib.call
    monkeypatch.setattr(ops._lib, "call", lambda fn, st, **kw: real(fn, st, **{**kw, **short}))
    with pytest.raises(VyomError, match="further inputs"):
        ops.causal_convs(batch, p.split(8, 1), ws, states)


@pytest.mark.parametrize("differ", ["weights", "inputs", "strides", "taps"])
def test_convolutions_that_no_launch_can_share(differ):
    """Inputs or weights of different types, strides or taps: what one call each gives."""
    from vyomai_b200 import ops
    from vyomai_b200.layers.mixers import GatedDeltaMixer
    g = torch.Generator(device=DEV).manual_seed(3)
    channels, tokens = (24, 24, 40), 50
    batch = ops.PackedBatch(_i32([0, tokens, tokens + 1]), _i32([0, 9]), _i32([1, 0]), tokens)
    xs = list(torch.randn(tokens + 1, sum(channels), generator=g, device=DEV).split(list(channels), 1))
    ws = [torch.randn(c, 4 if differ != "taps" or c == 24 else 3, generator=g, device=DEV) for c in channels]
    if differ == "weights":
        ws[1] = ws[1].bfloat16()
    elif differ == "inputs":
        xs[2] = torch.randn(tokens + 1, sum(channels), generator=g, device=DEV).bfloat16()[:, :40]
    elif differ == "strides":
        xs[0] = xs[0].contiguous()
    states = [torch.randn(2, *w.shape, generator=g, device=DEV)[..., 1:].contiguous() for w in ws]
    alone = [s.clone() for s in states]
    got = ops.causal_convs(batch, xs, ws, states).split(list(channels), 1)
    for x, w, s, y, t in zip(xs, ws, alone, got, states):
        assert torch.equal(y, ops.causal_conv(batch, x, w, s, out_dtype=torch.float32)) and torch.equal(s, t)
    if differ == "weights":
        cfg, w, _, forward = _delta_mixer(conv=torch.bfloat16)
        assert bool(torch.isfinite(forward(GatedDeltaMixer(cfg, w, 1e-6, torch.float32, False))).all())


@pytest.mark.parametrize("H,dk,dv", [(2, 20, 24), (1, 128, 64), (3, 64, 65), (2, 100, 130), (1, 8, 7)])
def test_linear_attention_all_chunks_at_once(monkeypatch, H, dk, dv):
    """Chunks of 64 tokens: portions of 64 (the walk), 65, 128, 130 and 1 token side by side, then a continuation of 66."""
    from vyomai_b200 import ops
    g = torch.Generator().manual_seed(dk)
    lengths, more = [64, 65, 128, 130, 1], [66, 1, 3, 64, 66]
    T = [a + b for a, b in zip(lengths, more)]
    q, k, v = ([torch.randn(t, H * w, generator=g) for t in T] for w in (dk, dk, dv))
    decay = torch.tensor([0.999, 0.5, 0.9][:H]).double().tolist()   # as fp32 holds them: 0.999 itself is 1.3e-8 off, 130 steps of it 1e-6
    want = [OH.lightning_attention(q[s].double().view(t, H, dk), k[s].double().view(t, H, dk), v[s].double().view(t, H, dv), decay).reshape(t, -1) for s, t in enumerate(T)]

    def walk():
        state = torch.full((6, H, dk, dv), float("nan"), device=DEV)
        out = []
        for at, take in (([0] * 5, lengths), (lengths, more)):
            cat = lambda src: torch.cat([src[s][at[s]:at[s] + take[s]] for s in range(5)]).to(DEV)  # noqa: E731
            batch = ops.PackedBatch(_i32([sum(take[:i]) for i in range(6)]), _i32(at), _i32([4, 1, 0, 5, 2]), max(take))
            out.append(ops.linear_attn(batch, cat(q), cat(k), cat(v), torch.tensor(decay, device=DEV), state, heads=H, dim=dk, vdim=dv).split(take))
        return [torch.cat([x, y]) for x, y in zip(*out)]

    for form in _both(monkeypatch, "vy_linear_attn_workspace_floats", walk):
        for s in range(5):
            assert _err(form[s], want[s]) < BOUND, s


@pytest.mark.parametrize("pool", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,d,dv,window,cap,sinks", [(4, 2, 20, 10, 0, 0.0, True), (8, 1, 64, 64, 31, 20.0, False), (2, 2, 96, 130, 65, 0.0, True), (16, 2, 128, 128, 0, 0.0, False),
                                                       (4, 4, 192, 192, 100, 0.0, False), (6, 2, 33, 256, 7, 5.0, True)])
def test_prompt_attention_on_the_tensor_cores(monkeypatch, pool, H, G, d, dv, window, cap, sinks):
    """Portions of 1 to 200 queries on contexts that end on and off the key tiles; pages that no query may read hold large numbers."""
    from vyomai_b200 import ops
    g = torch.Generator().manual_seed(d)
    new, pos0 = [200, 64, 17, 1], [0, 65, 130, 33]
    T = [n + p for n, p in zip(new, pos0)]
    q, k, v = ([(torch.randn(t, n, w, generator=g) / d ** (0.25 if i < 2 else 0)).to(pool).float() for t in T] for i, (n, w) in enumerate(((H, d), (G, d), (G, dv))))
    sink = torch.randn(H, generator=g) if sinks else None
    slopes = OZ.head_slopes(H)
    want = torch.cat([OZ.biased_attention(q[s].double(), k[s].double(), v[s].double(), scale=1.3, softcap=cap, window=window, slopes=slopes,
                                          sink=None if sink is None else sink.double())[pos0[s]:].reshape(new[s], -1) for s in range(4)])
    bs = 16
    batch, table, _, n_blocks, _ = shuffled_batch(new, pos0, bs, DEV, seed=d)
    kp, vp = torch.full((n_blocks, bs, G, d), 1e3, dtype=pool, device=DEV), torch.full((n_blocks, bs, G, dv), 1e3, dtype=pool, device=DEV)
    for s in range(4):
        for p in range(T[s]):
            kp[table[s][p // bs], p % bs], vp[table[s][p // bs], p % bs] = k[s][p].to(DEV, pool), v[s][p].to(DEV, pool)
    qq = torch.cat([q[s][pos0[s]:].reshape(new[s], -1) for s in range(4)]).to(DEV)
    call = lambda: ops.window_attn(batch, qq, kp, vp, heads=H, kv_heads=G, dim=d, vdim=dv, scale=1.3, window=window, keep_first=0, softcap=cap,  # noqa: E731
                                   head_slope=torch.tensor(slopes, device=DEV), sink=None if sink is None else sink.to(DEV), out_dtype=torch.float32)
    for got in _both(monkeypatch, "vy_window_attn_prompt_floats", call):
        assert _err(got, want) < BOUND


@pytest.mark.parametrize("H,G,d,dv,window", [(8, 2, 64, 64, 0), (16, 4, 20, 33, 37), (32, 8, 48, 16, 0), (8, 8, 7, 5, 16)])
def test_score_exchanging_prompts_on_the_tensor_cores(monkeypatch, H, G, d, dv, window):
    from vyomai_b200 import ops
    g = torch.Generator().manual_seed(H)
    new, pos0, scale, bs = [130, 17, 16], [0, 48, 1], 0.3, 4
    T = [n + p for n, p in zip(new, pos0)]
    q, k, v = ([torch.randn(t, n, w, generator=g) for t in T] for n, w in ((H, d), (G, d), (G, dv)))
    talk = torch.eye(H) + 0.3 * torch.randn(H, H, generator=g) / H ** 0.5
    want = []
    for s, t in enumerate(T):
        sc = torch.stack([q[s][:, a].double() @ k[s][:, a // (H // G)].double().T for a in range(H)]) * scale
        back = torch.arange(t)[:, None] - torch.arange(t)[None, :]
        p = OV.plus_one_softmax(OV.mix_heads(OV.capped(sc, 9.0), talk.double()), (back >= 0) & (back < window) if window else back >= 0)
        want.append(torch.stack([p[a] @ v[s][:, a // (H // G)].double() for a in range(H)], 1).reshape(t, -1)[pos0[s]:])
    batch, table, _, n_blocks, _ = shuffled_batch(new, pos0, bs, DEV, seed=H)
    kp, vp = torch.full((n_blocks, bs, G, d), 1e3, device=DEV), torch.full((n_blocks, bs, G, dv), 1e3, device=DEV)
    for s in range(3):
        for p in range(T[s]):
            kp[table[s][p // bs], p % bs], vp[table[s][p // bs], p % bs] = k[s][p].to(DEV), v[s][p].to(DEV)
    qq = torch.cat([q[s][pos0[s]:].reshape(new[s], -1) for s in range(3)]).to(DEV)
    call = lambda: ops.talk_attn(batch, qq, kp, vp, heads=H, kv_heads=G, dim=d, vdim=dv, scale=scale, softcap=9.0, talk=talk.to(DEV), zero_sink=True, window=window)  # noqa: E731
    for got in _both(monkeypatch, "vy_talk_attn_prompt_floats", call):
        assert _err(got, torch.cat(want)) < 4 * BOUND   # mixed scores: each is a sum over H capped ones, and the softmax takes its absolute error


@pytest.mark.parametrize("H,G,d,dv,window,cap,new,pos0,form", [
    (16, 4, 64, 64, 0, 9.0, [130, 17, 1], [0, 48, 200], "tc"), (16, 1, 64, 64, 70, 0.0, [129], [63], "tc"), (32, 4, 32, 48, 0, 30.0, [65, 4], [0, 60], "tc"),
    (32, 2, 7, 5, 3, 0.0, [70], [0], "tc"), (8, 4, 17, 64, 0, 4.0, [64, 128], [0, 1], "tc"), (8, 2, 48, 20, 0, 0.0, [16] * 148, [0, 5] * 74, "tc"),
    (8, 2, 48, 20, 0, 0.0, [16] * 149, [5] * 149, "mma"), (16, 2, 33, 33, 20, 9.0, [40] * 60, [3] * 60, "mma")])
@pytest.mark.parametrize("extras", [False, True])
def test_score_exchanging_on_both_sides_of_the_line(H, G, d, dv, window, cap, new, pos0, form, extras):
    """Tiles that end on, before and after an edge, few and many sequences; bare, or with bf16 inputs, scores to sink into and gates."""
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(H + d)
    bs, io, n = 4, torch.bfloat16 if extras else torch.float32, len(new)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    q, talk = rnd(sum(new), H * d).to(io), torch.eye(H, device=DEV) + 0.3 * rnd(H, H) / H ** 0.5 if not extras or H > 8 else None
    sink, per_channel = rnd(H) if extras else None, H != 16
    gate = rnd(sum(new), H * dv if per_channel else H) if extras else None
    batch, table, _, n_blocks, _ = shuffled_batch(new, pos0, bs, DEV, seed=H)
    kp, vp = rnd(n_blocks, bs, G, d).to(io), rnd(n_blocks, bs, G, dv).to(io)
    call = lambda: ops.talk_attn(batch, q, kp, vp, heads=H, kv_heads=G, dim=d, vdim=dv, scale=0.3, softcap=cap, talk=talk, window=window, sink=sink,  # noqa: E731
                                 gate=gate, gate_per_channel=per_channel and extras, out_dtype=torch.float32)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        got = call().double()
        torch.cuda.synchronize()
    assert any(f"talk_attn_{form}_kernel" in e.name for e in prof.events())
    at = 0
    for s in range(n):
        t = pos0[s] + new[s]
        pages = torch.tensor(table[s][:(t + bs - 1) // bs], device=DEV)
        k, v = (x[pages].reshape(-1, G, w)[:t].double().repeat_interleave(H // G, 1) for x, w in ((kp, d), (vp, dv)))
        sc = torch.einsum("qhd,khd->hqk", q[at:at + new[s]].double().view(-1, H, d), k) * 0.3
        if cap:
            sc = cap * torch.tanh(sc / cap)
        if talk is not None:
            sc = torch.einsum("hb,bqk->hqk", talk.double(), sc)
        back = torch.arange(pos0[s], t, device=DEV)[:, None] - torch.arange(t, device=DEV)[None, :]
        sc = sc.masked_fill(~((back >= 0) & (back < window) if window else back >= 0), -float("inf"))
        if sink is not None:
            sc = torch.cat([sc, sink.double().view(H, 1, 1).expand(-1, new[s], 1)], -1)
        want = torch.einsum("hqk,khd->qhd", torch.softmax(sc, -1)[..., :t], v)
        if gate is not None:
            want = want * torch.sigmoid(gate[at:at + new[s]].double()).view(new[s], H, -1)
        assert _err(got[at:at + new[s]], want.reshape(new[s], -1).cpu()) < 4 * BOUND   # as above
        at += new[s]


@pytest.mark.parametrize("H,G,d,dv,window,cap,new,pos0,form", [
    (16, 4, 48, 40, 0, 9.0, [40] * 40, [300] * 40, "tc"), (16, 4, 48, 40, 0, 9.0, [40] * 40, [200] * 40, "mma"), (16, 4, 48, 40, 256, 0.0, [40] * 40, [300] * 40, "tc"),
    (16, 4, 48, 40, 255, 0.0, [40] * 40, [300] * 40, "mma"), (8, 1, 16, 16, 0, 9.0, [40] * 60, [300] * 60, "mma"), (8, 2, 64, 64, 0, 9.0, [33] * 60 + [1], [0] * 60 + [400], "tc")])
def test_score_exchanging_form_by_the_keys_that_are_seen(H, G, d, dv, window, cap, new, pos0, form):
    """More CTAs than run at once: the line is at 256 keys on average, cached ones among them."""
    test_score_exchanging_on_both_sides_of_the_line(H, G, d, dv, window, cap, new, pos0, form, False)


@pytest.mark.parametrize("new,H,dk,dv,carried,form", [
    ([129], 3, 64, 64, False, "tc"), ([256, 1, 130, 127], 4, 36, 40, True, "tc"), ([300, 128], 2, 100, 132, True, "tc"), ([140] * 5, 5, 128, 96, False, "tc"),
    ([200, 65], 2, 33, 64, True, "mma"), ([200], 2, 64, 30, False, "mma"), ([200], 2, 32, 64, False, "mma"), ([700] + [2] * 15, 16, 64, 64, True, "mma")])
def test_linear_attention_of_activated_inputs(new, H, dk, dv, carried, form):
    """Chunks of 128 tokens with all columns of a head, and what stays with chunks of 64. Decays from 0 and far below one to one; inputs whose exponential overflows."""
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(dk)
    T, n = sum(new), len(new)
    q, k, v = (torch.randn(T, H * w, device=DEV, generator=g) for w in (dk, dk, dv))
    q[::7, 3], v[::5, 1] = -95.0, -1e4   # silu: below the smallest number, and 0
    decay = torch.tensor(([1.0, 0.97, 1e-3, 0.5, 0.0, 0.999, 0.9, 0.8] * 2)[:H], device=DEV)
    S0 = torch.randn(n, H, dk, dv, device=DEV, generator=g) if carried else torch.zeros(n, H, dk, dv, device=DEV)
    cu = [sum(new[:i]) for i in range(n + 1)]
    S = S0.clone()
    batch = ops.PackedBatch(_i32(cu), _i32([9 if carried else 0] * n), _i32(list(range(n))), max(new))
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        got = ops.linear_attn(batch, q, k, v, decay, S, heads=H, dim=dk, vdim=dv, in_act="silu")
        torch.cuda.synchronize()
    assert any("la_outputs_tc_kernel" in e.name for e in prof.events()) == (form == "tc")
    silu, d = torch.nn.functional.silu, decay.double()
    for s, t in enumerate(new):
        qq, kk, vv = (silu(x[cu[s]:cu[s + 1]].double()).view(t, H, -1) for x in (q, k, v))
        i = torch.arange(t, device=DEV)
        back = i[:, None] - i[None]
        P = torch.einsum("ihd,jhd->hij", qq, kk) * torch.where(back >= 0, d.view(H, 1, 1) ** back.clamp_min(0), 0.0)
        want = torch.einsum("hij,jhe->ihe", P, vv) + torch.einsum("ihd,hde->ihe", qq, S0[s].double()) * (d ** (i + 1).view(t, 1)).view(t, H, 1)
        assert _err(got[cu[s]:cu[s + 1]], want.reshape(t, -1).cpu()) < BOUND
        want = S0[s].double() * (d ** t).view(H, 1, 1) + torch.einsum("jhd,jhe,hj->hde", kk, vv, d.view(H, 1) ** (t - 1 - i))
        assert _err(S[s], want.cpu()) < BOUND


@pytest.mark.parametrize("taps", [1, 3, 4, 5, 16])
def test_causal_conv_over_portions_of_every_length(taps):
    """Portions shorter and longer than the taps and the kernel's token block, carried on; the taps that stay behind are the last inputs."""
    from vyomai_b200 import ops
    g = torch.Generator().manual_seed(taps)
    C, lengths, more = 130, [1, 15, 16, 17, 70], [33, 2, 16, 1, 15]
    x = [torch.randn(a + b, C, generator=g) for a, b in zip(lengths, more)]
    w = torch.randn(C, taps, generator=g)
    state = torch.full((6, C, max(taps - 1, 1)), float("nan"), device=DEV)
    slots, out = [4, 1, 0, 5, 2], []
    for at, take in (([0] * 5, lengths), (lengths, more)):
        batch = ops.PackedBatch(_i32([sum(take[:i]) for i in range(6)]), _i32(at), _i32(slots), max(take))
        out.append(ops.causal_conv(batch, torch.cat([x[s][at[s]:at[s] + take[s]] for s in range(5)]).to(DEV), w.to(DEV), state, act="silu").split(take))
    for s in range(5):
        assert _err(torch.cat([out[0][s], out[1][s]]), OH.causal_conv(x[s].double(), w.double())) < BOUND
        if taps > 1:
            last = torch.cat([torch.zeros(taps, C), x[s]])[-(taps - 1):]
            assert torch.equal(state[slots[s]].cpu(), last.T)


@pytest.mark.parametrize("M,N,K", [(33, 1, 256), (64, 64, 256), (65, 63, 260), (130, 200, 516), (40, 65, 1000)])
@pytest.mark.parametrize("aligned", [True, False])
def test_fp32_products_on_the_tensor_cores(M, N, K, aligned):
    """Edges of the 64 x 64 x 64 tiles and the shortest K of the rule, with epilogue; unaligned rows take the FMA form; infinities and NaN stay
    where a chain of FMAs has them, and rows of very large and very small numbers keep their precision."""
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(K)
    pad = 4 if aligned else 3
    x, w = (torch.randn(r, K + pad, generator=g, device=DEV)[:, :K] for r in (M, N))
    bias, addend = torch.randn(N, generator=g, device=DEV), torch.randn(M, N, generator=g, device=DEV)
    x[1] *= 1e30
    x[2] *= 1e-30
    want = torch.nn.functional.silu(x.double() @ w.double().T + bias.double()) * 0.5 + addend.double()
    got = ops.linear_plain(x, w, bias=bias, act="silu", scale=0.5, addend=addend)
    plain, exact = ops.linear_plain(x, w), x.double() @ w.double().T
    for a, b in ((got, want), (plain, exact)):
        for rows in (slice(0, 1), slice(1, 2), slice(2, 3), slice(3, M)):
            assert _err(a[rows], b[rows].cpu()) < 2 * BOUND   # a few rows of K terms: the sum may be smaller than its terms
    x[5, K - 1], x[6, 0], w[0, 3] = float("inf"), float("nan"), 0.0
    bad = ops.linear_plain(x, w)
    ref = x.double() @ w.double().T
    assert torch.equal(torch.isnan(bad), torch.isnan(ref)) and torch.equal(torch.isinf(bad), torch.isinf(ref))


@pytest.mark.parametrize("M,N,K", [(33, 9700, 516), (128, 4864, 512), (129, 3300, 580), (700, 2100, 260), (1300, 1000, 320), (9700, 33, 1028)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_fp32_products_split_once(monkeypatch, M, N, K, out_dtype):
    """Operands split ahead of the product: edges of the 128 x 128 tiles and of the stages of 64, with epilogue, large and small rows, infinities and NaN, and entries far below their rows'
    largest ones; beside the form that splits in every tile."""
    from vyomai_b200 import ops
    assert int(ops._lib.lib().vy_linear_plain_bytes(M, N, K)) > 0
    g = torch.Generator(device=DEV).manual_seed(M + K)
    x, w = (torch.randn(r, K + 4, generator=g, device=DEV)[:, :K] for r in (M, N))
    bias, addend = torch.randn(N, generator=g, device=DEV), torch.randn(M, N, generator=g, device=DEV)
    x[1] *= 1e30
    x[2] *= 1e-30
    x[3], w[4] = 0.0, 0.0
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        ops.linear_plain(x, w)
        torch.cuda.synchronize()
    assert any("linear_split_tc_kernel" in e.name for e in prof.events())
    exact = x.double() @ w.double().T
    for add in (None, addend):
        want = torch.nn.functional.silu(exact + bias.double()) * 0.5 + (0.0 if add is None else add.double())
        for got in _both(monkeypatch, "vy_linear_plain_bytes", lambda: ops.linear_plain(x, w, bias=bias, act="silu", scale=0.5, addend=add, out_dtype=out_dtype)):
            for rows in (slice(0, 1), slice(1, 2), slice(2, 4), slice(4, M)):
                assert _err(got[rows], want[rows].cpu()) < (2 * BOUND if out_dtype == torch.float32 else 2.0 ** -8)
    if out_dtype == torch.bfloat16:
        return
    x[5, K - 1], x[6, 0], w[0, 3] = float("inf"), float("nan"), 0.0
    bad, ref = ops.linear_plain(x, w), x.double() @ w.double().T
    assert torch.equal(torch.isnan(bad), torch.isnan(ref)) and torch.equal(torch.isinf(bad), torch.isinf(ref))
    for ratio in (2.0 ** 20, 1e12):
        x, w = torch.randn(M, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV)
        x[:, 7::64], w[:, 7::64] = ratio, 0.0
        assert _err(ops.linear_plain(x, w), (x.double() @ w.double().T).cpu()) < BOUND


@pytest.mark.parametrize("M,N,K", [(700, 1600, 512), (1300, 1001, 516)])
def test_fp32_products_split_once_of_rows_that_hold_nan(M, N, K):
    """Whole rows of NaN, one NaN in a row of either operand, infinities beside it: what float64 gives, and the other rows as without."""
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(N)
    x, w = torch.randn(M, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV)
    clean = ops.linear_plain(x, w)
    nan, inf = float("nan"), float("inf")
    x[3:90], x[200, 7], x[201, 5], x[202, 5:9], w[40, 9], w[41, 1], w[42:60] = nan, nan, inf, torch.tensor([inf, nan, 1.0, -inf], device=DEV), nan, -inf, nan
    got, want = ops.linear_plain(x, w), x.double() @ w.double().T
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want)) and torch.equal(got[torch.isinf(got)].sign(), want[torch.isinf(want)].sign().float())
    ok = torch.isfinite(got)
    assert torch.equal(got[ok], clean[ok])


@pytest.mark.parametrize("K", [512, 8192])
@pytest.mark.parametrize("ratio", [2.0 ** k for k in (12, 16, 18, 20, 21, 22, 24, 40)])
def test_fp32_products_split_once_beside_one_large_entry_per_row(monkeypatch, K, ratio):
    """One entry per row, in one stretch of 64, is `ratio` times the others and meets a zero: the unit of a whole row, results on both sides of the line below which they are computed again
    (about 2^16 sqrt(K) here). No bits fewer than where every tile is split by itself, whose units are its own."""
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(K)
    x, w = torch.randn(260, K, generator=g, device=DEV), torch.randn(2600, K, generator=g, device=DEV)
    x[:, 77], w[:, 77] = ratio, 0.0
    want = (x.double() @ w.double().T).cpu()
    ahead, tiles = (_err(y, want) for y in _both(monkeypatch, "vy_linear_plain_bytes", lambda: ops.linear_plain(x, w)))
    assert ahead < 1.02 * tiles and ahead < BOUND   # 2 %: errors of 676,000 results each


@pytest.mark.parametrize("ratio", [2.0 ** 16, 2.0 ** 20, 2.0 ** 24, 1e8, 1e12, 1e30])
def test_fp32_products_of_entries_far_below_their_row_s_largest(ratio):
    """One entry per row is `ratio` times the others and meets a zero: the sums consist of the small ones alone."""
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(5)
    x, w = torch.randn(65, 320, generator=g, device=DEV), torch.randn(70, 320, generator=g, device=DEV)
    x[:, 7::64] = ratio
    w[:, 7::64] = 0.0
    assert _err(ops.linear_plain(x, w), (x.double() @ w.double().T).cpu()) < BOUND
    w, x = torch.randn(70, 320, generator=g, device=DEV), torch.randn(65, 320, generator=g, device=DEV)
    w[:, 7::64] = ratio
    x[:, 7::64] = 0.0
    assert _err(ops.linear_plain(x, w), (x.double() @ w.double().T).cpu()) < BOUND


def _wide_case(g, T, H, G, d, dv, bad, what):
    """q, k, v of one sequence: one channel of one value row, or one channel of every key (and zeros there in the queries), far outside the others' range."""
    q, k, v = (torch.randn(T, n, w, generator=g) / d ** (0.25 if i < 2 else 0) for i, (n, w) in enumerate(((H, d), (G, d), (G, dv))))
    clean = v.clone()
    if what == "value":
        v[40, :, 5] = bad
    elif what == "row":
        v[40] *= bad
    else:
        k[:, :, 3] = bad
        q[:, :, 3] = 0.0
    return q, k, v, clean


@pytest.mark.parametrize("form", ["softmax", "sigmoid"])
@pytest.mark.parametrize("window", [0, 20])
@pytest.mark.parametrize("what,bad", [("value", 1e5), ("value", 1e9), ("value", float("inf")), ("value", float("nan")), ("row", 1e6), ("row", 1e12), ("key", 1e9), ("key", 1e15)])
def test_prompt_attention_keeps_large_numbers_to_where_they_are_seen(form, window, what, bad):
    """A value that a query does not see changes nothing for it, and one that it sees nothing in the other columns; large key channels that meet zeros
    change nothing. (An infinity or NaN may reach its own column of the queries that share a tile with it: a weight of zero times it.)"""
    from vyomai_b200 import ops
    g = torch.Generator().manual_seed(7)
    T, H, G, d, dv, bs = 70, 4, 2, 64, 40, 16
    q, k, v, clean = _wide_case(g, T, H, G, d, dv, bad, what)
    back = torch.arange(T)[:, None] - torch.arange(T)[None, :]
    seen = (back >= 0) & (back < window) if window else back >= 0
    want = torch.empty(T, H, dv, dtype=torch.float64)
    for h in range(H):
        sc = q[:, h].double() @ k[:, h // 2].double().T
        p = torch.softmax(sc.masked_fill(~seen, -torch.inf), 1) if form == "softmax" else torch.sigmoid(sc) * seen
        for c in range(dv):   # a column of its own: infinity times zero stays out of the others
            x = v[:, h // 2, c].double()
            want[:, h, c] = p @ (x if bool(torch.isfinite(x).all()) else clean[:, h // 2, c].double())
    batch, table, _, n_blocks, _ = shuffled_batch([T], [0], bs, DEV, seed=d)
    kp, vp = torch.zeros(n_blocks, bs, G, d, device=DEV), torch.zeros(n_blocks, bs, G, dv, device=DEV)
    for p in range(T):
        kp[table[0][p // bs], p % bs], vp[table[0][p // bs], p % bs] = k[p].to(DEV), v[p].to(DEV)
    got = ops.window_attn(batch, q.reshape(T, -1).to(DEV), kp, vp, heads=H, kv_heads=G, dim=d, vdim=dv, scale=1.0, window=window, keep_first=0, weights=form,
                          out_dtype=torch.float32).view(T, H, dv).cpu()
    sees = seen[:, 40]
    other = torch.arange(dv) != 5
    finite = bad == bad and abs(bad) < float("inf")
    for rows in (sees, ~sees):
        assert _err(got[rows][..., other], want[rows][..., other]) < BOUND
        if finite:
            assert _err(got[rows][..., 5], want[rows][..., 5]) < BOUND


@pytest.mark.parametrize("window", [0, 20])
@pytest.mark.parametrize("what,bad", [("value", 1e5), ("value", 1e9), ("value", float("inf")), ("value", float("nan")), ("row", 1e12), ("key", 1e9), ("talk", 1e9)])
def test_score_exchanging_prompts_keep_large_numbers_to_where_they_are_seen(window, what, bad):
    """As above. "talk": an exchange weight that meets a head whose scores are all zero."""
    from vyomai_b200 import ops
    g = torch.Generator().manual_seed(8)
    T, H, G, d, dv, bs = 70, 8, 2, 32, 24, 16
    q, k, v, clean = _wide_case(g, T, H, G, d, dv, bad, what)
    talk = torch.eye(H) + 0.3 * torch.randn(H, H, generator=g) / H ** 0.5
    if what == "talk":
        q[:, 6] = 0.0
        talk[:, 6] = bad
    back = torch.arange(T)[:, None] - torch.arange(T)[None, :]
    seen = (back >= 0) & (back < window) if window else back >= 0
    p = OV.plus_one_softmax(OV.mix_heads(OV.capped(torch.stack([q[:, a].double() @ k[:, a // 4].double().T for a in range(H)]) * 0.3, 9.0), talk.double()), seen)
    x = torch.where(torch.isfinite(v), v, clean).double()
    want = torch.stack([p[a] @ x[:, a // 4] for a in range(H)], 1)
    batch, table, _, n_blocks, _ = shuffled_batch([T], [0], bs, DEV, seed=H)
    kp, vp = torch.zeros(n_blocks, bs, G, d, device=DEV), torch.zeros(n_blocks, bs, G, dv, device=DEV)
    for t in range(T):
        kp[table[0][t // bs], t % bs], vp[table[0][t // bs], t % bs] = k[t].to(DEV), v[t].to(DEV)
    got = ops.talk_attn(batch, q.reshape(T, -1).to(DEV), kp, vp, heads=H, kv_heads=G, dim=d, vdim=dv, scale=0.3, softcap=9.0, talk=talk.to(DEV), zero_sink=True,
                        window=window).view(T, H, dv).cpu()
    other = torch.arange(dv) != 5
    for rows in (seen[:, 40], ~seen[:, 40]):
        assert _err(got[rows][..., other], want[rows][..., other]) < 4 * BOUND
        if bad == bad and abs(bad) < float("inf"):
            assert _err(got[rows][..., 5], want[rows][..., 5]) < 4 * BOUND


def _exchange_with_one_bad_entry(H, G, cap, window, what, bad):
    """A prompt of 70 tokens, one of whose query or key entries is `bad`: (this library's output, float64's), [tokens, heads, channels]."""
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(H)
    T, d, bs = 70, 32, 16
    q, talk = torch.randn(T, H, d, generator=g, device=DEV), torch.eye(H, device=DEV) + 0.3 * torch.randn(H, H, generator=g, device=DEV) / H ** 0.5
    batch, table, _, n_blocks, _ = shuffled_batch([T], [0], bs, DEV, seed=H)
    kp, vp = torch.randn(n_blocks, bs, G, d, generator=g, device=DEV), torch.randn(n_blocks, bs, G, d, generator=g, device=DEV)
    if what == "query":
        q[40, 3, 5] = bad
    else:
        kp[table[0][40 // bs], 40 % bs, G - 1, 2] = bad
    got = ops.talk_attn(batch, q.view(T, -1), kp, vp, heads=H, kv_heads=G, dim=d, vdim=d, scale=0.3, softcap=cap, talk=talk, window=window)
    pages = torch.tensor(table[0][:(T + bs - 1) // bs], device=DEV)
    k, v = (x[pages].reshape(-1, G, d)[:T].double().repeat_interleave(H // G, 1) for x in (kp, vp))
    sc = torch.einsum("qhd,khd->hqk", q.double(), k) * 0.3
    sc = torch.einsum("hb,bqk->hqk", talk.double(), cap * torch.tanh(sc / cap) if cap else sc)
    back = torch.arange(T, device=DEV)[:, None] - torch.arange(T, device=DEV)[None, :]
    seen = (back >= 0) & (back < window) if window else back >= 0
    p = torch.softmax(sc.masked_fill(~seen, -float("inf")), -1)
    return got.view(T, H, d), torch.einsum("hqk,khd->qhd", torch.where(seen, p, 0.0), v)


@pytest.mark.parametrize("H,G", [(16, 4), (8, 2), (16, 1)])
@pytest.mark.parametrize("window", [0, 20])
@pytest.mark.parametrize("cap", [0.0, 9.0])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
def test_score_exchanging_prompts_pass_a_bad_key_on_to_who_sees_it(H, G, window, cap, bad):
    """NaN under a cap too, which is no score of the cap's size."""
    got, want = _exchange_with_one_bad_entry(H, G, cap, window, "key", bad)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and bool(torch.isnan(want).any()) == (cap == 0.0 or bad != bad)
    ok = ~torch.isnan(want)
    assert _err(got[ok], want[ok].cpu()) < 4 * BOUND   # as above


@pytest.mark.parametrize("H,G", [(16, 4), (8, 2), (16, 1)])
@pytest.mark.parametrize("cap", [0.0, 9.0])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
def test_score_exchanging_prompts_keep_a_bad_query_to_itself(H, G, cap, bad):
    """128 / H queries share a CTA and its exchange."""
    got, want = _exchange_with_one_bad_entry(H, G, cap, 0, "query", bad)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and bool(torch.isnan(want).any()) == (cap == 0.0 or bad != bad)
    ok = ~torch.isnan(want)
    assert _err(got[ok], want[ok].cpu()) < 4 * BOUND   # as above


@pytest.mark.parametrize("std,most", [(1.0, 2.05e-7), (8.0, 5.55e-7)])
def test_score_exchanging_prompts_lose_no_bits_without_a_cap(std, most):
    """The error of the form on mma.sync at the same shape is 2.17e-7 and 5.6e-7; here it is 1.75e-7 and 5.3e-7 (three seeds within 2 %), and was 2.37e-7 and 5.8e-7 with every score
    multiplied out to an exponent before the row's largest was taken off and every query's heads in eight accumulations, each of which cuts off. The bound lies below both others."""
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(0)
    T, H, d = 600, 16, 64
    q, kp, vp = torch.randn(T, H * d, generator=g, device=DEV), torch.randn(1, T, 4, d, generator=g, device=DEV), torch.randn(1, T, 4, d, generator=g, device=DEV)
    batch = ops.PackedBatch(_i32([0, T]), _i32([0]), _i32([0]), T, _i32([[0]]), T)
    got = ops.talk_attn(batch, q, kp, vp, heads=H, kv_heads=4, dim=d, vdim=d, scale=std / 8)
    k, v = (x[0].double().repeat_interleave(H // 4, 1) for x in (kp, vp))
    sc = torch.einsum("qhd,khd->hqk", q.double().view(T, H, d), k) * (std / 8)
    p = torch.softmax(sc.masked_fill(torch.ones(T, T, dtype=torch.bool, device=DEV).triu(1), -float("inf")), -1)
    assert _err(got, torch.einsum("hqk,khd->qhd", p, v).reshape(T, -1).cpu()) < most


@pytest.mark.parametrize("small", [2.0 ** -k for k in (40, 28, 27, 26, 25, 24, 20, 10)])
def test_score_exchanging_prompts_of_scores_far_below_the_cap(small):
    """What the cap's arithmetic leaves of a score of `small` (up to 2^-23 of the cap, whatever the score) is within the scores' unit."""
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(12)
    T, H, d = 70, 16, 64
    q, kp, vp = torch.randn(T, H * d, generator=g, device=DEV) * small, torch.randn(1, T, 4, d, generator=g, device=DEV), torch.randn(1, T, 4, d, generator=g, device=DEV)
    batch = ops.PackedBatch(_i32([0, T]), _i32([0]), _i32([0]), T, _i32([[0]]), T)
    got = ops.talk_attn(batch, q, kp, vp, heads=H, kv_heads=4, dim=d, vdim=d, scale=0.125, softcap=30.0)
    k, v = (x[0].double().repeat_interleave(H // 4, 1) for x in (kp, vp))
    sc = 30.0 * torch.tanh(torch.einsum("qhd,khd->hqk", q.double().view(T, H, d), k) * 0.125 / 30.0)
    p = torch.softmax(sc.masked_fill(torch.ones(T, T, dtype=torch.bool, device=DEV).triu(1), -float("inf")), -1)
    assert _err(got, torch.einsum("hqk,khd->qhd", p, v).reshape(T, -1).cpu()) < 4 * BOUND   # as above


@pytest.mark.parametrize("bad", [1e5, 1e12, float("inf"), float("nan")])
@pytest.mark.parametrize("where", ["value", "state"])
def test_linear_attention_keeps_large_numbers_to_their_column(bad, where):
    """All chunks at once, then a continuation: a value, or an entry of the state that is carried in, changes its own column and nothing else."""
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(4)
    T, more, H, dk, dv, at, col = 200, 140, 2, 48, 80, 112, 5
    q, k, v = (torch.randn(T + more, H * w, generator=g, device=DEV) for w in (dk, dk, dv))
    S0 = torch.randn(1, H, dk, dv, generator=g, device=DEV)
    decay = torch.tensor([0.99, 0.9], device=DEV)

    def walk(v, S):
        S, out = S.clone(), []
        for a, n in ((0, T), (T, more)):
            batch = ops.PackedBatch(_i32([0, n]), _i32([a + 1]), _i32([0]), n)
            out.append(ops.linear_attn(batch, q[a:a + n], k[a:a + n], v[a:a + n], decay, S, heads=H, dim=dk, vdim=dv))
        return torch.cat(out).view(-1, H, dv), S

    clean, S_clean = walk(v, S0)
    vb, Sb = v.clone(), S0.clone()
    if where == "value":
        vb[at, col] = bad
    else:
        Sb[0, 0, 7, col] = bad
    got, S = walk(vb, Sb)
    hit = torch.zeros_like(got, dtype=torch.bool)
    hit[at if where == "value" else 0:, 0, col] = True
    hit_S = torch.zeros_like(S, dtype=torch.bool)
    hit_S[0, 0, :, col] = True
    assert float((got - clean)[~hit].norm() / clean[~hit].norm()) < BOUND and float((S - S_clean)[~hit_S].norm() / S_clean[~hit_S].norm()) < BOUND
    if not bad == bad or abs(bad) == float("inf"):
        assert not bool(torch.isfinite(got[hit][64:]).any())
    else:
        want = OH.lightning_attention(q.double().view(-1, H, dk).cpu(), k.double().view(-1, H, dk).cpu(), vb.double().view(-1, H, dv).cpu(), decay.double().tolist())
        if where == "value":   # from a state of zero: the column's own numbers
            got0, _ = walk(vb, torch.zeros_like(S0))
            assert _err(got0[:, 0, col], want[:, 0, col].cpu()) < BOUND


@pytest.mark.parametrize("bad", [1e6, 1e12, float("inf")])
def test_state_space_keeps_large_numbers_to_their_column(bad):
    """The same recurrence with a decay per token (vy_ssd): a large input channel of one head stays in its column of the state and out of the other heads."""
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(5)
    T, H, G, N, dv, taps, at, col = 200, 4, 2, 48, 32, 3, 112, 5
    inner, gn = H * dv, G * N
    x, b, c, dt, z = (torch.randn(T, w, generator=g, device=DEV) for w in (inner, gn, gn, H, inner))
    cw = torch.randn(inner + 2 * gn, taps, generator=g, device=DEV).abs() * 0.5

    def run(x):
        state, conv = torch.zeros(1, H, N, dv, device=DEV), torch.zeros(1, taps, inner + 2 * gn, device=DEV)
        out = ops.ssd(ops.PackedBatch(_i32([0, T]), _i32([0]), _i32([0]), T), x, b, c, dt, z, cw, None, conv, torch.zeros(H, device=DEV), torch.full((H,), -2.0, device=DEV),
                      torch.ones(H, device=DEV), torch.ones(inner, device=DEV), state, torch.zeros(1, 1, dtype=torch.int32, device=DEV), heads=H, groups=G, dim=N, vdim=dv,
                      taps=taps, norm_groups=H, norm_eps=1e-5)
        return out.view(T, H, dv), state

    clean, S_clean = run(x)
    xb = x.clone()
    xb[at, col] = bad
    got, S = run(xb)
    hit = torch.zeros_like(S, dtype=torch.bool)
    hit[0, 0, :, col] = True
    assert float((S - S_clean)[~hit].norm() / S_clean[~hit].norm()) < BOUND
    assert float((got - clean)[:, 1:].norm() / clean[:, 1:].norm()) < BOUND and float((got - clean)[:at].norm() / clean[:at].norm()) < BOUND


@pytest.mark.parametrize("bad", [1e6, 1e12, 1e30])
def test_delta_rule_keeps_a_large_value_to_later_tokens(bad):
    """The tokens before a large value that share its 16-token step read what they read without it."""
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(1)
    T, H, dk, dv, at, col = 40, 1, 48, 40, 29, 5
    q, k, v, a, b = (torch.randn(T, w, generator=g, device=DEV) for w in (dk, dk, dv, dk, H))
    batch = ops.PackedBatch(_i32([0, T]), _i32([0]), _i32([0]), T)
    run = lambda vv: ops.delta_rule(batch, q, k, vv, a, b, torch.zeros(1, device=DEV), torch.zeros(1, H, dk, dv, device=DEV), heads=H, kv_heads=H, dim=dk, vdim=dv)  # noqa: E731
    clean = run(v)
    vv = v.clone()
    vv[at, col] = bad
    got = run(vv)
    hit = torch.zeros(T, dv, dtype=torch.bool, device=DEV)
    hit[at:, col] = True
    assert float((got - clean)[16:at, col].norm() / clean[16:at, col].norm()) < BOUND
    assert float((got - clean)[~hit].norm() / clean[~hit].norm()) < BOUND
    unit = lambda x: OH.unit(x.double().cpu().view(T, 1, dk))  # noqa: E731
    decay = torch.exp(-torch.nn.functional.softplus(a.double().cpu(), threshold=1e9).view(T, 1, dk))
    want = OH.gated_delta_rule(unit(q) * dk ** -0.5, unit(k), vv.double().cpu().view(T, 1, dv), decay, torch.sigmoid(b.double().cpu()))[:, 0, col]
    assert _err(got[at:, col], want[at:]) < 4 * BOUND


@pytest.mark.parametrize("dim", [20, 48, 100])
@pytest.mark.parametrize("act", ["sigmoid", "silu", "relu2", "gelu_tanh"])
@pytest.mark.parametrize("T", [40, 150])
def test_linear_attention_activations_leave_padding_alone(dim, act, T):
    """Channel counts that no tile divides, with activations whose value at zero is not zero, chunk by chunk and all chunks at once."""
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(dim)
    q, k, v = (torch.randn(T, w, generator=g, device=DEV) for w in (dim, dim, 20))
    state = torch.zeros(1, 1, dim, 20, device=DEV)
    got = ops.linear_attn(ops.PackedBatch(_i32([0, T]), _i32([0]), _i32([0]), T), q, k, v, torch.tensor([0.9], device=DEV), state, heads=1, dim=dim, vdim=20, in_act=act)
    f = {"sigmoid": torch.sigmoid, "silu": torch.nn.functional.silu, "relu2": lambda x: torch.relu(x) ** 2, "gelu_tanh": lambda x: torch.nn.functional.gelu(x, approximate="tanh")}[act]
    x = [f(t.double().cpu()).view(T, 1, -1) for t in (q, k, v)]
    assert _err(got, OH.lightning_attention(*x, [float(torch.tensor(0.9))]).reshape(T, -1)) < 2 * BOUND   # activations in fp32


def test_a_wait_that_timed_out_stops_what_would_use_its_results():
    """The flag such a wait raises (here from the host): attention, delta rule, product and a serving step refuse until it is acknowledged, in fp32 models too."""
    from tests import hybrid_util as HU
    from vyomai_b200 import ops
    from vyomai_b200._lib import VyomError, lib
    model, _ = HU.build(HU.small_config())   # fp32: no vy_gemm
    engine, _ = HU.engine_for(model)
    for _ in range(3):
        engine.feed([("a", [3], [0])])   # from the third on a replayed step
    x = torch.randn(64, 64, device=DEV)
    batch = ops.PackedBatch(_i32([0, 64]), _i32([0]), _i32([0]), 64, _i32([[0]]), 64)
    calls = [lambda: ops.window_attn(batch, x, x.view(1, 64, 1, 64), x.view(1, 64, 1, 64), heads=1, kv_heads=1, dim=64, vdim=64, scale=1.0, window=0, keep_first=0),
             lambda: ops.delta_rule(batch, x, x, x, x, x[:, :1], torch.zeros(1, device=DEV), torch.zeros(1, 1, 64, 64, device=DEV), heads=1, kv_heads=1, dim=64, vdim=64),
             lambda: ops.gemm(x, x), lambda: engine.feed([("a", [3], [0])])]
    for call in calls:
        call()
    assert lib().vy_gemm_poison_raise() == 0
    try:
        for call in calls:
            with pytest.raises(VyomError, match="timed out"):
                call()
    finally:
        assert lib().vy_gemm_poisoned() == 1
    for call in calls:
        call()
    torch.cuda.synchronize()
    assert lib().vy_gemm_poison_peek() == 0


def test_every_op_whose_kernels_wait_looks_at_the_flag():
    """As above, for the others that launch such kernels: score-exchanging attention, linear attention, state space, grouped experts, products split once."""
    from vyomai_b200 import ops
    from vyomai_b200._lib import VyomError, lib
    x, one = torch.randn(256, 64, device=DEV), torch.ones(1, device=DEV)
    batch = ops.PackedBatch(_i32([0, 256]), _i32([0]), _i32([0]), 256, _i32([[0]]), 256)
    pool, h, big = x.view(1, 256, 1, 64), x.bfloat16(), torch.randn(2560, 512, device=DEV)
    need = ops.moe_grouped_bytes(256, 2, 1, 64, 64, 0)
    assert int(lib().vy_linear_plain_bytes(2560, 512, 512)) > 0
    calls = [lambda: ops.talk_attn(batch, x.repeat(1, 8), pool, pool, heads=8, kv_heads=1, dim=64, vdim=64, scale=1.0),
             lambda: ops.linear_attn(batch, x, x, x, one, torch.zeros(1, 1, 64, 64, device=DEV), heads=1, dim=64, vdim=64, in_act="silu"),
             lambda: ops.linear_attn(batch, x, x, x, one, torch.zeros(1, 1, 64, 64, device=DEV), heads=1, dim=64, vdim=64),
             lambda: ops.ssd(batch, x, x, x, x[:, :1], x, conv_w=torch.ones(192, 3, device=DEV), conv_b=None, dt_bias=one, a_log=one, skip=one, norm=torch.ones(64, device=DEV), heads=1, groups=1,
                             dim=64, vdim=64, taps=3, norm_groups=1, norm_eps=1e-5, conv_state=torch.zeros(1, 3, 192, device=DEV), state=torch.zeros(1, 1, 64, 64, device=DEV),
                             tickets=torch.zeros(1, 1, dtype=torch.int32, device=DEV)),
             lambda: ops.moe_grouped(h, torch.zeros(256, 1, dtype=torch.int32, device=DEV), torch.ones(256, 1, device=DEV), h, h[:64].repeat(1, 2), experts=2, ff=64,
                                     workspace=torch.empty(need, dtype=torch.uint8, device=DEV)),
             lambda: ops.linear_plain(big, big[:512])]
    for call in calls:
        call()
    assert lib().vy_gemm_poison_raise() == 0
    try:
        for call in calls:
            with pytest.raises(VyomError, match="timed out"):
                call()
    finally:
        assert lib().vy_gemm_poisoned() == 1
    for call in calls:
        call()
    torch.cuda.synchronize()


def test_causal_conv_over_very_many_channels():
    """More channels than a launch has blocks of 128 for."""
    from vyomai_b200 import ops
    C = 65535 * 128 + 130
    g = torch.Generator(device=DEV).manual_seed(2)
    x, w, state = torch.randn(2, C, generator=g, device=DEV), torch.randn(C, 2, generator=g, device=DEV), torch.zeros(1, C, 1, device=DEV)
    out = ops.causal_conv(ops.PackedBatch(_i32([0, 2]), _i32([0]), _i32([0]), 2), x, w, state, act=None)
    assert torch.equal(state[0, :, 0], x[1]) and torch.equal(out[0], x[0] * w[:, 1])
    assert float((out[1] - (x[1] * w[:, 1] + x[0] * w[:, 0])).abs().max()) < 1e-5


def test_scratch_that_cannot_be_had_is_done_without(monkeypatch):
    """A device without room for a prompt form's scratch: the step takes the form that needs none. Attention in a smaller scratch: a few sequences at a time."""
    from vyomai_b200 import ops
    assert ops._lend(1 << 50, torch.device(DEV)) is None and ops._lend(0, torch.device(DEV)) is None
    g = torch.Generator(device=DEV).manual_seed(6)
    R = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    new, bs, H = [70, 33, 130, 5], 16, 8
    cu = [sum(new[:i]) for i in range(5)]
    q, k, v, a, b = (R(cu[4], w) for w in (H * 32, H * 32, H * 32, H * 32, H))
    kp, vp = R(40, bs, 2, 32), R(40, bs, 2, 32)
    batch = ops.PackedBatch(_i32(cu), _i32([0, 20, 0, 30]), _i32([0, 1, 2, 3]), 130, torch.arange(40, dtype=torch.int32, device=DEV).view(4, 10), bs)
    x = {n: R(cu[4], w) for n, w in (("x", H * 32), ("b", 64), ("c", 64), ("dt", H), ("gate", H * 32))}
    ssd = dict(conv_w=R(H * 32 + 128, 3), conv_b=None, dt_bias=R(H), a_log=R(H), skip=R(H), norm=R(H * 32), heads=H, groups=2, dim=32, vdim=32, taps=3, norm_groups=H, norm_eps=1e-5)
    calls = [lambda: ops.window_attn(batch, q, kp, vp, heads=H, kv_heads=2, dim=32, vdim=32, scale=0.2, window=40, keep_first=3),
             lambda: ops.talk_attn(batch, q, kp, vp, heads=H, kv_heads=2, dim=32, vdim=32, scale=0.2, softcap=9.0, zero_sink=True),
             lambda: ops.linear_attn(batch, q, k, v, torch.full((H,), 0.9, device=DEV), torch.zeros(4, H, 32, 32, device=DEV), heads=H, dim=32, vdim=32),
             lambda: ops.delta_rule(batch, q, k, v, a, b, torch.zeros(H, device=DEV), torch.zeros(4, H, 32, 32, device=DEV), heads=H, kv_heads=H, dim=32, vdim=32),
             lambda: ops.ssd(batch, **x, **ssd, conv_state=torch.zeros(4, 3, H * 32 + 128, device=DEV), state=torch.zeros(4, H, 32, 32, device=DEV),
                             tickets=torch.zeros(4, 1, dtype=torch.int32, device=DEV))]
    whole = [c() for c in calls]
    monkeypatch.setattr(ops, "_prompt_attn_floats", lambda one, n_seqs: one)   # one sequence at a time
    for c, want in zip(calls[:2], whole):
        assert torch.equal(c(), want)
    monkeypatch.setattr(ops, "_lend", lambda floats, device: None)
    for c, want in zip(calls, whole):
        assert float((c() - want).norm() / want.norm()) < 4 * BOUND


def test_a_forced_form_is_taken_with_scratch_too(monkeypatch):
    """A caller that forces the tiled form of the score-exchanging attention and lends scratch gets the tiled form."""
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(9)
    q, kp, vp = torch.randn(64, 8 * 32, generator=g, device=DEV), torch.randn(4, 16, 2, 32, generator=g, device=DEV), torch.randn(4, 16, 2, 32, generator=g, device=DEV)
    batch = ops.PackedBatch(_i32([0, 64]), _i32([0]), _i32([0]), 64, _i32([[0, 1, 2, 3]]), 16)
    call = lambda: ops.talk_attn(batch, q, kp, vp, heads=8, kv_heads=2, dim=32, vdim=32, scale=0.2, softcap=9.0, form="tiled")  # noqa: E731
    want, real, ws = call(), ops._lib.call, torch.empty(1 << 22, device=DEV)
    monkeypatch.setattr(ops._lib, "call", lambda fn, st, **kw: real(fn, st, **{**kw, "workspace": ws.data_ptr(), "workspace_floats": ws.numel()}))
    assert torch.equal(call(), want)


@pytest.mark.parametrize("width,ff,experts,top,form,rows,want", [(1024, 256, 28, 3, "swiglu", 1024, False), (1024, 256, 28, 3, "swiglu", 4096, True), (512, 128, 28, 3, "swiglu", 4096, False),
                                                                 (1024, 512, 8, 2, "glu", 768, False), (1024, 512, 8, 2, "glu", 2048, True), (1024, 256, 16, 2, "plain", 1024, False),
                                                                 (1024, 256, 16, 2, "plain", 4096, True)])
def test_fp32_experts_are_sorted_where_that_is_faster(width, ff, experts, top, form, rows, want):
    """The estimate against what was measured (both forms at these sizes, the slower one at least a fifth behind)."""
    from vyomai_b200.layers.mixers import MoEFeedForward
    w = {"router": torch.zeros(experts, width, device=DEV)}
    for e in range(experts):
        w.update({f"e{e}.{k}": torch.zeros(ff, width, device=DEV) for k in (("up",) if form == "plain" else ("up", "gate"))})
        w[f"e{e}.down"] = torch.zeros(width, ff, device=DEV)
    assert MoEFeedForward(w, experts, top, 1.0, torch.float32, True, router="softmax", form=form)._sorted_is_faster(rows) is want


@pytest.mark.parametrize("form,H,G,d,dv,window,keep", [("softmax", 4, 4, 96, 128, 33, 5), ("sigmoid", 4, 4, 128, 72, 0, 0), ("softmax", 8, 2, 128, 128, 70, 0), ("sigmoid", 8, 2, 40, 100, 33, 5)])
def test_prompt_attention_in_blocks_of_192_rows(form, H, G, d, dv, window, keep):
    """Enough sequences of odd length for the wide form (window_attn_mma.cu: two rounds of its CTAs over the SMs), from position 0 and carried on."""
    from vyomai_b200 import ops
    g = torch.Generator().manual_seed(d)
    new = [193, 47, 49, 16, 97, 1] * 7
    pos0 = [(29 * i) % 90 for i in range(len(new))]
    rep = H // G
    hl = min(4, rep.bit_length() - 1)
    qn = 192 >> hl
    assert (max(new) + qn - 1) // qn * (H >> hl) * len(new) >= 2 * torch.cuda.get_device_properties(0).multi_processor_count
    T = [n + p for n, p in zip(new, pos0)]
    q, k, v = ([torch.randn(t, n, w, generator=g) / d ** (0.25 if i < 2 else 0) for t in T] for i, (n, w) in enumerate(((H, d), (G, d), (G, dv))))
    want, bs = [], 16
    for s, t in enumerate(T):
        i, j = torch.arange(pos0[s], t)[:, None], torch.arange(t)[None, :]
        seen = (j <= i) & ((i - j < window) | (j < keep)) if window else j <= i
        kk, vv = (x[s].double().repeat_interleave(rep, 1) for x in (k, v))
        sc = torch.einsum("ihd,jhd->hij", q[s][pos0[s]:].double(), kk)
        p = torch.softmax(sc.masked_fill(~seen, -torch.inf), 2) if form == "softmax" else torch.sigmoid(sc) * seen
        want.append(torch.einsum("hij,jhd->ihd", p, vv).reshape(new[s], -1))
    batch, table, _, n_blocks, _ = shuffled_batch(new, pos0, bs, DEV, seed=d)
    kp, vp = torch.full((n_blocks, bs, G, d), 1e3), torch.full((n_blocks, bs, G, dv), 1e3)
    for s, t in enumerate(T):
        at = torch.arange(t)
        rows = torch.tensor([table[s][p // bs] for p in range(t)])
        kp[rows, at % bs], vp[rows, at % bs] = k[s], v[s]
    got = ops.window_attn(batch, torch.cat([q[s][pos0[s]:].reshape(new[s], -1) for s in range(len(new))]).to(DEV), kp.to(DEV), vp.to(DEV), heads=H, kv_heads=G, dim=d, vdim=dv,
                          scale=1.0, window=window, keep_first=keep, weights=form, out_dtype=torch.float32)
    assert _err(got, torch.cat(want)) < BOUND


@pytest.mark.parametrize("form,H,G,d,dv,window,keep,chunk,cap,new,pos0", [
    ("softmax", 2, 2, 64, 64, 0, 0, 0, 0.0, [128, 127, 64, 1, 65], [0, 64, 65, 200, 63]),          # one tile, whole tiles, an odd number of them
    ("softmax", 8, 2, 128, 128, 70, 0, 0, 30.0, [193, 33, 130, 1], [0, 100, 31, 190]),              # bands that start inside a tile
    ("sigmoid", 8, 2, 128, 96, 0, 0, 0, 0.0, [131, 40, 257], [0, 90, 3]),
    ("softmax", 16, 1, 96, 64, 50, 70, 0, 0.0, [140, 9, 300], [0, 200, 77]),                         # kept tokens: two tiles of them, one of them inside the band
    ("sigmoid", 4, 1, 33, 7, 20, 5, 0, 0.0, [150, 16], [10, 300]),
    ("softmax", 3, 3, 112, 128, 0, 0, 48, 0.0, [200, 47, 96], [0, 50, 144]),                         # blocks of 48 positions
    ("softmax", 6, 3, 16, 24, 129, 0, 0, 5.0, [385, 66], [0, 130]),
    ("sigmoid", 4, 4, 128, 128, 0, 0, 0, 0.0, [100, 37, 64] * 25, [0, 3, 40] * 25),                  # fewer rows than a tile, many sequences: 192 rows on mma.sync
])
def test_prompt_attention_on_tcgen05(form, H, G, d, dv, window, keep, chunk, cap, new, pos0):
    """The edges of 64-key tiles, of pairs of them and of 128-row blocks, in every form of the scores, with sinks, gates and slopes; padded query rows."""
    from vyomai_b200 import ops
    g = torch.Generator().manual_seed(d + dv)
    rep, bs, T = H // G, 16, [n + p for n, p in zip(new, pos0)]
    q, k, v = ([torch.randn(t, n, w, generator=g) / d ** (0.25 if i < 2 else 0) for t in T] for i, (n, w) in enumerate(((H, d), (G, d), (G, dv))))
    sink, gate, slopes = torch.randn(H, generator=g), [torch.randn(n, H, generator=g) for n in new], torch.tensor(OZ.head_slopes(H), dtype=torch.float32)
    want = []
    for s, t in enumerate(T):
        i, j = torch.arange(pos0[s], t)[:, None], torch.arange(t)[None, :]
        seen = (j <= i) & ((i - j < window) | (j < keep)) if window else (j <= i) & (j >= i // chunk * chunk) if chunk else j <= i
        kk, vv = (x[s].double().repeat_interleave(rep, 1) for x in (k, v))
        sc = torch.einsum("ihd,jhd->hij", q[s][pos0[s]:].double(), kk) * 1.5
        if cap:
            sc = cap * torch.tanh(sc / cap) - slopes.double()[:, None, None] * (i - j)
        if form == "softmax":
            p = torch.softmax(torch.cat([sc.masked_fill(~seen, -torch.inf), sink.double()[:, None, None].expand(H, new[s], 1)], 2), 2)[:, :, :t]
        else:
            p = torch.sigmoid(sc) * seen
        want.append((torch.einsum("hij,jhd->ihd", p, vv) * torch.sigmoid(gate[s].double())[:, :, None]).reshape(new[s], -1))
    batch, table, _, n_blocks, _ = shuffled_batch(new, pos0, bs, DEV, seed=d)
    kp, vp = torch.full((n_blocks, bs, G, d), 1e3), torch.full((n_blocks, bs, G, dv), 1e3)
    for s, t in enumerate(T):
        rows = torch.tensor([table[s][p // bs] for p in range(t)])
        kp[rows, torch.arange(t) % bs], vp[rows, torch.arange(t) % bs] = k[s], v[s]
    wide = torch.cat([torch.cat([q[s][pos0[s]:].reshape(new[s], -1) for s in range(len(new))]), torch.zeros(sum(new), 3)], 1).to(DEV)[:, :-3]
    call = lambda: ops.window_attn(batch, wide, kp.to(DEV), vp.to(DEV), heads=H, kv_heads=G, dim=d, vdim=dv, scale=1.5, window=window, keep_first=keep, chunk=chunk,  # noqa: E731
                                   weights=form, softcap=cap, head_slope=slopes.to(DEV) if cap else None, sink=sink.to(DEV) if form == "softmax" else None,
                                   gate=torch.cat(gate).to(DEV), out_dtype=torch.float32)
    got = call()
    # a capped score is cap (1 - 2 r) with r in [0, 1] off by a unit in its last place: cap 2^-24 as an exponent, as much as that of the weight. Not this form's alone:
    # cap 30 with slopes and sinks, 2048 tokens, 8 heads of 128 over 2, window 512: 1.154e-6 of the 2-norm here, 1.159e-6 on mma.sync (without a cap 2.7e-7 and 3.3e-7)
    assert _err(got, torch.cat(want)) < BOUND + cap * 2.0 ** -24
    assert torch.equal(call(), got)


def test_delta_rule_form_for_one_prompt_beside_many_tokens():
    """One long portion beside many short ones takes the walk up to a length that grows with the rounds of CTAs; portions that are alike do not."""
    from vyomai_b200._lib import lib
    floats = lambda lengths, H, d: int(lib().vy_delta_rule_prompt_floats(sum(lengths), len(lengths), max(lengths), H, d, d))  # noqa: E731
    assert floats([32] + [1] * 31, 8, 128) == 0 and floats([100] + [1] * 31, 8, 128) > 0
    assert floats([70] + [1] * 63, 8, 128) == 0 and floats([200] + [1] * 63, 8, 128) > 0
    assert floats([32] * 32, 8, 128) > 0 and floats([32] + [1] * 7, 8, 128) > 0 and floats([48] + [1] * 31, 4, 64) > 0


def test_delta_rule_sums_are_not_cut_short():
    """A tensor-core accumulation cuts off where fp32 rounds; delta_rule_mma.cu adds back the share that costs on average. On a part that accumulates in another way the
    correction would itself be a bias: read-outs measure -0.4e-8 with it, -5.8e-8 without it, the serial walk +0.5e-8."""
    from vyomai_b200 import ops
    g = torch.Generator().manual_seed(11)
    T, H, d = 320, 4, 128
    q, k, v, a, b = (torch.randn(T, w, generator=g) for w in (H * d, H * d, H * d, H * d, H))
    unit = lambda x: OH.unit(x.double().view(T, H, d))  # noqa: E731
    decay = torch.exp(-torch.exp(torch.tensor(-3.0).double()) * torch.nn.functional.softplus(a.double(), threshold=1e9).view(T, H, d))
    want = OH.gated_delta_rule(unit(q) * d ** -0.5, unit(k), v.double().view(T, H, d), decay, torch.sigmoid(b.double())).reshape(T, -1)
    c = lambda x: x.to(DEV)  # noqa: E731
    got = ops.delta_rule(ops.PackedBatch(_i32([0, T]), _i32([0]), _i32([0]), T), c(q), c(k), c(v), c(a), c(b), torch.full((H,), -3.0, device=DEV),
                         torch.zeros(1, H, d, d, device=DEV), heads=H, kv_heads=H, dim=d, vdim=d).double().cpu()
    assert abs(float(((got - want) * want).sum() / (want * want).sum())) < 4e-8


def test_linear_attention_sums_are_not_cut_short():
    """The same in linear_attn_mma.cu: read-outs measure -1.1e-8 with the share added back, -1.4e-7 without it, the chunk walk -0.8e-8."""
    from vyomai_b200 import ops
    g = torch.Generator().manual_seed(12)
    T, H, d = 600, 4, 64
    q, k, v = (torch.randn(T, H * d, generator=g) for _ in range(3))
    decay = float(torch.tensor(0.9))
    want = OH.lightning_attention(*(x.double().view(T, H, d) for x in (q, k, v)), [decay] * H).reshape(T, -1)
    got = ops.linear_attn(ops.PackedBatch(_i32([0, T]), _i32([0]), _i32([0]), T), q.to(DEV), k.to(DEV), v.to(DEV), torch.full((H,), decay, device=DEV),
                          torch.zeros(1, H, d, d, device=DEV), heads=H, dim=d, vdim=d).double().cpu()
    assert abs(float(((got - want) * want).sum() / (want * want).sum())) < 4e-8


def test_linear_attention_form_for_one_prompt_beside_many_tokens():
    """One long portion beside many short ones takes the walk up to a length that grows with the chunks; portions that are alike do from three chunks on."""
    from vyomai_b200._lib import lib
    floats = lambda lengths, H, d, dv: int(lib().vy_linear_attn_workspace_floats(sum(lengths), len(lengths), max(lengths), H, d, dv))  # noqa: E731
    assert floats([128], 16, 128, 64) == 0 and floats([130], 16, 128, 64) > 0 and floats([130] * 32, 16, 128, 64) > 0
    assert floats([200] + [1] * 31, 16, 128, 64) == 0 and floats([512] + [1] * 31, 16, 128, 64) > 0 and floats([200] + [1] * 7, 16, 128, 64) > 0
    assert floats([400] + [1] * 31, 32, 128, 64) == 0 and floats([2000] + [1] * 31, 32, 128, 64) > 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_a_repeated_product_reads_its_own_operands(dtype):
    """Products of one shape share a prepared argument block: other addresses, strides and streams give what a first call gives."""
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(2)
    xs = [torch.randn(96, 264, generator=g, device=DEV).to(dtype) for _ in range(6)]
    ws = [torch.randn(128, 256, generator=g, device=DEV).to(dtype) for _ in range(6)]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    for i, (x, w) in enumerate(zip(xs, ws)):
        x = x[:, :256] if i % 2 else x[:, :256].contiguous()
        with torch.cuda.stream(side if i % 3 == 2 else torch.cuda.current_stream()):
            y = ops.gemm(x, w)
        torch.cuda.synchronize()
        want = x.double() @ w.double().T
        assert float((y.double() - want).norm() / want.norm()) < (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -9)   # the output's or the operands' rounding


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_norm_gradients_in_the_parameters_type(dtype):
    from vyomai_b200 import ops
    from vyomai_b200.autograd_train import _ln_bwd
    g = torch.Generator(device=DEV).manual_seed(3)
    W, rows = 264, 77
    s, dy = (torch.randn(rows, W, generator=g, device=DEV).to(dtype) for _ in range(2))
    gamma, beta, bias = (torch.nn.Parameter(torch.randn(W, generator=g, device=DEV).to(dtype)) for _ in range(3))
    mean = s.float().mean(1)
    rstd = torch.rsqrt(s.float().var(1, unbiased=False) + 1e-5)
    ds, dg, db, dbias = _ln_bwd(dy, s, gamma, beta, mean, rstd, bias)
    xhat = (s.double() - mean.double()[:, None]) * rstd.double()[:, None]
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else BOUND
    assert dg.dtype == db.dtype == dbias.dtype == dtype
    assert _err(dg, (dy.double() * xhat).sum(0).cpu()) < tol and _err(db, dy.double().sum(0).cpu()) < tol
    dx = gamma.double() * dy.double()
    dx = (dx - dx.mean(1, keepdim=True) - xhat * (dx * xhat).mean(1, keepdim=True)) * rstd.double()[:, None]
    assert _err(ds, dx.cpu()) < 2 * tol and _err(dbias, dx.sum(0).cpu()) < 32 * tol   # columns of dx nearly cancel

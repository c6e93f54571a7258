"""-m gpu: forms of the packed decoders' row kernels for fp32 rows on 16-byte boundaries (four neighbouring entries per thread), against the general forms, which the
same call takes on operands one element off. Both sum the same fp32 numbers in another order or round one operation otherwise: a few units in the last place, 8 * 2^-24
of the result's 2-norm."""
import pytest
import torch

from tests.hybrid_util import shuffled_batch

pytestmark = pytest.mark.gpu
DEV = "cuda"
BOUND = 8 * 2.0 ** -24


def _close(a, b):
    assert a.shape == b.shape and float((a.double() - b.double()).norm()) <= BOUND * float(b.double().norm())


def _off(t):
    """The same values, one element past a 16-byte boundary."""
    if t is None:
        return None
    buf = torch.zeros(t.numel() + t.shape[0] * 4 + 8, device=t.device, dtype=t.dtype)
    v = torch.as_strided(buf, t.shape, (t.shape[1] + 4 - t.shape[1] % 4, 1), 1)
    v.copy_(t)
    return v


def _ran(call, kernel):
    """The call's result, made by `kernel`."""
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        out = call()
        torch.cuda.synchronize()
    assert any(kernel in e.key for e in prof.key_averages()), kernel
    return out


@pytest.mark.parametrize("taps", [1, 2, 4])
@pytest.mark.parametrize("act", ["silu", "sigmoid", None])
def test_convolution_of_four_channels_per_thread(taps, act):
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(taps)
    C, pos0 = 20004, [0, 3, 0, 40, 2]   # enough channels for two CTAs per SM
    batch = ops.PackedBatch(torch.tensor([0, 1, 16, 32, 49, 119], dtype=torch.int32, device=DEV), torch.tensor(pos0, dtype=torch.int32, device=DEV),
                            torch.tensor([4, 1, 0, 5, 2], dtype=torch.int32, device=DEV), 70)
    x, w, state = torch.randn(119, C, generator=g, device=DEV) * 3, torch.randn(C, taps, generator=g, device=DEV), torch.randn(6, C, max(taps - 1, 1), generator=g, device=DEV)
    x[5, 7], x[6, 9], x[7, 11], w[11] = 200.0, -200.0, -1e30, w[11].abs()   # the exponentials there overflow or vanish
    if taps == 1:
        state = state[:, :, :0].contiguous()
    states = [state.clone(), state.clone()]
    a = _ran(lambda: ops.causal_conv(batch, x, w, states[0], act=act), "causal_conv_quads_kernel")
    b = _ran(lambda: ops.causal_conv(batch, _off(x), w, states[1], act=act), "causal_conv_kernel")
    _close(a, b)
    assert torch.equal(*states)


@pytest.mark.parametrize("taps", [1, 2, 3, 4])
def test_convolutions_keep_infinities_to_the_tokens_that_see_them(taps):
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(taps)
    C, n = 16384, 160
    batch = ops.PackedBatch(*(torch.tensor(t, dtype=torch.int32, device=DEV) for t in ([0, n], [0], [0])), n)
    x, w = torch.randn(n, C, generator=g, device=DEV), torch.randn(C, taps, generator=g, device=DEV)
    x[5, 3], x[33, 3], x[33, 8], x[47, 100], x[159, 7] = float("inf"), float("nan"), float("-inf"), float("inf"), float("inf")
    run = lambda t: ops.causal_conv(batch, t, w, torch.zeros(1, C, max(taps - 1, 1), device=DEV)[:, :, :taps - 1].contiguous(), act=None)  # noqa: E731
    a, b = _ran(lambda: run(x), "causal_conv_quads_kernel"), _ran(lambda: run(_off(x)), "causal_conv_kernel")
    seen = torch.zeros(n, C, dtype=torch.bool, device=DEV)
    for i, c in (~x.isfinite()).nonzero().tolist():
        seen[i:i + taps, c] = True
    assert torch.equal(~a.isfinite(), seen) and torch.equal(a.isnan(), b.isnan())
    _close(a.nan_to_num(0, 0, 0), b.nan_to_num(0, 0, 0))


@pytest.mark.parametrize("layout,rot,dim", [("half", 64, 128), ("half", 24, 48), ("pairs", 6, 20), ("pairs", 128, 128), ("pairs", 0, 128), ("half", 128, 128)])
@pytest.mark.parametrize("norm,pool", [("weight", torch.float32), ("unit", torch.float32), (None, torch.bfloat16), ("unit", None)])
def test_rotation_of_four_entries_per_lane(layout, rot, dim, norm, pool):
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(dim + rot)
    H, G, dv, new, pos0 = 5, 2, 36, [170, 1, 1247], [0, 300, 7]
    batch, _, _, blocks, _ = shuffled_batch(new, pos0, 16, DEV, seed=rot)
    q, k, v = (torch.randn(sum(new), n, generator=g, device=DEV) for n in (H * dim, G * dim, G * dv))
    freq = 100.0 ** -(torch.arange(max(rot // 2, 1), device=DEV) / max(rot // 2, 1))
    nw = torch.randn(dim, generator=g, device=DEV) if norm == "weight" else None

    def run(q, k, v):
        kp, vp = (None, None) if pool is None else (torch.zeros(blocks, 16, G, dim, device=DEV, dtype=pool), torch.zeros(blocks, 16, G, dv, device=DEV, dtype=pool))
        ko = k if pool is None else None
        ops.rope_kv_write(batch, q, k, v, freq, kp, vp, heads=H, kv_heads=G, dim=dim, vdim=dv, rot_dims=rot, layout=layout, rot_scale=1.5, unit_rms=norm == "unit", eps=1e-6,
                          q_scale=0.7, k_scale=1.3, k_out=ko, q_norm=nw, k_norm=nw, q_temp=(0.3, 9) if norm else None)
        return q, (ko if pool is None else kp.float()), (v if pool is None else vp.float())

    a, b = _ran(lambda: run(q.clone(), k.clone(), v), "rope_heads_rows_kernel"), _ran(lambda: run(_off(q), _off(k), _off(v)), "rope_heads_kernel")
    _close(a[0], b[0])
    if pool == torch.bfloat16:   # one rounding of a key may go the other way
        assert float((a[1] - b[1]).abs().max()) <= 2.0 ** -7 * float(b[1].abs().max())
    else:
        _close(a[1], b[1])
    assert torch.equal(a[2], b[2])


def _gates():
    """Arguments of SiLU and sigmoid over fp32's range, dense where e^-x leaves the range of the approximate reciprocal (2^126: x = -87.3) and of fp32 (-88.7)."""
    e = torch.tensor([float("inf"), float("-inf"), float("nan"), 0.0, -0.0, 3e38, -3e38, -1e30, 1e-30, -1e-30, -100.0, 100.0], device=DEV)
    x = torch.cat([e, torch.linspace(-89.0, -87.0, 2036, device=DEV), torch.linspace(-110.0, 110.0, 2048, device=DEV)])
    return x, {"silu": x.double() * torch.sigmoid(x.double()), "sigmoid": torch.sigmoid(x.double())}


def _gate_close(got, want, x, act):
    """A few roundings, and what fp32 flushes where e^-x is infinite: |x| 2^-128 (sigmoid: 2^-128)."""
    want = torch.where(x == float("-inf"), torch.full_like(want, float("nan") if act == "silu" else 0.0), want)   # x / (1 + e^-x) is -inf / inf there
    assert torch.equal(got.isnan(), want.isnan())
    fine = want.isfinite()
    assert torch.equal(got.double()[~fine].nan_to_num(1.0), want[~fine].nan_to_num(1.0))
    room = 2.0 ** -21 * want.abs() + 2.0 ** -128 * (x.abs().double().clamp(max=200.0) if act == "silu" else 1.0)
    assert bool(((got.double() - want).abs() <= room)[fine].all())


@pytest.mark.parametrize("act", ["silu", "sigmoid"])
def test_gates_over_the_whole_range(act):
    from vyomai_b200 import ops
    x, want = _gates()
    n = 640   # tokens: enough for the form with four channels per thread
    batch = ops.PackedBatch(*(torch.tensor(t, dtype=torch.int32, device=DEV) for t in ([0, n], [0], [0])), n)
    xs = x.expand(n, -1).contiguous()
    got = _ran(lambda: ops.causal_conv(batch, xs, torch.ones(x.numel(), 1, device=DEV), torch.zeros(1, x.numel(), 0, device=DEV), act=act), "causal_conv_quads_kernel")
    for row in (got[0], got[-1]):
        _gate_close(row, want[act], x, act)
    ones = torch.ones(3, x.numel(), device=DEV)
    got = ops.rms_norm(ones, None, eps=0.0, gate=xs[:3].contiguous(), gate_act=act)
    _gate_close(got[2], want[act], x, act)
    if act == "silu":   # the state-space convolution: x | b | c, one tap; what it gives shows in the read-out of a token with no state before it
        H, dim, vdim = 8, 16, 64
        v = x[:512].clone()
        v[:12] = -88.0
        xs, b = v.expand(4, -1).contiguous(), torch.full((4, dim), 30.0, device=DEV)   # silu(30) = 30 to 1e-13
        w = dict(conv_w=torch.ones(512 + 2 * dim, 1, device=DEV), conv_b=None, dt_bias=torch.full((H,), -50.0, device=DEV), a_log=torch.zeros(H, device=DEV), skip=torch.ones(H, device=DEV),
                 norm=torch.full((512,), 1.0, device=DEV), heads=H, groups=1, dim=dim, vdim=vdim, taps=1, norm_groups=1, norm_eps=1.0, out_dtype=torch.float32)
        batch = ops.PackedBatch(*(torch.tensor(t, dtype=torch.int32, device=DEV) for t in ([0, 4], [0], [0])), 4)
        got = ops.ssd(batch, xs, b, b.clone(), torch.zeros(4, H, device=DEV), None, **w, conv_state=torch.zeros(1, 1, 512 + 2 * dim, device=DEV), state=torch.zeros(1, H, dim, vdim, device=DEV),
                      tickets=torch.zeros(1, 1, dtype=torch.int32, device=DEV))
        _gate_close(got[0] if bool(got.isfinite().all()) else got[0] * float("nan"), v.double() * torch.sigmoid(v.double()), v, "silu")

"""-m gpu: state-space prompts in chunks of 128 tokens (csrc/linear_attn_tc.cu) against a token-by-token walk in 64 bits, and against the form in chunks of 64 that the same
call takes where the gate is one element off a 16-byte boundary. Either is within about 2^-22 of the result's 2-norm of 64-bit arithmetic (measured 1.4e-7 for outputs, 3.5e-7
for states): 8 * 2^-24 between them, 16 * 2^-24 from the walk (whose convolution and steps are in 64 bits too)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
BOUND = 8 * 2.0 ** -24


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def _inputs(lengths, H, G, dim, vdim, seed, dt_scale=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    R = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    T, n, inner = sum(lengths), len(lengths), H * vdim
    C = inner + 2 * G * dim
    x = dict(x=R(T, inner), b=R(T, G * dim), c=R(T, G * dim), dt=R(T, H) * dt_scale, gate=R(T, inner))
    w = dict(conv_w=R(C, 3) * 0.5, conv_b=R(C), dt_bias=R(H) - 1, a_log=R(H) * 0.3, skip=R(H), norm=torch.ones(inner, device=DEV), heads=H, groups=G, dim=dim, vdim=vdim, taps=3,
             norm_groups=H, norm_eps=1e-6, out_dtype=torch.float32)
    return x, w, R(n, 3, C), R(n, H, dim, vdim)


def _run(lengths, pos0, x, w, conv, state, off):
    from vyomai_b200 import ops
    cu = [0]
    for n in lengths:
        cu.append(cu[-1] + n)
    x = dict(x)
    if off:
        buf = torch.zeros(cu[-1], x["gate"].shape[1] + 4, device=DEV)
        buf[:, 1:-3] = x["gate"]
        x["gate"] = buf[:, 1:-3]
    conv, state = conv.clone(), state.clone()
    out = ops.ssd(ops.PackedBatch(_i32(cu), _i32(pos0), _i32(list(range(len(lengths)))), max(lengths)), **x, **w, conv_state=conv, state=state,
                  tickets=torch.zeros(len(lengths), 1, dtype=torch.int32, device=DEV))
    return out, state


def _walk(lengths, pos0, x, w, conv, state):
    """Token by token in 64 bits: (outputs, states)."""
    H, G, dim, vdim, taps = (w[k] for k in ("heads", "groups", "dim", "vdim", "taps"))
    f, outs, states, at = (lambda t: t.double()), [], [], 0
    rate, cw = torch.exp(f(w["a_log"])), f(w["conv_w"])
    for s, (n, p0) in enumerate(zip(lengths, pos0)):
        raw = torch.cat([f(x[k][at:at + n]) for k in ("x", "b", "c")], 1)
        before = torch.stack([f(conv[s, (p0 - lag) % taps]) if p0 - lag >= 0 else torch.zeros_like(raw[0]) for lag in range(taps - 1, 0, -1)])
        seq = torch.cat([before, raw])
        z = f(w["conv_b"]) + sum(seq[t:t + n] * cw[:, t] for t in range(taps))
        z = z * torch.sigmoid(z)
        xs, b, c = z[:, :H * vdim].view(n, H, vdim), *(z[:, H * vdim + i * G * dim:][:, :G * dim].view(n, G, dim).repeat_interleave(H // G, 1) for i in (0, 1))
        step = torch.nn.functional.softplus(f(x["dt"][at:at + n]) + f(w["dt_bias"]), threshold=1e9)
        S, o = f(state[s]).clone() if p0 else torch.zeros_like(f(state[s])), torch.empty(n, H, vdim, device=DEV, dtype=torch.float64)
        decay = torch.exp(-rate * step)
        for t in range(n):
            S = decay[t, :, None, None] * S + (step[t, :, None] * b[t])[:, :, None] * xs[t][:, None, :]
            o[t] = torch.einsum("hkv,hk->hv", S, c[t])
        g = f(x["gate"][at:at + n])
        y = (o + f(w["skip"])[:, None] * xs).reshape(n, -1) * g * torch.sigmoid(g)
        y = y.view(n, w["norm_groups"], -1)
        outs.append((y / torch.sqrt(y.square().mean(-1, keepdim=True) + w["norm_eps"])).reshape(n, -1) * f(w["norm"]))
        states.append(S)
        at += n
    return torch.cat(outs), torch.stack(states)


def _close(a, b, bound=BOUND):
    assert a.shape == b.shape and float((a.double() - b.double()).norm()) <= bound * float(b.double().norm())


def _forms(call):
    """(the call's result, which forms' kernels it launched)"""
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        out = call()
        torch.cuda.synchronize()
    names = " ".join(e.key for e in prof.key_averages())
    return out, [n for n in ("la_outputs_tc_kernel", "la_outputs_kernel") if n in names]


@pytest.mark.parametrize("H,G,dim,vdim", [(8, 1, 128, 64), (6, 2, 96, 40), (5, 5, 16, 64), (14, 2, 64, 132), (4, 1, 128, 32), (22, 2, 20, 68)])
@pytest.mark.parametrize("lengths,pos0", [([129], [0]), ([1, 127, 128, 129, 300], [7, 0, 3, 0, 1]), ([256, 5, 640], [0, 2, 9])])
def test_chunks_of_128_tokens(H, G, dim, vdim, lengths, pos0):
    from vyomai_b200._lib import lib
    assert lib().vy_linear_attn_workspace_floats(sum(lengths), len(lengths), max(lengths), H, dim, vdim) > 0   # 0: the walk alone, in either call
    args = _inputs(lengths, H, G, dim, vdim, H + dim)
    (a, ka), (b, kb) = (_forms(lambda: _run(lengths, pos0, *args, off)) for off in (False, True))
    assert ka == ["la_outputs_tc_kernel"] and kb == ["la_outputs_kernel"]
    want = _walk(lengths, pos0, *args)
    for got, other, exact in zip(a, b, want):
        _close(got, other)
        _close(got, exact, 2 * BOUND)


@pytest.mark.parametrize("what", ["steep decays", "flat decays", "wide rows", "infinite value", "infinite gates"])
def test_chunks_of_128_tokens_at_the_ends_of_their_range(what):
    """Decays that vanish within a chunk or never start; rows too far apart for fp16 halves and infinities, which leave their heads to the walk in either form."""
    lengths, pos0 = [400, 260], [0, 4]
    x, w, conv, state = _inputs(lengths, 8, 2, 64, 64, 3, dt_scale=30.0 if what == "steep decays" else 1.0)
    if what == "flat decays":
        w["dt_bias"] = torch.full_like(w["dt_bias"], -40.0)
    if what == "wide rows":
        x["x"][130:140] *= 1e9
        x["c"][50] *= 1e-12
    if what == "infinite value":
        x["x"][300, 70] = float("inf")
    if what == "infinite gates":
        x["gate"][5, 3], x["gate"][200, 65], x["gate"][7, 9], x["gate"][8, 9], x["gate"][9, 9] = float("inf"), float("-inf"), float("nan"), 200.0, -200.0
    a, b = (_run(lengths, pos0, x, w, conv, state, off) for off in (False, True))
    if what.endswith("decays"):
        for got, exact in zip(a, _walk(lengths, pos0, x, w, conv, state)):
            _close(got, exact, 2 * BOUND)
    for p, q in zip(a, b):
        assert torch.equal(p.isfinite(), q.isfinite())
        _close(p.nan_to_num(0, 0, 0), q.nan_to_num(0, 0, 0))


def test_gates_far_below_zero_and_where_their_exponential_leaves_fp32():
    """A read-out times silu(gate), entry by entry, against the same read-out times silu(1): gates around -88 (e^88 is past the approximate reciprocal), large negative ones, which give zero."""
    lengths, pos0 = [256, 130], [0, 0]
    x, w, conv, state = _inputs(lengths, 4, 1, 32, 64, 5)
    w["norm_eps"] = 1e12   # the norm behind the gate: a division by 1e6 (the rows' own squares are 1e-8 of it)
    gate = torch.cat([torch.linspace(-89.0, -87.0, 128), torch.tensor([-1e30, -3e38, -1e3, -100.0]), torch.linspace(-30.0, 80.0, 124)]).to(DEV)
    x["gate"] = gate.expand(386, -1).contiguous()
    got = _run(lengths, pos0, x, w, conv, state, False)[0].double() * 1e6
    x["gate"] = torch.ones_like(x["gate"])
    y = _run(lengths, pos0, x, w, conv, state, False)[0].double() * 1e6 / torch.sigmoid(torch.tensor(1.0, dtype=torch.float64))
    want, g = y * gate.double() * torch.sigmoid(gate.double()), gate.double().abs().clamp(max=200.0)
    assert bool(((got - want).abs() <= 2.0 ** -20 * want.abs() + y.abs() * g * 2.0 ** -128 + 1e6 * 2.0 ** -148).all())

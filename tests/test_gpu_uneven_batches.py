"""-m gpu: which form of the prompt kernels a step takes where one portion is long and the others are single tokens (the grids have the longest portion's CTAs for every sequence),
by the kernels that run, and that a sequence's results are the same to fp32 rounding as by itself: 16 * 2^-24 of the 2-norm, as for the forms themselves."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
BOUND = 16 * 2.0 ** -24


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def _batch(new, pos0):
    from vyomai_b200 import ops
    cu, table, at, width = [0], [], 0, max((a + b + 15) // 16 for a, b in zip(new, pos0))
    for n, p in zip(new, pos0):
        pages = (n + p + 15) // 16
        table.append(list(range(at, at + pages)) + [0] * (width - pages))
        at += pages
        cu.append(cu[-1] + n)
    return ops.PackedBatch(_i32(cu), _i32(pos0), _i32(list(range(len(new)))), max(new), _i32(table), 16), at


def _kernels(call):
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        out = call()
        torch.cuda.synchronize()
    return out, " ".join(e.key for e in prof.key_averages())


def _close(a, b):
    assert a.shape == b.shape and float((a.double() - b.double()).norm()) <= BOUND * float(b.double().norm())


@pytest.mark.parametrize("H,G,d,dv,window,tokens,alone,beside", [(16, 16, 96, 64, 64, 512, "tc", "mma"), (8, 2, 128, 128, 512, 2048, "tc", "tc"), (32, 8, 64, 64, 64, 512, "tc", "mma")])
def test_prompt_attention_beside_single_tokens(H, G, d, dv, window, tokens, alone, beside):
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(d)
    new, pos0 = [tokens] + [1] * 31, [0] + [700] * 31
    batch, pages = _batch(new, pos0)
    R = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    q, kp, vp = R(sum(new), H * d), R(pages, 16, G, d), R(pages, 16, G, dv)
    call = lambda b, q: ops.window_attn(b, q, kp, vp, heads=H, kv_heads=G, dim=d, vdim=dv, scale=d ** -0.5, window=window, keep_first=0, out_dtype=torch.float32)  # noqa: E731
    both, names = _kernels(lambda: call(batch, q))
    assert f"window_attn_{beside}_kernel" in names
    one, _ = _batch(new[:1], pos0[:1])
    first, names = _kernels(lambda: call(one, q[:tokens]))
    assert f"window_attn_{alone}_kernel" in names
    _close(both[:tokens], first)
    for s in (1, 31):   # a token by itself has its pages elsewhere in the table
        b1 = ops.PackedBatch(_i32([0, 1]), _i32([700]), _i32([0]), 1, batch.block_table[s:s + 1].contiguous(), 16)
        _close(both[tokens + s - 1:tokens + s], call(b1, q[tokens + s - 1:tokens + s]))


@pytest.mark.parametrize("new,channels,conv,heads,rope", [([300] + [20] * 7, 1024, "causal_conv_kernel", 32, "rope_heads_kernel"), ([512] + [1] * 31, 4096, "causal_conv_quads_kernel", 8, "rope_heads_rows_kernel"),
                                                          ([700, 600], 2048, "causal_conv_quads_kernel", 8, "rope_heads_rows_kernel"), ([700, 400], 1024, "causal_conv_kernel", 8, "rope_heads_kernel")])
def test_row_kernels_choose_by_the_tokens_that_are_there(new, channels, conv, heads, rope):
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(channels)
    batch, pages = _batch(new, [3] * len(new))
    R = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    T, n = sum(new), len(new)
    x, w, st = R(T, channels), R(channels, 4), R(n, channels, 3)
    (y, state), names = _kernels(lambda: (lambda s: (ops.causal_conv(batch, x, w, s), s))(st.clone()))
    assert conv in names
    one, _ = _batch(new[:1], [3])
    s1 = st[:1].clone()
    _close(y[:new[0]], ops.causal_conv(one, x[:new[0]], w, s1))
    assert torch.equal(state[:1], s1)
    d, G = 64, 4
    q, k, v, kp, vp, fr = R(T, heads * d), R(T, G * d), R(T, G * d), torch.zeros(pages, 16, G, d, device=DEV), torch.zeros(pages, 16, G, d, device=DEV), torch.rand(d // 2, device=DEV)
    turn = lambda b, q, k, v, kp, vp: ops.rope_kv_write(b, q, k, v, fr, kp, vp, heads=heads, kv_heads=G, dim=d, vdim=d, rot_dims=d, layout="half", unit_rms=True, eps=1e-6)  # noqa: E731
    q1, kp1, vp1, m = q[:new[0]].clone(), kp.clone(), vp.clone(), new[0]
    _, names = _kernels(lambda: turn(batch, q, k, v, kp, vp))
    assert rope in names
    turn(one, q1, k[:m].contiguous(), v[:m].contiguous(), kp1, vp1)
    rows = (m + 3 + 15) // 16
    _close(q[:m], q1)
    _close(kp[:rows], kp1[:rows])
    assert torch.equal(vp[:rows], vp1[:rows])


@pytest.mark.parametrize("H,G,beside", [(16, 16, "la_outputs_kernel"), (8, 1, "la_outputs_tc_kernel")])
def test_state_space_beside_single_tokens(H, G, beside):
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(H)
    new, pos0, dim, vdim = [512] + [1] * 31, [0] + [7] * 31, 64, 64
    T, n, C, inner = sum(new), len(new), H * vdim + 2 * G * dim, H * vdim
    R = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    x = dict(x=R(T, inner), b=R(T, G * dim), c=R(T, G * dim), dt=R(T, H), gate=R(T, inner))
    w = dict(conv_w=R(C, 4) * 0.5, conv_b=R(C), dt_bias=R(H) - 1, a_log=R(H) * 0.3, skip=R(H), norm=torch.ones(inner, device=DEV), heads=H, groups=G, dim=dim, vdim=vdim, taps=4, norm_groups=1,
             norm_eps=1e-6, out_dtype=torch.float32)
    conv, state = R(n, 4, C), R(n, H, dim, vdim)

    def run(lo, hi, a, b):
        cu = [0]
        for m in new[lo:hi]:
            cu.append(cu[-1] + m)
        cs, ss = conv[lo:hi].clone(), state[lo:hi].clone()
        out = ops.ssd(ops.PackedBatch(_i32(cu), _i32(pos0[lo:hi]), _i32(list(range(hi - lo))), max(new[lo:hi])), **{k: t[a:b] for k, t in x.items()}, **w, conv_state=cs, state=ss,
                      tickets=torch.zeros(hi - lo, 1, dtype=torch.int32, device=DEV))
        return out, ss

    (out, states), names = _kernels(lambda: run(0, n, 0, T))
    assert beside in names
    first, s0 = run(0, 1, 0, 512)
    _close(out[:512], first)
    _close(states[:1], s0)
    last, s1 = run(n - 1, n, T - 1, T)
    _close(out[-1:], last)
    _close(states[-1:], s1)

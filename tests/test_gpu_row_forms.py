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


@pytest.mark.parametrize("taps", [1, 2, 4])
@pytest.mark.parametrize("act", ["silu", "sigmoid", None])
def test_convolution_of_four_channels_per_thread(taps, act):
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(taps)
    C, pos0 = 8196, [0, 3, 0, 40, 2]   # enough channels for a CTA per SM
    batch = ops.PackedBatch(torch.tensor([0, 1, 16, 32, 49, 119], dtype=torch.int32, device=DEV), torch.tensor(pos0, dtype=torch.int32, device=DEV),
                            torch.tensor([4, 1, 0, 5, 2], dtype=torch.int32, device=DEV), 70)
    x, w, state = torch.randn(119, C, generator=g, device=DEV) * 3, torch.randn(C, taps, generator=g, device=DEV), torch.randn(6, C, max(taps - 1, 1), generator=g, device=DEV)
    x[5, 7], x[6, 9], x[7, 11], w[11] = 200.0, -200.0, -1e30, w[11].abs()   # the exponentials there overflow or vanish
    if taps == 1:
        state = state[:, :, :0].contiguous()
    states = [state.clone(), state.clone()]
    a, b = (ops.causal_conv(batch, t, w, s, act=act) for t, s in zip((x, _off(x)), states))
    _close(a, b)
    assert torch.equal(*states)


@pytest.mark.parametrize("layout,rot,dim", [("half", 64, 128), ("half", 24, 48), ("pairs", 6, 20), ("pairs", 128, 128), ("pairs", 0, 128), ("half", 128, 128)])
@pytest.mark.parametrize("norm,pool", [("weight", torch.float32), ("unit", torch.float32), (None, torch.bfloat16), ("unit", None)])
def test_rotation_of_four_entries_per_lane(layout, rot, dim, norm, pool):
    from vyomai_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(dim + rot)
    H, G, dv, new, pos0 = 5, 2, 36, [17, 1, 240], [0, 300, 7]
    batch, _, _, blocks, _ = shuffled_batch(new, pos0, 16, DEV, seed=rot)
    q, k, v = (torch.randn(258, n, generator=g, device=DEV) for n in (H * dim, G * dim, G * dv))
    freq = 100.0 ** -(torch.arange(max(rot // 2, 1), device=DEV) / max(rot // 2, 1))
    nw = torch.randn(dim, generator=g, device=DEV) if norm == "weight" else None

    def run(q, k, v):
        kp, vp = (None, None) if pool is None else (torch.zeros(blocks, 16, G, dim, device=DEV, dtype=pool), torch.zeros(blocks, 16, G, dv, device=DEV, dtype=pool))
        ko = k if pool is None else None
        ops.rope_kv_write(batch, q, k, v, freq, kp, vp, heads=H, kv_heads=G, dim=dim, vdim=dv, rot_dims=rot, layout=layout, rot_scale=1.5, unit_rms=norm == "unit", eps=1e-6,
                          q_scale=0.7, k_scale=1.3, k_out=ko, q_norm=nw, k_norm=nw, q_temp=(0.3, 9) if norm else None)
        return q, (ko if pool is None else kp.float()), (v if pool is None else vp.float())

    a, b = run(q.clone(), k.clone(), v), run(_off(q), _off(k), _off(v))
    _close(a[0], b[0])
    if pool == torch.bfloat16:   # one rounding of a key may go the other way
        assert float((a[1] - b[1]).abs().max()) <= 2.0 ** -7 * float(b[1].abs().max())
    else:
        _close(a[1], b[1])
    assert torch.equal(a[2], b[2])

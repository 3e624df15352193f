"""The one-tile and the two-tile CTA of the attention kernel, and the row kernels' groups of four, at the
sizes where they change hands."""
import numpy as np
import pytest

from tests._util import assert_parity, dev_bf16, host_bits, host_f32, normal_bits

pytestmark = pytest.mark.gpu


def _forward(q, k, v):
    import torch

    import f2k_cuda_b200 as f2k
    B, S, H, D = q.shape
    att = f2k.Attention(f2k.Attention.Config(B, S, H, D))
    o = torch.full_like(q, float("nan"))
    assert att.forward(q, k, v, o), att.last_error()
    assert att.device_status() == 0, att.last_error()
    return o


# Tiles per head 1, 2, 3, 4, 9: alone with few heads (every pair is split into one-tile CTAs), and as
# part of 160 heads (148 SMs: most pairs stay whole). Key tiles 1, 2, 3, ... make the first and the last
# use of every barrier.
@pytest.mark.parametrize("S", [1, 128, 129, 256, 300, 400, 1100])
def test_rows_do_not_depend_on_the_plan(S):
    import torch
    H = 160
    q, k, v = [dev_bf16(normal_bits(0x51A6 + i, S, (1, S, H, 128))) for i in range(3)]
    whole = _forward(q, k, v)
    few = [0, 77, 159]
    part = _forward(*[x[:, :, few].contiguous() for x in (q, k, v)])
    assert torch.equal(whole[:, :, few], part)          # the same arithmetic in both kinds of CTA
    for n, h in enumerate(few):
        s = (q[0, :, h].float() @ k[0, :, h].float().T) * 128 ** -0.5
        assert_parity(host_f32(part[0, :, n]), (torch.softmax(s, -1) @ v[0, :, h].float()).cpu().numpy(), f"head {h}")


# The lazy reference maximum moves (and O is rescaled in tensor memory) when a tile's maximum exceeds it by 8 in
# log2 units, 5.5 nats: score levels per key tile that rise by 8 nats and more from tile to tile in every second
# head, and lie anywhere from 0 to 40 in the others. Values within 4.7 (400 thousand N(0, 1)): 2^-9 of that for the rounding of P
# and as much for the output's stay below the gate.
@pytest.mark.parametrize("S", [256, 300, 400, 1100])
def test_moving_maximum_in_both_kinds_of_cta(S):
    import torch
    H, tiles = 160, -(-S // 128)
    q, k, v = [dev_bf16(normal_bits(0x3A71 + i, S, (1, S, H, 128))) for i in range(3)]
    level = np.random.default_rng(S).uniform(0, 40, (H, tiles))
    level[1::2] = 12 * np.arange(tiles) + level[1::2] / 10
    q[..., 0] = 128 ** 0.5
    k[..., 0] = torch.from_numpy(level.T.repeat(128, axis=0)[:S].astype(np.float32)).cuda()
    whole = _forward(q, k, v)
    few = [0, 77, 159]
    part = _forward(*[x[:, :, few].contiguous() for x in (q, k, v)])
    assert torch.equal(whole[:, :, few], part)
    for n, h in enumerate(few):
        s = (q[0, :, h].double() @ k[0, :, h].double().T) * 128 ** -0.5
        assert_parity(host_f32(part[0, :, n]), (torch.softmax(s, -1) @ v[0, :, h].double()).cpu().numpy(), f"head {h}")


@pytest.mark.parametrize("rows", [1, 2, 3, 4, 5, 63, 64, 65, 148 * 8 * 64 + 3]
                         + [148 * 8 * 16 + n for n in (0, 1, 2, 3, 4)])       # one row at a time up to here, then four
def test_row_kernels_at_the_edges_of_their_groups(rows):
    """Every row alone gives the same bits as the row inside a call (a half-warp takes one or four at a time), and
    nothing behind the last row is written."""
    import torch

    import f2k_cuda_b200 as f2k
    seq = 37
    x = dev_bf16(normal_bits(0x2B, rows, (rows, 128)))
    g = dev_bf16(normal_bits(0x2C, 0, (128,)))
    cos, sin = [torch.from_numpy(t).cuda() for t in
                f2k.build_rope_4axis_tables((32,) * 4, np.arange(seq * 4).reshape(seq, 4) % 11, 2000.0)]
    pos = torch.from_numpy(((np.arange(rows) * 7) // 3 % (seq + 2) - 1).astype(np.int32)).cuda()   # some out of range
    y = torch.full((rows + 4, 128), 3.0, dtype=torch.bfloat16, device="cuda")
    assert f2k.rmsnorm_bf16(x, g, y, rows, 128, 1e-6)
    normed = y.clone()
    assert f2k.rope_4axis_inplace_bf16(y, cos, sin, pos, rows, 128, seq)
    torch.cuda.synchronize()
    assert torch.all(y[rows:] == 3.0) and torch.all(normed[rows:] == 3.0)
    xf = x.double()
    ref = xf * torch.rsqrt((xf * xf).mean(-1, keepdim=True) + 1e-6) * g.double()
    # one bf16 rounding of a value computed in fp32: half a unit in the last place, 2^-8 relative
    assert torch.all((normed[:rows].double() - ref).abs() <= ref.abs() * 2.0 ** -8 * 1.01)
    for r in sorted({0, rows // 2, rows - 1}):
        one = torch.empty(1, 128, dtype=torch.bfloat16, device="cuda")
        assert f2k.rmsnorm_bf16(x[r:r + 1].clone(), g, one, 1, 128, 1e-6)
        assert torch.equal(one[0], normed[r])
        assert f2k.rope_4axis_inplace_bf16(one, cos, sin, pos[r:r + 1].clone(), 1, 128, seq)
        assert np.array_equal(host_bits(one[0]), host_bits(y[r]))

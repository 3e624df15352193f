"""Performance cases of the joint-attention engine: what is timed, on which inputs, and how close
two correct implementations have to agree.

A case names an entry point ("path") and its sizes. Paths:

  joint    JointAttention.forward_fused        a double-stream block: text and image streams
  single   Attention.forward_fused_single      a single-stream block: Q, K, V are columns of the fused
                                               projection output, O goes into the [attn | mlp] buffer
  plain    Attention.forward                   inputs already normalised and rotated
  step     StepAttention, as a CUDA graph      every attention call of one denoise step (8 joint, 24 single)
  host     JointAttention.forward_fused_host   pinned host buffers in and out
  rows     rmsnorm_bf16, rope_4axis_inplace_bf16   the stand-alone row kernels on one Q or K tensor

The image tokens are `images` grids of `rows` x `cols`. All heads are 128 wide, all tensors bf16.
"""
import numpy as np
import torch

import f2k_cuda_b200 as f2k
from f2k_cuda_b200.inputs import AXES_DIM, RMS_EPS, ROPE_THETA
from f2k_cuda_b200.step import DoubleCall, SingleCall, StepAttention

D = 128
N_DOUBLE, N_SINGLE = 8, 24      # attention calls of one model forward


def _case(name, path, txt, rows, cols, heads=32, batch=1, images=1):
    c = {"path": path, "batch": batch, "txt": txt, "images": images, "rows": rows, "cols": cols, "heads": heads}
    return {"name": name, **c} if name else c


def listed():
    return [
        # The smallest call: a thumbnail latent with a short prompt on four heads (one GPU's share of
        # 32 heads over eight). Launches and latency are all there is.
        _case("joint_192_h4", "joint", 64, 8, 16, heads=4),
        # Ordinary small generation: 512 x 512 pixels, 128 text tokens.
        _case("joint_1152", "joint", 128, 32, 32),
        # Two prompts at once (guidance in one batch), an odd crop and an unpadded prompt: every tile
        # at a stream's end is ragged, and the head count is not a multiple of eight.
        _case("joint_ragged_b2_h12", "joint", 77, 37, 53, heads=12, batch=2),
        # The headline: 1024 x 1024 pixels, 512 text tokens.
        _case("joint_4608", "joint", 512, 64, 64),
        # Four of them in one batch.
        _case("joint_4608_b4", "joint", 512, 64, 64, batch=4),
        # The largest: 2048 x 2048 pixels.
        _case("joint_16896", "joint", 512, 128, 128),
        # The same picture with its heads spread over eight GPUs: one GPU's share. Few heads, long rows.
        _case("joint_16896_h4", "joint", 512, 128, 128, heads=4),
        # A single-stream block at the headline size, reading the projection output in place.
        _case("single_4608", "single", 512, 64, 64),
        # Attention alone on a combined stream whose length is no multiple of anything.
        _case("plain_2125", "plain", 77, 32, 64),
        # All 32 attention calls of one denoise step at the small generation size, replayed as a graph.
        _case("step_1152", "step", 128, 32, 32),
        # Host buffers in and out at the headline size: bound by the bus.
        _case("host_4608", "host", 512, 64, 64),
        # The stand-alone row kernels on one tensor of the headline size, for callers that keep the
        # separate calls.
        _case("rows_4608", "rows", 512, 64, 64),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    """Another case of the same ranges: 40 to 16896 tokens of odd and even sizes, 1 to 32 heads, 1 to 4
    batch elements, never costlier than the largest listed case of its path."""
    path = rng.choice(["joint", "joint", "joint", "joint", "single", "single", "plain", "plain", "step", "host", "rows"])
    top = {"step": 1200, "host": 4608, "single": 8704}.get(path, 16384)
    while True:
        img = _log_int(rng, 128, top)
        rows = max(4, int(round(img ** 0.5 * rng.uniform(0.6, 1.6))))
        cols = max(4, img // rows)
        txt = _log_int(rng, 32, 512)
        images = 2 if img >= 512 and rng.random() < 0.15 else 1
        heads = rng.choice([4, 8, 16, 24, 32, 32, 32]) if rng.random() < 0.85 else rng.randint(1, 32)
        batch = rng.choice([1, 1, 1, 2, 4]) if path not in ("step", "host") else 1
        c = _case(None, path, txt, rows, cols, heads, batch, images)
        seq = _seq(c)
        limit = {"step": 1152.0, "host": 4608.0}.get(path, 16896.0)
        if batch * heads * seq ** 2 <= 32 * limit ** 2 and batch * heads * seq <= 32 * 18432 and seq <= 16896:
            return c


def _img(c):
    return c["images"] * c["rows"] * c["cols"]


def _seq(c):
    return c["txt"] + _img(c)


def _positions(c):
    """Token positions (t, h, w, l) of the text and of the image stream."""
    txt = np.zeros((c["txt"], 4), np.int32)
    txt[:, 3] = np.arange(c["txt"])
    i, r, w = np.meshgrid(np.arange(c["images"]), np.arange(c["rows"]), np.arange(c["cols"]), indexing="ij")
    img = np.zeros((_img(c), 4), np.int32)
    img[:, 0], img[:, 1], img[:, 2] = i.ravel(), r.ravel(), w.ravel()
    return txt, img


def _tables(positions):
    return tuple(torch.from_numpy(t).cuda() for t in f2k.build_rope_4axis_tables(AXES_DIM, positions, ROPE_THETA))


class _Inputs:
    """Seeded device tensors: projections N(0, 1), gains 1 + U(-0.1, 0.1)."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(int(seed))

    def normal(self, *shape):
        return torch.randn(*shape, device="cuda", dtype=torch.bfloat16, generator=self.gen)

    def gain(self):
        return (0.9 + 0.2 * torch.rand(D, device="cuda", generator=self.gen)).to(torch.bfloat16)


def prepare(case, seed):
    c, inp = case, _Inputs(seed)
    B, H, St, Si, S = c["batch"], c["heads"], c["txt"], _img(c), _seq(c)
    pos_t, pos_i = _positions(c)
    s = {"path": c["path"]}

    if c["path"] in ("joint", "host"):
        s["module"] = m = f2k.JointAttention(f2k.JointAttention.Config(B, St, Si, H, D))
        s["args"] = [inp.normal(B, n, H, D) for n in (St, St, St, Si, Si, Si)]
        s["gains"] = tuple(inp.gain() for _ in range(4))
        s["tables"] = (*_tables(pos_t), *_tables(pos_i))
        s["out"] = [torch.empty_like(s["args"][0]), torch.empty_like(s["args"][3])]
        if c["path"] == "joint":
            s["workspace"] = torch.empty(m.fused_workspace_size_bytes(), dtype=torch.uint8, device="cuda")
        else:
            s["args"] = [x.cpu().pin_memory() for x in s["args"]]
            s["out"] = [torch.empty(x.shape, dtype=x.dtype).pin_memory() for x in s["out"]]
    elif c["path"] == "single":
        # One token's row of the projection output: Q, K, V (H * 128 each), then the MLP's 6 * H * 128.
        hd = H * D
        wide = torch.zeros(B, S, 9 * hd, device="cuda", dtype=torch.bfloat16)
        wide[:, :, :3 * hd] = inp.normal(B, S, 3 * hd)
        s["module"] = m = f2k.Attention(f2k.Attention.Config(B, S, H, D))
        s["args"] = [wide[:, :, i * hd:(i + 1) * hd].view(B, S, H, D) for i in range(3)]
        s["gains"] = (inp.gain(), inp.gain())
        s["tables"] = _tables(np.concatenate([pos_t, pos_i]))
        s["out"] = torch.zeros(B, S, 4 * hd, device="cuda", dtype=torch.bfloat16)[:, :, :hd].view(B, S, H, D)
        s["workspace"] = torch.empty(m.fused_workspace_size_bytes(), dtype=torch.uint8, device="cuda")
    elif c["path"] == "plain":
        s["module"] = f2k.Attention(f2k.Attention.Config(B, S, H, D))
        s["args"] = [inp.normal(B, S, H, D) for _ in range(3)]
        s["out"] = torch.empty_like(s["args"][0])
    elif c["path"] == "step":
        doubles = [DoubleCall(*[inp.normal(B, n, H, D) for n in (St, St, St, Si, Si, Si)],
                              *[torch.empty(B, n, H, D, device="cuda", dtype=torch.bfloat16) for n in (St, Si)])
                   for _ in range(N_DOUBLE)]
        singles = [SingleCall(*[inp.normal(B, S, H, D) for _ in range(3)],
                              torch.empty(B, S, H, D, device="cuda", dtype=torch.bfloat16)) for _ in range(N_SINGLE)]
        gains = tuple(inp.gain() for _ in range(4))
        tables = (*_tables(pos_t), *_tables(pos_i))
        combined = _tables(np.concatenate([pos_t, pos_i]))
        s["step"] = StepAttention(B, St, Si, H, D)
        s["graph"], _ = s["step"].capture([(doubles, singles)], gains, tables, combined, RMS_EPS)
        s["keep"] = (doubles, singles, gains, tables, combined)
        s["out"] = [o for call in doubles for o in (call.o_txt, call.o_img)] + [call.o for call in singles]
    else:
        s["x"], s["gain"] = inp.normal(B, S, H, D), inp.gain()
        s["cos"], s["sin"] = _tables(np.concatenate([pos_t, pos_i]))
        s["out"] = torch.empty_like(s["x"])
        n_rows = B * S * H
        s["pos"] = ((torch.arange(n_rows, device="cuda") // H) % S).to(torch.int32)
        s["n_rows"], s["seq"] = n_rows, S
    return s


def run(s):
    path = s["path"]
    if path == "joint":
        ok = s["module"].forward_fused(*s["args"], s["gains"], s["tables"], RMS_EPS, *s["out"], s["workspace"])
    elif path == "single":
        ok = s["module"].forward_fused_single(*s["args"], *s["gains"], *s["tables"], RMS_EPS, s["out"], s["workspace"],
                                              strided=True)
    elif path == "plain":
        ok = s["module"].forward(*s["args"], s["out"])
    elif path == "step":
        s["graph"].replay()
        ok = True
    elif path == "host":
        ok = s["module"].forward_fused_host(*s["args"], s["gains"], s["tables"], RMS_EPS, *s["out"])
    else:
        ok = f2k.rmsnorm_bf16(s["x"], s["gain"], s["out"], s["n_rows"], D, RMS_EPS) and \
            f2k.rope_4axis_inplace_bf16(s["out"], s["cos"], s["sin"], s["pos"], s["n_rows"], D, s["seq"])
    if not ok:
        raise RuntimeError(s["module"].last_error() if "module" in s else "the call was refused")
    return s["out"]


def work(case):
    """Each input read once and each output written once; two products of S x S x 128 per head."""
    c = case
    B, H, S = c["batch"], c["heads"], _seq(c)
    tensor = B * S * H * D * 2
    tables = 2 * S * (D // 2) * 4
    if c["path"] == "rows":
        return {"bytes": 2 * tensor + tables + 4 * B * S * H, "flops": 8 * B * S * H * D}
    calls = N_DOUBLE + N_SINGLE if c["path"] == "step" else 1
    return {"bytes": calls * 4 * tensor + (0 if c["path"] == "plain" else tables), "flops": calls * 4 * B * H * S * S * D}


def tolerance(case):
    """Relative 2-norm error and the largest single one. Against a 64-bit computation of the same inputs the
    attention paths show 0.0023 to 0.0034 and 0.012 to 0.026 (Q and K rounded to bf16 after the norm and the
    rotation, P and O rounded to bf16), the row kernels 0.0020 and 0.013 (two roundings)."""
    return {"rel": 8e-3, "max": 5e-2} if case["path"] == "rows" else {"rel": 1.2e-2, "max": 8e-2}


def _turned(x, gain, cos, sin):
    """RMSNorm over each head row times the gain, then the rotation of interleaved pairs, in 64 bits."""
    x = x.cuda().double()
    x = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + RMS_EPS) * gain.double()
    even, odd = x[..., 0::2], x[..., 1::2]
    c, s = cos.double()[:, None, :], sin.double()[:, None, :]
    return torch.stack([even * c - odd * s, even * s + odd * c], dim=-1).flatten(-2)


def _attended(q, k, v):
    """softmax(Q K^T / sqrt(128)) V of [batch, tokens, heads, 128], in 64 bits, a block of rows of one head at a time."""
    out = torch.empty_like(q)
    for b in range(q.shape[0]):
        for h in range(q.shape[2]):
            keys, values = k[b, :, h].T.contiguous(), v[b, :, h].cuda().double()
            for r in range(0, q.shape[1], 4096):
                scores = (q[b, r:r + 4096, h] @ keys).mul_(D ** -0.5)
                out[b, r:r + 4096, h] = torch.softmax(scores, -1) @ values
    return out


def exact(case, seed):
    """The outputs of run() for these inputs in 64 bits, without the bf16 roundings between the steps."""
    s = prepare(case, seed)
    St = case["txt"]

    def joint(a, gains, tables):
        q = torch.cat([_turned(a[0], gains[0], *tables[:2]), _turned(a[3], gains[2], *tables[2:])], 1)
        k = torch.cat([_turned(a[1], gains[1], *tables[:2]), _turned(a[4], gains[3], *tables[2:])], 1)
        o = _attended(q, k, torch.cat([a[2], a[5]], 1))
        return [o[:, :St], o[:, St:]]

    if case["path"] in ("joint", "host"):
        return joint(s["args"], s["gains"], s["tables"])
    if case["path"] == "single":
        q, k, v = s["args"]
        return _attended(_turned(q, s["gains"][0], *s["tables"]), _turned(k, s["gains"][1], *s["tables"]), v)
    if case["path"] == "plain":
        q, k, v = s["args"]
        return _attended(q.double(), k.double(), v)
    if case["path"] == "step":
        doubles, singles, gains, tables, combined = s["keep"]
        outs = []
        for c in doubles:
            outs += joint((c.q_txt, c.k_txt, c.v_txt, c.q_img, c.k_img, c.v_img), gains, tables)
        for c in singles:
            outs.append(_attended(_turned(c.q, gains[2], *combined), _turned(c.k, gains[3], *combined), c.v))
        return outs
    return _turned(s["x"], s["gain"], s["cos"], s["sin"])

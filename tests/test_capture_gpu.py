"""Calls behind something other than a kernel of the same stream - a copy, a memset, a stream joined by an
event - eagerly and inside a captured graph, with work on a second stream behind them. The kernels are
launched so that they may overlap the kernel in front: that must neither break a capture nor let a call start
before what it depends on is there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TXT, IMG, H, D = 40, 130, 4, 128


def _state(seed):
    import torch

    import f2k_cuda_b200 as f2k
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen).to(torch.bfloat16)  # noqa: E731
    t = {f"{x}_{s}": rnd(1, n, H, D) for s, n in (("txt", TXT), ("img", IMG)) for x in "qkv"}
    t["gamma"] = (1 + 0.2 * rnd(D).float()).to(torch.bfloat16)
    for s, n in (("txt", TXT), ("img", IMG)):
        pos = np.arange(n * 4).reshape(n, 4) % 23
        t[f"cos_{s}"], t[f"sin_{s}"] = [torch.from_numpy(a).cuda() for a in
                                        f2k.build_rope_4axis_tables((32,) * 4, pos, 2000.0)]
    t["pos_ids"] = (torch.arange(IMG * H, device="cuda") // H).to(torch.int32)
    return t


def _call(kind, t):
    """(the call, its outputs, the handle) on the buffers of t."""
    import torch

    import f2k_cuda_b200 as f2k
    if kind == "joint":
        m = f2k.JointAttention(f2k.JointAttention.Config(1, TXT, IMG, H, D))
        ws = torch.empty(m.fused_workspace_size_bytes(), dtype=torch.uint8, device="cuda")
        out = [torch.empty_like(t["q_txt"]), torch.empty_like(t["q_img"])]
        return lambda: m.forward_fused(*[t[f"{x}_{s}"] for s in ("txt", "img") for x in "qkv"], [t["gamma"]] * 4,
                                       [t[n] for n in ("cos_txt", "sin_txt", "cos_img", "sin_img")], 1e-6, *out, ws), out, m
    out = [torch.empty_like(t["q_img"])]
    if kind == "plain":
        m = f2k.Attention(f2k.Attention.Config(1, IMG, H, D))
        return lambda: m.forward(t["q_img"], t["k_img"], t["v_img"], out[0]), out, m
    if kind == "rmsnorm":
        return lambda: f2k.rmsnorm_bf16(t["q_img"], t["gamma"], out[0], IMG * H, D, 1e-6), out, None
    return lambda: f2k.rope_4axis_inplace_bf16(t["q_img"], t["cos_img"], t["sin_img"], t["pos_ids"], IMG * H, D, IMG), \
        [t["q_img"]], None


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("before", ["copy", "memset", "joined"])
@pytest.mark.parametrize("kind", ["joint", "plain", "rmsnorm", "rope"])
def test_behind_copies_memsets_and_joined_streams(kind, before, captured):
    import torch
    sources = [_state(s) for s in (1, 2)]
    names = ["q_img"] if kind in ("rmsnorm", "rope") else ["q_img", "k_img", "v_img"]

    def expected(src):
        t = _state(0)
        for n in names:
            t[n].copy_(src[n])
        if before == "memset":
            t[names[-1]].zero_()
        go, out, _ = _call(kind, t)
        torch.cuda.synchronize()
        assert go()
        torch.cuda.synchronize()
        return [o.clone() for o in out]

    want = [expected(s) for s in sources]
    t = _state(0)
    src = {n: sources[0][n].clone() for n in names}
    go, out, module = _call(kind, t)
    seen = [torch.empty_like(o) for o in out]
    side = torch.cuda.Stream()

    def sequence():
        cur = torch.cuda.current_stream()
        if before == "joined":
            side.wait_stream(cur)
            with torch.cuda.stream(side):
                for n in names:
                    torch.mul(src[n], 1.0, out=t[n])
            cur.wait_stream(side)
        else:
            for n in names:
                t[n].copy_(src[n])
            if before == "memset":
                t[names[-1]].zero_()
        assert go()
        side.wait_stream(cur)                     # a reader on another stream behind the call
        with torch.cuda.stream(side):
            for a, b in zip(seen, out):
                a.copy_(b)
        cur.wait_stream(side)

    main = torch.cuda.Stream()
    main.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(main):
        if captured:
            sequence()                            # first use outside the capture
            main.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=main):
                sequence()
        for k in (0, 1, 0):
            for n in names:
                src[n].copy_(sources[k][n])
            for a in seen:
                a.fill_(float("nan"))
            graph.replay() if captured else sequence()
            main.synchronize()
            assert all(torch.equal(a, b) for a, b in zip(want[k], seen)), f"inputs {k}"
    assert module is None or module.device_status() == 0

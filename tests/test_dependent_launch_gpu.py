"""Calls right behind a kernel that lets its successor start early and writes one of the call's inputs late:
every input - rows, gains, tables, positions - must be read as that kernel leaves it."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = Path(__file__).resolve().parent
LATE_CLOCKS = 600_000       # some 0.3 ms: the call behind is enqueued, and its blocks are resident, long before


@pytest.fixture(scope="module")
def late_copy(tmp_path_factory):
    from f2k_cuda_b200.build import NVCC_FLAGS, _nvcc
    so = tmp_path_factory.mktemp("late") / "late_copy.so"
    subprocess.run([_nvcc(), *NVCC_FLAGS, "-shared", str(HERE / "cpp" / "late_copy.cu"), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    lib.late_copy.argtypes = [C.c_void_p, C.c_void_p, C.c_longlong, C.c_longlong, C.c_void_p]

    def copy(dst, src):
        import torch
        assert dst.is_contiguous() and src.is_contiguous() and dst.nbytes == src.nbytes
        assert lib.late_copy(dst.data_ptr(), src.data_ptr(), dst.nbytes, LATE_CLOCKS,
                             torch.cuda.current_stream().cuda_stream) == 0
    return copy


def _inputs(seed):
    """Inputs of every call below, by name, for 130 + 40 tokens x 4 heads. Another seed: other values throughout."""
    import torch

    import f2k_cuda_b200 as f2k
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen).to(torch.bfloat16)  # noqa: E731
    t = {}
    for stream, n in (("txt", 40), ("img", 130)):
        for x in "qkv":
            t[f"{x}_{stream}"] = rnd(1, n, 4, 128)
        for x in "qk":
            t[f"gamma_{x}_{stream}"] = (1 + 0.2 * rnd(128).float()).to(torch.bfloat16)
        pos = (np.arange(n * 4).reshape(n, 4) * (seed + 3)) % 29
        t[f"cos_{stream}"], t[f"sin_{stream}"] = [torch.from_numpy(a).cuda() for a in
                                                  f2k.build_rope_4axis_tables((32,) * 4, pos, 2000.0)]
    t["pos_ids"] = ((torch.arange(520, device="cuda") * (seed + 2)) % 130).to(torch.int32)
    return t


def _joint(f2k, t):
    import torch
    ja = f2k.JointAttention(f2k.JointAttention.Config(1, 40, 130, 4, 128))
    ws = torch.empty(ja.fused_workspace_size_bytes(), dtype=torch.uint8, device="cuda")
    out = [torch.empty_like(t["q_txt"]), torch.empty_like(t["q_img"])]
    return ja, ws, out, lambda: ja.forward_fused(
        *[t[f"{x}_{s}"] for s in ("txt", "img") for x in "qkv"],
        [t[n] for n in ("gamma_q_txt", "gamma_k_txt", "gamma_q_img", "gamma_k_img")],
        [t[n] for n in ("cos_txt", "sin_txt", "cos_img", "sin_img")], 1e-6, *out, ws)


def _plain(f2k, t):
    import torch
    att = f2k.Attention(f2k.Attention.Config(1, 130, 4, 128))
    out = torch.empty_like(t["q_img"])
    return att, None, [out], lambda: att.forward(t["q_img"], t["k_img"], t["v_img"], out)


STREAMS = [f"{n}_{s}" for s in ("txt", "img") for n in ("q", "k", "v", "gamma_q", "gamma_k", "cos", "sin")]


@pytest.mark.parametrize("call,late", [("rmsnorm", n) for n in ("q_img", "gamma_q_img")]
                         + [("rope", n) for n in ("q_img", "cos_img", "sin_img", "pos_ids")]
                         + [("joint", n) for n in STREAMS] + [("plain", n) for n in ("q_img", "k_img", "v_img")])
def test_a_late_input_is_read_as_written(late_copy, call, late):
    import torch

    import f2k_cuda_b200 as f2k

    def run(t, before=lambda: None):
        if call in ("joint", "plain"):        # handle, workspace and outputs are there before the writer starts
            module, _, out, go = (_joint if call == "joint" else _plain)(f2k, t)
            torch.cuda.synchronize()
            before()
            assert go(), module.last_error()
            torch.cuda.synchronize()
            assert module.device_status() == 0
            return out
        y = torch.empty_like(t["q_img"])
        torch.cuda.synchronize()
        before()
        if call == "rmsnorm":
            assert f2k.rmsnorm_bf16(t["q_img"], t["gamma_q_img"], y, 520, 128, 1e-6)
        else:
            assert f2k.rope_4axis_inplace_bf16(t["q_img"], t["cos_img"], t["sin_img"], t["pos_ids"], 520, 128, 130)
            y = t["q_img"]
        torch.cuda.synchronize()
        return [y]

    fresh = _inputs(1)[late]
    want = run(dict(_inputs(0), **{late: fresh.clone()}))
    stale_result = run(_inputs(0))
    assert any(not torch.equal(a, b) for a, b in zip(want, stale_result))      # the input matters
    t = _inputs(0)
    got = run(t, lambda: late_copy(t[late], fresh))
    assert all(torch.equal(a, b) for a, b in zip(want, got))

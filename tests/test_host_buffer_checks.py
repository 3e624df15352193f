"""The host-buffer call takes contiguous bf16 tensors only, like every other attention call of the mirror: the copies
behind it move heads * 128 * 2 bytes a token from the address they are given, whatever the tensor there is."""
from types import SimpleNamespace

import pytest
import torch

SHAPE = (1, 8, 2, 128)


@pytest.fixture
def call(monkeypatch):
    """forward_fused_host of a module that was never created on a GPU, with the C call behind it recorded."""
    from f2k_cuda_b200 import api
    reached = []
    m = api.JointAttention.__new__(api.JointAttention)
    m._rc, m._h = 0, None
    monkeypatch.setattr(api, "lib", SimpleNamespace(f2k_attn_forward_fused_host=lambda *a: reached.append(a) or 0))

    def run(tensors, gains):
        tables = [torch.zeros(8, 64) for _ in range(4)]
        ok = m.forward_fused_host(*tensors[:6], gains, tables, 1e-6, *tensors[6:], stream=0)
        return ok, reached

    return run


def _tensors():
    return [torch.zeros(SHAPE, dtype=torch.bfloat16) for _ in range(8)], [torch.zeros(128, dtype=torch.bfloat16) for _ in range(4)]


def test_contiguous_bf16_reaches_the_library(call):
    ok, reached = call(*_tensors())
    assert ok and len(reached) == 1


def test_no_text_stream(call):
    t, g = _tensors()
    ok, reached = call([None] * 3 + t[3:6] + [None] + t[7:], [None, None, *g[2:]])
    assert ok and len(reached) == 1


@pytest.mark.parametrize("which", range(12))
@pytest.mark.parametrize("bad", ["float32", "float16", "int8", "strided"])
def test_others_are_refused(call, which, bad):
    t, g = _tensors()
    group, i = (t, which) if which < 8 else (g, which - 8)
    x = group[i]
    group[i] = x.repeat_interleave(2, -1)[..., ::2] if bad == "strided" else x.to(getattr(torch, bad))
    with pytest.raises(TypeError):
        call(t, g)

"""The `stream` argument means the same in every part of the package: None is the current stream, a stream object its
handle, an integer the handle itself, 0 included (the legacy default stream)."""
import importlib
from types import SimpleNamespace

import pytest
import torch

CURRENT = 0x7000
ARGUMENTS = [(None, CURRENT), (0, 0), (0x55, 0x55), (SimpleNamespace(cuda_stream=0x99), 0x99), (SimpleNamespace(cuda_stream=0), 0)]


def _calls():
    """Each call with a `stream` argument that goes through one of the package's three modules, and the position of
    the stream among the arguments of the C function behind it."""
    from f2k_cuda_b200 import api, headswap, seqpar
    x = torch.zeros(1, 8, 1, 128, dtype=torch.bfloat16)
    hx = headswap.HeadExchangeAttention.__new__(headswap.HeadExchangeAttention)
    sp = seqpar.SequenceParallelAttention.__new__(seqpar.SequenceParallelAttention)
    at = api.Attention.__new__(api.Attention)
    hx._h = sp._h = at._h = None
    at._rc = 0
    tensors = (x,) * 7
    return {
        "api": (api, "f2k_attn_forward", -1, lambda s: at.forward(x, x, x, x, stream=s)),
        "seqpar_forward": (seqpar, "f2k_seqpar_forward", -2, lambda s: sp.forward(x, x, stream=s)),
        "qk_norm_rope": (seqpar, "f2k_qk_norm_rope_bf16", -1, lambda s: seqpar.qk_norm_rope(x, x, x, x, x, 1e-6, stream=s)),
        "hx_exchange_in": (headswap, "f2k_hx_exchange_in", -1, lambda s: hx.exchange_in(*tensors, 1e-6, stream=s)),
        "hx_exchange_in_copy": (headswap, "f2k_hx_exchange_in_copy", -1, lambda s: hx.exchange_in_copy(*tensors, 1e-6, stream=s)),
        "hx_forward": (headswap, "f2k_hx_forward", -1, lambda s: hx.forward(*tensors, 1e-6, stream=s)),
        "hx_attend": (headswap, "f2k_hx_attend", -1, lambda s: hx.attend(stream=s)),
        "hx_output": (headswap, "f2k_hx_output", -1, lambda s: hx.output(stream=s)),
    }


@pytest.mark.parametrize("call", ["api", "seqpar_forward", "qk_norm_rope", "hx_exchange_in", "hx_exchange_in_copy",
                                  "hx_forward", "hx_attend", "hx_output"])
@pytest.mark.parametrize("given,handle", ARGUMENTS, ids=["none", "zero", "handle", "stream", "default-stream"])
def test_stream_argument(monkeypatch, call, given, handle):
    module, function, position, run = _calls()[call]
    seen = []

    def c_function(*args):
        seen.append(args[position])
        return 1                                   # an error code: nothing further is done with the outputs

    monkeypatch.setattr(module, "lib", SimpleNamespace(**{function: c_function}))
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: CURRENT, raising=False)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: SimpleNamespace(cuda_stream=CURRENT))
    from f2k_cuda_b200 import _stream
    monkeypatch.setattr(_stream, "_current_handle", lambda device: CURRENT)
    assert not run(given)
    got = seen[0]
    assert (getattr(got, "value", got) or 0) == handle


def test_without_the_private_function(monkeypatch):
    from f2k_cuda_b200 import _stream
    try:
        with monkeypatch.context() as m:
            m.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
            m.setattr(torch.cuda, "current_device", lambda: 0)
            m.setattr(torch.cuda, "current_stream", lambda device=None: SimpleNamespace(cuda_stream=CURRENT))
            importlib.reload(_stream)
            assert _stream.stream_handle(None) == CURRENT
    finally:
        importlib.reload(_stream)


@pytest.mark.gpu
def test_current_stream_on_the_gpu():
    from f2k_cuda_b200._stream import stream_handle
    side = torch.cuda.Stream()
    assert stream_handle(None) == torch.cuda.current_stream().cuda_stream
    with torch.cuda.stream(side):
        assert stream_handle(None) == side.cuda_stream == stream_handle(side)

"""The `stream` argument of the package's calls, as the handle that the C ABI takes."""
from __future__ import annotations

import torch

# The current stream's handle without a torch.cuda.Stream around it (192 tokens x 4 heads: 15.5 us a call with the
# object, 12.0 without). A private function of torch, checked with 2.11; a torch without it gives the same handle
# the public way.
_current_handle = getattr(torch._C, "_cuda_getCurrentRawStream", None) or \
    (lambda device: torch.cuda.current_stream(device).cuda_stream)


def stream_handle(stream) -> int:
    """None is the current stream of the current device; a torch stream, or any object with a `cuda_stream`,
    is its handle; an integer is taken as it is (0: the legacy default stream)."""
    if stream is None:
        return _current_handle(torch.cuda.current_device())
    return stream.cuda_stream if hasattr(stream, "cuda_stream") else int(stream)

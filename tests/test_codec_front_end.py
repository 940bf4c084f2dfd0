"""The torch front end of the device codec, as far as it runs without a GPU."""
import importlib.util

import torch

from tirocinio_triennale_b200.ops import codec


def test_torch_without_the_private_functions(monkeypatch):
    """Stream and device are looked up by private functions of torch where there are any, else by the public ones."""
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    monkeypatch.delattr(torch._C, "_cuda_getDevice", raising=False)
    spec = importlib.util.spec_from_file_location(codec.__name__ + "_public", codec.__file__)
    public = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(public)
    asked = []

    class Stream:
        cuda_stream = 77

    monkeypatch.setattr(torch.cuda, "current_stream", lambda index: asked.append(index) or Stream)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    c = public.Codec.__new__(public.Codec)
    c._index = 3
    seen = []
    c._call("call", lambda *a: seen.append(a) or 0, 1, 2)
    assert seen == [(1, 2, 77)] and asked == [3]

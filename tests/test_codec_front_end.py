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


def test_size_words_made_during_a_capture_are_not_kept(monkeypatch):
    """A replay zeroes what was filled during the capture, so later calls must not get their words from it."""
    monkeypatch.setattr(codec, "_raw_stream", lambda index: 77)
    c = codec.Codec.__new__(codec.Codec)
    c._index, c._sizes, c.device = 0, {}, torch.device("cpu")
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    captured = c._size_words(8)
    assert captured.numel() == 8 and not c._sizes
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    words = [c._size_words(k) for k in (1, 8, 247, 8)]
    spans = [(w.data_ptr(), w.data_ptr() + 8 * w.numel()) for w in words + [captured]]
    for i, a in enumerate(spans):
        assert all(a[1] <= b[0] or b[1] <= a[0] for b in spans[i + 1:])
    assert all(int(w.abs().sum()) == 0 for w in words)

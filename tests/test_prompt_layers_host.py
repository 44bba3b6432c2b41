"""The native call of a Llama prompt portion's layers, on the host side alone."""
import ctypes
import struct
import threading

import pytest
import torch

from fastkernels_b200 import _lib, ops, prompt_layers

FIELDS = tuple(range(0x1000, 0x100f)) + (1e-5, 1e-6, 1e-5, 0.125)
TAIL = struct.pack("26Q", *range(0x2000, 0x201a))


def _run_to(native, monkeypatch):
    """A run on host tensors whose native call is the Python function `native`."""
    # as the prototype has them: two structs, and the stream
    proto = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_int, ctypes.c_int,
                             ctypes.c_void_p, ctypes.c_void_p)
    assert _lib.PROTOTYPES["fk_llama_prompt_layers"][1] == list(proto._argtypes_)
    stub = type("Stub", (), {"fk_llama_prompt_layers": staticmethod(proto(native))})
    monkeypatch.setattr(_lib, "lib", stub)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(prompt_layers, "_pack_layer", lambda *a: ("sizes", FIELDS))
    run = prompt_layers.PromptRun()
    run.rope = None
    run.shape, run.device = torch.Size((3, 8)), torch.device("cpu")
    run.sizes, run.fits, run.many, run.tail = "sizes", True, False, TAIL
    return run


def _expected(residual, hidden):
    return (struct.pack("15Q4d", *FIELDS),
            struct.pack("2Q", residual.data_ptr(), hidden.data_ptr()) + TAIL)


@pytest.mark.parametrize("threads", [0, 2])
def test_structs_live_until_the_call_returns(threads, monkeypatch):
    """Objects of the structs' sizes that are made during the call, by the thread itself or by
    others, do not land where the native side reads."""
    sizes = [len(s) for s in _expected(torch.empty(0), torch.empty(0))]
    stop, others = threading.Event(), []

    def allocate():
        keep = []
        while not stop.is_set():
            keep = [bytes([0xa5]) * n for n in sizes for _ in range(64)]
        return keep
    for _ in range(threads):
        others.append(threading.Thread(target=allocate, daemon=True))
        others[-1].start()
    seen = []

    def native(layer, count, first, prompt, stream):
        made = []
        for _ in range(50):
            made += [bytes([0x5a]) * n for n in sizes for _ in range(20)]
            seen.append((count, first, ctypes.string_at(layer, sizes[0]),
                         ctypes.string_at(prompt, sizes[1])))
        return 0
    run = _run_to(native, monkeypatch)
    hidden = torch.zeros((3, 8), dtype=torch.bfloat16)
    try:
        for residual in (None, torch.zeros_like(hidden)):
            seen.clear()
            out, res = run.layer(object(), hidden, residual)
            want = (1, int(residual is None), *_expected(res, out))
            assert len(seen) == 50 and all(s == want for s in seen)
    finally:
        stop.set()
        for t in others:
            t.join()

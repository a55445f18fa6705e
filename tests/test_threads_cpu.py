"""Calls of several threads share the cached workspaces: no two of them may be inside the library on
one buffer.  The library's entry points are replaced by ones that only look at the addresses."""
import contextlib
import threading
import time

import pytest
import torch


class _Stream:
    cuda_stream = 0

    def synchronize(self):
        pass


class _Lib:
    """Entry points that take a while and record whether another call is on the same workspace."""

    def __init__(self, real):
        self.real, self.busy, self.clash, self.calls = real, {}, [], 0
        self.lock = threading.Lock()

    def __getattr__(self, name):
        real = getattr(self.real, name)
        if "workspace_size" in name:
            return real
        at = {"nsgb_bwareaopen": 13, "nsgb_imfill_holes": 8, "nsgb_recon_f32_bwd": 9, "nsgb_bounding_boxes": 9}[name]

        def call(*args):
            lo, hi = args[at], args[at] + args[at + 1]
            with self.lock:
                self.calls += 1
                self.clash += [n for n, (a, b) in self.busy.values() if a < hi and lo < b]
                key = (threading.get_ident(), self.calls)
                self.busy[key] = (name, (lo, hi))
            time.sleep(0.01)
            with self.lock:
                del self.busy[key]
            return 0

        return call


def _calls(m, side):
    u8, i32 = torch.zeros((side, side), dtype=torch.uint8), torch.zeros((side, side), dtype=torch.int32)
    f32 = torch.zeros((side, side))
    return {
        "area": lambda: m.bwareaopen2(u8, False, True, 1, 2, 8),
        "fill": lambda: m.imfillHoles(u8, False, 4),
        "boxes": lambda: m.bounding_boxes(i32),
        "adjoint": lambda: m.recon_f32_backward(f32, i32),
    }


@pytest.mark.parametrize("names", [("area", "fill"), ("fill", "boxes"), ("adjoint", "adjoint")])
def test_threads_do_not_share_a_buffer(monkeypatch, names):
    import nsgb

    fake = _Lib(nsgb.lib)
    monkeypatch.setattr(nsgb, "lib", fake)
    monkeypatch.setattr(nsgb, "workspace", nsgb._Workspace())  # host buffers: not the cache of other tests
    monkeypatch.setattr(nsgb, "_check_image", lambda t, name: None)
    monkeypatch.setattr(nsgb, "_stack3", lambda t, name: t.unsqueeze(0))
    monkeypatch.setattr(nsgb, "_stream", lambda: 0)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: _Stream())
    start, errors = threading.Barrier(len(names)), []

    def work(name, k):
        try:
            start.wait(timeout=10)
            for n in range(6):  # sizes rise, so that a buffer in use is also asked to grow
                _calls(nsgb, 64 * (1 + n + k))[name]()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(n, k)) for k, n in enumerate(names)]
    with contextlib.ExitStack() as done:
        done.callback(lambda: [t.join() for t in threads])
        for t in threads:
            t.start()
    assert not errors and fake.calls == 6 * len(names)
    assert not fake.clash, fake.clash

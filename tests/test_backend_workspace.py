"""Scratch buffers of the host mirrors, on the CPU: what a captured graph was recorded with has to stay."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_cpp_mirror(tmp_path):
    """The C++ mirror over fakes of the CUDA runtime and the library (tests/cpp/workspace_tests.cpp)."""
    from aidotnet.tensors_b200 import build
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc())))
    exe = str(tmp_path / "workspace_tests")
    # the entry points that no case reaches have no fake
    subprocess.run([build._host_cxx(), "-std=c++17", "-O1", "-g", "-I", os.path.join(cuda, "include"), "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "workspace_tests.cpp"),
                    os.path.join(build.CSRC, "host", "direct_gpu_backend.cpp"), "-Wl,--unresolved-symbols=ignore-in-object-files"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "all cases passed" in r.stdout, r.stdout + r.stderr


class _Stream:
    def __init__(self, handle):
        self.cuda_stream = handle


class _Memory:
    """Stands in for torch: hands out numbered buffers, knows which the backend still holds and can run out of memory."""

    def __init__(self, monkeypatch):
        import contextlib
        import torch
        from aidotnet.tensors_b200 import backend, native
        self.capture, self.left, self.live, self.count, self.gone = None, 1 << 40, {}, 0, set()
        memory = self

        class Tensor:
            def __init__(self, n):
                memory.count += 1
                self.n, self.address = n, memory.count
                memory.live[self.address] = n

            def numel(self):
                return self.n

            def data_ptr(self):
                return self.address

            def __del__(self):
                memory.live.pop(self.address, None)

        def empty(n, **_):
            if n > memory.left:
                raise torch.OutOfMemoryError("fake")
            return Tensor(n)

        class Capture:
            def __init__(self, ident, graph):
                self.id = ident

            @property
            def gone(self):
                return self.id in memory.gone

            @staticmethod
            def of(stream):
                return (memory.capture, 1) if memory.capture else None

        monkeypatch.setattr(torch, "empty", empty)
        monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
        monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: memory.capture is not None)
        monkeypatch.setattr(native, "Capture", Capture, raising=False)
        self.backend = object.__new__(backend.CudaBackend)
        self.backend.device, self.backend._stream, self.backend._scratch, self.backend._captured = 0, None, {}, {}


def test_python_mirror_keeps_what_graphs_were_recorded_with(monkeypatch):
    memory = _Memory(monkeypatch)
    stream = _Stream(100)
    ws = lambda n, s=stream: memory.backend._workspace(n, s)[0]
    eager = ws(100)
    memory.capture = 7
    first = ws(100)
    assert ws(50) == first                  # the layers of one graph take turns with one buffer
    grown = ws(300)
    memory.capture = 8                      # a second graph on the same stream: may be replayed beside the first
    second = ws(100)
    memory.capture = None
    recorded = {first, grown, second}
    assert len(recorded) == 3 and eager not in recorded
    assert ws(5000) not in recorded
    for handle in range(200, 220):          # more streams than the backend keeps a buffer for
        assert ws(100, _Stream(handle)) not in recorded
    assert recorded <= set(memory.live) and eager not in memory.live
    memory.gone = {7}
    ws(6000)
    assert second in memory.live and not {first, grown} & set(memory.live)


def test_python_mirror_gives_back(monkeypatch):
    memory = _Memory(monkeypatch)
    for ident in range(1, 51):              # a program that captures again and again
        memory.capture = ident
        memory.backend._workspace(100, _Stream(100))
        memory.gone.add(ident - 1)
    assert len(memory.live) <= 2


def test_python_mirror_runs_a_prefill_without_memory_for_its_workspace(monkeypatch):
    import torch
    memory = _Memory(monkeypatch)
    ws = lambda n, optional=False: memory.backend._workspace(n, _Stream(100), optional)[0]
    eager = ws(100)
    memory.left = 1000
    assert ws(2000, optional=True) is None and ws(100) == eager
    memory.capture = 9
    assert ws(2000, optional=True) is None and ws(100) in memory.live
    memory.capture = None
    with pytest.raises(torch.OutOfMemoryError):
        ws(2000)
    assert ws(500) in memory.live


def test_only_a_prefill_does_without(monkeypatch):
    """What the mirror's calls pass on: a decode asks, a prefill may."""
    from aidotnet.tensors_b200.backend import CudaBackend

    class Handle:
        last_launch_count = last_path = 0

        def workspace_bytes(self, *_):
            return 100

        def launch(self, **kw):
            self.kw = kw

    class Buffer:
        Handle = 1

    asked = []
    backend = object.__new__(CudaBackend)
    backend._stream, backend.launch_count = _Stream(100), 0
    backend._workspace = lambda n, stream, optional=False: asked.append(optional) or (None, 0)
    for rows in (1, 2):
        backend._run(Handle(), query=Buffer, key=Buffer, value=Buffer, output=Buffer, batch=1, seqQ=rows, seqK=9, scale=1.0)
    assert asked == [False, True]

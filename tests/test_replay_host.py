"""Host side of compiled calls (``transforms/compile.py``, ``transforms/tape.py``) with stand-ins for the GPU's part."""
import importlib

import pytest
import torch

import nabla_b200 as nb
from nabla_b200 import native
from nabla_b200.transforms import tape

C = importlib.import_module("nabla_b200.transforms.compile")


class _Owned:
    """A GPU tensor that a recording owns, as far as the host sees it."""
    is_cuda, device = True, torch.device("cuda", 0)

    def __init__(self, log):
        self.log = log

    def record_stream(self, stream):
        self.log.append(("told", stream))


class _Impl:
    literal = None

    def __init__(self, log):
        self._buffers = [_Owned(log)]


@pytest.fixture
def gpu(monkeypatch):
    """(log, set the current stream, say whether it is capturing) of a GPU that is not there."""
    state, log = {"stream": 1, "capturing": False}, []
    monkeypatch.setattr(native, "raw_stream", lambda device: state["stream"], raising=False)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: state["stream"])
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: state["capturing"])
    return state, log


class _Module:
    def __init__(self, log, out):
        self.log, self.out = log, out

    def call(self, handle, args, deterministic):
        self.log.append(("call", handle))
        return self.out


def _taped_function(monkeypatch, log):
    f = nb.compile(lambda x: x)
    rec = C._Recorded()
    rec.constants = [_Impl(log)]
    rec.tape, rec.tape_counts = "handle", ()
    f._taped = (rec.tape, rec, f.use_cuda_graph)
    monkeypatch.setattr(tape, "module", lambda: _Module(log, "out"))
    return f, rec


def test_each_stream_is_told_of_the_constants_before_a_taped_call(gpu, monkeypatch):
    """What was made with the plan may be freed while another stream still reads it: once per stream, ahead of the launches."""
    state, log = gpu
    f, _ = _taped_function(monkeypatch, log)
    x = nb.Tensor.from_torch(torch.zeros(2))
    for stream in (1, 1, 2, 1):
        state["stream"] = stream
        assert f(x) == "out"
    assert log == [("told", 1), ("call", "handle"), ("call", "handle"), ("told", 2), ("call", "handle"), ("call", "handle")]


def test_a_graph_of_the_callers_gets_constants_of_its_own(gpu, monkeypatch):
    """It may outlive the function, so nothing that goes with the recording is in it."""
    state, log = gpu
    f, rec = _taped_function(monkeypatch, log)
    state["capturing"] = True
    assert f._call_taped(f._taped, (nb.Tensor.from_torch(torch.zeros(2)),)) is NotImplemented and log == []

    class Op:
        def __init__(self, execute):
            self.execute = execute

    class Node:
        def __init__(self, out, execute):
            self.out, self.op, self.out_refs = out, Op(execute), []

        def outputs(self):
            return [self.out]

    class Impl:
        literal = _buffers = None

    constant, helper, seen = Impl(), Impl(), []
    rec.nodes = [Node(helper, lambda n: [[torch.ones(3)]]), Node(constant, lambda n: [[helper._buffers[0] + 1]]),
                 Node(None, lambda n: seen.append(constant._buffers[0]) or [])]
    rec.constants, rec.constant_nodes, rec.steps, rec.free_after = [constant], [0, 1], [("op", (2,))], [[]]
    constant._buffers = [made := torch.full((3,), 2.0)]
    f._run(rec)
    state["capturing"] = False
    f._run(rec)
    assert seen[0] is not made and torch.equal(seen[0], made) and seen[1] is made and constant._buffers[0] is made
    assert helper._buffers is None


@pytest.mark.parametrize("what", ["garbage", "other version"])
def test_an_extension_that_does_not_load_is_one_that_is_not_there(what, tmp_path, monkeypatch):
    """Built for another Python or torch, or broken: said once, and calls go on by Python."""
    path = native.lib_path("libnb_replay.so")
    if what == "garbage":
        path = tmp_path / "libnb_replay.so"
        path.write_bytes(b"no library")
        monkeypatch.setattr(native, "lib_path", lambda name: path)
    else:
        if not path.exists():
            pytest.skip("not built")
        from nabla_b200.csrc import build

        monkeypatch.setattr(build, "replay_built_for", lambda: "another", raising=False)
    monkeypatch.setattr(tape, "_module", None)
    with pytest.warns(UserWarning, match="replayed by Python"):
        assert tape.module() is None
    assert tape.module() is None                     # and not a second time


def test_a_recording_that_cannot_be_taped_says_so_once(monkeypatch):
    """Without the extension being looked for, and without its nodes being looked over on every call."""
    def unexpected():
        raise AssertionError("looked for the extension")

    monkeypatch.setattr(tape, "module", unexpected)
    f = nb.compile(lambda x: x * 2.0 + 1.0)
    x = nb.Tensor.from_torch(torch.ones(3))
    for _ in range(3):
        assert f(x).to_torch().tolist() == [3.0, 3.0, 3.0]
    (entry,) = f._cache.values()
    (rec,) = entry.values()
    assert rec.tape is False


def test_build_leaves_the_extension_out_where_it_cannot_be_built(tmp_path, monkeypatch):
    import platform

    from nabla_b200.csrc import build

    monkeypatch.setattr(platform, "machine", lambda: "aarch64")
    monkeypatch.setattr(build, "LIB", tmp_path)
    monkeypatch.setattr(build, "TARGETS", {"libnb_replay.so": build.TARGETS["libnb_replay.so"]})
    assert build.build_all() == [] and not list(tmp_path.iterdir())

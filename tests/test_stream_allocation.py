"""Where the tensor helpers allocate when a stream is given: on that stream.

torch's allocator hands a freed block out again in the order of the stream it
was allocated on, so an output (or a temporary) of a helper that launches on
`stream` has to be allocated there: a block of the current stream could still
be in use by work pending on it, and could be reused by it while `stream`
reads.  The caller's stream is recorded on the outputs, so a dropped one is
not reused while the caller's own work still reads it.  Host logic only: tensors, streams and the C ABI are stand-ins, so the
ordering itself is not run here."""

import contextlib

import pytest

torch = pytest.importorskip("torch")


class FakeStream:
    def __init__(self, name):
        self.cuda_stream = hash(name) & 0xFFFF
        self.name = name

    def synchronize(self):
        pass


class FakeTensor:
    dtype, device = torch.uint64, "cuda"

    def __init__(self, shape, log, made_on=None, is_cuda=True):
        self.is_cuda, self.copies = is_cuda, []
        self.shape, self.log, self.made_on, self.recorded = tuple(shape), log, made_on, []

    def record_stream(self, s):
        self.recorded.append(s)

    def is_contiguous(self):
        return True

    def dim(self):
        return len(self.shape)

    def numel(self):
        n = 1
        for s in self.shape:
            n *= s
        return n

    def data_ptr(self):
        return 1 << 20

    def view(self, *shape):
        if isinstance(shape[0], torch.dtype):
            return self
        t = FakeTensor(shape, self.log, self.made_on)
        t.recorded = self.recorded  # one block
        return t

    def contiguous(self):
        return self

    def to(self, **kw):
        self.log.append(("to", self.log.current()))
        self.copies.append(FakeTensor(self.shape, self.log, self.log.current()))
        return self.copies[-1]

    def cpu(self):
        self.log.append(("cpu", self.log.current()))
        return self

    def numpy(self):
        return self


class Log(list):
    def __init__(self, current):
        super().__init__()
        self.current = current


@pytest.fixture
def fakes(monkeypatch):
    import zeknox_b200 as zk

    caller = FakeStream("caller")
    stack = [caller]
    log = Log(lambda: stack[-1])

    @contextlib.contextmanager
    def on(s):
        stack.append(s)
        try:
            yield
        finally:
            stack.pop()

    def alloc(shape, **kw):
        log.append(("alloc", stack[-1]))
        return FakeTensor(shape, log, stack[-1])

    class Lib:
        def __getattr__(self, name):
            return lambda *args: zk.capi.RustError(0, None)

    monkeypatch.setattr(torch, "empty", alloc)
    monkeypatch.setattr(torch, "zeros", alloc)
    monkeypatch.setattr(torch.cuda, "Stream", FakeStream)
    monkeypatch.setattr(torch.cuda, "stream", on)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: stack[-1])
    monkeypatch.setattr(zk.capi, "LIB", Lib())
    return zk, log, caller


CALLS = {
    "lde": lambda zk, t, s: zk.lde(t(4, 64), 3, stream=s),
    "transpose_rev": lambda zk, t, s: zk.transpose_rev(t(4, 64), stream=s),
    "lde_leaves": lambda zk, t, s: zk.lde_leaves(t(4, 64), 3, stream=s),
    "lde_leaves_coset": lambda zk, t, s: zk.lde_leaves_coset(t(4, 64), 3, 49, stream=s),
    "commit": lambda zk, t, s: zk.commit(t(4, 64), 3, 2, stream=s),
    "merkle_tree": lambda zk, t, s: zk.merkle_tree(t(64, 9), 2, stream=s),
    "merkle_tree, zeroed": lambda zk, t, s: zk.merkle_tree(t(64, 3), 2, zk.HashKeccak, stream=s),
    "merkle_open": lambda zk, t, s: zk.merkle_open(t(64, 9), t(120, 4), 2, t(5), stream=s),
    "fri_fold": lambda zk, t, s: zk.fri_fold(t(2, 64), 2, (1, 2), stream=s),
}


@pytest.mark.parametrize("name", CALLS)
def test_outputs_belong_to_the_given_stream(fakes, name):
    zk, log, caller = fakes
    side = FakeStream("side")
    out = CALLS[name](zk, lambda *shape: FakeTensor(shape, log), side)
    assert log and all(s is side for _, s in log), [(what, s.name) for what, s in log]
    outs = vars(out).values() if isinstance(out, zk.CommitBuffers) else out if isinstance(out, tuple) else (out,)
    assert all(t.made_on is side and t.recorded == [caller] for t in outs)
    log.clear()
    CALLS[name](zk, lambda *shape: FakeTensor(shape, log), None)
    assert log and all(s is caller for _, s in log)


def test_fri_commit_rounds_belong_to_the_given_stream(fakes):
    """Leaves, trees, the copies of the caps and the folded coefficients; the callback runs on the caller's stream."""
    zk, log, caller = fakes
    side = FakeStream("side")
    seen = []

    def challenge(i, cap):
        seen.append(torch.cuda.current_stream())
        return (1, 2)

    com = zk.fri_commit(FakeTensor((2, 1 << 8), log), 1, [2, 2], 1, challenge, stream=side)
    assert [what for what, _ in log].count("cpu") == 2 and all(s is side for _, s in log)
    assert seen == [caller, caller]
    for t in [com.final_poly] + [x for r in com.rounds for x in (r.leaves, r.digests, r.cap)]:
        assert t.made_on is side and t.recorded == [caller]


@pytest.mark.parametrize("on_device", [False, True])
def test_open_indices_outlive_the_call_on_the_given_stream(fakes, on_device):
    """Host indices are copied on the caller's stream, so that pending work on `stream` does not block the call."""
    zk, log, caller = fakes
    side = FakeStream("side")
    idx = FakeTensor((5,), log, is_cuda=on_device)
    zk.merkle_open(FakeTensor((64, 9), log), FakeTensor((120, 4), log), 2, idx, stream=side)
    (copy,) = idx.copies
    assert copy.made_on is (side if on_device else caller) and copy.recorded == [side]

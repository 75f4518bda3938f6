"""knn_distances and the index it keeps per thread, as far as that goes
without a GPU: what is refused."""
import pytest
import torch


@pytest.mark.parametrize("queries,points,error", [
    (torch.rand(5, 3), torch.rand(5, 3), "CUDA"),
    (torch.rand(5, 3), torch.tensor(1.0), "CUDA"),
    (torch.tensor(1.0), torch.rand(5, 3), "CUDA"),
])
def test_knn_distances_refuses_host_tensors(rtd, queries, points, error):
    from rtdsl import torch_ops
    with pytest.raises(TypeError, match=error):
        torch_ops.knn_distances(queries, points, 2)


class FakeCuda:
    """torch.cuda with two devices, each with a current stream."""

    def __init__(self):
        self.now, self.log = 0, []

    def current_stream(self, device=None):
        return FakeStream(self, self.now if device is None else torch.device(device).index)

    def device(self, device):
        import contextlib

        @contextlib.contextmanager
        def use():
            before, self.now = self.now, torch.device(device).index
            try:
                yield
            finally:
                self.now = before
        return use()

    def Event(self):
        return FakeEvent(self)


class FakeStream:
    def __init__(self, cuda, device):
        self.cuda, self.device = cuda, device

    def wait_event(self, event):
        self.cuda.log.append(("wait", self.device, event.recorded_on))


class FakeEvent:
    def __init__(self, cuda):
        self.cuda, self.recorded_on = cuda, None

    def record(self, stream):
        self.recorded_on = stream.device
        self.cuda.log.append(("record", stream.device))


@pytest.fixture
def fake(rtd, monkeypatch):
    from rtdsl import api
    cuda = FakeCuda()

    class FakeIndex:
        def __init__(self):
            self.made_on, self.points = cuda.now, None

        def use(self):   # as build and knn: on the current device's current stream
            cuda.log.append(("use", cuda.current_stream().device, self.made_on))

    for name in ("current_stream", "device", "Event"):
        monkeypatch.setattr(torch.cuda, name, getattr(cuda, name))
    monkeypatch.setattr(api, "Index", FakeIndex)
    api.release_kept_index()
    yield cuda
    api.release_kept_index()


def test_kept_index_lives_on_the_device_of_its_points(fake):
    from rtdsl.api import short_lived_index
    one = torch.device("cuda", 1)
    for _ in range(2):   # the current device is 0
        with short_lived_index(one, 10, 10, 5) as ix:
            ix.use()
    assert fake.now == 0
    fake.now = 1
    with short_lived_index(one, 10, 10, 5) as ix:
        ix.use()
    fake.now = 0
    with short_lived_index(torch.device("cuda", 0), 10, 10, 5) as ix:
        ix.use()
    # made, used, awaited and marked on one and the same device
    assert fake.log == [("use", 1, 1), ("record", 1), ("wait", 1, 1), ("use", 1, 1), ("record", 1),
                        ("wait", 1, 1), ("use", 1, 1), ("record", 1), ("use", 0, 0), ("record", 0)]


@pytest.mark.parametrize("n,nq,k,kept", [(5_000, 10, 2048, True), (5_000, 10, 2049, False), (2_048, 10, 9_000, True),
                                         (1 << 21, 1 << 21, 1, True), ((1 << 21) + 1, 1, 1, False),
                                         (1, (1 << 21) + 1, 1, False)])
def test_kept_index_is_bounded(fake, n, nq, k, kept):
    """Lists above 2,048 entries take a slab of up to 1 GiB on the index."""
    from rtdsl import api
    with api.short_lived_index(torch.device("cuda", 0), n, nq, k) as ix:
        ix.use()
    assert (api._kept.entry is not None) == kept

"""run_layers against the loop it stands for, trk_out.copy_(trk_in) and one call pair per layer: what
the copy refused, recorded or converted. The library is replaced by a recorder, so no GPU is needed."""
import pytest

torch = pytest.importorskip("torch")

NLAYER = 3


@pytest.fixture
def loop(p2r, monkeypatch):
    """run_layers over CPU tensors; returns what the first propagation would read."""
    from p2r_tests_b200 import api
    cfg = p2r.Config(bsize=4, nlayer=NLAYER, nevts=1, nb=2)
    hits = torch.zeros(cfg.nblocks * NLAYER, 9, 4)
    calls = []

    class Recorder:
        @staticmethod
        def p2r_propagate_to_r(c, src, h, layer, out, dr, st):
            calls.append((layer, src, out))
            return 0

        @staticmethod
        def p2r_kalman_update(c, out, h, layer, chi2, st):
            return 0

    monkeypatch.setattr(api, "lib", lambda: Recorder)
    monkeypatch.setattr(api, "_ptr", lambda t: t.data_ptr())
    monkeypatch.setattr(api, "_stream", lambda s: 0)

    def run(trk_in, trk_out):
        calls.clear()
        p2r.run_layers(cfg, trk_in, hits, trk_out)
        assert [c[0] for c in calls] == list(range(NLAYER))
        assert all(c[2] == trk_out.data_ptr() for c in calls)
        assert all(c[1] == trk_out.data_ptr() for c in calls[1:])
        return trk_in if calls[0][1] == trk_in.data_ptr() else trk_out

    run.calls = calls
    return run


def tracks(*shape):
    return torch.arange(2 * 28 * 4, dtype=torch.float32).reshape(shape or (2, 28, 4)) + 1


@pytest.mark.parametrize("shape", [(2, 28, 4), (224,)])
def test_plain_input_is_read_in_place(loop, shape):
    t, out = tracks(*shape), torch.zeros(shape)
    assert loop(t, out) is t


@pytest.mark.parametrize("shape", [(2, 4, 28), (4, 28, 2), (8, 28)])
def test_other_shape_of_the_same_count_is_refused(loop, shape):
    out = torch.zeros(2, 28, 4)
    with pytest.raises(RuntimeError):
        loop(tracks(*shape), out)
    assert not loop.calls and not out.any()


@pytest.mark.parametrize("form", ["broadcast", "flat", "strided", "double", "negative", "in_place", "overlapping"])
def test_converted_forms_are_copied(loop, form):
    t, out = tracks(), torch.zeros(2, 28, 4)
    if form == "flat":
        t, out = tracks(224), torch.zeros(1, 224)
    src = {"broadcast": lambda: t[:1], "flat": lambda: t, "strided": lambda: torch.stack([t, t], -1)[..., 0],
           "double": lambda: t.double(), "negative": lambda: torch._neg_view(t), "in_place": lambda: out,
           "overlapping": lambda: None}[form]()
    if form == "in_place":
        out.copy_(t)
    if form == "overlapping":  # contiguous, shifted by one element within the same memory
        base = torch.zeros(225)
        src, out = base[:224].view(2, 28, 4), base[1:].view(2, 28, 4)
        with pytest.raises(RuntimeError):
            out.copy_(src)
        with pytest.raises(RuntimeError):
            loop(src, out)
        return
    want = torch.zeros_like(out).copy_(src)
    loop(src, out)
    assert loop.calls[0][1] == out.data_ptr()
    assert torch.equal(out, want)


def test_the_write_is_seen_by_autograd(loop):
    t, out = tracks(), torch.zeros(2, 28, 4)
    before = out._version
    loop(t, out)
    assert out._version > before
    w = torch.ones(2, 28, 4, requires_grad=True)
    loss = (w * out).sum()
    loop(t, out)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        loss.backward()


def test_autograd_refuses_and_records_as_the_copy_does(loop):
    with pytest.raises(RuntimeError):
        loop(tracks(), torch.zeros(2, 28, 4, requires_grad=True))
    out = torch.zeros(2, 28, 4)
    loop(tracks().requires_grad_(), out)
    assert out.requires_grad
    with torch.inference_mode():
        out = torch.zeros(2, 28, 4)
    with pytest.raises(RuntimeError):
        loop(tracks(), out)


def test_forward_mode_tangent_goes_with_the_copy(loop):
    import torch.autograd.forward_ad as fwd
    out = torch.zeros(2, 28, 4)
    with fwd.dual_level():
        loop(fwd.make_dual(tracks(), torch.ones(2, 28, 4)), out)
        assert torch.equal(fwd.unpack_dual(out).tangent, torch.ones(2, 28, 4))


def test_no_layers_is_the_copy(loop, p2r):
    t, out = tracks(), torch.zeros(2, 28, 4)
    p2r.run_layers(p2r.Config(bsize=4, nlayer=0, nevts=1, nb=2), t, None, out)
    assert torch.equal(out, t)


class FakeStreams:
    """torch.cuda's stream calls over handles: the current stream is 0; `log` takes what happens where."""

    class Stream:
        def __init__(self, handle, device=None):
            self.cuda_stream = handle

    def __init__(self, monkeypatch):
        from p2r_tests_b200 import api
        self.log, self.now, self.captured = [], self.Stream(0), set()
        cuda = torch.cuda

        class On:
            def __init__(ctx, s):
                ctx.s = s

            def __enter__(ctx):
                ctx.before, self.now = self.now, ctx.s

            def __exit__(ctx, *exc):
                self.now = ctx.before

        copy, record = torch.Tensor.copy_, self.log.append
        self.Stream.record_event = lambda s: (record(("event", s.cuda_stream)), s.cuda_stream)[1]
        self.Stream.wait_event = lambda s, e: record(("wait", s.cuda_stream, e))
        monkeypatch.setattr(cuda, "Stream", self.Stream)
        monkeypatch.setattr(cuda, "ExternalStream", self.Stream)
        monkeypatch.setattr(cuda, "stream", On)
        monkeypatch.setattr(cuda, "current_stream", lambda device=None: self.now)
        monkeypatch.setattr(cuda, "is_current_stream_capturing", lambda: self.now.cuda_stream in self.captured)
        monkeypatch.setattr(torch.Tensor, "copy_",
                            lambda t, src: (record(("copy", self.now.cuda_stream)), copy(t, src))[1], raising=False)
        monkeypatch.setattr(torch.Tensor, "record_stream",
                            lambda t, s: record(("used", s.cuda_stream)), raising=False)
        monkeypatch.setattr(api, "_stream", lambda s: s.cuda_stream if hasattr(s, "cuda_stream") else int(s or 0))


@pytest.mark.parametrize("form,kind,expected", [
    ("plain", "current", []),
    ("plain", "legacy handle", []),
    ("plain", "torch", [("used", 640)]),
    ("plain", "handle", [("copy", 640), ("event", 640), ("wait", 0, 640)]),
    ("strided", "current", [("copy", 0)]),
    ("strided", "torch", [("copy", 640), ("used", 640)]),
    ("strided", "handle", [("copy", 640), ("event", 640), ("wait", 0, 640)]),
    ("strided", "captured handle", [("copy", 640)]),
    ("strided", "handle under capture", [("copy", 640)]),
])
def test_copy_and_lifetime_on_another_stream(loop, p2r, monkeypatch, form, kind, expected):
    """The copy belongs to the kernels' stream: on torch's current one it races with the first layer."""
    fake = FakeStreams(monkeypatch)
    t, out = tracks(), torch.zeros(2, 28, 4)
    if form == "strided":
        t = torch.stack([t, t], -1)[..., 0]
    stream = {"current": fake.now, "legacy handle": 1, "torch": fake.Stream(640)}.get(kind, 640)
    fake.captured = {"captured handle": {640}, "handle under capture": {0}}.get(kind, set())
    fake.log.clear()
    p2r.run_layers(p2r.Config(bsize=4, nlayer=NLAYER, nevts=1, nb=2), t, torch.zeros(2 * NLAYER, 9, 4), out,
                   stream=stream)
    assert fake.log == expected and len(loop.calls) == NLAYER


def gpu_case(p2r, mode):
    cfg = p2r.Config(bsize=24, nlayer=5, nevts=2, nb=3, bz=3.8, mode=mode)
    trk, hit = p2r.generate_helix(cfg, p2r.gen_params(bz=3.8, seed=12))
    t, h = torch.from_numpy(trk).cuda(), torch.from_numpy(hit).cuda()
    want = torch.empty_like(t)
    p2r.forward(cfg, t, h, want)
    torch.cuda.synchronize()
    return cfg, t, h, want


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["plain", "host", "strided", "broadcast"])
@pytest.mark.parametrize("kind", ["torch", "handle"])
def test_side_stream_that_holds_earlier_work(p2r, form, kind):
    cfg, t, h, want = gpu_case(p2r, p2r.MODE_CHAINED)
    if form == "broadcast":
        t[:] = t[0].clone()
        p2r.forward(cfg, t, h, want)
        torch.cuda.synchronize()
    src = {"plain": t.clone, "host": t.cpu, "strided": lambda: torch.stack([t, t], -1)[..., 0],
           "broadcast": lambda: t[:1].clone()}[form]()
    side, out = torch.cuda.Stream(), torch.empty_like(t)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)  # about 10 ms
        out.fill_(5.0)  # earlier work on the side stream that writes the output
    p2r.run_layers(cfg, src, h, out, stream=side if kind == "torch" else side.cuda_stream)
    shape, on_gpu = src.shape, src.is_cuda
    del src  # free at once: the next allocation of its size may not land in it before it is read
    if on_gpu:
        torch.full(shape, float("nan"), device="cuda")
    torch.cuda.synchronize()
    assert torch.equal(out.view(torch.int32), want.view(torch.int32))


@pytest.mark.gpu
@pytest.mark.parametrize("handle", [0, 1, 2])  # the default stream: torch's, the legacy one by name, this thread's
@pytest.mark.parametrize("form", ["plain", "strided"])
def test_default_stream_handles(p2r, handle, form):
    cfg, t, h, want = gpu_case(p2r, p2r.MODE_CHAINED)
    src = t if form == "plain" else torch.stack([t, t], -1)[..., 0]
    out, fused = torch.empty_like(t), torch.empty_like(t)
    torch.cuda.synchronize()
    p2r.run_layers(cfg, src, h, out, stream=handle)
    p2r.forward(cfg, t, h, fused, stream=handle)
    torch.cuda.synchronize()
    assert torch.equal(out.view(torch.int32), want.view(torch.int32))
    assert torch.equal(fused.view(torch.int32), want.view(torch.int32))

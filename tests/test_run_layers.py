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

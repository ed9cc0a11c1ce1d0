"""The stride forward_backward chooses itself, on a device whose memory runs out: a refused stride-1
workspace is replaced by the stride-5 one, once per output dict; a stride that the caller names, or one
that is refused as well, raises. The library's call is replaced by a recorder, so no GPU is needed."""
import pytest

torch = pytest.importorskip("torch")


@pytest.fixture
def call(p2r, monkeypatch):
    from p2r_tests_b200 import autograd
    cfg = p2r.Config(bsize=32, nlayer=20, nevts=1, nb=2, bz=3.8)
    need = {ck: p2r.workspace_size(cfg, ck) for ck in (1, 5)}
    assert need[5] < need[1]
    real, empty, used, limit = autograd.lib(), torch.empty, [], [need[1]]

    class Recorder:
        def __getattr__(self, name):
            return getattr(real, name)

        @staticmethod
        def p2r_forward_backward(c, *args):
            used.append(dict(stride=args[-4], bytes=args[-2]))
            return 0

    def bounded_empty(*shape, **kw):
        if kw.get("dtype") is torch.uint8 and shape[0] > limit[0]:
            raise torch.cuda.OutOfMemoryError("no memory")
        return empty(*shape, **kw)

    monkeypatch.setattr(autograd, "lib", lambda: Recorder())
    monkeypatch.setattr(autograd, "_ptr", lambda t: None if t is None else t.data_ptr())
    monkeypatch.setattr(autograd, "_arg", lambda t, dtype, n, name: None if t is None else t.data_ptr())
    monkeypatch.setattr(autograd, "_stream", lambda s: None)
    monkeypatch.setattr(torch, "empty", bounded_empty)
    trk, hit = torch.zeros(cfg.ntracks * 28), torch.zeros(cfg.ntracks * 20 * 9)

    def run(allowed, **kw):
        limit[0] = allowed
        o = p2r.forward_backward(cfg, trk, hit, **kw)
        return o, used[-1]

    run.need = need
    return run


def test_stride_one_where_it_fits(call):
    o, used = call(call.need[1])
    assert o["ckpt_stride"] == used["stride"] == 1 and used["bytes"] == call.need[1]


def test_refused_workspace_takes_stride_five_and_keeps_it(call):
    o, used = call(call.need[5])
    assert o["ckpt_stride"] == used["stride"] == 5
    assert used["bytes"] == o["workspace"].numel() == call.need[5]
    again, used = call(call.need[1], out=o)  # memory is there again: the dict's stride stays
    assert again is o and o["ckpt_stride"] == used["stride"] == 5 and used["bytes"] == call.need[5]


@pytest.mark.parametrize("kw", [dict(ckpt_stride=1), dict()])
def test_named_stride_and_second_refusal_raise(call, kw):
    allowed = call.need[5] if kw else call.need[5] - 1
    with pytest.raises(torch.cuda.OutOfMemoryError):
        call(allowed, **kw)

"""The host side of run_layers and of the adjoint's stride choice: every form of input the copy of
the layer loop used to take, and the free-memory query only where the workspace is large."""
import numpy as np
import pytest


def test_small_workspace_asks_no_free_memory(monkeypatch):
    import torch

    import p2r_tests_b200 as p2r
    asked = []
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda dev: (asked.append(dev), (40 << 30, 180 << 30))[1])
    small = p2r.Config(bsize=32, nlayer=20, nevts=1, nb=300, bz=3.8)
    assert p2r.auto_ckpt_stride(small, "cuda") == 1 and not asked
    assert p2r.auto_ckpt_stride(small, "cuda", tape=False) == 5 and not asked
    large = p2r.Config(bsize=32, nlayer=20, nevts=100, nb=300, bz=3.8)  # 4.2 GB of 20 allowed
    assert p2r.auto_ckpt_stride(large, "cuda") == 1 and len(asked) == 1
    huge = p2r.Config(bsize=32, nlayer=40, nevts=100, nb=3125, bz=3.8)  # 86 GB
    assert p2r.auto_ckpt_stride(huge, "cuda") == 5 and len(asked) == 2


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["chained", "restart"])
@pytest.mark.parametrize("form", ["plain", "host", "strided", "in_place"])
def test_run_layers_input_forms(form, mode):
    import torch

    import p2r_tests_b200 as p2r
    cfg = p2r.Config(bsize=24, nlayer=5, nevts=2, nb=3, bz=3.8,
                     mode=p2r.MODE_CHAINED if mode == "chained" else p2r.MODE_RESTART)
    trk, hit = p2r.generate_helix(cfg, p2r.gen_params(bz=3.8, seed=12))
    t, h = torch.from_numpy(trk).cuda(), torch.from_numpy(hit).cuda()
    want = torch.empty_like(t)
    p2r.forward(cfg, t, h, want)
    out = torch.full_like(t, 7.0)
    src = {"plain": t, "host": t.cpu(), "in_place": out,
           "strided": torch.stack([t, t], -1)[..., 0]}[form]
    if form == "in_place":
        out.copy_(t)
    if mode == "restart" and form != "plain":
        if form == "in_place":
            return  # every layer would start from the last one's output
        with pytest.raises(p2r.P2RError):
            p2r.run_layers(cfg, src, h, out)
        return
    p2r.run_layers(cfg, src, h, out)
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy().view(np.int32), want.cpu().numpy().view(np.int32))

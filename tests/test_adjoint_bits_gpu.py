"""The grid adjoint and the persistent one run the same arithmetic: per-track results equal bit for
bit, at the block width the grid's forward has compiled in (32) and at one taken at run time."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("bsize", [32, 64])
@pytest.mark.parametrize("nlayer,r_first,r_last", [(20, 20.0, 100.0), (40, 4.0, 110.0)])
@pytest.mark.parametrize("ordered", [False, True])
def test_grid_and_queue_adjoint_agree_to_the_bit(p2r, bsize, nlayer, r_first, r_last, ordered):
    import torch
    nevts, nb = 4, 8192 // bsize
    cfg = p2r.Config(bsize=bsize, nlayer=nlayer, nevts=nevts, nb=nb, bz=3.8)
    trk, hit = p2r.generate_helix_device(cfg, p2r.gen_params(bz=3.8, seed=91, r_first=r_first, r_last=r_last))
    rng = np.random.default_rng(91)
    nlay = rng.integers(0, nlayer + 1, cfg.ntracks).astype(np.int32)
    off = np.arange(nevts + 1, dtype=np.int64) * nb
    w = dict(nlay_lane=nlay, event_block_offset=off, ntrk_event=np.full(nevts, nb * bsize), nblocks=cfg.nblocks,
             bsize=bsize, nlayer=nlayer, bz=cfg.bz, updates=int(nlay.sum()))
    gen = torch.Generator(device="cuda").manual_seed(5)
    g_trk = torch.randn(trk.shape, generator=gen, device="cuda")
    g_chi2 = torch.rand(cfg.ntracks, generator=gen, device="cuda")
    dr = (torch.rand(nlayer, generator=gen, device="cuda") - 0.5) * 0.02
    flags = p2r.FLAG_ORDER_BY_LAYERS if ordered else 0
    cfg.flags = flags
    grid = p2r.forward_backward(cfg, trk, hit, dr=dr, nlay_lane=torch.from_numpy(nlay).cuda(), grad_trk_out=g_trk,
                                grad_chi2=g_chi2, ckpt_stride=1)
    q = p2r.Queue(w, blocks_per_item=3, flags=flags)
    queue = q.run_adjoint(trk, hit, dr=dr, grad_trk_out=g_trk, grad_chi2=g_chi2)
    assert q.error_bits() == 0
    for k in ("trk_out", "chi2", "grad_trk_in", "grad_hits"):
        a, b = (o[k].cpu().numpy().reshape(-1).view(np.int32) for o in (grid, queue))
        assert np.array_equal(a, b), (k, int((a != b).sum()))

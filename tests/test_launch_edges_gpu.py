"""Edges of the launch plumbing and of the small kernels around the hot path, on the GPU: chunk
boundaries of the host-buffer pipeline, the rows of the gradient totals, layer counts around the
hit prefetch, and capture of dependent launches. All comparisons are bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits(t):
    return t.detach().cpu().contiguous().numpy().reshape(-1).view(np.int32)


def make(bsize, nb, nevts, nlayer, seed=5):
    import torch

    import p2r_tests_b200 as p2r
    cfg = p2r.Config(bsize=bsize, nlayer=nlayer, nevts=nevts, nb=nb, bz=3.8)
    trk, hit = p2r.generate_helix_device(cfg, p2r.gen_params(bz=3.8, seed=seed))
    return p2r, torch, cfg, trk, hit


# (blocks, chunks): one chunk, two (no shorter last one), a last chunk of a quarter, more chunks than
# blocks, and a block count that no chunk count divides; 20 layers of 512 lanes are 0.4 MB a block
@pytest.mark.parametrize("nb,nevts,nchunks", [(1, 1, 8), (22, 1, 2), (11, 7, 8), (3, 5, 100), (101, 1, 7)])
@pytest.mark.parametrize("mode", [0, 1])
def test_host_chunks(nb, nevts, nchunks, mode):
    p2r, torch, cfg, trk, hit = make(512, nb, nevts, 20)
    cfg.mode = mode
    want = torch.empty_like(trk)
    p2r.forward(cfg, trk, hit, want)
    host = [trk.cpu().pin_memory(), hit.cpu().pin_memory(), torch.full(trk.shape, 7.0).pin_memory()]
    dev = [torch.full_like(trk, 3.0), torch.full_like(hit, 3.0), torch.full_like(trk, 3.0)]
    p2r.forward_host(cfg, *[h.numpy() for h in host], *dev, nchunks=nchunks)
    torch.cuda.synchronize()
    assert np.array_equal(bits(host[2]), bits(want))


@pytest.mark.parametrize("nevts", [1, 255, 256, 257, 600])
def test_totals_are_the_events_in_order(nevts):
    p2r, torch, cfg, trk, hit = make(32, 1, nevts, 3)
    o = p2r.forward_backward(cfg, trk, hit, grad_chi2=torch.ones(cfg.ntracks, device="cuda"), per_event=True)
    torch.cuda.synchronize()
    for total, event in (("grad_dr", "grad_dr_event"), ("grad_bz", "grad_bz_event")):
        rows = o[event].cpu().numpy().reshape(nevts, -1)
        s = np.zeros(rows.shape[1])
        for r in rows:
            s = s + r
        assert np.array_equal(o[total].cpu().numpy(), s)


@pytest.mark.parametrize("bsize", [1, 20, 33, 96])
@pytest.mark.parametrize("nlayer", [1, 2, 3])
def test_fused_equals_layer_by_layer(bsize, nlayer):
    p2r, torch, cfg, trk, hit = make(bsize, 5, 2, nlayer)
    fused, layers, masked = (torch.empty_like(trk) for _ in range(3))
    p2r.forward(cfg, trk, hit, fused)
    p2r.run_layers(cfg, trk, hit, layers)
    full = torch.full((cfg.ntracks,), nlayer, dtype=torch.int32, device="cuda")
    p2r.forward(cfg, trk, hit, masked, nlay_lane=full)
    torch.cuda.synchronize()
    assert np.array_equal(bits(fused), bits(layers)) and np.array_equal(bits(fused), bits(masked))
    p2r.forward(cfg, trk, hit, masked, nlay_lane=torch.zeros_like(full))
    assert np.array_equal(bits(masked), bits(trk))


def test_dependent_launches_under_capture():
    p2r, torch, cfg, trk, hit = make(32, 40, 1, 6)
    want, out = torch.empty_like(trk), torch.empty_like(trk)
    p2r.forward(cfg, trk, hit, want)
    side, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=side):
        p2r.run_layers(cfg, trk, hit, out, stream=side)
    for _ in range(3):
        out.fill_(0.0)
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(bits(out), bits(want))


# below, at and above the size from which a masked batch is ordered (12 groups of 32 tracks per SM)
@pytest.mark.parametrize("groups", [1, 12 * 148 - 1, 12 * 148, 12 * 148 + 1, 16 * 148 + 5])
@pytest.mark.parametrize("bsize,options", [(32, False), (64, True), (256, False)])
def test_ordered_flag_around_its_line(groups, bsize, options):
    import p2r_tests_b200 as p2r
    p2r, torch, cfg, trk, hit = make(bsize, max(1, groups * 32 // bsize), 1, 5)
    if options:
        cfg.flags = p2r.FLAG_SQUASH_PHI
    nlay = torch.randint(0, 7, (cfg.ntracks,), dtype=torch.int32, device="cuda")  # 6: more than there are
    dr = torch.linspace(-0.01, 0.01, 5, device="cuda") if options else None
    outs = []
    for flag in (0, p2r.FLAG_ORDER_BY_LAYERS):
        cfg.flags = (cfg.flags & ~p2r.FLAG_ORDER_BY_LAYERS) | flag
        for threads in (0, 128):
            cfg.block_threads = threads
            out, chi2 = torch.empty_like(trk), torch.empty(cfg.ntracks, device="cuda")
            p2r.forward(cfg, trk, hit, out, chi2=chi2, dr=dr, nlay_lane=nlay)
            outs.append((bits(out), bits(chi2)))
    for o, c in outs[1:]:
        assert np.array_equal(o, outs[0][0]) and np.array_equal(c, outs[0][1])

"""p2r_forward_host with several chunks: batches large enough that the pipeline splits them (a chunk for
every 4 MiB of input), in both modes, from pinned and unpinned host arrays, at odd block widths, with
more chunks asked for than there are blocks, from two threads, and between guard regions. Bit for bit
against the device-resident forward."""
import threading

import numpy as np
import pytest

from tests.test_guard_gpu import Guarded

pytestmark = pytest.mark.gpu
CHUNK = 4 << 20


@pytest.fixture(scope="module")
def torch():
    import torch as t
    return t


def bits(a):
    return (a.numpy() if hasattr(a, "numpy") else a).reshape(-1).view(np.int32)


def make(p2r, torch, bsize, nb, nevts, nlayer, mode, chunks, seed=5):
    """A batch whose input is at least `chunks` * 4 MiB, its host copies and the device's result."""
    cfg = p2r.Config(bsize=bsize, nlayer=nlayer, nevts=nevts, nb=nb, bz=3.8, mode=mode)
    block = (28 + 9 * (1 if mode == p2r.MODE_RESTART else nlayer)) * 4 * bsize
    assert cfg.nblocks * block >= chunks * CHUNK
    trk, hit = p2r.generate_helix_device(cfg, p2r.gen_params(bz=3.8, seed=seed))
    want = torch.empty_like(trk)
    p2r.forward(cfg, trk, hit, want)
    return cfg, trk.cpu(), hit.cpu(), bits(want.cpu())


# chained: 0.43 MB a block of 512 lanes x 20 layers; restart: 0.076 MB, so more blocks
@pytest.mark.parametrize("bsize,nb,nevts,nlayer,mode,nchunks,chunks", [
    (512, 31, 1, 20, 1, 3, 3), (512, 11, 7, 20, 1, 8, 7), (512, 10, 2, 20, 1, 2, 2), (33, 101, 9, 20, 1, 5, 5),
    (1, 4000, 7, 20, 1, 8, 5), (20, 700, 3, 17, 1, 100, 7), (4096, 2, 1, 40, 1, 100, 3), (4096, 1, 3, 40, 1, 3, 4),
    (512, 170, 1, 20, 0, 3, 3), (512, 61, 7, 20, 0, 8, 7), (33, 700, 4, 20, 0, 5, 3), (4096, 7, 1, 2, 0, 100, 1),
    (4096, 2, 11, 3, 0, 100, 3), (1, 9000, 9, 2, 0, 4, 2),
])
@pytest.mark.parametrize("pinned", [True, False])
def test_chunks_equal_one_device_run(p2r, torch, bsize, nb, nevts, nlayer, mode, nchunks, chunks, pinned):
    cfg, trk, hit, want = make(p2r, torch, bsize, nb, nevts, nlayer, mode, chunks)
    host = [trk, hit, torch.full_like(trk, 7.0)]
    if pinned:
        host = [t.pin_memory() for t in host]
    dev = [Guarded(torch, t.numel(), torch.float32) for t in host]
    for d in dev:
        d.t.fill_(float("nan"))  # what is not copied may not be read
    p2r.forward_host(cfg, *[h.numpy() for h in host], *[d.t for d in dev], nchunks=nchunks)
    torch.cuda.synchronize()
    assert np.array_equal(bits(host[2]), want)
    assert all(d.intact() for d in dev)
    copied = np.isfinite(dev[1].t.cpu().numpy().reshape(cfg.nblocks, nlayer, -1)).all(2)
    assert copied[:, -1].all()
    assert copied[:, :-1].all() if mode == p2r.MODE_CHAINED else not copied[:, :-1].any()


@pytest.mark.parametrize("mode", [0, 1])
def test_two_threads_in_place_on_the_host(p2r, torch, mode):
    """Both threads' calls share the pool; the output overwrites the host's input tracks."""
    cases = []
    for seed in (11, 12):
        cfg, trk, hit, want = make(p2r, torch, 512, 60 if mode else 250, 1, 20, mode, 4, seed)
        dev = [torch.empty(t.shape, device="cuda") for t in (trk, hit, trk)]
        cases.append((cfg, trk, trk.pin_memory(), hit.pin_memory(), dev, torch.cuda.Stream(), want))
    torch.cuda.synchronize()
    bad = []

    def work(cfg, trk, h_t, h_h, dev, stream, want):
        try:
            for _ in range(4):
                h_t.copy_(trk)
                p2r.forward_host(cfg, h_t.numpy(), h_h.numpy(), h_t.numpy(), *dev, nchunks=4, stream=stream)
                stream.synchronize()
                if not np.array_equal(bits(h_t), want):
                    bad.append("result")
        except Exception as exc:  # reported below
            bad.append(exc)

    threads = [threading.Thread(target=work, args=c) for c in cases]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad

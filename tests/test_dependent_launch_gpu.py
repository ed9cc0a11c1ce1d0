"""Kernels are launched so that each may be set up while the one before it on the stream runs, and begin by
waiting for it. These tests hold memory to the stream's order where the predecessor is something else:
work of the legacy default stream before and after a blocking stream, an event of another stream, and, in
a captured graph, copies, memsets and the join of two branches. Bit for bit against the plain order."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SLEEP = 4_000_000  # clocks, about 2 ms


@pytest.fixture(scope="module")
def torch():
    import torch as t
    return t


def bits(t):
    return t.detach().cpu().contiguous().numpy().reshape(-1).view(np.int32)


def same(a, b):
    return np.array_equal(bits(a), bits(b))


@pytest.fixture
def case(p2r, torch):
    cfg = p2r.Config(bsize=32, nlayer=6, nevts=1, nb=40, bz=3.8)
    trk, hit = p2r.generate_helix_device(cfg, p2r.gen_params(bz=3.8, seed=8))
    want = torch.empty_like(trk)
    p2r.forward(cfg, trk, hit, want)
    torch.cuda.synchronize()
    return cfg, trk, hit, want


@pytest.fixture
def blocking_stream(torch):
    """A stream that the legacy default stream waits for and that waits for it (torch's own do not)."""
    path = next(line.split()[-1] for line in open("/proc/self/maps") if "libcudart.so" in line)
    rt, handle = ctypes.CDLL(path), ctypes.c_void_p()
    torch.cuda.synchronize()
    assert rt.cudaStreamCreate(ctypes.byref(handle)) == 0
    yield handle.value
    torch.cuda.synchronize()
    assert rt.cudaStreamDestroy(handle) == 0


@pytest.mark.parametrize("call", ["forward", "layers"])
def test_legacy_default_and_blocking_stream(p2r, torch, case, blocking_stream, call):
    cfg, trk, hit, want = case
    assert torch.cuda.current_stream().cuda_stream == 0
    run = p2r.forward if call == "forward" else p2r.run_layers
    src, out = torch.full_like(trk, float("nan")), torch.empty_like(trk)
    for _ in range(3):
        src.fill_(float("nan"))
        torch.cuda._sleep(SLEEP)
        src.copy_(trk)
        run(cfg, src, hit, out, stream=blocking_stream)
        src2 = out.clone()  # on the default stream: after the call's kernels
        src.fill_(float("nan"))
        run(cfg, trk, hit, out, stream=blocking_stream)
        torch.cuda.synchronize()
        assert same(src2, want) and same(out, want)


def test_event_of_another_stream_between_two_kernels(p2r, torch, case):
    cfg, trk, hit, want = case
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    mid, src, out = torch.empty_like(trk), torch.full_like(trk, float("nan")), torch.empty_like(trk)
    torch.cuda.synchronize()
    p2r.forward(cfg, trk, hit, mid, stream=a)
    with torch.cuda.stream(b):
        torch.cuda._sleep(SLEEP)
        src.copy_(trk)
    a.wait_stream(b)
    p2r.forward(cfg, src, hit, out, stream=a)  # its predecessor on the stream is a kernel of the library
    torch.cuda.synchronize()
    assert same(mid, want) and same(out, want)


def test_capture_after_memory_nodes_and_a_join(p2r, torch, case):
    """Copy and memset nodes before the kernels, a fork and a join around them, adjoint and queue after."""
    cfg, trk, hit, want = case
    gc = torch.ones(cfg.ntracks, device="cuda")
    ref = p2r.forward_backward(cfg, trk, hit, grad_chi2=gc, ckpt_stride=1)
    off = np.array([0, 15, cfg.nblocks], np.int64)
    w = dict(nlay_lane=np.full(cfg.ntracks, cfg.nlayer, np.int32), event_block_offset=off,
             ntrk_event=np.array([15 * 32, 25 * 32]), nblocks=cfg.nblocks, bsize=32, nlayer=cfg.nlayer, bz=cfg.bz,
             updates=cfg.ntracks * cfg.nlayer)
    q = p2r.Queue(w, blocks_per_item=3)
    src, fwd, lay, que = (torch.full_like(trk, 5.0) for _ in range(4))
    adj = p2r.forward_backward(cfg, trk, hit, grad_chi2=gc, ckpt_stride=1)  # its buffers are reused below
    qadj = q.run_adjoint(trk, hit, grad_chi2=gc)
    side, fork, g = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=side):
        src.copy_(trk)
        fwd.zero_()
        fork.wait_stream(side)
        p2r.forward(cfg, src, hit, fwd, stream=side)
        p2r.run_layers(cfg, src, hit, lay, stream=fork)
        side.wait_stream(fork)
        p2r.forward_backward(cfg, src, hit, grad_chi2=gc, ckpt_stride=1, out=adj)
        que.zero_()
        q.run(src, hit, que)
        q.run_adjoint(src, hit, grad_chi2=gc, out=qadj)
        src.zero_()
    names = ("trk_out", "chi2", "grad_trk_in", "grad_hits")
    for _ in range(3):
        for t in (src, fwd, lay, que, *(o[k] for o in (adj, qadj) for k in names)):
            t.fill_(5.0)
        g.replay()
        torch.cuda.synchronize()
        assert same(fwd, want) and same(lay, want) and same(que, want) and not src.any()
        for o in (adj, qadj):
            assert all(same(o[k], ref[k]) for k in names)
        assert torch.equal(adj["grad_dr"], ref["grad_dr"])

"""The masked forward ordered by layer count, at batch sizes above the line from which it is ordered at
all (12 groups of 32 tracks per SM; below it the flag runs the unordered kernel): every block width that
has an instance of its own and widths taken at run time, both CTA sizes, chunks that are partly filled,
with and without chi2, radius offsets and wrapped phi. Bit for bit against the unordered kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def line():
    import torch
    return 12 * 32 * torch.cuda.get_device_properties(0).multi_processor_count


def compare(p2r, bsize, ntracks_over, threads, chi2, options, nlayer=4):
    """Ordered against unordered on the fewest blocks that hold line() + ntracks_over tracks."""
    import torch
    nb = -(-(line() + ntracks_over) // bsize)
    cfg = p2r.Config(bsize=bsize, nlayer=nlayer, nevts=1, nb=nb, bz=3.8, block_threads=threads)
    assert cfg.ntracks > line()
    trk, hit = p2r.generate_helix_device(cfg, p2r.gen_params(bz=3.8, seed=17))
    nlay = torch.randint(0, nlayer + 2, (cfg.ntracks,), dtype=torch.int32, device="cuda")  # one more than there are
    dr = torch.linspace(-0.01, 0.01, nlayer, device="cuda") if options else None
    got = []
    for flag in (0, p2r.FLAG_ORDER_BY_LAYERS):
        cfg.flags = flag | (p2r.FLAG_SQUASH_PHI if options else 0)
        out = torch.full_like(trk, float("nan"))
        c2 = torch.full((cfg.ntracks,), float("nan"), device="cuda") if chi2 else None
        p2r.forward(cfg, trk, hit, out, chi2=c2, dr=dr, nlay_lane=nlay)
        got.append([t.cpu().numpy().reshape(-1).view(np.int32) for t in (out, c2) if t is not None])
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("chi2,options", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("threads", [64, 128])
@pytest.mark.parametrize("bsize", [32, 64, 96, 128, 256])
def test_ordered_equals_unordered(p2r, bsize, threads, chi2, options):
    compare(p2r, bsize, 5 * bsize + 1, threads, chi2, options)


@pytest.mark.parametrize("bsize,threads", [(32, 128), (64, 128), (128, 64), (512, 64)])
def test_smallest_ordered_batch(p2r, bsize, threads):
    compare(p2r, bsize, 1, threads, True, False)


@pytest.mark.parametrize("nlayer", [1, 64])
def test_fewest_and_most_layers(p2r, nlayer):
    compare(p2r, 128, 1000, 128, True, True, nlayer=nlayer)

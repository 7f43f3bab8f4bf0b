"""The y passes of the prime-factor lengths (478 and 678 points) where they can
go wrong: odd and even depths, rows whose planes start on different halves of a
word, cut and thin tiles, uint16 and float32, with and without a flat field,
whole rows with and without the box mean, and the read windows."""
import numpy as np
import pytest
import torch

from oracle import deconv as od

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _volume(Z, X, Y, seed):
    from mermake_gb300 import synth
    return synth.hyb_stack(Z, X, Y, max(20, X * Y // 2000), seed, device="cpu", sigma_z=2.0)


@pytest.mark.parametrize("ts,Z,X,Y,zpad,dtype,flat,blur", [
    (300, 3, 351, 413, 2, "uint16", True, 30),   # X Y odd: the two planes of a line differ in alignment
    (300, 4, 300, 389, 3, "uint16", False, None),  # one tile along x, a last tile of 89
    (300, 5, 302, 640, 1, "float32", True, 31),  # a last tile of two rows
    (500, 2, 501, 530, 1, "uint16", True, None),
    (500, 3, 612, 502, 2, "float32", False, 50),
])
def test_tiles_of_the_prime_factor_lengths_match_the_oracle(ts, Z, X, Y, zpad, dtype, flat, blur):
    """Every voxel of every tile.  The passes do about 3 transforms of 50
    roundings (6e-8) in sequence, each on values below the largest: 1e-5 of the
    largest voxel leaves them all adding up."""
    from mermake_gb300 import deconvolver, synth
    img = _volume(Z, X, Y, 7 * ts + Z)
    if dtype == "float32":
        img = img.to(torch.float32)
    gain = synth.flat_gain(X, Y) if flat else None
    psf = synth.gaussian_psf((5, 9, 9), 1.2, 1.3)
    args = dict(tile_size=ts, zpad=zpad, overlap=89, beta=0.01)
    dec = deconvolver.Deconvolver(psf, (Z, X, Y), **args)
    ref = od.Deconvolver(psf, (Z, X, Y), **args)
    got = dec.tile_wise(img.cuda(), None if gain is None else torch.from_numpy(gain).cuda(), blur)
    for (x, y, tile, _), (_, _, want, _) in zip(got, ref.tile_wise(img.numpy(), gain, blur)):
        err = np.abs(tile.cpu().numpy() - want).max() / np.abs(want).max()
        assert tile.shape == want.shape and err < 1e-5, (x, y, err)


@pytest.mark.parametrize("ts,Z,X,Y", [(300, 5, 613, 701), (500, 10, 1003, 590)])
def test_read_windows_hold_the_same_voxels_as_whole_rows(ts, Z, X, Y):
    """The DAPI block stitches from the windowed pass; apply with the folded
    blur stitches whole rows: the same transforms, so the same bits.  The hyb
    rows of the windowed pass are those of the tiles of the whole-row pass."""
    from mermake_gb300 import _lib, deconvolver, maxima, pipeline, synth
    img = _volume(Z, X, Y, ts).cuda()
    a = dict(tile_size=ts, zpad=Z - 1, overlap=89, beta=0.01, blur_radius=30, threshold=2000.0, delta=1, delta_fit=3)
    dec = deconvolver.Deconvolver(synth.gaussian_psf((5, 9, 9), 1.2, 1.3), (Z, X, Y), **a)
    buf = torch.empty((Z, X, Y), dtype=torch.float32, device="cuda")
    pipeline.dapi_spots(dec, img, None, buffer=buf, **dict(a, threshold=3.0))
    whole = torch.zeros_like(buf)
    with _lib.blur_mode(_lib.MM_BLUR_SPECTRAL):
        dec.apply(img, None, blur_radius=30, output=whole)
        rows = []
        for x, y, tile, raw in dec.tile_wise(img, None, 30):
            r = maxima.find_local_maxima(tile, raw=raw, **a)
            hi = torch.tensor([tile.shape[1] - 89, tile.shape[2] - 89], device=r.device)
            r = r[torch.all((r[:, 1:3] >= 89) & (r[:, 1:3] < hi), dim=-1)]
            r[:, 1] += x - 89
            r[:, 2] += y - 89
            rows.append(r.cpu().numpy())
    assert torch.equal(buf, whole)
    got = pipeline.hyb_spots(dec, img, None, **a).cpu().numpy()
    want = np.concatenate(rows)
    assert len(want) > 20 and got.shape == want.shape
    np.testing.assert_array_equal(got[np.lexsort(got.T)], want[np.lexsort(want.T)])

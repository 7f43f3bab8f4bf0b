"""The stitched centre: written straight from the inverse pass with the blur
folded, none, or truncated, at fields whose tiles cover them and that leave
gaps."""
import numpy as np
import pytest
import torch

from oracle import deconv as od

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("X,Y,ts,ov", [(130, 97, 40, 12),   # covered
                                       (45, 90, 40, 12),    # a cut first tile: columns that no tile writes
                                       (311, 401, 300, 89), (400, 505, 500, 89)])
@pytest.mark.parametrize("blur", [None, 9])
def test_apply_and_dapi_buffer_match_the_oracle_where_tiles_write(X, Y, ts, ov, blur):
    """float32 passes against the 64-bit oracle: 1e-5 of the largest voxel, as for
    the tiles.  The DAPI buffer is zero where no tile writes, apply leaves the
    caller's values there."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mermake_gb300 import deconvolver, pipeline, synth
    Z = 5
    img = synth.hyb_stack(Z, X, Y, X * Y // 400, seed=X, sigma_z=2.0)
    psf = synth.gaussian_psf((5, 7, 7), 1.2, 1.3)
    args = dict(tile_size=ts, zpad=4, overlap=ov, beta=0.01)
    want = od.Deconvolver(psf, (Z, X, Y), **args).apply(img.numpy(), None, blur)
    there = ~np.isnan(want)
    dec = deconvolver.Deconvolver(psf, (Z, X, Y), **args)
    for batch in (None, 1):
        out = torch.full((Z, X, Y), -7.0, device="cuda")
        dec.apply(img.cuda(), None, blur_radius=blur, output=out, batch=batch)
        got = out.cpu().numpy()
        assert np.abs(got[there] - want[there]).max() < 1e-5 * np.abs(want[there]).max()
        assert np.all(got[~there] == -7.0)
    buf = torch.full((Z, X, Y), -7.0, device="cuda")
    pipeline.dapi_spots(dec, img.cuda(), None, buffer=buf, blur_radius=blur, threshold=3.0, delta=1, delta_fit=1)
    got = buf.cpu().numpy()
    assert np.abs(got[there] - want[there]).max() < 1e-5 * np.abs(want[there]).max()
    assert np.all(got[~there] == 0.0)


@pytest.mark.parametrize("Z,X,Y", [(2, 40, 40), (5, 80, 77), (7, 123, 131), (30, 300, 256)])
def test_dapi_rms_over_whole_and_cut_rounds_of_the_sum(Z, X, Y):
    """The divisor is the root of a sum of squares accumulated beyond float32,
    rounded to float32 three times: 2e-7 of it."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mermake_gb300 import deconvolver, pipeline, synth
    img = synth.dapi_stack(Z, X, Y, seed=X, n_nuclei=6)
    dec = deconvolver.Deconvolver(synth.gaussian_psf((5, 7, 7), 1.2, 1.3), (Z, X, Y), tile_size=40, zpad=1, overlap=9,
                                  beta=0.01)
    _, _, buf, rms = pipeline.dapi_spots(dec, img.cuda(), None, threshold=3.0, delta=1, delta_fit=1)
    v = buf.cpu().numpy().astype(np.float64)
    want = np.sqrt((v * v).sum() / v.size)
    assert abs(rms - want) <= 2e-7 * want

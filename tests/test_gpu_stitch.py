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

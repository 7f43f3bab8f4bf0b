"""The register z operator over one spectrum at every batch size its plans
differ for, at depths of whole and of cut row groups."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Z,zpad", [(50, 49), (50, 24), (37, 36), (37, 18), (12, 11), (7, 2), (3, 1), (64, 63)])
@pytest.mark.parametrize("ts,ov", [(14, 3), (30, 9)])  # planes of 2 and of 0 mod 8 frequencies
def test_register_form_over_batch_sizes(Z, zpad, ts, ov):
    """Against the transforms over the padded depth (2e-5 of the largest voxel,
    as for the other forms).  Where the matrix forms take every batch, the same
    bits for every batch size: each output sums its columns in the same order."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mermake_gb300 import _lib, deconvolver, synth
    X, Y = 4 * ts - 1, 4 * ts
    img = synth.hyb_stack(Z, X, Y, 40, seed=Z + ts).cuda()
    dec = deconvolver.Deconvolver(synth.gaussian_psf((5, 7, 7), 1.2, 1.3), (Z, X, Y), tile_size=ts, zpad=zpad, overlap=ov,
                                  beta=0.01)
    with _lib.zform(_lib.MM_ZFORM_TRANSFORMS):
        want = dec.apply(img, None)
    transforms = 26 <= Z <= 56 and (zpad == Z - 1 or 2 * zpad == Z - 2)  # from four tiles on
    first = None
    with _lib.zform(_lib.MM_ZFORM_REGISTERS):
        for batch in (1, 2, 3, 4, 5, 6, 9, 11, 16):
            got = dec.apply(img, None, batch=batch)
            err = (got - want).abs().max() / want.abs().max()
            assert err < 2e-5, (batch, float(err))
            first = got if first is None else first
            assert transforms or torch.equal(got, first), batch
    # the library's own choice: one tile takes the per-tile form where it can
    assert torch.equal(dec.apply(img, None, batch=1), first)


@pytest.mark.parametrize("Z", [25, 26, 30, 31, 35, 36, 40, 41, 45, 46, 50, 51, 56, 57])
@pytest.mark.parametrize("near", [False, True])
def test_short_transforms_at_the_edges_of_their_lengths(Z, near):
    """The first and last depth of every length (and the depths beside them),
    both paddings, planes that end inside a group of 64 frequencies, batches of
    whole and of cut rounds, with and without the folded blur: against the
    transforms over the padded depth, 2e-5 of the largest voxel as above.  A
    tile's bits do not depend on its batch."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mermake_gb300 import _lib, deconvolver, synth
    if near and Z % 2:
        pytest.skip("no such padding at an odd depth")
    for ts, ov in ((14, 3), (30, 9)):
        X, Y = 4 * ts - 1, 3 * ts
        img = synth.hyb_stack(Z, X, Y, 40, seed=Z + ts).cuda()
        dec = deconvolver.Deconvolver(synth.gaussian_psf((5, 7, 7), 1.2, 1.3), (Z, X, Y), tile_size=ts,
                                      zpad=(Z - 2) // 2 if near else Z - 1, overlap=ov, beta=0.01)
        for blur in (None, 6):
            mode = _lib.MM_BLUR_EXACT if blur is None else _lib.MM_BLUR_SPECTRAL
            got = {}
            with _lib.blur_mode(mode):
                with _lib.zform(_lib.MM_ZFORM_DIRECT):
                    want = dec.apply(img, None, blur_radius=blur)
                for batch in (4, 6, 12):
                    got[batch] = dec.apply(img, None, blur_radius=blur, batch=batch)
            err = (got[12] - want).abs().max() / want.abs().max()
            assert err < 2e-5, (ts, blur, float(err))
            assert torch.equal(got[4], got[12]) and torch.equal(got[6], got[12]), (ts, blur)


@pytest.mark.parametrize("Z", [26, 31, 37, 39, 41, 46, 49, 51, 56])  # no multiples of 5: those have their own form
@pytest.mark.parametrize("near", [False, True])
def test_short_transforms_with_a_kernel_per_tile(Z, near):
    """A PSF per tile at depths of every length: against the direct sum (2e-5 of
    the largest voxel), planes that end inside a group of 32 frequencies, batches
    past tile 0, and the same bits for every batch."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mermake_gb300 import _lib, deconvolver, synth
    if near and Z % 2:
        pytest.skip("no such padding at an odd depth")
    for ts, ov in ((14, 3), (30, 9)):
        X, Y = 3 * ts - 1, 2 * ts
        img = synth.hyb_stack(Z, X, Y, 40, seed=Z + ts).cuda()
        psfs = {i: synth.gaussian_psf((5, 7, 7), 1.0 + 0.1 * i, 1.1 + 0.05 * i) for i in range(6)}
        dec = deconvolver.Deconvolver(psfs, (Z, X, Y), tile_size=ts, zpad=(Z - 2) // 2 if near else Z - 1, overlap=ov,
                                      beta=0.01)
        for blur in (None, 6):
            with _lib.blur_mode(_lib.MM_BLUR_EXACT if blur is None else _lib.MM_BLUR_SPECTRAL):
                with _lib.zform(_lib.MM_ZFORM_DIRECT):
                    want = dec.apply(img, None, blur_radius=blur)
                got = {b: dec.apply(img, None, blur_radius=blur, batch=b) for b in (1, 4, 6)}
            err = (got[6] - want).abs().max() / want.abs().max()
            assert err < 2e-5, (ts, blur, float(err))
            assert torch.equal(got[1], got[6]) and torch.equal(got[4], got[6]), (ts, blur)

"""The register z operator over one spectrum at every batch size its plans
differ for, at depths of whole and of cut row groups."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Z,zpad", [(50, 49), (50, 24), (37, 36), (37, 18), (12, 11), (7, 2), (3, 1), (64, 63)])
@pytest.mark.parametrize("ts,ov", [(14, 3), (30, 9)])  # planes of 2 and of 0 mod 8 frequencies
def test_register_form_over_batch_sizes(Z, zpad, ts, ov):
    """Against the transforms over the padded depth (2e-5 of the largest voxel,
    as for the other forms), and the same bits for every batch size: each
    output sums its columns in the same order."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mermake_gb300 import _lib, deconvolver, synth
    X, Y = 4 * ts - 1, 4 * ts
    img = synth.hyb_stack(Z, X, Y, 40, seed=Z + ts).cuda()
    dec = deconvolver.Deconvolver(synth.gaussian_psf((5, 7, 7), 1.2, 1.3), (Z, X, Y), tile_size=ts, zpad=zpad, overlap=ov,
                                  beta=0.01)
    with _lib.zform(_lib.MM_ZFORM_TRANSFORMS):
        want = dec.apply(img, None)
    first = None
    with _lib.zform(_lib.MM_ZFORM_REGISTERS):
        for batch in (1, 2, 3, 4, 5, 6, 9, 11, 16):
            got = dec.apply(img, None, batch=batch)
            err = (got - want).abs().max() / want.abs().max()
            assert err < 2e-5, (batch, float(err))
            first = got if first is None else first
            assert torch.equal(got, first), batch
    # the library's own choice: one tile takes the per-tile form where it can
    assert torch.equal(dec.apply(img, None, batch=1), first)

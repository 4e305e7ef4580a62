"""Split batches whose scales take both ways through the transform stages (large
ones map by map, the small ones a chunk of maps per launch), with maps left
over from whole chunks and groups, and single maps: against the FP64 form on the same
maps, at test_gpu_split.py's bounds."""
import pytest
from test_gpu_split import TOL_RECON, TOL_W, _run


@pytest.mark.gpu
@pytest.mark.parametrize("B,N,alpha,nmaps", [
    (512, 4, 2.0, 3),   # bl = 512 alone (33 MB per map), the rest in one chunk
    (512, 4, 2.0, 5),
    (256, 5, 2.0, 5),   # chunks of two maps and one left over
    (150, 8, 2.0, 34),  # two groups of maps, the second smaller than a chunk
    (300, 1, 2.0, 1),   # one map: the larger scales apart
    (300, 4, 2.0, 1),
    (512, 1, 2.0, 1),
])
def test_split_batches_match_fp64(B, N, alpha, nmaps):
    worst, recon, syn = _run(B, N, alpha, nmaps)
    assert worst <= TOL_W, f"max|dw|/max|w| = {worst:.3e}"
    assert syn <= TOL_W, f"max|dflm|/max|flm| = {syn:.3e}"
    assert recon <= TOL_RECON, f"recon {recon:.3e}"

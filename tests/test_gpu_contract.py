"""The contraction kernels, which walk all scales of a transform at once: band
limits around their tiles (16 m', 8 S m, 16 P l, chunks of 16 l and 4 m'),
scales that end inside a chunk (alpha that gives ragged band limits), scales
that meet at one l, few scales (J < Jmax), and every number of n values.

Tolerance: the repository's bar for the FP64 form, 1e-12 of each scale's
max|w| and of max|flm| (about 5000 units of rounding, an l-walk of 200 steps
adds a few hundred)."""
import numpy as np
import pytest

from oracle import oracle as O
from s2dw_b200 import core
from s2dw_b200.workload import gaussian_flm, transform_setup

CASES = [
    (15, 4, 2.0, None), (16, 4, 2.0, None), (17, 4, 2.0, None), (31, 2, 1.5, None), (33, 3, 3.0, None),
    (48, 5, 1.7, None), (63, 7, 2.0, 3), (64, 8, 2.0, 1), (65, 1, 2.0, 2), (96, 6, 2.5, None), (130, 4, 3.0, 2),
    (40, 12, 2.0, None), (34, 16, 1.3, None), (431, 3, 2.0, None), (433, 4, 3.0, None), (495, 2, 2.0, None),
    (497, 1, 2.0, None), (450, 10, 2.0, 1),
]


@pytest.mark.gpu
@pytest.mark.parametrize("B,N,alpha,J", CASES)
def test_all_scale_walks_match_the_oracle(B, N, alpha, J):
    t = transform_setup(B, N, alpha, J)
    J = t["J"]
    a = (t["K_gamma"], t["Slm"], J, B, N, t["bl_scoeff"], alpha)
    f = gaussian_flm(B, seed=B + N)
    got, sc = core.s2dw_core_analysis_flm2wav_dynamic(f, *a)
    ref, scr = O.analysis_dynamic(f, *a)
    top = max(np.abs(r).max() for r in ref)
    for j, (w, r) in enumerate(zip(got, ref)):
        assert np.abs(w - r).max() <= 1e-12 * max(np.abs(r).max(), 1e-3 * top), f"scale {j}"
    np.testing.assert_array_equal(sc, scr)
    rng = np.random.default_rng(B * N)
    wav = [np.asfortranarray(rng.standard_normal(w.shape)) for w in got]
    s = (t["K_gamma"], t["Phi2"], t["Slm"], J, B, N, t["bl_scoeff"], alpha)
    fg = core.s2dw_core_synthesis_wav2flm_dynamic([w.copy(order="F") for w in wav], sc, *s)
    fo = O.synthesis_dynamic([w.copy(order="F") for w in wav], sc, *s)
    assert np.abs(fg - fo).max() <= 1e-12 * np.abs(fo).max()


@pytest.mark.gpu
@pytest.mark.parametrize("B,l", [(64, 16), (64, 17), (64, 32), (48, 12), (50, 13)])
def test_a_nan_stays_in_its_scales(B, l):
    """A coefficient that is not a number reaches only the scales whose range
    (bl_lo, bl) holds its l (at l = bl_lo of scale j that is scale j + 1
    alone), and not-a-number wavelets of one scale reach only its l."""
    N, alpha = 4, 2.0
    t = transform_setup(B, N, alpha)
    J = t["J"]
    lim = [core.band_limits(j, B, alpha) for j in range(J + 1)]
    f = gaussian_flm(B, seed=1)
    f[l, 3] = np.nan
    a = (t["K_gamma"], t["Slm"], J, B, N, t["bl_scoeff"], alpha)
    wav, sc = core.s2dw_core_analysis_flm2wav_dynamic(f, *a)
    for j, (hi, lo) in enumerate(lim):
        assert np.isnan(wav[j]).any() == (lo < l < hi), f"scale {j}: range ({lo}, {hi})"
    good, sc = core.s2dw_core_analysis_flm2wav_dynamic(gaussian_flm(B, seed=1), *a)
    s = (t["K_gamma"], t["Phi2"], t["Slm"], J, B, N, t["bl_scoeff"], alpha)
    for j, (hi, lo) in enumerate(lim):
        if hi - lo < 2:
            continue
        w = [x.copy(order="F") for x in good]
        w[j][:] = np.nan
        g = core.s2dw_core_synthesis_wav2flm_dynamic(w, sc, *s)
        rows = np.isnan(g).any(axis=1)
        for k in range(B):
            assert not rows[k] or lo < k < hi, f"scale {j}: l={k}"
        assert rows[lo + 1:hi].all()

"""The grouped transform stages at every transform length they have: beta FFTs
of 16 to 1024 points (bl = 8 ... 512), Bluestein transforms of 16 to 2048
points (other band limits, bl = 16 and 64 for alpha), the prime-factor alpha
rows, row counts that leave CTAs partly empty (odd N, odd bl), and a launch of
more scales than one holds (J = 30).

Tolerance: the repository's bar for the FP64 form, 1e-12 of each scale's
max|w| and of max|flm|."""
import numpy as np
import pytest

from oracle import oracle as O
from s2dw_b200 import core
from s2dw_b200.workload import gaussian_flm, transform_setup

CASES = [
    (5, 1, 2.0), (9, 3, 2.0), (16, 1, 2.0), (32, 5, 2.0), (37, 2, 3.0), (64, 2, 2.0), (70, 3, 1.5), (128, 3, 2.0),
    (129, 1, 2.0), (200, 2, 2.5), (256, 1, 2.0), (257, 2, 3.0), (16, 2, 1.1),
]


@pytest.mark.gpu
@pytest.mark.parametrize("B,N,alpha", CASES)
def test_stages_match_the_oracle(B, N, alpha):
    t = transform_setup(B, N, alpha)
    J = t["J"]
    f = gaussian_flm(B, seed=B)
    a = (t["K_gamma"], t["Slm"], J, B, N, t["bl_scoeff"], alpha)
    got, sc = core.s2dw_core_analysis_flm2wav_dynamic(f, *a)
    ref, _ = O.analysis_dynamic(f, *a)
    top = max(np.abs(r).max() for r in ref)
    for j, (w, r) in enumerate(zip(got, ref)):
        assert np.abs(w - r).max() <= 1e-12 * max(np.abs(r).max(), 1e-3 * top), f"scale {j}"
    rng = np.random.default_rng(B)
    wav = [np.asfortranarray(rng.standard_normal(w.shape)) for w in got]
    s = (t["K_gamma"], t["Phi2"], t["Slm"], J, B, N, t["bl_scoeff"], alpha)
    fg = core.s2dw_core_synthesis_wav2flm_dynamic([w.copy(order="F") for w in wav], sc, *s)
    fo = O.synthesis_dynamic([w.copy(order="F") for w in wav], sc, *s)
    assert np.abs(fg - fo).max() <= 1e-12 * np.abs(fo).max()


@pytest.mark.gpu
@pytest.mark.parametrize("B,N", [(512, 3), (400, 2)])
def test_grouped_and_single_scales_agree(B, N):
    """The device plan runs the scales of these sizes in one launch per
    stage, the host entry points scale by scale: the same values, bit for
    bit, and the round trip returns the map."""
    import torch

    from s2dw_b200.device import Plan

    t = transform_setup(B, N, 2.0)
    J = t["J"]
    f = gaussian_flm(B, seed=3)
    a = (t["K_gamma"], t["Slm"], J, B, N, t["bl_scoeff"], 2.0)
    host, _ = core.s2dw_core_analysis_flm2wav_dynamic(f, *a)
    plan = Plan(B, N, 2.0, J)
    plan.set_tables(t["K_gamma"], t["Phi2"], t["Slm"], t["bl_scoeff"])
    d_flm = torch.from_numpy(np.ascontiguousarray(f.T)).cuda()
    wav = torch.empty(plan.wav_size, dtype=torch.float64, device="cuda")
    sc = torch.empty(t["bl_scoeff"] ** 2, dtype=torch.complex128, device="cuda")
    out = torch.empty_like(d_flm)
    plan.analysis(d_flm, wav, sc)
    plan.synthesis(wav, sc, out)
    torch.cuda.synchronize()
    for j in range(J + 1):
        np.testing.assert_array_equal(plan.scale_view(wav, j).cpu().numpy().transpose(2, 1, 0), host[j])
    assert np.abs(out.cpu().numpy().T - f).max() <= 1e-10
    plan.close()


@pytest.mark.gpu
@pytest.mark.parametrize("B,N", [(48, 2), (1024, 1)])
def test_priority_plan_on_other_streams(B, N):
    """A plan with a priority runs on its own stream when the caller's has
    another: the same values bit for bit, ordered with the caller's stream,
    directly and from a CUDA graph."""
    import torch

    from s2dw_b200.device import Plan

    t = transform_setup(B, N, 2.0)
    plan = Plan(B, N, 2.0, t["J"])
    plan.set_tables(t["K_gamma"], t["Phi2"], t["Slm"], t["bl_scoeff"])
    bs = t["bl_scoeff"]
    src = torch.from_numpy(np.ascontiguousarray(gaussian_flm(B, seed=4).T)).cuda()
    flm = torch.zeros_like(src)
    wav = torch.empty(plan.wav_size, dtype=torch.float64, device="cuda")
    sc = torch.empty((bs, bs), dtype=torch.complex128, device="cuda")
    back = torch.empty_like(src)

    def run():
        flm.copy_(src)
        plan.analysis(flm, wav, sc)
        plan.synthesis(wav, sc, back)
        out = wav.clone(), back.clone()
        wav.zero_()
        flm.zero_()
        return out

    ref = run()
    plan.set_priority(-1)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        got = run()
    s.synchronize()
    assert all(torch.equal(x, y) for x, y in zip(got, ref))
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = run()
    g.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(x, y) for x, y in zip(got, ref))

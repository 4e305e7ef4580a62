"""The contractions' larger tiles and the walks per scale, which the oracle
is too slow for, against direct sums in 64 bits on the GPU (perf/cases.py:
Wigner d functions at the sample angles and torch.fft, no code of the library):
every tile of the analysis and the synthesis kernel at NP = 3 ... 8, and the
band limits on both sides of the rules that choose them.

Tolerance 1e-11 of each scale's max|w| and of max|flm|: the repository's bar
against the oracle is 1e-12, and the direct sums' own three-term recurrence
adds about ten units of rounding per step, 840 x 10 x 1.1e-16 = 1e-12, on either
side of a product."""
import numpy as np
import pytest

CASES = [
    # B, N, alpha
    (440, 5, 3.0), (500, 8, 3.0), (440, 7, 4.0), (840, 6, 4.0), (840, 8, 4.0),  # NP = 3, 4: 2 x 2 and 2 x 4 tiles
    (840, 9, 4.0), (832, 12, 4.0),                                             # NP = 5, 6, the largest tile
    (512, 14, 4.0), (513, 13, 4.0), (520, 15, 4.0), (833, 14, 4.0), (840, 16, 4.0),  # NP = 7, 8: one walk, one per scale
]


@pytest.mark.gpu
@pytest.mark.parametrize("B,N,alpha", CASES)
def test_large_tiles_match_direct_sums(B, N, alpha):
    from perf import cases

    case = {"kind": "pair", "B": B, "N": N, "alpha": alpha, "maps": 1}
    state = cases.prepare(case, 7)
    got = {k: v.cpu() for k, v in cases.run(state).items()}
    plan = state["plan"]
    ref = {k: v.cpu() for k, v in cases.exact(case, 7).items()}
    off = plan.wav_offsets
    for j in range(plan.J + 1):
        w, r = got["wav"][off[j]:off[j + 1]], ref["wav"].reshape(-1)[off[j]:off[j + 1]]
        assert float((w - r).abs().max()) <= 1e-11 * float(r.abs().max()), f"scale {j}"
    assert float((got["flm"] - ref["flm"]).abs().max()) <= 1e-11 * float(ref["flm"].abs().max())
    np.testing.assert_array_equal(got["scoeff"].numpy(), ref["scoeff"].numpy().reshape(got["scoeff"].shape))
    plan.close()


@pytest.mark.gpu
def test_walks_per_scale_of_a_general_slm():
    """The second pass of the walks per scale (a complex Slm that
    init_directionality does not make): the coefficients are real-linear in S, so those of
    a + i b are the sum of those of a (one pass) and of i b (both passes, the first with
    zero tables); and every launch alone (timing mode) gives the same values."""
    import torch

    from s2dw_b200.device import Plan
    from s2dw_b200.workload import gaussian_flm, transform_setup

    B, N = 520, 14
    t = transform_setup(B, N, 4.0)
    bs = t["bl_scoeff"]
    rng = np.random.default_rng(3)
    a, b = (np.asfortranarray(t["Slm"] * rng.uniform(0.5, 1.5, (B, 1))) for _ in range(2))
    flm = torch.from_numpy(np.ascontiguousarray(gaussian_flm(B, seed=2).T)).cuda()
    wav = {}
    for name, S, timing in (("a", a, False), ("ab", a + 1j * b, False), ("again", a + 1j * b, True),
                            ("jb", 1j * b, False)):
        plan = Plan(B, N, 4.0, t["J"])
        plan.set_tables(t["K_gamma"], t["Phi2"], S, bs)
        plan.set_timing(timing)
        w = torch.empty(plan.wav_size, dtype=torch.float64, device="cuda")
        sc = torch.empty(bs * bs, dtype=torch.complex128, device="cuda")
        plan.analysis(flm, w, sc)
        wav[name] = w.cpu().numpy()
        plan.close()
    np.testing.assert_array_equal(wav["ab"], wav["again"])
    top = np.abs(wav["ab"]).max()
    assert np.abs(wav["ab"] - wav["a"] - wav["jb"]).max() <= 1e-12 * top
    assert np.abs(wav["jb"]).max() > 0.1 * top


@pytest.mark.gpu
@pytest.mark.parametrize("B,N,alpha", [(520, 14, 4.0), (450, 2, 2.0), (512, 4, 2.0)])
def test_scales_on_their_own_streams_in_host_calls_and_graphs(B, N, alpha):
    """Walks per scale and full-band scales as groups of their own: the host entry
    points, whose groups follow their copies, and a CUDA graph of both directions give the
    device calls' values bit for bit."""
    import torch

    from s2dw_b200 import core
    from s2dw_b200.device import Plan
    from s2dw_b200.workload import gaussian_flm, transform_setup

    t = transform_setup(B, N, alpha)
    J, bs = t["J"], t["bl_scoeff"]
    f = gaussian_flm(B, seed=5)
    plan = Plan(B, N, alpha, J)
    plan.set_tables(t["K_gamma"], t["Phi2"], t["Slm"], bs)
    flm = torch.from_numpy(np.ascontiguousarray(f.T)).cuda()
    wav = torch.empty(plan.wav_size, dtype=torch.float64, device="cuda")
    sc = torch.empty(bs * bs, dtype=torch.complex128, device="cuda")
    out = torch.empty_like(flm)
    plan.analysis(flm, wav, sc)
    plan.synthesis(wav, sc, out)
    torch.cuda.synchronize()
    host, hsc = core.s2dw_core_analysis_flm2wav_dynamic(f, t["K_gamma"], t["Slm"], J, B, N, bs, alpha)
    for j in range(J + 1):
        np.testing.assert_array_equal(plan.scale_view(wav, j).cpu().numpy().transpose(2, 1, 0), host[j])
    back = core.s2dw_core_synthesis_wav2flm_dynamic(host, hsc, t["K_gamma"], t["Phi2"], t["Slm"], J, B, N, bs, alpha)
    np.testing.assert_array_equal(back, out.cpu().numpy().T)
    w2, s2, o2 = torch.zeros_like(wav), torch.zeros_like(sc), torch.zeros_like(out)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        plan.analysis(flm, w2, s2)
        plan.synthesis(w2, s2, o2)
    for _ in range(2):
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(w2, wav) and torch.equal(o2, out)
    del g
    plan.close()

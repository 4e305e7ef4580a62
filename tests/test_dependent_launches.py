"""Programmatic dependent launches: a kernel may start before the one in front
of it on its stream has finished, and may touch what earlier kernels write
only after its own griddepcontrol.wait (pdl_wait)."""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "s2dw_b200", "csrc")


def _kernels():
    """{name: body} of the __global__ functions."""
    out = {}
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
            for m in re.finditer(r"__global__ void (?:__launch_bounds__\((?:[^()]|\((?:[^()]|\([^()]*\))*\))*\) )?(\w+)\(",
                                 src):
                i = src.index("{", m.end())
                depth, k = 1, i + 1
                while depth:
                    depth += {"{": 1, "}": -1}.get(src[k], 0)
                    k += 1
                out[m.group(1)] = src[i:k]
    return out


def test_every_dependent_kernel_waits_unconditionally():
    """The kernels that launch_dep launches: a wait at the top level of the
    kernel or of what it calls first, never behind a condition on an argument."""
    src = "".join(open(os.path.join(CSRC, f)).read() for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh", ".h")))
    assert not re.search(r"\bif\s*\([^;{}]*\)\s*pdl_wait", src)
    k = _kernels()
    for name in ("pfa1023_kernel", "alpha_kernel"):
        body = k[name]
        assert re.search(r"^    pdl_wait\(\);", body, re.M), name
        assert body.index("pdl_wait();") < body.index("alpha_rows_in" if name == "pfa1023_kernel" else "rows_run"), name


@pytest.mark.gpu
@pytest.mark.parametrize("B,N", [(512, 1), (512, 2), (1024, 1)])
def test_overlapped_stages_see_the_new_input(B, N):
    """Transforms whose stages are several dependent launches, with other
    inputs each time and nothing waited for between them: the same values, bit for
    bit, as with every launch alone (timing mode), never those of the call before."""
    import torch

    from s2dw_b200.device import Plan
    from s2dw_b200.workload import gaussian_flm, transform_setup

    t = transform_setup(B, N, 2.0)
    bs = t["bl_scoeff"]
    reps = 12
    plan = Plan(B, N, 2.0, t["J"])
    plan.set_tables(t["K_gamma"], t["Phi2"], t["Slm"], bs)
    base = torch.from_numpy(np.ascontiguousarray(gaussian_flm(B, seed=6).T)).cuda()
    flm = [base * (1.0 + 0.25 * k) for k in range(reps)]
    wav = [torch.empty(plan.wav_size, dtype=torch.float64, device="cuda") for _ in range(reps)]
    sc = [torch.empty(bs * bs, dtype=torch.complex128, device="cuda") for _ in range(reps)]
    out = [torch.empty_like(base) for _ in range(reps)]
    torch.cuda.synchronize()
    for k in range(reps):
        plan.analysis(flm[k], wav[k], sc[k])
        plan.synthesis(wav[k], sc[k], out[k])
    plan.set_timing(True)
    w, s, o = torch.empty_like(wav[0]), torch.empty_like(sc[0]), torch.empty_like(base)
    for k in range(reps):
        plan.analysis(flm[k], w, s)
        plan.synthesis(w, s, o)
        assert torch.equal(w, wav[k]) and torch.equal(o, out[k]), k
    plan.close()

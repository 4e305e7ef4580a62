"""The host side of the library on a stand-in CUDA runtime (fake_cudart.cpp,
preloaded into a child process): what a call leaves behind when the runtime
refuses one of its steps, which launches it queues and how they are ordered.
Nothing here needs a GPU and no kernel runs."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fake") / "fake_cudart.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I/usr/local/cuda/include",
                    os.path.join(HERE, "fake_cudart.cpp"), "-o", out], check=True)
    return out


def run(fake, name, *args):
    r = subprocess.run([sys.executable, os.path.abspath(__file__), name, *map(str, args)], capture_output=True, text=True,
                       env=dict(os.environ, LD_PRELOAD=fake, OMP_NUM_THREADS="2", PYTHONPATH=os.path.dirname(HERE)))
    assert r.returncode == 0, r.stdout + r.stderr


# ---- in the child ----------------------------------------------------------
def _fake():
    f = ctypes.CDLL(None)
    f.fake_log.restype = ctypes.c_char_p
    f.fake_fail.argtypes = [ctypes.c_char_p, ctypes.c_int]
    f.fake_pin.argtypes = [ctypes.c_void_p, ctypes.c_size_t]
    return f


class Plan:
    """s2dw_b200.device.Plan without torch, on host buffers."""

    def __init__(self, B, N, form=0):
        from s2dw_b200._lib import check, lib
        from s2dw_b200.workload import transform_setup

        self.t = t = transform_setup(B, N, 2.0)
        self.B, self.J, self.bs = B, t["J"], t["bl_scoeff"]
        self.L, self.check, self.h = lib(), check, ctypes.c_void_p()
        check(self.L.s2dwc_plan_create(ctypes.byref(self.h), B, N, 2.0, self.J, form, 0))
        offs = (ctypes.c_longlong * (self.J + 2))()
        check(self.L.s2dwc_plan_wav_offsets(self.h, offs))
        self.size = offs[self.J + 1]
        check(self.set_tables(t["Slm"]))

    def set_tables(self, S):
        dp = ctypes.POINTER(ctypes.c_double)
        K, P = (np.asfortranarray(self.t[k]) for k in ("K_gamma", "Phi2"))
        S = np.asfortranarray(S, dtype=np.complex128)
        return self.L.s2dwc_plan_set_tables(self.h, K.ctypes.data_as(dp), P.ctypes.data_as(dp), S.ctypes.data_as(dp),
                                            self.bs)

    def reserve(self, maps):
        return self.L.s2dwc_plan_reserve(self.h, maps, None)

    def bytes(self):
        return self.L.s2dwc_plan_workspace_bytes(self.h)

    def buffers(self, maps=1):
        self.keep = [np.zeros(n * maps + 2) for n in (self.size, 2 * self.bs ** 2, 2 * self.B ** 2)]
        return [ctypes.c_void_p(a.ctypes.data) for a in self.keep]

    def close(self):
        self.L.s2dwc_plan_destroy(self.h)


def _launches(f):
    """(stream, priority, programmatic, name, grid, block) of the kernels since the last call."""
    out = []
    for line in f.fake_log().decode().splitlines():
        if line != "event":
            s, prio, dep, rest = line.split(" ", 3)
            name, grid, block = rest.rsplit(" ", 2)
            out.append((int(s), int(prio), dep == "1", name, grid, block))
    return out


def failed_reserve():
    f = _fake()

    def batch(p):
        w, s, x = p.buffers(4)
        f.fake_log()
        p.check(p.L.s2dwc_plan_analysis_batch(p.h, 4, w, s, x, None))
        p.check(p.L.s2dwc_plan_synthesis_batch(p.h, 4, x, w, s, None))
        return [k[3:] for k in _launches(f)]

    p = Plan(64, 5, form=1)
    base = p.bytes()
    assert p.reserve(4) == 0
    want, size = batch(p), p.bytes()
    p.close()
    assert len(want) > 0
    # the plan memory limit refuses the first reserve
    for extra in (1, 20000, (size - base) // 2, size - base - 1):
        p = Plan(64, 5, form=1)
        p.L.s2dwc_set_plan_memory_limit(base + extra)
        st = p.reserve(4)
        p.L.s2dwc_set_plan_memory_limit(0)
        if st:
            assert st == 4
            assert p.reserve(4) == 0
            assert p.bytes() == size and batch(p) == want, extra
        p.close()
    # so does the device, at any allocation
    failed = 0
    for n in range(1, 1000):
        p = Plan(64, 5, form=1)
        f.fake_fail(b"cudaMalloc", n)
        st = p.reserve(4)
        if f.fake_armed():  # fewer than n allocations: done
            f.fake_fail(b"cudaMalloc", 1 << 30)
            break
        if st:
            failed += 1
            assert st == 4, n
            assert p.reserve(4) == 0
            assert p.bytes() == size and batch(p) == want, n
        else:  # (the stages' workspace fell back to a smaller one)
            assert p.bytes() < size
            batch(p)
        p.close()
    assert failed > 8


def failed_buffers():
    """Tables of a general Slm, moments' and host calls' buffers: every
    allocation fails once, and the call works when it is repeated."""
    f = _fake()
    dp = ctypes.POINTER(ctypes.c_double)

    def slm():
        rng = np.random.default_rng(0)
        return rng.standard_normal((24, 4)) + 1j * rng.standard_normal((24, 4))

    def general(p):
        return p.set_tables(slm())

    def moments(p):
        w, s, x = p.buffers()
        m = ctypes.c_void_p(np.zeros((p.J + 1) * 6).ctypes.data)
        return p.L.s2dwc_plan_stat_moments(p.h, 1, w, None, m, None)

    def host(p):
        t, B = p.t, p.B
        K, S = np.asfortranarray(t["K_gamma"]), np.asfortranarray(t["Slm"])
        out = [np.zeros(p.size) for _ in range(p.J + 1)]
        sc, flm = np.zeros(2 * p.bs ** 2), np.zeros(2 * B * B)
        ptrs = (dp * (p.J + 1))(*[o.ctypes.data_as(dp) for o in out])
        return p.L.s2dwc_analysis_flm2wav_dynamic(ptrs, sc.ctypes.data_as(dp), flm.ctypes.data_as(dp), K.ctypes.data_as(dp),
                                                  S.ctypes.data_as(dp), p.J, B, 4, p.bs, 2.0)

    for call in (general, moments, host):
        p = Plan(24, 4)
        assert call(p) == 0
        size = p.bytes()
        p.close()
        for n in range(1, 1000):
            p = Plan(24, 4)
            p.L.s2dwc_finalize()
            held = f.fake_allocations()
            f.fake_fail(b"cudaMalloc", n)
            st = call(p)
            if f.fake_armed():
                f.fake_fail(b"cudaMalloc", 1 << 30)
                break
            assert st == 4
            assert call is host or f.fake_allocations() == held
            assert call(p) == 0, (call.__name__, n)
            assert p.bytes() == size
            p.close()
        assert n > 3


def failed_host_calls(alpha10):
    """Host calls on page-locked and pageable arrays in which any one runtime
    call fails: nothing of the caller's memory is still to be copied afterwards."""
    from s2dw_b200._lib import check, lib
    from s2dw_b200.workload import transform_setup

    f = _fake()
    B, N, alpha = 24, 2, alpha10 / 10
    t = transform_setup(B, N, alpha)
    J, bs = t["J"], t["bl_scoeff"]
    dp = ctypes.POINTER(ctypes.c_double)
    L = lib()
    size = [L.s2dwc_wav_scale_size(j, B, N, alpha) for j in range(J + 1)]
    K, S, P = np.asfortranarray(t["K_gamma"]), np.asfortranarray(t["Slm"]), np.ascontiguousarray(t["Phi2"])

    def arrays(pin):
        a = [np.zeros(n) for n in size] + [np.zeros(2 * B * B), np.zeros(2 * bs * bs)]
        if pin:
            for x in a:
                f.fake_pin(x.ctypes.data, x.nbytes)
        return a

    def ptr(x):
        return x.ctypes.data_as(dp)

    for pin in (True, False):
        a = arrays(pin)
        w = (dp * (J + 1))(*[ptr(x) for x in a[:J + 1]])
        flm, sc = a[-2:]
        calls = [
            lambda: L.s2dwc_analysis_flm2wav_dynamic(w, ptr(sc), ptr(flm), ptr(K), ptr(S), J, B, N, bs, alpha),
            lambda: L.s2dwc_synthesis_wav2flm_dynamic(ptr(flm), w, ptr(sc), ptr(K), ptr(P), ptr(S), J, B, N, bs, alpha),
        ]
        for call in calls:
            check(call())
            assert f.fake_pending_copies() == 0
            for name in (b"cudaLaunchKernel", b"cudaLaunchKernelExC", b"cudaMemcpyAsync", b"cudaMemcpy", b"cudaEventRecord",
                         b"cudaStreamWaitEvent", b"cudaStreamSynchronize"):
                for n in range(1, 400):
                    f.fake_fail(name, n)
                    st = call()
                    if f.fake_armed():
                        f.fake_fail(name, 1 << 30)
                        break
                    assert st != 0 and f.fake_pending_copies() == 0, (pin, name, n, st)
                    check(call())


def noalloc_timing():
    """s2dwc_plan_analysis_noalloc creates nothing, with the plan's timing on
    too, and leaves its records alone."""
    f = _fake()
    p = Plan(24, 4)
    w, s, x = p.buffers()
    p.check(p.L.s2dwc_plan_analysis_noalloc(p.h, w, s, x, None))
    f.fake_log()
    p.check(p.L.s2dwc_plan_analysis_noalloc(p.h, w, s, x, None))
    plain = f.fake_log().decode()
    assert plain and "event" not in plain
    p.L.s2dwc_plan_set_timing(p.h, 1)
    p.check(p.L.s2dwc_plan_analysis_noalloc(p.h, w, s, x, None))
    assert f.fake_log().decode() == plain
    n, ms = ctypes.c_longlong(), ctypes.c_double()
    for kind in range(7):
        p.check(p.L.s2dwc_plan_timing(p.h, kind, ctypes.byref(n), ctypes.byref(ms)))
        assert n.value == 0
    p.close()


def alpha_stage_choice(B):
    """The alpha stages' transforms are the plan's own choice (S2DW_PFA at its
    creation), whatever plans come after it, and the tables are those it needs."""
    f = _fake()

    def create(pfa):
        os.environ["S2DW_PFA"] = pfa
        p = Plan(B, 2)
        need = ctypes.c_longlong()
        p.check(p.L.s2dwc_plan_footprint(B, 2, 2.0, p.J, 0, ctypes.byref(need)))
        assert p.bytes() == need.value
        return p

    def launches(p):
        w, s, x = p.buffers()
        f.fake_log()
        p.check(p.L.s2dwc_plan_analysis(p.h, w, s, x, None))
        p.check(p.L.s2dwc_plan_synthesis(p.h, x, w, s, None))
        return [k[3:] for k in _launches(f)]

    blue = create("0")
    first = launches(blue)
    prime = create("1")
    second = launches(prime)
    assert launches(blue) == first != second
    assert prime.bytes() < blue.bytes()
    again = create("0")
    assert launches(prime) == second and launches(again) == first


def priority(form):
    f = _fake()
    p = Plan(24, 4, form=form)
    p.check(p.L.s2dwc_plan_set_priority(p.h, -3))
    w, s, x = p.buffers(3)
    p.check(p.reserve(3))
    f.fake_log()
    for maps in (1, 3):
        p.check(p.L.s2dwc_plan_analysis_batch(p.h, maps, w, s, x, None))
        p.check(p.L.s2dwc_plan_synthesis_batch(p.h, maps, x, w, s, None))
    got = _launches(f)
    assert len(got) > 6
    assert all(k[1] == -3 for k in got), [k for k in got if k[1] != -3]


# ---- tests -----------------------------------------------------------------
def test_a_failed_reserve_leaves_the_plan_as_it_was(fake):
    """Split workspaces that do not fit: whichever allocation fails, the next
    reserve succeeds, holds no more memory than on a fresh plan, and the batches
    after it make a fresh plan's launches (every scale once in each grouped one)."""
    run(fake, "failed_reserve")


def test_a_failed_buffer_allocation_can_be_repeated(fake):
    """No pointer of a group of buffers stays set while another of it is
    missing: a kernel would get the null one on the next call."""
    run(fake, "failed_buffers")


@pytest.mark.parametrize("alpha10", [20, 11])  # 1.1: no scale large enough for a stream of its own
def test_no_copy_outlives_a_failed_host_call(fake, alpha10):
    run(fake, "failed_host_calls", alpha10)


def test_noalloc_creates_nothing_in_timing_mode(fake):
    run(fake, "noalloc_timing")


@pytest.mark.parametrize("B", [128, 256, 1024])
def test_alpha_stages_are_the_plan_s_choice(fake, B):
    run(fake, "alpha_stage_choice", B)


@pytest.mark.parametrize("form", [0, 1])
def test_every_kernel_has_the_plan_s_priority(fake, form):
    """On a stream of another priority, in both forms."""
    run(fake, "priority", form)


if __name__ == "__main__":
    globals()[sys.argv[1]](*map(int, sys.argv[2:]))

"""Host-buffer calls on pageable arrays (staged through page-locked slots by
several threads) form the device call's image bit for bit; GPU tests."""
import os
import threading

import numpy as np
import pytest

import sarbp_b200 as sb
from sarbp_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    return pytest.importorskip("torch")


def _data(nu, nv, P, S, seed):
    d = synth.make_from(dict(P=P, S=S, f0=9.6e9, df=1.5e6, R0=4e3, dep=35.0, span=3.0, nscat=5, half=10.0, clutter=0,
                             snr=20.0, n=32, extent=20.0, taylor=20, upsample=2, db=(-40.0, 0.0), seed=seed))
    d["u"], d["v"] = (np.arange(nu) - nu // 2) * 0.1, (np.arange(nv) - nv // 2) * 0.1
    d["r"] = sb.pixel_locs(d["u"], d["v"], d["u_hat"], d["v_hat"])
    return d


def _host(ctx, d, f64):
    t = np.float64 if f64 else np.float32
    return ctx.backprojection_cuda(d["phs"], d["k_r"].astype(t), 20, d["N_fft"], d["delta_r"], d["u"], d["v"],
                                   d["pos"].astype(t), d["r"])


def _device(ctx, torch, d, f64):
    c = lambda a, t: torch.from_numpy(np.ascontiguousarray(a, t)).cuda()
    nu, nv = d["u"].size, d["v"].size
    keep = [c(d["phs"].view(np.float32), np.float32), c(d["k_r"], np.float32), c(d["pos"], np.float32),
            c(d["r"], np.float64), c(d["k_r"], np.float64), c(d["pos"], np.float64),
            torch.zeros((nv, nu, 2), dtype=torch.float64, device="cuda")]
    p = [k.data_ptr() for k in keep]
    P, S = d["phs"].shape
    ctx.run_jobs([sb.make_job(S, P, d["N_fft"], 20, nu, nv, d["delta_r"], p[0], p[1], p[2], p[6], r=p[3], k_r64=p[4],
                              pos64=p[5], precision=sb.PREC_PRECISE if f64 else sb.PREC_COMPAT)])
    ctx.synchronize()
    return keep[6].cpu().numpy().view(np.complex128)[..., 0]


# nothing staged; positions only; all arrays, in one piece and in slabs; more
# than the slots hold at once, ragged
@pytest.mark.parametrize("nu,nv,P,S", [(100, 90, 20, 60), (300, 200, 33, 64), (500, 480, 300, 200), (640, 601, 40, 64),
                                       (1301, 903, 30, 1100)])
@pytest.mark.parametrize("f64", [False, True])
def test_pageable_arrays_equal_device_call(ctx, torch, nu, nv, P, S, f64):
    d = _data(nu, nv, P, S, seed=nu)
    want = _device(ctx, torch, d, f64)
    for _ in range(3):
        assert np.array_equal(_host(ctx, d, f64), want)


def test_contexts_on_several_threads():
    """Each context stages with its own slots and threads."""
    data = [_data(700 + 64 * i, 600, 30, 80, seed=i) for i in range(3)]
    out, errors = [None] * 3, []

    def work(i):
        try:
            with sb.Context(0) as c:
                first = _host(c, data[i], False)
                for _ in range(4):
                    assert np.array_equal(_host(c, data[i], False), first)
                out[i] = first
        except Exception as e:
            errors.append(e)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not errors, errors
    with sb.Context(0) as c:
        for i in range(3):
            assert np.array_equal(_host(c, data[i], False), out[i])


# page-locked inputs: none staged; the image is, from 4 MB on
@pytest.mark.parametrize("nu,nv", [(100, 90), (300, 200), (500, 480), (640, 601)])
def test_page_locked_arrays_equal_device_call(ctx, torch, nu, nv):
    d = _data(nu, nv, 40, 64, seed=nu)
    want = _device(ctx, torch, d, False)
    pinned = {k: torch.from_numpy(np.ascontiguousarray(d[k], t)).pin_memory().numpy()
              for k, t in (("k_r", np.float32), ("pos", np.float32), ("r", np.float64))}
    phs = torch.from_numpy(np.ascontiguousarray(d["phs"], np.complex64).view(np.float32)).pin_memory().numpy()
    for _ in range(3):
        got = ctx.backprojection_cuda(phs.view(np.complex64), pinned["k_r"], 20, d["N_fft"], d["delta_r"], d["u"],
                                      d["v"], pinned["pos"], pinned["r"])
        assert np.array_equal(got, want)


def test_a_small_image_alone_wakes_no_copy_threads(torch):
    """Waking them takes longer than the driver's copy."""
    d = _data(300, 200, 33, 64, seed=6)
    d["r"] = torch.from_numpy(np.ascontiguousarray(d["r"])).pin_memory().numpy()
    threads = lambda: len(os.listdir("/proc/self/task"))
    with sb.Context(0) as c:
        _host(c, _data(40, 40, 33, 64, seed=6), False)  # whatever the driver starts
        before = threads()
        _host(c, d, False)
        assert threads() == before

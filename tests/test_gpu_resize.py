"""Resampling of platform data (the reference's data/resize.py) on the
device, against the CPU restatement of skimage.transform.resize on
scipy.ndimage (oracle/resize_oracle.py):

* 2-D arrays shrinking on both axes, growing, and shrinking on one axis
  only (pos: (P, 3) -> (p, 3)); 1-D arrays (k_r); f32 and f64; complex
  arrays resampled as real and imaginary parts.  The f64 accumulation runs
  in scipy's order, so the results agree to the last bits: relative
  1e-6 of the array's range for f32, 1e-12 for f64.
* The resize tool on the AFRL platform files writes the same arrays, with
  the reference's dtypes, as the restated tool.
"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(got, want):
    assert got.shape == want.shape and got.dtype == want.dtype, (got.shape, want.shape, got.dtype, want.dtype)
    tol = (1e-6 if want.real.dtype == np.float32 else 1e-12) * max(1e-30, float(np.abs(want).max()))
    np.testing.assert_allclose(got, want, rtol=0, atol=tol)


@pytest.mark.parametrize("shape_in,shape_out", [
    ((469, 424), (300, 256)),   # both axes shrink
    ((97, 130), (200, 333)),    # both grow
    ((469, 424), (469, 212)),   # one axis
    ((1999, 3), (777, 3)),      # pos
    ((40, 7), (13, 2)),
])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_resize_2d_matches_oracle(ctx, shape_in, shape_out, dtype):
    from resize_oracle import sk_resize
    a = np.random.default_rng(3).normal(size=shape_in).astype(dtype)
    _check(ctx.resize(a, shape_out), sk_resize(a, shape_out))


@pytest.mark.parametrize("n_in,n_out", [(424, 212), (424, 1000), (1024, 333), (5, 1)])
def test_resize_1d_matches_oracle(ctx, n_in, n_out):
    from resize_oracle import sk_resize
    k = np.linspace(380.0, 395.0, n_in).astype(np.float32)
    _check(ctx.resize(k, (n_out,)), sk_resize(k, (n_out,)))
    _check(ctx.resize(k.astype(np.float64) * 0.5, (n_out,)), sk_resize(k.astype(np.float64) * 0.5, (n_out,)))


def test_resize_complex_is_real_and_imaginary_parts(ctx):
    from resize_oracle import sk_resize
    rng = np.random.default_rng(5)
    z = (rng.normal(size=(123, 77)) + 1j * rng.normal(size=(123, 77))).astype(np.complex64)
    want = sk_resize(np.real(z), (50, 90)) + 1j * sk_resize(np.imag(z), (50, 90))
    _check(ctx.resize(z, (50, 90)), want)


def test_resize_tool_on_afrl_files(ctx, afrl_input, tmp_path):
    from resize_oracle import resize_platform
    from sarbp_b200.resize import resize
    src = tmp_path / "in"
    src.mkdir()
    for k in ("delta_r", "k_r", "npulses", "nsamples", "phs", "pos", "R_c"):
        np.save(str(src / (k + ".npy")), afrl_input[k])
    for p, s, sp, ss, name in ((300, 256, 1.0, 1.0, "a"), (None, None, 0.5, 1.5, "b")):
        dst = str(tmp_path / name)
        resize(str(src), dst, p, s, scale_p=sp, scale_s=ss, ctx=ctx)
        d_r, k_r, P, S, phs, pos = resize_platform(afrl_input["delta_r"], afrl_input["k_r"],
                                                   afrl_input["npulses"], afrl_input["nsamples"],
                                                   afrl_input["phs"], afrl_input["pos"], p, s, sp, ss)
        got = {k: np.load(os.path.join(dst, k + ".npy")) for k in
               ("delta_r", "k_r", "npulses", "nsamples", "phs", "pos", "R_c")}
        assert np.array_equal(got["delta_r"], d_r) and got["delta_r"].dtype == d_r.dtype
        assert int(got["npulses"]) == P and int(got["nsamples"]) == S
        assert np.array_equal(got["R_c"], afrl_input["R_c"])
        _check(got["k_r"], k_r)
        _check(got["phs"], phs)
        _check(got["pos"], pos)


def _device(ctx, torch, a, shape, shift=0, over=False):
    """sarbp_resize_device of a [rows][cols][ncomp] array; `shift` puts the
    output that many elements off its alignment, `over` over the input."""
    import ctypes

    from sarbp_b200._lib import check, lib
    t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    n = shape[0] * shape[1] * a.shape[2]
    buf = torch.zeros(max(n, t.numel()) + 4, dtype=t.dtype, device="cuda")
    src = t
    if over:
        buf[:t.numel()] = t.reshape(-1)
        src = buf
    p = lambda x, o=0: ctypes.c_void_p(x.data_ptr() + o * x.element_size())
    check(lib().sarbp_resize_device(ctx.handle, t.element_size(), a.shape[2], p(src), a.shape[0], a.shape[1],
                                    shape[0], shape[1], p(buf, shift)))
    ctx.synchronize()
    return buf[shift:shift + n].reshape(shape[0], shape[1], a.shape[2]).cpu().numpy()


# one output row or column, tiles and remainders, the largest filters of the
# tile kernel and the ones beyond it, one axis each way, single rows and columns
@pytest.mark.parametrize("shape_in,shape_out", [
    ((300, 260), (150, 130)), ((131, 129), (33, 127)), ((500, 40), (140, 40)), ((520, 64), (130, 16)),
    ((40, 900), (41, 110)), ((64, 700), (64, 80)), ((33, 70), (200, 515)), ((1, 1000), (1, 260)), ((1000, 1), (301, 1)),
    ((2, 2), (5, 5)), ((7, 5), (1, 1)), ((90, 90), (89, 91)), ((257, 300), (70, 1)),
])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("nc", [1, 2])
def test_tile_kernel_matches_oracle_and_steps(ctx, shape_in, shape_out, dtype, nc):
    import torch
    from resize_oracle import sk_resize
    a = np.random.default_rng(11).normal(size=shape_in + (nc,)).astype(dtype)
    got = _device(ctx, torch, a, shape_out)
    for k in range(nc):
        _check(got[..., k], sk_resize(a[..., k], shape_out))
    # an output over its input is formed step by step
    steps = _device(ctx, torch, a, shape_out, over=True) if np.prod(shape_out) <= np.prod(shape_in) else got
    tol = (1e-6 if dtype == np.float32 else 1e-14) * np.abs(a).max()
    np.testing.assert_allclose(got, steps, rtol=0, atol=tol)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape_out", [(30, 21), (100, 90), (61, 20)])
def test_tile_kernel_clips_like_the_steps(ctx, dtype, shape_out):
    """Constant arrays stay constant; NaN and infinities come out as the
    step-by-step kernels leave them (clipped to the extremes)."""
    import torch
    c = np.full((61, 43, 2), 0.1, dtype)
    assert np.array_equal(_device(ctx, torch, c, shape_out), np.full(shape_out + (2,), 0.1, dtype))
    a = np.random.default_rng(2).normal(size=(61, 43, 2)).astype(dtype)
    a[5, 7, 0] = np.nan
    a[40, 30, 1] = np.inf
    a[0, 0, 1] = -np.inf
    for b in (a, np.full_like(a, np.nan)):
        got, want = _device(ctx, torch, b, shape_out), _device(ctx, torch, b, shape_out, shift=1)
        tol = (1e-6 if dtype == np.float32 else 1e-14) * 5
        np.testing.assert_allclose(got, want, rtol=0, atol=tol)


def test_contexts_on_several_threads_resize_different_shapes(sb):
    """Shapes whose tiles need different amounts of shared memory from the same
    kernel, each from a context and a thread of its own."""
    import threading

    import torch
    jobs = [((80, 70, 2), (640, 700)), ((9, 7, 2), (12, 10)), ((5, 40, 2), (7, 90))]
    errors = []

    def work(shape_in, shape_out):
        try:
            a = np.random.default_rng(4).normal(size=shape_in)
            with sb.Context(0) as c:
                first = _device(c, torch, a, shape_out)
                for _ in range(400):
                    assert np.array_equal(_device(c, torch, a, shape_out), first)
        except Exception as e:
            errors.append(e)

    ts = [threading.Thread(target=work, args=j) for j in jobs for _ in range(2)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not errors, errors[:2]


@pytest.mark.parametrize("shape_in,shape_out", [((300, 260), (150, 130)), ((131, 129), (40, 37)), ((90, 90), (89, 91)),
                                                ((64, 300), (64, 80)), ((70, 33), (200, 115))])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("nc", [1, 2])
def test_tile_kernel_rounds_like_the_steps(ctx, shape_in, shape_out, dtype, nc):
    import torch
    a = np.random.default_rng(12).normal(size=shape_in + (nc,)).astype(dtype)
    # an output off its elements' alignment is formed step by step
    if nc == 2:
        want = _device(ctx, torch, a, shape_out, shift=1)
    else:
        three = np.repeat(a, 3, axis=2)
        want = _device(ctx, torch, three, shape_out)[..., :1]
    assert np.array_equal(_device(ctx, torch, a, shape_out), want)


# many tiles of few rows: beyond the line the steps, below it tiles
@pytest.mark.parametrize("shape_in,shape_out", [((1, 600000), (1, 240000)), ((1, 100000), (1, 40000)),
                                                ((3, 700001), (3, 350000)), ((4, 120000), (7, 240001))])
@pytest.mark.parametrize("nc", [1, 2])
def test_long_rows(ctx, shape_in, shape_out, nc):
    import torch
    a = np.random.default_rng(13).normal(size=shape_in + (nc,))
    # three components always go step by step
    want = _device(ctx, torch, np.concatenate([a, a, a], axis=2)[..., :3], shape_out)[..., :nc]
    assert np.array_equal(_device(ctx, torch, a, shape_out), want)


# few tiles, split by rows down to four
@pytest.mark.parametrize("shape_in,shape_out", [((64, 64), (64, 1000)), ((9, 1000), (5, 400)), ((2000, 2), (1000, 2)),
                                                ((300, 300), (77, 75)), ((3, 40), (2, 900)), ((469, 3), (301, 3))])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_split_tiles_round_like_the_steps(ctx, shape_in, shape_out, dtype):
    import torch
    a = np.random.default_rng(14).normal(size=shape_in + (2,)).astype(dtype)
    assert np.array_equal(_device(ctx, torch, a, shape_out), _device(ctx, torch, a, shape_out, shift=1))


# without filters, on both sides of their line; one row has its own
@pytest.mark.parametrize("shape_in,shape_out", [((2, 350000), (3, 350000)), ((2, 700000), (3, 700000)),
                                                ((1, 100000), (1, 200000)), ((1, 400001), (1, 800000)),
                                                ((7, 500000), (8, 500000))])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_long_rows_without_filters(ctx, shape_in, shape_out, dtype):
    import torch
    a = np.random.default_rng(15).normal(size=shape_in + (1,)).astype(dtype)
    want = _device(ctx, torch, np.repeat(a, 3, axis=2), shape_out)[..., :1]
    assert np.array_equal(_device(ctx, torch, a, shape_out), want)

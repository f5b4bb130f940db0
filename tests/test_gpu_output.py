"""dB and u8 images at the edges of their f32 and f64 ranges; GPU tests."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    return pytest.importorskip("torch")


def _images(rng):
    z = rng.normal(size=(37, 53)) + 1j * rng.normal(size=(37, 53))
    bright = z.copy()
    bright[5, 7] *= 1e4  # most pixels far below the display range
    mixed = z * 10.0 ** rng.uniform(-20, 0, size=z.shape)
    mixed[::3] = 0.0
    return {"speckle": z, "bright": bright, "mixed": mixed, "one": z[:1, :1], "odd": bright[:1, :1023 // 23],
            "tiny": bright * 1e-30, "huge": mixed * 1e30, "f32_min": mixed * 1e-19, "f64_min": z * 1e-160,
            "f64_max": z * 1e150, "equal": np.full((8, 9), 3.0 - 4.0j), "zero": np.zeros((4, 6), np.complex128)}


@pytest.mark.parametrize("lo,hi", [(-45.0, 0.0), (-30.0, -10.0), (-400.0, 5.0)])
@pytest.mark.parametrize("name", sorted(_images(np.random.default_rng(0))))
def test_db_and_u8_match_oracle(ctx, oracle, torch, name, lo, hi):
    """u8 exactly the oracle's, from the image at once and through the dB
    image; dB within 1e-12 of it (three roundings of the square, times 5 / ln
    10, are 8e-16; a square below 1e-290 is left to the oracle's formula)."""
    img = np.ascontiguousarray(_images(np.random.default_rng(3))[name], np.complex128)
    nv, nu = img.shape
    want_dB = oracle.img_output_to_dB(img)
    want = oracle.img_output_u8(want_dB, lo, hi)
    dB = ctx.img_output_to_dB(img)
    fine = np.isfinite(want_dB)
    assert np.array_equal(fine, np.isfinite(dB)) and np.array_equal(np.isnan(want_dB), np.isnan(dB))
    if fine.any():
        assert np.abs(dB[fine] - want_dB[fine]).max() < 1e-12 and dB[fine].max() == want_dB[fine].max() == 0.0
    assert np.array_equal(ctx.img_output_u8(dB, lo, hi), want)
    t = torch.from_numpy(img.view(np.float64)).cuda()
    for off in (0, 1):  # aligned and unaligned destination
        out = torch.zeros(nu * nv + 8, dtype=torch.uint8, device="cuda")
        ctx.img_output_u8_from_img_device(t.data_ptr(), nu, nv, lo, hi, out.data_ptr() + off)
        ctx.synchronize()
        assert np.array_equal(out.cpu().numpy()[off:off + nu * nv].reshape(nv, nu), want)


def test_unaligned_db_destination(ctx, sb, torch):
    from sarbp_b200._lib import check, lib
    img = torch.randn(5, 7, 2, dtype=torch.float64, device="cuda")
    a, b = torch.zeros(40, dtype=torch.float64, device="cuda"), torch.zeros(40, dtype=torch.float64, device="cuda")
    p = lambda t, o=0: ctypes.c_void_p(t.data_ptr() + o)
    check(lib().sarbp_img_output_to_dB_device(ctx.handle, p(img), 7, 5, p(a)))
    check(lib().sarbp_img_output_to_dB_device(ctx.handle, p(img), 7, 5, p(b, 8)))
    ctx.synchronize()
    assert torch.equal(a[:35], b[1:36]) and float(a[35]) == 0.0 == float(b[36])


# |z|^2 ordinary f32 numbers whose ratio to the maximum's is subnormal or zero there
@pytest.mark.parametrize("lo,hi", [(-300.0, 0.0), (-500.0, 0.0), (-230.0, -190.0)])
def test_u8_over_thirty_decades(ctx, oracle, torch, lo, hi):
    rng = np.random.default_rng(8)
    img = (rng.normal(size=(61, 47)) + 1j * rng.normal(size=(61, 47))) * 10.0 ** rng.uniform(-20, 9, size=(61, 47))
    img[0, 0], img[3, 4] = 1e-15, 1e10
    want = oracle.img_output_u8(oracle.img_output_to_dB(img), lo, hi)
    t = torch.from_numpy(img.view(np.float64)).cuda()
    out = torch.zeros(img.size, dtype=torch.uint8, device="cuda")
    ctx.img_output_u8_from_img_device(t.data_ptr(), 47, 61, lo, hi, out.data_ptr())
    ctx.synchronize()
    assert np.array_equal(out.cpu().numpy().reshape(61, 47), want)


def test_db_where_the_squares_ratio_leaves_the_f64_range(ctx, oracle):
    """Pixels down to 280 decades below the maximum: the logarithm of each
    side is good to an ulp and three roundings follow it (4 x 2.2e-16)."""
    rng = np.random.default_rng(9)
    img = (1 + rng.uniform(size=(40, 30)) + 1j * rng.normal(size=(40, 30))) * 10.0 ** rng.uniform(-140, 140, (40, 30))
    want, got = oracle.img_output_to_dB(img), ctx.img_output_to_dB(img)
    assert np.isfinite(want).all()
    np.testing.assert_allclose(got, want, rtol=9e-16, atol=1e-12)


def test_db_error_is_not_above_the_f64_formulas(ctx, oracle):
    """Against 80-bit values, for the image's own maximum |z|."""
    rng = np.random.default_rng(10)
    img = rng.normal(size=(700, 600)) + 1j * rng.normal(size=(700, 600))
    re, im = img.real.astype(np.longdouble), img.imag.astype(np.longdouble)
    a = np.sqrt(re * re + im * im)
    exact = 10 * np.log(a / a.max()) / np.longdouble(np.log(np.float32(10.0)))
    err = lambda d: float(np.sqrt(np.mean((d - exact) ** 2)))
    assert err(ctx.img_output_to_dB(img)) <= err(oracle.img_output_to_dB(img))


@pytest.mark.parametrize("n", [1, 700, 5000, 300001, 3000001])
def test_maximum_wherever_it_lies(ctx, sb, torch, n):
    """The partial maxima of every CTA and lane count, low bits included."""
    from sarbp_b200._lib import check, lib
    import ctypes
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    img = torch.ones(n, 2, dtype=torch.float64, device="cuda")
    dB = torch.empty(n, dtype=torch.float64, device="cuda")
    u8 = torch.empty(n, dtype=torch.uint8, device="cuda")
    for at in sorted({0, n // 7, n // 3, n // 2, max(0, n - 257), n - 1}):
        img[at, 0] = 1.0 + 2.0 ** -40  # the high words of |z|^2 are equal
        img[at, 1] = 1.0 + 2.0 ** -40
        torch.cuda.synchronize()
        check(lib().sarbp_img_output_to_dB_device(ctx.handle, p(img), n, 1, p(dB)))
        ctx.img_output_u8_from_img_device(img.data_ptr(), n, 1, -1e-12, 0.0, u8.data_ptr())
        ctx.synchronize()
        assert float(dB[at]) == 0.0 and int(u8[at]) == 255
        if n > 1:
            rest = torch.cat([dB[:at], dB[at + 1:]])
            assert float(rest.max()) < 0.0 and float(rest.min()) == float(rest.max())
            assert int(torch.cat([u8[:at], u8[at + 1:]]).max()) == 0
        img[at] = 1.0

"""The backprojection's work list: persistent CTAs that claim further items
(with even shares of the end of the list) form the same image, bit for bit,
as one CTA per tile; GPU tests."""
import numpy as np
import pytest

import sarbp_b200 as sb
from sarbp_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    return pytest.importorskip("torch")


def _cfg(P, seed, **kw):
    c = dict(P=P, S=96, f0=9.6e9, df=1.5e6, R0=4e3, dep=35.0, span=3.0, nscat=5, half=10.0, clutter=0, snr=20.0,
             n=32, extent=20.0, taylor=20, upsample=2, db=(-40.0, 0.0), seed=seed)
    c.update(kw)
    return c


class _Job:
    """A device-resident job of nu x nv pixels at 0.3 m."""

    def __init__(self, torch, nu, nv, P, seed, precise=False):
        d = synth.make_from(_cfg(P, seed))
        t = lambda a, k: torch.from_numpy(np.ascontiguousarray(a, k)).cuda()
        self.a = [t(d["phs"].view(np.float32), np.float32), t(d["k_r"], np.float32), t(d["pos"], np.float32),
                  t((np.arange(nu) - nu // 2) * 0.3, np.float64), t((np.arange(nv) - nv // 2) * 0.3, np.float64),
                  t(d["k_r"], np.float64), t(d["pos"], np.float64)]
        self.out = torch.full((nv, nu, 2), -7.0, dtype=torch.float64, device="cuda")
        self.u8 = torch.zeros((nv, nu), dtype=torch.uint8, device="cuda")
        p = [x.data_ptr() for x in self.a]
        self.job = sb.make_job(d["S"], P, d["N_fft"], 20, nu, nv, d["delta_r"], p[0], p[1], p[2],
                               self.out.data_ptr(), u=p[3], v=p[4], u_hat=d["u_hat"], v_hat=d["v_hat"], k_r64=p[5],
                               pos64=p[6], out_u8=self.u8.data_ptr(), dB_min=-40.0, dB_max=0.0,
                               precision=sb.PREC_PRECISE if precise else sb.PREC_COMPAT)

    def run(self, ctx, jobs=None, **tune):
        ctx.run_jobs(jobs or [self.job], **tune)
        ctx.synchronize()
        return self.out.cpu().numpy().copy(), self.u8.cpu().numpy().copy()


@pytest.fixture(scope="module")
def ctx():
    with sb.Context(0) as c:
        yield c


# tiles: one; all resident (3 x 148) less and more one; between one and two
# rounds; above two rounds; pulses: fewer and more than a chunk, odd
@pytest.mark.parametrize("tx,ty,P", [(1, 1, 3), (443, 1, 65), (37, 12, 40), (89, 5, 129), (23, 32, 70), (33, 31, 11)])
def test_claimed_items_equal_one_cta_per_tile(ctx, torch, tx, ty, P):
    j = _Job(torch, 32 * tx - 5, 32 * ty - 3, P, seed=tx)
    want = j.run(ctx, persistent=2, pulse_parts=1)
    assert np.isfinite(want[0]).all() and np.abs(want[0]).max() > 0
    got = j.run(ctx, pulse_parts=1)
    assert np.array_equal(want[0], got[0]) and np.array_equal(want[1], got[1])


@pytest.mark.parametrize("precise", [False, True])
def test_uneven_list_equals_each_job_alone(ctx, torch, precise):
    sizes = [(700, 500, 211), (96, 96, 17), (513, 130, 90), (64, 1000, 64), (40, 30, 1), (300, 300, 150)]
    jobs = [_Job(torch, nu, nv, P, seed=i, precise=precise) for i, (nu, nv, P) in enumerate(sizes)]
    alone = [j.run(ctx) for j in jobs]
    for j in jobs:
        j.out.fill_(-7.0)
        j.u8.fill_(0)
    jobs[0].run(ctx, jobs=[j.job for j in jobs])
    for j, (img, u8) in zip(jobs, alone):
        assert np.array_equal(img, j.out.cpu().numpy()) and np.array_equal(u8, j.u8.cpu().numpy())


# the fewest and the most parts, odd counts, parts of one pulse
@pytest.mark.parametrize("parts,P", [(2, 65), (5, 97), (16, 16), (16, 200)])
def test_parts_summed_by_the_last_item(ctx, torch, parts, P):
    """The same bits whichever CTA completes a tile, alone and in a batch; the
    sum over parts differs from one item per tile by f32 rounding only (P
    terms: about sqrt(P) 2^-24 of the sum, well below 1e-5)."""
    a, b = _Job(torch, 200, 130, P, seed=P), _Job(torch, 90, 300, P + 3, seed=P + 1)
    whole = a.run(ctx, pulse_parts=1)[0]
    first = a.run(ctx, pulse_parts=parts)
    assert np.linalg.norm(first[0] - whole) < 1e-5 * np.linalg.norm(whole)
    for _ in range(10):
        a.out.fill_(-7.0)
        again = a.run(ctx, jobs=[a.job, b.job], pulse_parts=parts)
        assert np.array_equal(first[0], again[0]) and np.array_equal(first[1], again[1])


# range windows wholly or partly below and above the profile: the clamped edge
# pairs; narrow and wide windows
@pytest.mark.parametrize("upsample,pixel", [(2, 0.8), (6, 1.6), (1, 2.5)])
def test_tiles_off_the_range_swath(ctx, oracle, torch, upsample, pixel):
    nu, nv, P = 230, 190, 70
    d = synth.make_from(_cfg(P, 3, S=64, upsample=upsample))
    u, v = (np.arange(nu) - nu // 2) * pixel, (np.arange(nv) - nv // 2) * pixel
    r = sb.pixel_locs(u, v, d["u_hat"], d["v_hat"])
    got = ctx.backprojection_cuda(d["phs"], d["k_r"], 20, d["N_fft"], d["delta_r"], u, v, d["pos"], r)
    idx = np.random.default_rng(1).choice(nu * nv, 4000, replace=False)
    want = oracle.backprojection(d["phs"], d["k_r"], 20, d["N_fft"], d["delta_r"], d["pos"], r, nu, nv,
                                 mode=oracle.MODE_FP64, out_idx=idx)
    assert np.linalg.norm(got.reshape(-1)[idx] - want) < 1e-4 * np.linalg.norm(want)


def test_parts_summed_in_place_beside_parts_combined(ctx, torch):
    """One round of items: a job in two parts (added by a tile's last item)
    and one in many (the combine kernel), as alone."""
    a, b = _Job(torch, 300, 300, 90, seed=31), _Job(torch, 70, 60, 620, seed=32)
    alone = [a.run(ctx), b.run(ctx)]
    for _ in range(3):
        a.out.fill_(-7.0)
        b.out.fill_(-7.0)
        a.run(ctx, jobs=[a.job, b.job])
        for j, (img, u8) in zip((a, b), alone):
            assert np.array_equal(img, j.out.cpu().numpy()) and np.array_equal(u8, j.u8.cpu().numpy())

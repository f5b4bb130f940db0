"""Range profiles: windows longer than the set-up kernel's clusters hold at
once, and where the profiles may be stored; GPU tests."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    return pytest.importorskip("torch")


def _job(sb, torch, phs, N, offset=0):
    """A range-compression job; its phase history starts `offset` floats into a larger buffer."""
    P, S = phs.shape
    rng = np.random.default_rng(S)
    k_r = rng.uniform(350, 400, size=S).astype(np.float32)
    buf = torch.zeros(offset + max(2 * P * S, 2 * P * N) + 64, dtype=torch.float32, device="cuda")
    buf[offset:offset + 2 * P * S] = torch.from_numpy(phs.view(np.float32).reshape(-1)).cuda()
    k, pos = torch.from_numpy(k_r).cuda(), torch.zeros(P, 3, device="cuda")
    j = sb.make_job(S, P, N, 20, 0, 0, 1.0, buf.data_ptr() + 4 * offset, k.data_ptr(), pos.data_ptr(), 0)
    return j, buf, k_r, (k, pos)


def _phs(P, S):
    rng = np.random.default_rng(P + S)
    return (rng.normal(size=(P, S)) + 1j * rng.normal(size=(P, S))).astype(np.complex64)


# one element per thread of the cluster (2048) and one more; all that its
# threads keep (8192) and more
@pytest.mark.parametrize("P,S,N", [(2048, 40, 64), (2049, 33, 64), (8192, 20, 32), (8201, 17, 32), (9, 9000, 16384)])
def test_long_windows(sb, ctx, oracle, torch, P, S, N):
    phs = _phs(P, S)
    j, buf, k_r, keep = _job(sb, torch, phs, N)
    q = torch.empty(P, N, 2, device="cuda")
    ctx.range_compress_device(j, q.data_ptr())
    ctx.synchronize()
    ref = oracle.range_compress(phs, k_r.astype(np.float64), 20, N, mode=oracle.MODE_REF)
    assert rel_l2(q.cpu().numpy().view(np.complex64)[..., 0], ref) < 2e-6


@pytest.mark.parametrize("N", [128, 32768])
@pytest.mark.parametrize("where", ["odd", "over_input", "after_input", "pinned"])
def test_profiles_stored_anywhere(sb, ctx, torch, N, where):
    """Unaligned and page-locked destinations and ones over the phase history
    take the same values as an ordinary one."""
    P, S = 37, 100
    phs = _phs(P, S)
    j, buf, _, keep = _job(sb, torch, phs, N, offset=2)
    want = torch.empty(P * N * 2, device="cuda")
    ctx.range_compress_device(j, want.data_ptr())
    ctx.synchronize()
    n = P * N * 2
    big = torch.empty(n + 8, device="cuda")
    if where == "odd":
        got = big[1:1 + n]
    elif where == "over_input":
        got = buf[4:4 + n]
    elif where == "after_input":
        big = torch.empty(2 * P * S + n + 2, device="cuda")
        big[:2 * P * S] = torch.from_numpy(phs.view(np.float32).reshape(-1)).cuda()
        j.phs = big.data_ptr()
        got = big[2 * P * S:2 * P * S + n]
    else:
        got = torch.empty(n, dtype=torch.float32).pin_memory()
    ctx.range_compress_device(j, got.data_ptr())
    ctx.synchronize()
    assert np.array_equal(got.cpu().numpy(), want.cpu().numpy())

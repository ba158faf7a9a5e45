"""The standalone fits at the edges of their warps and blocks: a tuple's
result does not depend on how many tuples are fitted with it, and nothing is
written past the last one.

Tolerance: none.  A tuple's arithmetic is the same whatever warp, block size
or position it has, so the results are compared bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = {"state": 5, "cov": 15, "pt": 1, "eta": 1, "chi2": 1}
GUARD = 64


def _fit(chain, entry, N, hits, ge, n):
    import torch
    import pixgpu
    h = torch.from_numpy(np.ascontiguousarray(hits[:n, :N])).cuda()
    g = torch.from_numpy(np.ascontiguousarray(ge[:n, :N])).cuda()
    out = {k: torch.full(((n + GUARD) * w,), -77.0, dtype=torch.float32, device="cuda") for k, w in SIZES.items()}
    rc = getattr(pixgpu.gpu_lib(), entry)(chain._h, N, n, h.data_ptr(), g.data_ptr(), pixgpu.B_FIELD,
                                          *[out[k].data_ptr() for k in SIZES],
                                          torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    return {k: v.cpu().numpy().view(np.uint32).reshape(n + GUARD, -1) for k, v in out.items()}


@pytest.mark.parametrize("entry", ["pg_fit_broken_line", "pg_fit_broken_line_mixed", "pg_fit_riemann",
                                   "pg_fit_riemann_mixed"])
@pytest.mark.parametrize("N", [3, 4])
def test_fit_of_any_number_of_tuples(default_detector, entry, N):
    import pixgpu
    chain = pixgpu.Chain(default_detector.es, max_events=1, max_words_per_batch=300000)
    most = 148 * 256 + 33  # one block more than the SMs, at the largest block
    hits, ge, _ = pixgpu.fit_tuples(99 + N, most, N)
    want = _fit(chain, entry, N, hits, ge, most)
    sentinel = np.float32(-77.0).view(np.uint32)
    for n in (1, 31, 32, 33, 255, 257, 147 * 32 + 1, 148 * 64 + 5, 148 * 128 - 31):
        got = _fit(chain, entry, N, hits, ge, n)
        for k in SIZES:
            assert np.array_equal(got[k][:n], want[k][:n]), (n, k)
            assert (got[k][n:] == sentinel).all(), (n, k)
    chain.close()


@pytest.mark.parametrize("entry,block", [("pg_fit_broken_line", 256), ("pg_fit_broken_line_mixed", 256),
                                         ("pg_fit_riemann", 128), ("pg_fit_riemann_mixed", 128)])
@pytest.mark.parametrize("N", [3, 4])
def test_fit_of_more_tuples_than_one_pass_of_the_grid(default_detector, entry, block, N):
    """The grid has at most 16 blocks per SM: with one block's tuples and a
    ragged warp more than that, the first blocks take a second tile, into the
    shared memory that still held the first one's results."""
    import pixgpu
    chain = pixgpu.Chain(default_detector.es, max_events=1, max_words_per_batch=300000)
    one = 148 * 16 * block
    n, some = one + block + 33, 4 * block
    base, ge, _ = pixgpu.fit_tuples(199 + N, some, N)
    times = n // some + 1  # the same tuples over and over: every repetition has the same results
    got = _fit(chain, entry, N, np.tile(base, (times, 1, 1)), np.tile(ge, (times, 1, 1)), n)
    want = _fit(chain, entry, N, base, ge, some)
    sentinel = np.float32(-77.0).view(np.uint32)
    for k in SIZES:
        assert np.array_equal(got[k][:n], np.tile(want[k][:some], (times, 1))[:n]), k
        assert (got[k][n:] == sentinel).all(), k
    chain.close()

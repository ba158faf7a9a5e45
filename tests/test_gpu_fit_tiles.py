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

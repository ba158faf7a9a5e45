"""The vertex finder at the edges of its groupings and of its split over CTAs.

Tolerance: whole numbers equal; the floating results within 1e-5 relative of
the serial vertex finder, as everywhere in these tests (the sums run in the
serial order in single precision; only divisions and the conversion of the
inputs could differ).  Clusters of different sizes are compared bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
RTOL = 1e-5


def _tracks(n, n_vertices, seed, spread):
    """n four-hit loose tracks from n_vertices vertices on a grid of `spread` cm (narrow errors, so that they stay apart)."""
    rng = np.random.default_rng(seed)
    vz = (np.arange(n_vertices) - n_vertices / 2) * spread
    z = (vz[rng.integers(0, n_vertices, n)] + rng.normal(0, 0.0015, n)).astype(np.float32)
    st, cv = np.zeros((n, 5), np.float32), np.zeros((n, 15), np.float32)
    st[:, 4] = z
    cv[:, 14] = (rng.uniform(0.0015, 0.002, n) ** 2).astype(np.float32)
    return {"tupleOff": (np.arange(n + 1) * 4).astype(np.uint32), "quality": np.full(n, 2, np.uint8),
            "pt": (0.5 + rng.exponential(1.0, n)).astype(np.float32), "state": st.ravel(), "cov": cv.ravel()}


# tracks, vertices: none to one warp, one CTA's threads, the last size in shared memory and the first beyond it;
# one vertex, a warp's worth, so many that the grouping's table has fewer rows than warps
@pytest.mark.parametrize("n,n_vertices", [(1, 1), (2, 1), (31, 1), (33, 2), (1023, 1), (1025, 33), (5500, 64), (5501, 64),
                                          (5400, 860), (9000, 300)])
def test_vertices_of_any_number_of_tracks(default_detector, n, n_vertices):
    import oracle
    import torch
    import pixgpu
    t = _tracks(n, n_vertices, 7 + n, min(0.5, 22.0 / n_vertices))
    want = oracle.Oracle(default_detector.es).vertices(*[t[k] for k in ("tupleOff", "quality", "pt", "state", "cov")])
    ins = [torch.from_numpy(t[k].view(np.int32) if t[k].dtype == np.uint32 else t[k]).cuda()
           for k in ("tupleOff", "quality", "pt", "state", "cov")]
    idv = torch.full((n,), 12345, dtype=torch.int16, device="cuda")
    outs = [torch.zeros(1024, dtype=torch.float32, device="cuda") for _ in range(4)]
    ndof = torch.zeros(1024, dtype=torch.int32, device="cuda")
    order = torch.zeros(1024, dtype=torch.int16, device="cuda")
    nv, _ = pixgpu.vertices_noalloc(*ins, idv, *outs, ndof, order)
    assert nv == want["nVertices"]
    assert np.array_equal(idv.cpu().numpy(), want["idv"])
    assert np.array_equal(ndof.cpu().numpy()[:nv], want["ndof"])
    if nv:
        assert np.array_equal(order.cpu().numpy().view(np.uint16)[:nv], want["sortInd"])
    for k, o in zip(("zv", "wv", "vchi2", "ptv2"), outs):
        np.testing.assert_allclose(o.cpu().numpy()[:nv], want[k], rtol=RTOL, atol=0, err_msg=k)


@pytest.mark.parametrize("algo", [0, 1, 2])
def test_vertices_do_not_depend_on_the_batch(default_detector, algo):
    """Batches of 1, 20 and 40 events run the vertex finder on 8, 4 and 2 CTAs per event, and the results are
    packed by 8 CTAs per event or one."""
    import pixgpu
    raws = [default_detector.event(4000 + k, 2 + k % 7 * 4) for k in range(40)]
    chain = pixgpu.Chain(default_detector.es, max_events=40, vertex_algo=algo)
    got = {}
    for n in (1, 20, 40):
        slot = chain.submit(raws[:n])
        chain.wait(slot)
        got[n] = [chain.result(slot, k) for k in range(n)]
        chain.release(slot)
    chain.close()
    for a, b in ((got[1], got[20]), (got[20], got[40])):
        for k, x in enumerate(a):
            for name, v in x.items():
                assert np.array_equal(np.asarray(v).view(np.uint8) if np.ndim(v) else v,
                                      np.asarray(b[k][name]).view(np.uint8) if np.ndim(v) else b[k][name]), (k, name)

"""The chain's fits on a batch with more tuples than their blocks take in one
go, so that every block goes from tiles of one multiplicity to the next.

Tolerance: none.  A tuple's fit is the same whichever thread of whichever
block does it, so the batch's events equal their own runs alone bit for bit
(alone, an event's tuples fit into one tile per block)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ONE_PASS = 148 * 4 * 128  # tuples that one pass of the fits' blocks takes in a batch of more than four events


@pytest.mark.parametrize("riemann", [False, True])
@pytest.mark.parametrize("mixed", [False, True])
def test_a_batch_of_several_tiles_equals_its_events_alone(default_detector, riemann, mixed):
    import pixgpu
    raws = [default_detector.event(7100 + k, 44) for k in range(8)]  # dense model
    chain = pixgpu.Chain(default_detector.es, max_events=len(raws), max_words_per_batch=len(raws) * 300000,
                         riemann_fit=riemann, mixed_fit=mixed)
    names = ("tupleOff", "quality", "state", "cov", "pt", "eta", "chi2")
    try:
        alone = []
        for r in raws:
            chain.process([r])
            assert chain.counts(0)["flags"] == 0
            alone.append({k: chain.product(0, k) for k in names})
        # the hits of every fitted tuple (the others' results are zero)
        fitted = np.concatenate([np.diff(a["tupleOff"])[a["pt"][:len(a["tupleOff"]) - 1] != 0] for a in alone])
        assert len(fitted) > 1.2 * ONE_PASS and all((fitted == n).sum() > 128 for n in (3, 4, 5))
        for _ in range(3):
            chain.process(raws)
            for e, want in enumerate(alone):
                for k in names:
                    got = chain.product(e, k)
                    assert got.tobytes() == want[k].tobytes(), (e, k)
    finally:
        chain.close()

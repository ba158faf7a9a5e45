"""More and larger batches in flight than run side by side: a batch that waits
for an earlier one (six million FED words, and always three batches, run at
once) gives the same results, and the slots can be waited for in any order.

Tolerance: none.  The packed results are compared byte for byte with the same
batch alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SLOTS, BATCH = 5, 40


def _results(chain, slot, n):
    return [{k: np.asarray(v).tobytes() for k, v in chain.result(slot, e).items()} for e in range(n)]


@pytest.mark.parametrize("graphs", [True, False])
def test_batches_beyond_those_that_run_at_once(default_detector, graphs):
    import pixgpu
    raws = [default_detector.event(8800 + k, 50, model="calibrated") for k in range(BATCH)]
    chain = pixgpu.Chain(default_detector.es, max_events=BATCH, max_words_per_batch=BATCH * 120000, slots=SLOTS,
                         use_graphs=graphs, pool_words=BATCH * 120000)
    try:
        handles = []
        for r in raws:
            while (h := chain.pool_put(r)) is None:
                pass
            handles.append(h)
        info = chain.pool_info()
        assert SLOTS * (info["cap_words"] - info["free_words"]) > 6 << 20  # no room for all of them at once
        # whole batches, with single events between them
        batches = [handles, handles[:1], handles[::-1], handles[5:] + handles[:5], handles[7:8], handles]
        alone = []
        for b in batches:
            s = chain.submit_pooled(b, keep=True)
            chain.wait(s)
            alone.append(_results(chain, s, len(b)))
            chain.release(s)
        for order in (1, -1):
            held = []
            for k in list(range(len(batches))) * 3:
                while (s := chain.submit_pooled(batches[k], keep=True)) is None:
                    j, o = held.pop(0 if order == 1 else -1)
                    chain.wait(o)
                    assert _results(chain, o, len(batches[j])) == alone[j], j
                    chain.release(o)
                held.append((k, s))
            for j, o in held[::order]:
                chain.wait(o)
                assert _results(chain, o, len(batches[j])) == alone[j], j
                chain.release(o)
    finally:
        chain.close()

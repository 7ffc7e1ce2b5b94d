"""lst_batch_get_output of batches on both sides of its pinned staging (1 MiB): the
output of a batch is its events' outputs one after the other, whichever way it
takes; a caller's arrays that are too small are refused and stay as they were."""
import numpy as np
import pytest

from tracklooper_b200 import gen, lst

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("events", [
    [(1, 41, 0.0), (5, 42, 0.0)],                            # a few bytes
    [(2, 43, 200.0)] * 3,                                    # below 1 MiB
    [(2, 44, 200.0)] * 10 + [(1, 45, 0.0)],                  # above
])
def test_batch_output_is_the_events_outputs(events):
    inputs = [gen.generate_event(*e) for e in events]
    es = lst.ES(device=0)
    s = lst.EventSet(es, len(inputs), max(i.n_hits for i in inputs) + 1024)
    try:
        s.upload_packed(0, *lst.pack_events(inputs))
        s.run(0, len(inputs))
        n = len(inputs)
        hits, ln, seed, typ, tco, hco = s.output(0, n, 31000 * n, 31000 * 14 * n)
        for i in range(n):
            one = s.output(i, 1)
            t0, t1, h0, h1 = (int(v) for v in (tco[i], tco[i + 1], hco[i], hco[i + 1]))
            for a, b in zip((hits[h0:h1], ln[t0:t1], seed[t0:t1], typ[t0:t1]), one[:4]):
                assert a.tobytes() == b.tobytes()
            assert int(one[1].sum()) == one[0].size
        if tco[-1] > 1:
            with pytest.raises(lst.LSTError):
                s.output(0, n, int(tco[-1]) - 1, 31000 * 14 * n)
    finally:
        s.close()
        es.close()

"""Mini-doublets, segments and triplets of a large batch, whose warps take several
lower modules at a time (from 32 events per launch), against each event on its
own: the same stores, every value equal.  Empty, one-muon and dense events, so
that tasks hold modules with no, few and many candidates."""
import numpy as np
import pytest

from tracklooper_b200 import gen, geometry, lst

pytestmark = pytest.mark.gpu

STORES = {"md": ("nMDs", "totOccupancyMDs"), "ls": ("nSegments", "totOccupancySegments")}


def objects(s, slot):
    out = {}
    for store, (n, tot) in STORES.items():
        counts = s.field(slot, f"{store}.{n}").astype(np.int64)
        out[f"{store}.{n}"], out[f"{store}.{tot}"] = counts, s.field(slot, f"{store}.{tot}").copy()
        lo = s.field(slot, "ranges.mdRanges" if store == "md" else "ranges.segmentRanges").reshape(-1, 2)[:, 0]
        n_lower = s.es.info["nLowerModules"]
        first = lo.astype(np.int64)
        live = np.concatenate([np.arange(first[m], first[m] + counts[m]) for m in np.nonzero(counts[:n_lower])[0]]
                              or [np.zeros(0, np.int64)])
        room = s.field(slot, f"{store}.anchorHitIndices" if store == "md" else f"{store}.dPhis").size
        for name in lst.field_names():
            if name.startswith(store + ".") and name not in out:
                a = s.field(slot, name)
                if a.size % room == 0:
                    out[name] = a.reshape(room, -1)[live]
    return out


@pytest.mark.parametrize("geo", ["OT800_IT615_pt0.8", "OT800_IT615_pt0.6"])
def test_large_batch_equals_single_events(geo):
    kinds = [(1, 0.0), (5, 0.0), (3, 20.0), (1, 0.0)]
    events = [(kinds[i % 4][0], 50 + i, kinds[i % 4][1]) for i in range(32)] + [(2, 90, 200.0)]
    inputs = [gen.generate_event(*e) for e in events]
    es = lst.ES(device=0, geometry_dir=geometry.geometry_dir(geo))
    hits = max(i.n_hits for i in inputs) + 1024
    batch, one = lst.EventSet(es, len(inputs), hits), lst.EventSet(es, 1, hits)
    try:
        batch.upload_packed(0, *lst.pack_events(inputs))
        batch.run(0, len(inputs))
        for i in (0, 1, 2, 7, 31, 32):
            one.upload_packed(0, *lst.pack_events(inputs[i:i + 1]))
            one.run(0, 1)
            a, b = objects(batch, i), objects(one, 0)
            for name, x in a.items():
                assert x.tobytes() == b[name].tobytes(), (i, name)
            assert batch.counts(i)["nSegments"] == one.counts(0)["nSegments"]
    finally:
        batch.close()
        one.close()
        es.close()

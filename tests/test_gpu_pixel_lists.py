"""The list paths of the quintuplet and pixel stages against the fallback walks
(lst_event_set_walk), which evaluate every candidate in the reference's loop
order: the same pT5s, pT3s and track candidates, every stored value equal.
Events from no candidates at all to PU400, both geometries (pt0.6 events have
several times the candidates), ragged batches included."""
import numpy as np
import pytest

from tracklooper_b200 import gen, geometry, lst

pytestmark = pytest.mark.gpu

FIELDS = {"pt5": ("nPixelQuintuplets", "totOccupancyPixelQuintuplets"),
          "pt3": ("nPixelTriplets", "totOccupancyPixelTriplets"),
          "tc": ("nTrackCandidates", None)}


def stores(s, slot):
    out = {}
    for store, (count, found) in FIELDS.items():
        n = int(s.field(slot, f"{store}.{count}")[0])
        out[f"{store}.{count}"] = n
        if found:
            out[f"{store}.{found}"] = int(s.field(slot, f"{store}.{found}")[0])
        room = {"pt5": 15000, "pt3": 5000, "tc": 31000}[store]
        for name in lst.field_names():
            if not name.startswith(store + ".") or name.startswith((f"{store}.n", f"{store}.totOcc")):
                continue
            a = s.field(slot, name)
            out[name] = a.reshape(room, -1)[:n].copy()
    # the quintuplets of every module, and how many were found
    counts = s.field(slot, "t5.nQuintuplets").astype(np.int64)
    first = s.field(slot, "ranges.quintupletModuleIndices").astype(np.int64)
    out["t5.nQuintuplets"], out["t5.totOccupancyQuintuplets"] = counts, s.field(slot, "t5.totOccupancyQuintuplets")
    live = np.concatenate([np.arange(first[m], first[m] + counts[m]) for m in np.nonzero(counts)[0]]
                          or [np.zeros(0, np.int64)])
    room = s.es.info["maxQuintuplets"]
    for name in lst.field_names():
        if name.startswith("t5.") and name not in out:
            a = s.field(slot, name)
            if a.size % room == 0:
                out[name] = a.reshape(room, -1)[live]
    return out


@pytest.mark.parametrize("geo,events", [
    ("OT800_IT615_pt0.8", [(1, 21, 0.0)]),
    ("OT800_IT615_pt0.8", [(3, 22, 20.0), (1, 23, 0.0), (2, 24, 0.0)]),
    ("OT800_IT615_pt0.8", [(5, 25, 0.0)]),
    ("OT800_IT615_pt0.8", [(2, 920, 400.0)]),
    ("OT800_IT615_pt0.6", [(5, 26, 0.0), (3, 27, 60.0)]),
])
def test_lists_equal_walk(geo, events):
    inputs = [gen.generate_event(*e) for e in events]
    es = lst.ES(device=0, geometry_dir=geometry.geometry_dir(geo))
    got = []
    try:
        for walk in (False, True):
            s = lst.EventSet(es, len(inputs), max(i.n_hits for i in inputs) + 1024)
            try:
                s.set_walk(walk)
                blob, offsets = lst.pack_events(inputs)
                s.upload_packed(0, blob, offsets)
                s.run(0, len(inputs))
                got.append([stores(s, i) for i in range(len(inputs))])
            finally:
                s.close()
    finally:
        es.close()
    for a, b in zip(*got):
        for name, x in a.items():
            y = b[name]
            if isinstance(x, np.ndarray):
                assert x.tobytes() == y.tobytes(), name
            else:
                assert x == y, name

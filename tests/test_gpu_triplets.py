"""Triplets made by blocks of one, two and four warps over several modules at a
time: the same stores, every value equal (one warp takes a task's candidates
strictly one step after the other), and in each module the reference's order
(inner segment, then outer segment) over segments that share a mini-doublet.
Batches of 1 (8 modules per task) and 5 events (16), from empty events and single
muons to modules with several times more inner segments than a block has threads."""
import numpy as np
import pytest

from tracklooper_b200 import gen, geometry, lst

pytestmark = pytest.mark.gpu


def triplets(s, slot, n_lower):
    counts = s.field(slot, "t3.nTriplets")[:n_lower].astype(np.int64)
    first = s.field(slot, "ranges.tripletModuleIndices")[:n_lower].astype(np.int64)
    live = np.concatenate([np.arange(first[m], first[m] + counts[m]) for m in np.nonzero(counts)[0]]
                          or [np.zeros(0, np.int64)])
    room = s.es.info["maxTriplets"]
    out = {"counts": counts, "found": s.field(slot, "t3.totOccupancyTriplets")[:n_lower]}
    for name in lst.field_names():
        if name.startswith("t3.") and not name.startswith(("t3.n", "t3.totOcc")):
            a = s.field(slot, name)
            assert a.size % room == 0
            out[name] = a.reshape(room, -1)[live]
    return out


@pytest.mark.parametrize("geo,events", [
    ("OT800_IT615_pt0.8", [(1, 31, 0.0)]),
    ("OT800_IT615_pt0.8", [(2, 32, 250.0)]),
    ("OT800_IT615_pt0.8", [(5, 33, 0.0), (1, 34, 0.0), (3, 35, 20.0), (2, 36, 0.0), (1, 37, 0.0)]),
    ("OT800_IT615_pt0.6", [(2, 38, 200.0)]),
])
def test_block_width_changes_nothing(geo, events):
    inputs = [gen.generate_event(*e) for e in events]
    es = lst.ES(device=0, geometry_dir=geometry.geometry_dir(geo))
    n_lower = es.info["nLowerModules"]
    got = []
    try:
        for warps in (1, 2, 4):
            s = lst.EventSet(es, len(inputs), max(i.n_hits for i in inputs) + 1024)
            try:
                s.set_launch_shape("kCreateT3", warps, 32)
                s.upload_packed(0, *lst.pack_events(inputs))
                s.run(0, len(inputs))
                got.append([triplets(s, i, n_lower) for i in range(len(inputs))])
                segs = [s.field(i, "ls.mdIndices").reshape(-1, 2) for i in range(len(inputs))]
            finally:
                s.close()
    finally:
        es.close()
    for other in got[1:]:
        for a, b in zip(got[0], other):
            for name, x in a.items():
                assert x.tobytes() == b[name].tobytes(), name
    for a, md in zip(got[0], segs):
        pair = a["t3.segmentIndices"].astype(np.int64)
        assert (md[pair[:, 0], 1] == md[pair[:, 1], 0]).all()
        module = np.repeat(np.arange(n_lower), a["counts"])
        same = module[1:] == module[:-1]
        up = (pair[1:, 0] > pair[:-1, 0]) | ((pair[1:, 0] == pair[:-1, 0]) & (pair[1:, 1] > pair[:-1, 1]))
        assert (up | ~same).all()

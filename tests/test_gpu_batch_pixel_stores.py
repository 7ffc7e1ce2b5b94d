"""A batch's triplets, pixel mini-doublets and pixel segments against each event's
on its own: a few events per launch take other task widths for the triplets than
many do, and the pixel stores are written by a thread per mini-doublet, then per
segment.  Every value equal; batches on both sides of the widths' boundaries."""
import numpy as np
import pytest

from tracklooper_b200 import gen, geometry, lst

pytestmark = pytest.mark.gpu


COUNTS = {f"{store}.{f}" for store, fields in (("md", ("nMDs", "totOccupancyMDs")),
                                               ("ls", ("nSegments", "totOccupancySegments")),
                                               ("t3", ("nTriplets", "totOccupancyTriplets"))) for f in fields}
PER_PLS = {"ls." + f for f in ("seedIdx", "charge", "superbin", "pLSHitsIdxs", "pixelType", "isQuad", "isDup", "partOfPT5",
                               "ptIn", "ptErr", "px", "py", "pz", "etaErr", "eta", "phi", "score", "circleCenterX",
                               "circleCenterY", "circleRadius")}
# segment fields that are not stored for pixel segments (SDL/Segment.h:392-453)
PLS_UNSET = {"ls.dPhis", "ls.dPhiMins", "ls.dPhiMaxs", "ls.dPhiChangeMins", "ls.dPhiChangeMaxs"}


def objects(s, slot, n_pls):
    """The live triplets of a slot, and its pixel module's objects, every field."""
    info = s.es.info
    n_lower = info["nLowerModules"]
    found = {name: s.field(slot, name)[:n_lower + 1].copy() for name in COUNTS}
    assert found["md.nMDs"][n_lower] == 2 * n_pls and found["ls.nSegments"][n_lower] == n_pls
    counts = found["t3.nTriplets"][:n_lower].astype(np.int64)
    first = s.field(slot, "ranges.tripletModuleIndices")[:n_lower].astype(np.int64)
    md0 = int(s.field(slot, "ranges.miniDoubletModuleIndices")[n_lower])
    ls0 = int(s.field(slot, "ranges.segmentModuleIndices")[n_lower])
    rows = {"md": np.arange(md0, md0 + 2 * n_pls), "ls": np.arange(ls0, ls0 + n_pls), "pls": np.arange(n_pls),
            "t3": np.concatenate([np.arange(first[m], first[m] + counts[m]) for m in np.nonzero(counts)[0]]
                                 or [np.zeros(0, np.int64)])}
    room = {"md": info["nTotalMDs"], "ls": info["nTotalSegments"], "pls": 50000, "t3": info["maxTriplets"]}
    out = found
    for name in lst.field_names():
        store = "pls" if name in PER_PLS else name.split(".")[0]
        if store in rows and name not in COUNTS | PLS_UNSET:
            out[name] = s.field(slot, name).reshape(room[store], -1)[rows[store]]
    return out


@pytest.mark.parametrize("geo,n", [("OT800_IT615_pt0.8", 3), ("OT800_IT615_pt0.8", 4), ("OT800_IT615_pt0.8", 9),
                                   ("OT800_IT615_pt0.6", 5)])
def test_batch_equals_single_events(geo, n):
    kinds = [(2, 200.0), (1, 0.0), (5, 0.0), (3, 20.0)]
    inputs = [gen.generate_event(kinds[i % 4][0], 60 + i, kinds[i % 4][1]) for i in range(n)]
    es = lst.ES(device=0, geometry_dir=geometry.geometry_dir(geo))
    hits = max(i.n_hits for i in inputs) + 1024
    batch, one = lst.EventSet(es, n, hits), lst.EventSet(es, 1, hits)
    try:
        batch.upload_packed(0, *lst.pack_events(inputs))
        batch.run(0, n)
        for i, inp in enumerate(inputs):
            # (the event on its own through the Event members: another ingest path)
            one.add_inputs(0, inp)
            for st in lst.STAGE_ORDER:
                one.run_stage(0, st)
            a, b = objects(batch, i, inp.n_pls), objects(one, 0, inp.n_pls)
            assert len(a) == 3 * 2 + 34 + 6 + 20 + 11
            for name, x in a.items():
                assert x.tobytes() == b[name].tobytes(), (i, name)
    finally:
        batch.close()
        one.close()
        es.close()

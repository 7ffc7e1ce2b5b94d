"""Stages left out, run again and fed in another order: what a stage reads of an
event must be that event's own, whatever the slot held before."""
import numpy as np
import pytest

from tracklooper_b200 import gen, lst

pytestmark = pytest.mark.gpu

ROOM = {"pt5": 15000, "pt3": 5000, "tc": 31000}
COUNT = {"pt5": "pt5.nPixelQuintuplets", "pt3": "pt3.nPixelTriplets", "tc": "tc.nTrackCandidates"}


def stores(s, slot):
    """The live pT5s, pT3s and track candidates of a slot, every field."""
    out = {}
    for store, count in COUNT.items():
        n = int(s.field(slot, count)[0])
        out[count] = np.array([n])
        for name in lst.field_names():
            if name.startswith(store + ".") and not name.startswith((f"{store}.n", f"{store}.totOcc")):
                out[name] = s.field(slot, name).reshape(ROOM[store], -1)[:n].copy()
    return out


def same(a, b):
    for name, x in a.items():
        assert x.tobytes() == b[name].tobytes(), name


@pytest.fixture(scope="module")
def es():
    e = lst.ES(device=0)
    yield e
    e.close()


@pytest.fixture(scope="module")
def inputs():
    return gen.generate_event(2, 70, 200.0), gen.generate_event(2, 71, 200.0)


# the pLS alone; the pT3s with them; segments and triplets but no quintuplets
@pytest.mark.parametrize("stages", [("tc",), ("pls_clean", "tc"), ("md", "ls", "t3", "pls_clean", "pt5", "pt3", "tc")])
def test_candidates_without_the_quintuplet_stage(es, inputs, stages):
    """On a slot that another event has filled, as on a fresh one; and the
    quintuplets that the other event left behind are not touched."""
    before, inp = inputs
    hits = max(i.n_hits for i in inputs) + 1024
    got = []
    for used in (False, True):
        s = lst.EventSet(es, 1, hits)
        try:
            if used:
                s.add_inputs(0, before)
                for st in lst.STAGE_ORDER:
                    s.run_stage(0, st)
                assert s.counts(0)["nQuintuplets"] > 100
                s.reset(0)
            s.add_inputs(0, inp)
            left = s.field(0, "t5.isDup") if used else None
            for st in stages:
                s.run_stage(0, st)
            if used:
                assert s.field(0, "t5.isDup").tobytes() == left.tobytes()
            got.append(stores(s, 0))
        finally:
            s.close()
    assert got[0]["tc.nTrackCandidates"][0] > 1000
    if "pt3" in stages:
        assert got[0]["pt3.nPixelTriplets"][0] > 100
    same(*got)


def shuffled(pls, rng):
    order = rng.permutation(len(pls["hitIndices0"]))
    return {name: a[order] for name, a in pls.items()}


@pytest.mark.parametrize("walk", [False, True])
@pytest.mark.parametrize("twice", [False, True])
def test_pixel_segments_after_the_mini_doublets(es, inputs, twice, walk):
    """Added after createMiniDoublets on a slot that another event has filled, or
    added in another order first and again then: the candidates of the usual order."""
    before, inp = inputs
    got = []
    for late in (False, True):
        s = lst.EventSet(es, 1, max(i.n_hits for i in inputs) + 1024)
        try:
            s.set_walk(walk)
            if late:
                s.add_inputs(0, before)
                for st in lst.STAGE_ORDER:
                    s.run_stage(0, st)
            s.add_hits(0, inp.x, inp.y, inp.z, inp.detId, inp.idxInNtuple)
            if late:
                if twice:
                    s.add_pixel_segments(0, shuffled(inp.pls, np.random.default_rng(5)))
                s.run_stage(0, "md")
                s.add_pixel_segments(0, inp.pls)
            else:
                s.add_pixel_segments(0, inp.pls)
                s.run_stage(0, "md")
            for st in lst.STAGE_ORDER[1:]:
                s.run_stage(0, st)
            got.append(stores(s, 0))
        finally:
            s.close()
    assert got[0]["pt5.nPixelQuintuplets"][0] > 100 and got[0]["pt3.nPixelTriplets"][0] > 100
    same(*got)


def test_candidates_again_and_again(es, inputs):
    """The track-candidate stage run on one event until its candidates fill the
    store (it appends to them): they end there, the first ones stay, the event in
    the next slot too, and a reset gives the first run's candidates again."""
    s = lst.EventSet(es, 2, max(i.n_hits for i in inputs) + 1024)
    try:
        for slot, inp in enumerate(inputs):
            s.add_inputs(slot, inp)
            for st in lst.STAGE_ORDER:
                s.run_stage(slot, st)
        first, other = stores(s, 0), stores(s, 1)
        n = int(first["tc.nTrackCandidates"][0])
        last = n
        for _ in range(24):
            s.run_stage(0, "tc")
            now = int(s.field(0, "tc.nTrackCandidates")[0])
            assert last <= now <= ROOM["tc"]
            last = now
        assert last >= 30000 and s.counts(0)["status"] & lst.STATUS_TC_TRUNCATED
        again = stores(s, 0)
        for name, x in first.items():
            if name.startswith("tc.") and name != "tc.nTrackCandidates":
                assert again[name][:n].tobytes() == x.tobytes(), name
        same(other, stores(s, 1))
        s.add_inputs(0, inputs[0])
        for st in lst.STAGE_ORDER:
            s.run_stage(0, st)
        same(first, stores(s, 0))
    finally:
        s.close()

"""Places of the kept seeds in the event at the edges of the conversion's chunks
(256 seeds) and on uneven batches: which seeds are kept, in which order, and the
pseudo-hits each appends, against a plain restatement of LST::prepareInput's
selection (SDL/LST.cc:193-262).  Whole numbers, so they must be equal."""
import numpy as np
import pytest

from tracklooper_b200 import gen, lst

pytestmark = pytest.mark.gpu


def cut(seeds, n, short=()):
    """The first n seeds; the ones in `short` lose their hits but two."""
    lens = np.diff(seeds.hit_offsets.astype(np.int64))[:n]
    lists = [seeds.hit_idx[seeds.hit_offsets[i]:seeds.hit_offsets[i + 1]][:2 if i in short else None] for i in range(n)]
    lens = np.array([len(h) for h in lists], np.int64)
    off = np.zeros(n + 1, np.uint32)
    off[1:] = np.cumsum(lens)
    see = {k: v[:n].copy() for k, v in seeds.see.items()}
    idx = np.concatenate(lists).astype(np.int32) if n else np.zeros(0, np.int32)
    return gen.SeedInput(see, off, idx, seeds.ph2_detId, seeds.ph2_x, seeds.ph2_y, seeds.ph2_z)


def expected(s):
    px, py = (s.see[f"see_stateTrajGlbP{c}"].astype(np.float64) for c in "xy")
    pt = np.sqrt(px * px + py * py).astype(np.float32)
    err = (np.float32(2) * s.see["see_ptErr"]).astype(np.float64)
    passes = pt.astype(np.float64) > 0.8 - err
    lens = np.diff(s.hit_offsets.astype(np.int64))
    keep = passes & (lens >= 3)
    pseudo = np.where(lens > 3, 4, 3)[keep]
    first = s.n_ph2 + np.concatenate(([0], np.cumsum(pseudo)[:-1])) if keep.any() else np.zeros(0, np.int64)
    starts = s.hit_offsets[:-1].astype(np.int64)[keep]
    idx = np.concatenate([s.hit_idx[a:a + k] for a, k in zip(starts, pseudo)]) if keep.any() else np.zeros(0)
    return np.nonzero(keep)[0], first, pseudo, idx, bool((passes & (lens < 3)).any())


@pytest.mark.parametrize("sizes", [[0], [1], [255], [256], [257], [1000], [1, 0, 513, 2971], [2971] * 3])
def test_kept_seeds_and_pseudo_hits(sizes):
    full = gen.generate_event(3, 1, 40.0).seeds
    events = [cut(full, n, short={5, 300} if n > 600 else ()) for n in sizes]
    es = lst.ES(device=0)
    s = lst.EventSet(es, len(events), full.n_ph2 + 4 * full.n_seeds + 16)
    try:
        blob, offsets = lst.pack_seed_events(events)
        s.upload_seeds(0, blob, offsets)
        counts = s.batch_counts(0, len(events))
        for slot, e in enumerate(events):
            kept, first, pseudo, idx, short = expected(e)
            c = counts[slot]
            assert c["nPixelSegments"] == kept.size and c["nHits"] == e.n_ph2 + idx.size
            assert bool(c["status"] & lst.STATUS_INVALID_INPUT) == short
            assert np.array_equal(s.field(slot, "ls.seedIdx", kept.size), kept)
            assert np.array_equal(s.field(slot, "hits.idxs", c["nHits"])[e.n_ph2:], idx)
            assert np.array_equal(s.field(slot, "ls.isQuad", kept.size) != 0, pseudo == 4)
            base = es.info["nTotalSegments"] - 50000
            hit0 = s.field(slot, "ls.innerMiniDoubletAnchorHitIndices")[base:base + kept.size]
            assert np.array_equal(hit0, first)
    finally:
        s.close()
        es.close()

"""Duplicate removal of quintuplets within a module and of pT5s, against a
plain numpy restatement of the reference's pair loops (SDL/Kernels.h:202-249,
:356-382) on the stored objects.  The marks are whole numbers: they must be
equal.  Events from one muon to PU400, so that modules hold from none to
several hundred quintuplets (tiles of 32 pairs: full, ragged, diagonal) and
events hold from none to a few thousand pT5s."""
import numpy as np
import pytest

from tracklooper_b200 import gen, lst

pytestmark = pytest.mark.gpu

EVENTS = [(1, 7, 0.0), (3, 11, 20.0), (2, 645000, 0.0), (5, 921, 0.0), (2, 920, 400.0)]


@pytest.fixture(scope="module")
def es():
    e = lst.ES(device=0)
    yield e
    e.close()


def matched(a, b):
    """For every pair (i, j): how many of a[i]'s hits are among b[j]'s."""
    return (a[:, None, :, None] == b[None, :, None, :]).any(axis=3).sum(axis=2)


def wrap(d):
    pi = np.float32(np.pi)
    d = np.where(d > pi, d - np.float32(2) * pi, np.where(d < -pi, d + np.float32(2) * pi, d))
    return d.astype(np.float32)


@pytest.mark.parametrize("config,index,pileup", EVENTS)
def test_module_quintuplet_duplicates(es, config, index, pileup):
    inp = gen.generate_event(config, index, pileup)
    s = lst.EventSet(es, 1, inp.n_hits + 1024)
    try:
        s.add_inputs(0, inp)
        for st in ("md", "ls", "t3", "t5"):
            s.run_stage(0, st)
        n_t5 = s.field(0, "t5.nQuintuplets")
        first = s.field(0, "ranges.quintupletModuleIndices")
        last = int((first + n_t5.astype(np.int64))[n_t5 > 0].max(initial=1))
        eta, phi, score, is_dup = (s.field(0, f"t5.{f}", last) for f in ("eta", "phi", "score_rphisum", "isDup"))
        hits = s.field(0, "t5.hitIndices", 10 * last).reshape(-1, 10)
    finally:
        s.close()
    if pileup > 300:
        assert n_t5.max() > 64  # modules of several tiles
    for m in np.nonzero(n_t5)[0]:
        o = slice(int(first[m]), int(first[m]) + int(n_t5[m]))
        e, p, sc, h = eta[o], phi[o], score[o], hits[o]
        near = (np.abs(e[:, None] - e[None, :]) <= np.float32(0.1)) & (
            np.abs(wrap(p[:, None] - p[None, :])) <= np.float32(0.1))
        pair = np.triu(near & (matched(h, h) >= 7), 1)
        keep_second = sc[:, None] >= sc[None, :]  # the first of the pair goes
        expected = (pair & keep_second).any(axis=1) | (pair & ~keep_second).any(axis=0)
        assert np.array_equal(is_dup[o] != 0, expected), f"module {m} with {n_t5[m]} quintuplets"


@pytest.mark.parametrize("config,index,pileup", EVENTS)
def test_pt5_duplicates(es, config, index, pileup):
    inp = gen.generate_event(config, index, pileup)
    s = lst.EventSet(es, 1, inp.n_hits + 1024)
    try:
        s.add_inputs(0, inp)
        for st in ("md", "ls", "t3", "t5", "pls_clean", "pt5"):
            s.run_stage(0, st)
        n = int(s.field(0, "pt5.nPixelQuintuplets")[0])
        score, is_dup = (s.field(0, f"pt5.{f}", n) for f in ("score", "isDup"))
        hits = s.field(0, "pt5.hitIndices", 14 * n).reshape(-1, 14)
    finally:
        s.close()
    if pileup > 300:
        assert n > 1170
    i = np.arange(n)
    for a0 in range(0, n, 64):
        a = i[a0:a0 + 64]
        worse = (score[a][:, None] > score[None, :]) | ((score[a][:, None] == score[None, :]) & (a[:, None] > i[None, :]))
        expected = (worse & (matched(hits[a], hits) >= 7)).any(axis=1)
        assert np.array_equal(is_dup[a] != 0, expected), f"pT5s {a0}.. of {n}"

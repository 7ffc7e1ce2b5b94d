"""The workloads whose speed this framework is judged by.

A case is one pass of a user's program through the public entry points: the
C ABI of include/lst_b200.h (directly, or through tracklooper_b200.lst) for the
object-building chain, and tracklooper_b200.t5dnn for training the quintuplet
classifier.  Events come from the package's seeded generator with the
multiplicities of the chain's real use: single muons, light pileup, PU200, and
PU250 with displaced tracks.

Kinds of pass (the case's "api"):
  lst_run   lst_run: one event's CMSSW seed and hit vectors in host memory ->
            the track-candidate lists, as a producer calls it once per event
  event     the Event members one after the other on one event (addHitToEvent,
            addPixelSegmentToEvent, the eight stages), then its output lists
  batch     packed events in pinned host memory -> lst_batch_upload, all
            stages, output lists
  resident  events resident on the device: lst_batch_ingest, the stages as a
            CUDA graph, output lists
  stream    several batches of packed CMSSW seed events through two event sets
            in turn, each batch's copy staged while the other's stages run
  train     one step of the quintuplet classifier's training: logits, binary
            cross-entropy, gradient of all 2337 weights
"""
import ctypes
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from tracklooper_b200 import gen, geometry, lst, t5dnn

GEOMETRIES = {"pt0.8": "OT800_IT615_pt0.8", "pt0.6": "OT800_IT615_pt0.6"}
TC_PER_EVENT = 12000  # room for track candidates per event in the output buffers (a PU200 event has about 6000)
HITS_PER_TC = 8  # and for hits, on the average candidate
STREAM_SETS = 2


def chain(name, api, config, events, pileup, geometry="pt0.8", cuts=False, batches=1):
    """`events` per batch; `pileup`: mean number of vertices (0: the
    generator's own for the configuration); `cuts`: cut-only T5 selection."""
    return {"name": name, "api": api, "config": config, "events": events, "pileup": pileup, "geometry": geometry,
            "cuts": cuts, "batches": batches}


def listed():
    return [
        # The smallest call there is: one muon's hits; launches and copies count.
        chain("lst_run_muon", "lst_run", 1, 1, 0.0),
        # The reference's own use, one PU200 event per call, from CMSSW vectors.
        chain("lst_run_pu200", "lst_run", 2, 1, 200.0),
        # The reference's standalone driver: stage by stage on one lighter event.
        chain("event_pu60", "event", 3, 1, 60.0),
        # A few light events, an odd number of them: the GPU is far from full.
        chain("batch5_pu30", "batch", 3, 5, 30.0),
        # A producer that gathers a few PU200 events before it calls.
        chain("batch8_pu200", "batch", 2, 8, 200.0),
        # The densest events (PU250, 5% displaced), cut-only T5 selection.
        chain("batch13_pu250_cuts", "batch", 5, 13, 250.0, cuts=True),
        # The looser pt0.6 maps: more segments and triplets per event.
        chain("resident16_pt06", "resident", 2, 16, 200.0, geometry="pt0.6"),
        # The headline benchmark: 64 PU200 events per launch.
        chain("resident64_pu200", "resident", 2, 64, 200.0),
        # Serving: uneven events (PU140-250), copies overlapped with the stages.
        chain("stream4x12_pu140_250", "stream", 3, 12, 0.0, batches=4),
        # Training the classifier: the shipped batch size, and one large odd batch.
        {"name": "train_8192", "api": "train", "candidates": 8192},
        {"name": "train_262143", "api": "train", "candidates": 262143},
    ]


def _log_uniform(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def draw(rng):
    api = rng.choice(("lst_run", "event", "batch", "batch", "resident", "resident", "stream", "train"))
    if api == "train":
        return {"api": api, "candidates": int(_log_uniform(rng, 2048, 262143))}
    config = rng.choice((2, 2, 3, 5))
    pileup = round(_log_uniform(rng, 20.0, 250.0), 2)
    geo = rng.choice(("pt0.8", "pt0.8", "pt0.8", "pt0.6"))
    # no more work than the largest listed case
    most = 64 * 200.0 / pileup / (2.5 if geo == "pt0.6" else 1.25)
    batches = 1
    events = 1
    if api in ("batch", "resident"):
        events = max(1, int(_log_uniform(rng, 1, min(64.0, most))))
    elif api == "stream":
        batches = rng.randint(2, 4)
        events = max(1, int(_log_uniform(rng, 2, min(16.0, most / batches))))
    case = chain("", api, config, events, pileup, geo, rng.random() < 0.25, batches)
    del case["name"]
    return case


# ---------------------------------------------------------------- inputs
_setups = {}


def _setup(geo):
    """The event setup: a program loads it once."""
    if geo not in _setups:
        _setups[geo] = lst.ES(device=0, geometry_dir=geometry.geometry_dir(GEOMETRIES[geo]))
    return _setups[geo]


def _events(case, seed):
    n = case["events"] * case["batches"]
    first = (int(seed) * 1009 + 17) % (1 << 24) * 128
    with ThreadPoolExecutor(max(1, min(16, os.cpu_count() or 1))) as pool:
        return list(pool.map(lambda i: gen.generate_event(case["config"], first + i, case["pileup"]), range(n)))


def _pinned(a):
    t = torch.empty(max(int(a.nbytes), 1), dtype=torch.uint8, pin_memory=True)
    v = t.numpy()[:a.nbytes]
    v[:] = a
    return t, v


class Lists:
    """Output buffers of one lst_batch_get_output call, in pinned host memory:
    the lists end where the offsets say, zeros follow."""

    def __init__(self, events):
        tc = TC_PER_EVENT * events
        self.keep = [torch.zeros(n, dtype=dt, pin_memory=True)
                     for n, dt in ((tc * HITS_PER_TC, torch.int32), (tc, torch.int32), (tc, torch.int32),
                                   (tc, torch.int16))]
        self.hits, self.len, self.seed, self.type = (t.numpy() for t in self.keep)
        self.tc_offsets = np.zeros(events + 1, np.uint64)
        self.hit_offsets = np.zeros(events + 1, np.uint64)
        self.c = lst.Output(self.hits.ctypes.data, self.hits.size, self.len.ctypes.data, self.seed.ctypes.data,
                            self.type.ctypes.data, self.len.size, self.tc_offsets.ctypes.data,
                            self.hit_offsets.ctypes.data)

    def arrays(self):
        return {"hits": self.hits, "len": self.len, "seedIdx": self.seed, "type": self.type,
                "tc_offsets": self.tc_offsets.view(np.int64), "hit_offsets": self.hit_offsets.view(np.int64)}


def _read(eset, events, lists):
    lst._check(lst.library().lst_batch_get_output(eset.handle, 0, events, ctypes.byref(lists.c)),
               "lst_batch_get_output")
    return lists.arrays()


def _event_set(case, inputs):
    hits = max(i.n_hits for i in inputs)
    eset = lst.EventSet(_setup(case["geometry"]), n_slots=case["events"], max_hits=(hits + 4095) // 4096 * 4096)
    if case["cuts"]:
        eset.set_t5_method(lst.T5_CUTS)
    return eset


class State:
    pass


def prepare(case, seed):
    torch.cuda.init()
    s = State()
    s.case = case
    s.api = case["api"]
    if s.api == "train":
        s.x, s.y, s.w = (t.cuda() for t in _training_inputs(case, seed))
        s.w.requires_grad_(True)
        return s
    inputs = _events(case, seed)
    n = case["events"]
    s.events = n
    s.sets = [_event_set(case, inputs) for _ in range(STREAM_SETS if s.api == "stream" else 1)]
    s.set = s.sets[0]
    s.out = [Lists(n) for _ in range(case["batches"])]
    if s.api == "lst_run":
        s.seeds, s.keep = lst.seed_struct(inputs[0].seeds)
    elif s.api == "event":
        s.input = inputs[0]
    elif s.api == "stream":
        packed = [lst.pack_seed_events([i.seeds for i in inputs[b * n:(b + 1) * n]]) for b in range(case["batches"])]
        s.keep, s.blobs = zip(*[_pinned(blob) for blob, _ in packed])
        s.offsets = [off for _, off in packed]
    else:
        blob, s.offsets = lst.pack_events(inputs)
        s.keep, s.blob = _pinned(blob)
        if s.api == "resident":
            s.set.upload_packed(0, s.blob, s.offsets)
    for e in s.sets:
        e.sync()
    return s


def run(s):
    if s.api == "train":
        logit = t5dnn.t5dnn_logits(s.x, s.w)
        loss = torch.nn.functional.binary_cross_entropy_with_logits(logit, s.y)
        grad, = torch.autograd.grad(loss, s.w)
        return {"logit": logit.detach(), "loss": loss.detach(), "grad": grad}
    e, n = s.set, s.events
    if s.api == "lst_run":
        lst._check(lst.library().lst_run(e.handle, 0, ctypes.byref(s.seeds), ctypes.byref(s.out[0].c)), "lst_run")
        return s.out[0].arrays()
    if s.api == "event":
        e.add_inputs(0, s.input)
        for stage in lst.STAGE_ORDER:
            e.run_stage(0, stage)
        return _read(e, n, s.out[0])
    if s.api == "batch":
        e.upload_packed(0, s.blob, s.offsets)
        e.run(0, n)
        return _read(e, n, s.out[0])
    if s.api == "resident":
        e.ingest(0, n)
        e.run_graph(0, n)
        return _read(e, n, s.out[0])
    # stream
    outs = []
    s.sets[0].stage(0, s.blobs[0], s.offsets[0], seed_layout=True)
    for b in range(len(s.blobs)):
        cur = s.sets[b % STREAM_SETS]
        cur.ingest_staged()
        cur.run_graph(0, n)
        if b + 1 < len(s.blobs):
            s.sets[(b + 1) % STREAM_SETS].stage(0, s.blobs[b + 1], s.offsets[b + 1], seed_layout=True)
        if b > 0:
            outs.append(_read(s.sets[(b - 1) % STREAM_SETS], n, s.out[b - 1]))
    outs.append(_read(cur, n, s.out[len(s.blobs) - 1]))
    return outs


# ------------------------------------------------------- classifier training
def _training_inputs(case, seed):
    """Standardised features as the training loop feeds them (a common spread
    per candidate on top of independent ones, as track features have), labels
    and He-initialised weights."""
    rng = np.random.default_rng([int(seed) & 0xffffffff, 38])
    n = case["candidates"]
    x = (0.8 * rng.standard_normal((n, t5dnn.N_FEATURES), dtype=np.float32)
         + 0.6 * rng.standard_normal((n, 1), dtype=np.float32))
    y = (rng.random(n, dtype=np.float32) < 0.6).astype(np.float32)
    return torch.from_numpy(x), torch.from_numpy(y), torch.from_numpy(t5dnn.random_weights(int(seed) & 0xffffffff))


def exact(case, seed):
    """The training step in 64 bits; the chain's outputs are whole numbers."""
    if case["api"] != "train":
        return None
    x, y, w = (t.double() for t in _training_inputs(case, seed))
    w.requires_grad_(True)
    w0, b0, w2, b2, w4, b4 = torch.split(w, [38 * 32, 32, 32 * 32, 32, 32, 1])
    h1 = torch.relu(x @ w0.reshape(38, 32) + b0)
    h2 = torch.relu(h1 @ w2.reshape(32, 32) + b2)
    logit = h2 @ w4 + b4
    loss = torch.nn.functional.binary_cross_entropy_with_logits(logit, y)
    grad, = torch.autograd.grad(loss, w)
    return {"logit": logit.detach(), "loss": loss.detach(), "grad": grad}


def work(case):
    """Training: features, labels and logits once, the multiply-adds of the
    forward and backward passes.  Chain: each event's packed inputs (20 B per
    hit, 66 B per pixel segment) read and its output lists (10 B per track
    candidate and 4 B per hit on it) written once, at the generator's mean
    multiplicities per pileup vertex."""
    if case["api"] == "train":
        n = case["candidates"]
        forward = 2 * (38 * 32 + 32 * 32 + 32)
        backward = 2 * (38 * 32 + 2 * 32 * 32 + 2 * 32)
        return {"bytes": n * (38 * 4 + 4 + 4) + 2 * 4 * t5dnn.N_PARAMS, "flops": n * (forward + backward)}
    events = case["events"] * case["batches"]
    if case["config"] == 1:
        return {"bytes": events * (20 * 20 + 66 + 50)}
    vertices = case["pileup"] or {2: 200.0, 3: 195.0, 5: 250.0}[case["config"]]
    per_vertex = 752 * 20 + 73 * 66 + 31 * (10 + 9 * 4)
    return {"bytes": int(events * vertices * per_vertex)}

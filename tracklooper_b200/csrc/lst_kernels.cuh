// CUDA kernels of the LST object-building chain.  Every kernel takes the
// device event setup by value and an array of per-event views; blockIdx.y
// selects the event, so one launch processes a whole batch of events.
//
// Ordering.  The reference appends objects with atomic counters; its serial
// CPU backend therefore stores them in loop-nest order, and per-module
// occupancy caps keep the first N in that order.  Here each module (or pixel
// seed) is owned by one warp that walks the flattened loop nest in order,
// 32 candidates at a time, and places accepted objects with a warp ballot
// prefix, so object indices equal the reference CPU backend's.
#pragma once

#include <cuda_runtime.h>

#include "lst_device.h"

namespace lst {

  constexpr unsigned int kFullMask = 0xffffffffu;

  // T5 classifier weights (uploaded once per process from the weight file).
  __constant__ T5DnnWeights c_t5dnn;
  __constant__ float c_t5dnnWP = kT5DnnWP;  // DNN working point of the loaded weights

  __device__ T5DnnWeights g_t5dnn;         // the same weights in memory (kT5Classify stages them in shared memory)

  struct ConstDnn {
    __device__ __forceinline__ const T5DnnWeights& get() const { return c_t5dnn; }
  };

  // First statement of every kernel that LST_LAUNCH launches.  Those launches let
  // a kernel's blocks in as soon as the last block of the stream's previous kernel
  // has exited (programmatic dependent launch), so that the launch overlaps the
  // previous kernel's completion: a batch is 44 kernels from its unpacking to its
  // candidates, most of them a few microseconds long.  The wait returns when the
  // previous kernel has completed and its writes are visible; since every block of
  // every kernel waits here before it does anything (or exits), that holds for all
  // kernels before it as well.  One muon's lst_run 437 -> 289 us, five PU30 events 865 -> 750, one
  // PU200 event 1734 -> 1582, 64 PU200 events unchanged.  Letting the next kernel
  // in at the start of the previous one brought no more, and blocks waiting
  // behind a one-block kernel kept other streams' kernels off the SMs (two event
  // sets in turn 9.36 -> 11.0 ms).
  __device__ __forceinline__ void kernelEntry() { cudaGridDependencySynchronize(); }

  __device__ __forceinline__ unsigned int laneId() { return threadIdx.x & 31u; }
  __device__ __forceinline__ unsigned int lanesBelowMask() { return (1u << laneId()) - 1u; }

  // Rank of this lane's flag among the set flags of lower lanes; total = set flags in the warp.
  __device__ __forceinline__ unsigned int warpRank(bool flag, unsigned int& total) {
    unsigned int b = __ballot_sync(kFullMask, flag);
    total = __popc(b);
    return __popc(b & lanesBelowMask());
  }

  // Exclusive prefix sums of countOf(0..n-1) into pre[0..n] (pre[n] = total),
  // computed by one warp.  pre must be warp-private shared memory.
  template <typename F>
  __device__ __forceinline__ unsigned int warpPrefix(unsigned int* pre, int n, F countOf) {
    unsigned int carry = 0;
    for (int base = 0; base < n; base += 32) {
      int i = base + int(laneId());
      unsigned int c = (i < n) ? countOf(i) : 0u;
      unsigned int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        unsigned int y = __shfl_up_sync(kFullMask, incl, o);
        if (int(laneId()) >= o)
          incl += y;
      }
      if (i < n)
        pre[i] = carry + incl - c;
      carry += __shfl_sync(kFullMask, incl, 31);
    }
    if (laneId() == 0)
      pre[n] = carry;
    __syncwarp();
    return carry;
  }

  // Largest k in [0, n) with pre[k] <= f (pre[n] > f).
  __device__ __forceinline__ int findSlot(const unsigned int* pre, int n, unsigned int f) {
    int lo = 0, hi = n;
    while (hi - lo > 1) {
      int mid = (lo + hi) >> 1;
      if (pre[mid] <= f)
        lo = mid;
      else
        hi = mid;
    }
    return lo;
  }

  __device__ __forceinline__ unsigned int laneInclusiveSum(unsigned int v) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned int y = __shfl_up_sync(kFullMask, v, o);
      if (int(laneId()) >= o)
        v += y;
    }
    return v;
  }

  // Block-wide exclusive scan (blockDim.x a multiple of 32, <= 1024).
  __device__ __forceinline__ unsigned int blockExclusiveScan(unsigned int v, unsigned int& total) {
    __shared__ unsigned int sWarp[32];
    __shared__ unsigned int sTotal;
    unsigned int lane = laneId(), wid = threadIdx.x >> 5;
    unsigned int nw = blockDim.x >> 5;
    unsigned int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      unsigned int y = __shfl_up_sync(kFullMask, incl, o);
      if (int(lane) >= o)
        incl += y;
    }
    if (lane == 31)
      sWarp[wid] = incl;
    __syncthreads();
    if (wid == 0) {
      unsigned int w = (lane < nw) ? sWarp[lane] : 0u;
      unsigned int wi = w;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        unsigned int y = __shfl_up_sync(kFullMask, wi, o);
        if (int(lane) >= o)
          wi += y;
      }
      if (lane < nw)
        sWarp[lane] = wi - w;
      if (lane == 31)
        sTotal = wi;
    }
    __syncthreads();
    unsigned int excl = sWarp[wid] + incl - v;
    total = sTotal;
    __syncthreads();
    return excl;
  }

  // The lower modules' cut constants, once per event setup.
  __global__ void kModuleCuts(Modules m, MDCut* mdCuts, LSCut* lsCuts) {
    const unsigned int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.nLowerModules)
      return;
    mdCuts[i] = mdCut(m, static_cast<uint16_t>(i));
    lsCuts[i] = lsCut(m, static_cast<uint16_t>(i));
  }

  // =============================================================== reset
  // Hit -> pLS index of the pLS cleaning: chains of (pLS, hit slot) entries
  // e = 4 pLS + slot in a hash table keyed by the stored pixel hit
  // (pLSHitsIdxs[e]): a head per bucket, a next entry per entry.  The heads are
  // empty when kPixelIngest inserts every entry once: kResetEvent empties them,
  // and for pixel segments added to an event on their own kPLSHitReset does.
  constexpr unsigned int kPLSHitBucketBits = 15;
  constexpr unsigned int kPLSHitBuckets = 1u << kPLSHitBucketBits;
  constexpr unsigned int kPLSHitNone = 0xffffffffu;
  LST_DEV unsigned int plsHitBucket(unsigned int h) { return (h * 2654435761u) >> (32 - kPLSHitBucketBits); }

  __global__ void kPLSHitReset(const EventView* evs) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    for (unsigned int i = blockIdx.x * blockDim.x + threadIdx.x; i < kPLSHitBuckets; i += gridDim.x * blockDim.x)
      ev.plsHitHead[i] = kPLSHitNone;
  }

  LST_DEV void pixCountersClear(const EventView& ev) {
    ev.sc->pixNext = 0;
    ev.sc->pixQueueCount = 0;
    ev.sc->pixPassCount = 0;
    ev.sc->pixOverflow = 0;
  }

  __global__ void kResetEvent(DeviceES es, const EventView* evs) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    for (unsigned int i = blockIdx.x * blockDim.x + threadIdx.x; i < kPLSHitBuckets; i += gridDim.x * blockDim.x)
      ev.plsHitHead[i] = kPLSHitNone;
    const unsigned int nMod = es.nModules, nLower = es.nLowerModules;
    for (unsigned int i = blockIdx.x * blockDim.x + threadIdx.x; i < 2u * nMod; i += gridDim.x * blockDim.x) {
      ev.hits.hitRanges[i] = -1;
      ev.rg.mdRanges[i] = -1;
      ev.rg.segmentRanges[i] = -1;
      ev.rg.tripletRanges[i] = -1;
      ev.rg.quintupletRanges[i] = -1;
      if (i < nMod) {
        ev.hits.hitRangesLower[i] = -1;
        ev.hits.hitRangesUpper[i] = -1;
        ev.hits.hitRangesnLower[i] = -1;
        ev.hits.hitRangesnUpper[i] = -1;
      }
      if (i <= nLower) {
        ev.md.nMDs[i] = 0;
        ev.md.totOccupancyMDs[i] = 0;
        ev.ls.nSegments[i] = 0;
        ev.ls.totOccupancySegments[i] = 0;
        ev.rg.miniDoubletModuleIndices[i] = es.mdOffset[i];
        ev.rg.miniDoubletModuleOccupancy[i] = es.mdCap[i];
        ev.rg.segmentModuleIndices[i] = es.lsOffset[i];
        ev.rg.segmentModuleOccupancy[i] = es.lsCap[i];
      }
      if (i < nLower) {
        ev.t3.nTriplets[i] = 0;
        ev.t3.totOccupancyTriplets[i] = 0;
        ev.t5.nQuintuplets[i] = 0;
        ev.t5.totOccupancyQuintuplets[i] = 0;
        ev.rg.quintupletModuleIndices[i] = -1;
        ev.rg.quintupletModuleOccupancy[i] = 0;
        ev.rg.tripletModuleIndices[i] = 0;
        ev.rg.tripletModuleOccupancy[i] = 0;
      }
      if (i == 0) {
        ev.sc->status = 0;
        ev.sc->mdNext = 0;
        ev.sc->lsNext = 0;
        ev.sc->t3Next = 0;
        pixCountersClear(ev);
        // (the track-candidate stage walks this list, also of an event whose
        // quintuplet stage has not run)
        ev.sc->t5ListCount = 0;
        ev.sc->walkDone = 0;
        ev.sc->plsTCDone = 0;
        ev.sc->nPT5Total = 0;
        ev.sc->nPT3Total = 0;
        *ev.pt3.nPixelTriplets = 0;
        *ev.pt3.totOccupancyPixelTriplets = 0;
        *ev.pt5.nPixelQuintuplets = 0;
        *ev.pt5.totOccupancyPixelQuintuplets = 0;
        *ev.tc.nTrackCandidates = 0;
        *ev.tc.nTrackCandidatespT3 = 0;
        *ev.tc.nTrackCandidatespT5 = 0;
        *ev.tc.nTrackCandidatespLS = 0;
        *ev.tc.nTrackCandidatesT5 = 0;
        *ev.rg.nEligibleT5Modules = 0;
        *ev.rg.device_nTotalMDs = es.mdOffset[nLower];
        *ev.rg.device_nTotalSegs = es.lsOffset[nLower];
        *ev.rg.device_nTotalTrips = 0;
        *ev.rg.device_nTotalQuints = 0;
      }
    }
  }

  // ================================================================ hits
  // SDL/Hit.h:217-269
  // (64 PU200 events with 3 / 4 / 5 / 6 blocks per SM: 503 / 414 / 407 / 386 us)
  __global__ void __launch_bounds__(256, 6) kHitPrep(DeviceES es, const EventView* evs) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    const unsigned int nHits = ev.sc->nHits;
    const Modules& m = es.m;
    Hits h = ev.hits;
    for (unsigned int ihit = blockIdx.x * blockDim.x + threadIdx.x; ihit < nHits; ihit += gridDim.x * blockDim.x) {
      float x = h.xs[ihit], y = h.ys[ihit], z = h.zs[ihit];
      unsigned int detId = h.detid[ihit];
      float rt = fsqrt(x * x + y * y);
      h.rts[ihit] = rt;
      h.phis[ihit] = phiOf(x, y);
      h.etas[ihit] = ((z > 0) - (z < 0)) * facosh(fsqrt(x * x + y * y + z * z) / rt);
      float hex = 0.f, hey = 0.f, lex = 0.f, ley = 0.f;
      int mIdx = -1;  // module of detId: the ES hash (linear probing)
      {
        const unsigned int mask = (1u << es.detHashBits) - 1;
        unsigned int slot = (detId * 2654435761u) >> (32 - es.detHashBits);
        for (unsigned int probe = 0; probe <= mask; ++probe) {
          const uint16_t val = es.detHashVal[slot];
          if (val == 0xffff)
            break;
          if (es.detHashKey[slot] == detId) {
            mIdx = val;
            break;
          }
          slot = (slot + 1) & mask;
        }
      }
      if (mIdx < 0) {
        atomicOr(&ev.sc->status, kStatusUnknownDetId);
        h.moduleIndices[ihit] = 0xffff;
        h.highEdgeXs[ihit] = hex;
        h.highEdgeYs[ihit] = hey;
        h.lowEdgeXs[ihit] = lex;
        h.lowEdgeYs[ihit] = ley;
        continue;
      }
      uint16_t mi = static_cast<uint16_t>(mIdx);
      h.moduleIndices[ihit] = mi;
      // Per-hit parts of the mini-doublet cuts of the module pair this hit
      // belongs to (lower module lm): the dphi-threshold slope, and the strip
      // shift of the hit it moves (tilted barrel and endcap modules).
      ev.hitMiniSlope[ihit] = mdMiniSlope(rt, m.ptCut);
      if (mi != es.pixelModule) {
        const bool isLowerHit = m.isLower[mi];
        const uint16_t lm = isLowerHit ? mi : m.partnerModuleIndices[mi];
        const bool shifted = m.subdets[lm] == Endcap || (m.subdets[lm] == Barrel && m.sides[lm] != Center);
        if (shifted && shiftMovesLower(m, lm) == isLowerHit) {
          float xa, ya, zn;
          shiftStripPrep(m, lm, x, y, z, rt, xa, ya, zn);
          ev.hitShiftXa[ihit] = xa;
          ev.hitShiftYa[ihit] = ya;
          ev.hitShiftZn[ihit] = zn;
        }
      }
      if (m.subdets[mi] == Endcap && m.moduleType[mi] == TwoS) {
        const int f = m.geoMapIndex[mi];  // sortedFind(m.geoMapDetId, detId, m.nEndCapMap), per module
        if (f < 0) {
          atomicOr(&ev.sc->status, kStatusUnknownEndcapDetId);
        } else {
          float phi = m.geoMapPhi[f];
          float cos_phi = fcos(phi);
          hex = x + 2.5f * cos_phi;
          lex = x - 2.5f * cos_phi;
          float sin_phi = fsin(phi);
          hey = y + 2.5f * sin_phi;
          ley = y - 2.5f * sin_phi;
        }
      }
      h.highEdgeXs[ihit] = hex;
      h.highEdgeYs[ihit] = hey;
      h.lowEdgeXs[ihit] = lex;
      h.lowEdgeYs[ihit] = ley;
      // The module's hit range [first, last]: the lanes of this warp on the
      // same module combine first, and one lane per module updates it.  The
      // first index starts at -1, the largest value as unsigned, so an
      // unsigned minimum takes the place of the reference's set-or-minimum.
      const unsigned int peers = __match_any_sync(__activemask(), static_cast<unsigned int>(mi));
      const unsigned int first = __reduce_min_sync(peers, ihit), last = __reduce_max_sync(peers, ihit);
      if (static_cast<unsigned int>(__ffs(peers) - 1) == (threadIdx.x & 31u)) {
        atomicMin(reinterpret_cast<unsigned int*>(&h.hitRanges[mi * 2]), first);
        atomicMax(&h.hitRanges[mi * 2 + 1], static_cast<int>(last));
      }
    }
  }

  // SDL/Hit.h:194-215
  __device__ __forceinline__ void moduleRanges(DeviceES const& es, const EventView& ev) {
    Hits h = ev.hits;
    for (unsigned int lower = blockIdx.x * blockDim.x + threadIdx.x; lower < es.nLowerModules;
         lower += gridDim.x * blockDim.x) {
      uint16_t upper = es.m.partnerModuleIndices[lower];
      if (h.hitRanges[lower * 2] != -1 && h.hitRanges[upper * 2] != -1) {
        h.hitRangesLower[lower] = h.hitRanges[lower * 2];
        h.hitRangesUpper[lower] = h.hitRanges[upper * 2];
        h.hitRangesnLower[lower] = static_cast<int8_t>(h.hitRanges[lower * 2 + 1] - h.hitRanges[lower * 2] + 1);
        h.hitRangesnUpper[lower] = static_cast<int8_t>(h.hitRanges[upper * 2 + 1] - h.hitRanges[upper * 2] + 1);
      }
    }
  }

  __global__ void kModuleRanges(DeviceES es, const EventView* evs) {
    kernelEntry();
    moduleRanges(es, evs[blockIdx.y]);
  }

  // ========================================================= pixel segments
  // SDL/Segment.h:1031-1117
  // A thread per mini-doublet, whose stores then lie side by side, and then one per
  // segment (64 PU200 events: with both of a segment's mini-doublets in its thread
  // 320 us, then 184; 220 since the mini-doublets' records are written here too, so
  // that they are this event's whenever the segments are added, and no longer by
  // kMDDerived, which takes 617 instead of 646).  Register budget: three 256-thread
  // blocks per SM (before the records 184 us; 2: 197, 4: 197, 5: 217).
  // withRanges: sets the modules' hit ranges as well (batched ingest).
  __global__ void __launch_bounds__(256, 3) kPixelIngest(DeviceES es, const EventView* evs, bool withRanges) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    if (withRanges)
      moduleRanges(es, ev);
    const unsigned int nPLS = ev.sc->nPLS;
    const uint16_t pix = es.pixelModule;
    MiniDoublets md = ev.md;
    Segments ls = ev.ls;
    const unsigned int mdBase = es.mdOffset[es.nLowerModules];
    const unsigned int lsBase = es.lsOffset[es.nLowerModules];
    const unsigned int nHits = ev.sc->nHits;
    const unsigned int first = blockIdx.x * blockDim.x + threadIdx.x, nThreads = gridDim.x * blockDim.x;
    // The reference indexes the hit store with a seed's hits unchecked; an index
    // outside the event is flagged and replaced by hit 0 (the host rejects pixel
    // segments for events without hits).
    auto hitOf = [&](unsigned int hit) {
      if (hit < nHits)
        return hit;
      atomicOr(&ev.sc->status, kStatusInvalidInput);
      return 0u;
    };
    // a thread per mini-doublet, then one per segment
    for (unsigned int k = first; k < 2 * nPLS; k += nThreads) {
      const unsigned int tid = k >> 1;
      const unsigned int lower = (k & 1) ? ev.plsHit2[tid] : ev.plsHit0[tid];
      const unsigned int upper = (k & 1) ? ev.plsHit3[tid] : ev.plsHit1[tid];
      storePixelMD(es.m, ev.hits, md, pix, mdBase + k, hitOf(lower), hitOf(upper));
    }
    for (unsigned int tid = first; tid < nPLS; tid += nThreads) {
      storePixelLS(es.m, ev.hits, ls, pix, mdBase, lsBase, tid, hitOf(ev.plsHit0[tid]), hitOf(ev.plsHit1[tid]),
                   hitOf(ev.plsHit2[tid]), hitOf(ev.plsHit3[tid]), ev.plsDPhiChange[tid]);
      ls.partOfPT5[tid] = 0;
      ev.plsPhiP[tid] = phiOf(ls.px[tid], ls.py[tid]);
      ev.plsFlag[tid] = 0;
      for (unsigned int slot = 0; slot < 4; ++slot) {
        const unsigned int e = 4 * tid + slot;
        ev.plsHitNext[e] = atomicExch(&ev.plsHitHead[plsHitBucket(ls.pLSHitsIdxs[e])], e);
      }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      md.nMDs[pix] = 2 * nPLS;
      md.totOccupancyMDs[pix] = 2 * nPLS;
      ls.nSegments[pix] = nPLS;
      ls.totOccupancySegments[pix] = nPLS;
    }
  }

  // Work counters of the kernels whose warps take their next task from the
  // event's counter, so that a warp that drew light tasks takes more: the work per
  // module or pLS is very uneven.  A counter is zero before its kernel runs:
  // kResetEvent clears them all, and the kernel after the one that counts clears
  // its counter again, in case the stage is run again.
  // The tasks of the calling warp: first the one of its own number among the
  // event's warps, then from counter *next, which numbers the tasks after those
  // (the same value on every lane).  Without the first, thousands of warps start
  // with an atomic on one address.
  struct WarpTasks {
    unsigned int* next;
    unsigned int nWarps, own;
    bool started = false;
    __device__ __forceinline__ explicit WarpTasks(unsigned int* counter)
        : next(counter),
          nWarps(gridDim.x * (blockDim.x >> 5)),
          own(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) {}
    __device__ __forceinline__ unsigned int take() {
      if (!started) {
        started = true;
        return own;
      }
      unsigned int t = 0;
      if (laneId() == 0)
        t = atomicAdd(next, 1u);
      return nWarps + __shfl_sync(kFullMask, t, 0);
    }
  };

  // The same for the calling block's tasks.  (The barriers also end the use of
  // the shared memory of the task before.)
  struct BlockTasks {
    unsigned int* next;
    bool started = false;
    __device__ __forceinline__ explicit BlockTasks(unsigned int* counter) : next(counter) {}
    __device__ __forceinline__ unsigned int take() {
      if (!started) {
        started = true;
        return blockIdx.x;
      }
      __shared__ unsigned int sTask;
      __syncthreads();
      if (threadIdx.x == 0)
        sTask = gridDim.x + atomicAdd(next, 1u);
      __syncthreads();
      return sTask;
    }
  };

  // A block's queue of candidates, in order: the calling thread's place (if it
  // adds one), and the queue's new length.  Every thread calls it; the entries
  // may be written when it returns and read after a barrier.
  __device__ __forceinline__ unsigned int blockQueuePlace(bool add, unsigned int* warpCount, unsigned int& queued) {
    unsigned int n;
    unsigned int at = queued + warpRank(add, n);
    const unsigned int wid = threadIdx.x >> 5;
    if (laneId() == 0)
      warpCount[wid] = n;
    __syncthreads();
    for (unsigned int w = 0; w < blockDim.x >> 5; ++w) {
      const unsigned int c = warpCount[w];
      at += w < wid ? c : 0u;
      queued += c;
    }
    return at;
  }

  // The rank of a passing candidate among its module's, over the block's tasks of
  // up to 32 modules (module j's count so far in count[j]).  passing[] holds 32
  // words per warp.  Every thread calls it, then blockRankDone.
  __device__ __forceinline__ unsigned int blockModuleRank(bool ok, unsigned int j, unsigned int* passing,
                                                          const unsigned int* count) {
    const unsigned int wid = threadIdx.x >> 5;
    passing[32u * wid + laneId()] = 0;
    __syncwarp();
    const unsigned int peers = __match_any_sync(kFullMask, ok ? j : 32u + laneId());
    const unsigned int rank = __popc(peers & lanesBelowMask());
    if (ok && rank == 0)
      passing[32u * wid + j] = __popc(peers);
    __syncthreads();
    unsigned int r = count[j] + rank;
    for (unsigned int w = 0; w < wid; ++w)
      r += passing[32u * w + j];
    return r;
  }
  // Ends with a barrier.
  __device__ __forceinline__ void blockRankDone(const unsigned int* passing, unsigned int* count) {
    __syncthreads();
    if (threadIdx.x < 32)
      for (unsigned int w = 0; w < blockDim.x >> 5; ++w)
        count[threadIdx.x] += passing[32u * w + threadIdx.x];
    __syncthreads();
  }

  // ======================================================== mini-doublets
  // SDL/MiniDoublet.h:896-992: every (lower hit, upper hit) pair of a lower
  // module is a candidate; passing ones are stored in the module's arena at
  // their rank in the reference's serial loop order (lower hit outer, upper
  // hit inner), the first mdCap of them.
  //
  // A warp takes up to 32 consecutive lower modules at a time (most hold
  // fewer than 32 pairs, the median 14) and deals their pairs out in order, 32
  // per step, across module boundaries: lane l of step s takes the task's pair
  // 32 s + l, finds its module by a binary search over the lanes' exclusive
  // prefix of pair counts, and its hits by dividing by the module's upper
  // hit count.  A passing pair's rank is the module's running count (one
  // word per module in shared memory) plus the passing lanes of the same
  // module below it (__match_any_sync).  So the lanes stay busy on small
  // modules, and a large module simply spans several steps.
  constexpr int kMDMaxWarps = 8;  // warps per block the kernel is launched with (at most)
  __device__ __forceinline__ void mdTask(DeviceES const& es, const EventView& ev, unsigned int task,
                                         unsigned int modulesPerTask, unsigned int* count) {
    const Hits& h = ev.hits;
    const unsigned int lane = laneId();
    const unsigned int lmU = task * modulesPerTask + lane;
    const bool valid = lane < modulesPerTask && lmU < es.nLowerModules && h.hitRangesLower[lmU] != -1;
    const int nL = valid ? int(h.hitRangesnLower[lmU]) : 0;
    const int nU = valid ? int(h.hitRangesnUpper[lmU]) : 0;
    const int loHit0 = valid ? h.hitRangesLower[lmU] : 0;
    const int upHit0 = valid ? h.hitRangesUpper[lmU] : 0;
    const int cap = valid ? es.mdCap[lmU] : 0;
    const unsigned int base = valid ? es.mdOffset[lmU] : 0u;
    // (the reference's counts are int8; a negative one means no pairs here)
    const int pairs = (nL > 0 && nU > 0) ? nL * nU : 0;
    int incl = pairs;  // inclusive prefix of the pair counts over the lanes
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int o = __shfl_up_sync(kFullMask, incl, d);
      if (int(lane) >= d)
        incl += o;
    }
    const int excl = incl - pairs;
    const int total = __shfl_sync(kFullMask, incl, 31);
    count[lane] = 0;
    __syncwarp();
    MiniDoublets md = ev.md;
    const MDHitPre pre{ev.hitMiniSlope, ev.hitShiftXa, ev.hitShiftYa, ev.hitShiftZn};
    for (int start = 0; start < total; start += 32) {
      const int g = start + int(lane);
      // the module of pair g: the last lane whose exclusive prefix is <= g
      // (a lane without pairs shares its prefix with the next one)
      int j = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const int e = __shfl_sync(kFullMask, excl, (j + step) & 31);
        if (j + step < 32 && e <= g)
          j += step;
      }
      const int exj = __shfl_sync(kFullMask, excl, j);
      const int nUj = __shfl_sync(kFullMask, nU, j);
      const int loj = __shfl_sync(kFullMask, loHit0, j);
      const int upj = __shfl_sync(kFullMask, upHit0, j);
      const int capj = __shfl_sync(kFullMask, cap, j);
      const unsigned int basej = __shfl_sync(kFullMask, base, j);
      bool ok = false;
      MDValues v;
      unsigned int lowerIdx = 0, upperIdx = 0;
      const uint16_t lm = static_cast<uint16_t>(task * modulesPerTask + unsigned(j));
      if (g < total) {
        const int local = g - exj;
        lowerIdx = unsigned(loj + local / nUj);
        upperIdx = unsigned(upj + local % nUj);
        ok = mdSelect(es.mdCuts[lm], h.xs[lowerIdx], h.ys[lowerIdx], h.zs[lowerIdx], h.rts[lowerIdx], h.xs[upperIdx],
                      h.ys[upperIdx], h.zs[upperIdx], h.rts[upperIdx], h.phis[lowerIdx], h.phis[upperIdx], pre,
                      lowerIdx, upperIdx, v);
      }
      const unsigned int peers = __match_any_sync(kFullMask, ok ? unsigned(j) : 32u + lane);
      const unsigned int rank = __popc(peers & lanesBelowMask());
      if (ok) {
        const unsigned int r = count[j] + rank;
        if (int(r) < capj)
          storeMDPair(es.m, md, lowerIdx, upperIdx, lm, v, basej + r);
      }
      __syncwarp();
      if (ok && rank == 0)
        count[j] += __popc(peers);
      __syncwarp();
    }
    if (valid) {
      const unsigned int n = count[lane];
      md.nMDs[lmU] = (int(n) < cap) ? n : (cap > 0 ? unsigned(cap) : 0u);
      md.totOccupancyMDs[lmU] = n;
      if (int(n) > cap)
        atomicOr(&ev.sc->status, kStatusCapOverflow);
    }
    __syncwarp();
  }

  // Register budgets of the cut kernels, as resident blocks per SM.  The cut
  // kernels wait mostly on dependent loads, so they run faster with more warps
  // resident even where the tighter budget spills a little; the values are
  // the fastest of a sweep over 2..14 blocks on B200 (PU200 batches, launch
  // shapes autotuned for each setting).
#ifndef LST_LB_MD_B
#define LST_LB_MD_B 6
#endif
#ifndef LST_LB_LS_B
#define LST_LB_LS_B 12
#endif
#ifndef LST_LB_T3_B
#define LST_LB_T3_B 14
#endif
#ifndef LST_LB_EVAL_B
#define LST_LB_EVAL_B 7
#endif
#ifndef LST_LB_T5EVAL_B
#define LST_LB_T5EVAL_B 8
#endif
#ifndef LST_LB_PIXMID_B
#define LST_LB_PIXMID_B 10
#endif
#define LST_LB_MD 256, LST_LB_MD_B
#define LST_LB_LS 128, LST_LB_LS_B
#define LST_LB_T3 128, LST_LB_T3_B
#define LST_LB_EVAL 128, LST_LB_EVAL_B
#define LST_LB_T5EVAL 128, LST_LB_T5EVAL_B
#define LST_LB_PIXMID 128, LST_LB_PIXMID_B
  // modulesPerTask (1..32): 8 for batches; fewer for a single event, whose
  // 13 000 lower modules would otherwise make only ~400 warp tasks.
  __global__ void __launch_bounds__(LST_LB_MD) kCreateMD(DeviceES es, const EventView* evs, unsigned int modulesPerTask) {
    kernelEntry();
    __shared__ unsigned int sCount[kMDMaxWarps][32];
    const EventView& ev = evs[blockIdx.y];
    const int w = threadIdx.x >> 5;
    const unsigned int nTasks = (es.nLowerModules + modulesPerTask - 1u) / modulesPerTask;
    // tasks from the event's counter (zero before the kernel)
    WarpTasks tasks(&ev.sc->mdNext);
    for (unsigned int task = tasks.take(); task < nTasks; task = tasks.take())
      mdTask(es, ev, task, modulesPerTask, sCount[w]);
  }

  // SDL/MiniDoublet.h:1084-1104
  __device__ __forceinline__ void mdRanges(DeviceES const& es, const EventView& ev) {
    for (unsigned int i = blockIdx.x * blockDim.x + threadIdx.x; i < es.nLowerModules; i += gridDim.x * blockDim.x) {
      if (ev.md.nMDs[i] == 0 or ev.hits.hitRanges[i * 2] == -1) {
        ev.rg.mdRanges[i * 2] = -1;
        ev.rg.mdRanges[i * 2 + 1] = -1;
      } else {
        ev.rg.mdRanges[i * 2] = es.mdOffset[i];
        ev.rg.mdRanges[i * 2 + 1] = es.mdOffset[i] + ev.md.nMDs[i] - 1;
      }
    }
  }

  // The hits' values of every MD of the lower modules, and its record for the
  // later cuts (the pixel module's are whole when kPixelIngest has stored them).
  // A warp takes 32 lower modules at a time (a module holds a few MDs) and shares
  // their MDs out over its lanes: a lane-level prefix of the modules' counts, and
  // per MD the owning lane by a search over it.
  // Also sets the modules' mini-doublet ranges and clears kCreateMD's counter.
  // Waits for scattered sectors (a warp's 32 mini-doublets lie in a dozen modules'
  // places of some 25 arrays), with all of a mini-doublet's loads in flight: held
  // to 64 registers a thread instead of its 122 it took 746 us instead of 646, now
  // 617 (64 PU200 events; kCreateMD, which stored all of it, was 1128 and is 477, and
  // this kernel 177).
  __global__ void kMDDerived(DeviceES es, const EventView* evs) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    mdRanges(es, ev);
    if (blockIdx.x == 0 && threadIdx.x == 0)
      ev.sc->mdNext = 0;
    const unsigned int nWarps = gridDim.x * (blockDim.x >> 5);
    const unsigned int lane = laneId();
    MiniDoublets md = ev.md;
    for (unsigned int w0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32u; w0 < es.nLowerModules;
         w0 += nWarps * 32u) {
      const unsigned int w = w0 + lane;
      const unsigned int n = w < es.nLowerModules ? md.nMDs[w] : 0u;
      const unsigned int base = w < es.nLowerModules ? static_cast<unsigned int>(es.mdOffset[w]) : 0u;
      unsigned int incl = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned int y = __shfl_up_sync(kFullMask, incl, o);
        if (int(lane) >= o)
          incl += y;
      }
      const unsigned int total = __shfl_sync(kFullMask, incl, 31);
      for (unsigned int f0 = 0; f0 < total; f0 += 32) {
        const unsigned int f = f0 + lane;
        // owner: the first lane whose inclusive count exceeds f
        int owner = 0;
#pragma unroll
        for (int step = 16; step > 0; step >>= 1) {
          const unsigned int c = __shfl_sync(kFullMask, incl, owner + step - 1);
          if (c <= f)
            owner += step;
        }
        const unsigned int ownerIncl = __shfl_sync(kFullMask, incl, owner);
        const unsigned int ownerN = __shfl_sync(kFullMask, n, owner);
        const unsigned int ownerBase = __shfl_sync(kFullMask, base, owner);
        if (f < total)
          storeMDRest(es.m, ev.hits, md, static_cast<uint16_t>(w0 + owner), ownerBase + (f - (ownerIncl - ownerN)));
      }
    }
  }

  // ======================================================== line segments
  // Segments (SDL/Segment.h:798-910): a warp walks (connected module, inner
  // MD, outer MD) of up to kLSTaskModules inner lower modules in order.  The
  // (module, connected module) pairs are dealt out over the lanes, kLSChunk at a
  // time; the warp's shared memory then has the prefix of the candidates over the
  // pairs, and per pair the connected module, its MD count and first MD, so that
  // a candidate finds its MDs without a global load.  A passing segment's place
  // is its module's running count plus the passing lanes of the same module below.
  //
  // Bound by the gathers' latency and the L1 (72 % busy with them); a module's
  // own chain of dependent loads is shared by the task's modules (64 PU200 events:
  // a module per warp 1142 us, 4 modules 953).  A block per task with a queue
  // between the window and the rest, as in kCreateT3, has lanes 84 % busy instead
  // of 64 but loses it at the barriers (1066; one event 70 instead of 50).
  constexpr int kLSWarps = 4;
  constexpr int kLSChunk = 64;
  constexpr unsigned int kLSTaskModules = 8;  // modules per task (at most)
  struct LSScratch {
    unsigned int pre[kLSChunk + 1];
    unsigned int outerBase[kLSChunk];
    unsigned int modulePre[kLSTaskModules + 1];  // prefix of the task's pairs over its modules
    unsigned int innerBase[kLSTaskModules], nInnerMDs[kLSTaskModules], count[kLSTaskModules];
    LSCut cut[kLSTaskModules];
    uint16_t nOuterMDs[kLSChunk];
    uint16_t outer[kLSChunk];
    uint8_t module[kLSChunk];
  };
  __device__ __forceinline__ void lsTask(DeviceES const& es, const EventView& ev, unsigned int firstModule,
                                         unsigned int nModules, LSScratch& sc) {
    const Modules& m = es.m;
    const unsigned int lane = laneId();
    const unsigned int own = firstModule + lane;  // the lane's module
    const bool valid = lane < nModules && own < es.nLowerModules;
    const unsigned int nMDsOwn = valid ? ev.md.nMDs[own] : 0u;
    const int capOwn = valid ? es.lsCap[own] : 0;
    const unsigned int baseOwn = valid ? static_cast<unsigned int>(es.lsOffset[own]) : 0u;
    const unsigned int nConnOwn = valid ? m.nConnectedModules[own] : 0u;
    const unsigned int incl = laneInclusiveSum(nMDsOwn != 0 ? nConnOwn : 0u);
    const unsigned int nPairs = __shfl_sync(kFullMask, incl, 31);
    if (lane < kLSTaskModules) {
      sc.innerBase[lane] = valid ? static_cast<unsigned int>(es.mdOffset[own]) : 0u;
      sc.nInnerMDs[lane] = nMDsOwn;
      if (valid)
        sc.cut[lane] = es.lsCuts[own];
      sc.count[lane] = 0;
      sc.modulePre[lane + 1] = incl;
    }
    if (lane == 0)
      sc.modulePre[0] = 0;
    __syncwarp();
    Segments ls = ev.ls;
    for (unsigned int c0 = 0; c0 < nPairs; c0 += kLSChunk) {
      const int n = int(min(nPairs - c0, unsigned(kLSChunk)));
      const unsigned int total = warpPrefix(sc.pre, n, [&](int i) {
        const unsigned int g = c0 + unsigned(i);
        const int j = findSlot(sc.modulePre, kLSTaskModules, g);
        const uint16_t o = m.moduleMap[(firstModule + j) * kMaxConnectedModules + (g - sc.modulePre[j])];
        const unsigned int nOuter = ev.md.nMDs[o];
        sc.outer[i] = o;
        sc.nOuterMDs[i] = static_cast<uint16_t>(nOuter);
        sc.outerBase[i] = static_cast<unsigned int>(es.mdOffset[o]);
        sc.module[i] = static_cast<uint8_t>(j);
        return sc.nInnerMDs[j] * nOuter;
      });
      for (unsigned int start = 0; start < total; start += 32) {
        const unsigned int f = start + lane;
        bool ok = false;
        LSValues v;
        unsigned int innerMD = 0, outerMD = 0, j = 0;
        uint16_t outerLM = 0;
        if (f < total) {
          const int k = findSlot(sc.pre, n, f);
          outerLM = sc.outer[k];
          j = sc.module[k];
          const unsigned int nOuterMDs = sc.nOuterMDs[k], local = f - sc.pre[k];
          innerMD = sc.innerBase[j] + local / nOuterMDs;
          outerMD = sc.outerBase[k] + local % nOuterMDs;
          ok = lsSelect(sc.cut[j], es.lsCuts[outerLM], m.ptCut, ev.md.rec[innerMD], ev.md.rec[outerMD], v);
        }
        const unsigned int peers = __match_any_sync(kFullMask, ok ? j : 32u + lane);
        const unsigned int rank = __popc(peers & lanesBelowMask());
        const int cap = __shfl_sync(kFullMask, capOwn, j);
        const unsigned int base = __shfl_sync(kFullMask, baseOwn, j);
        const unsigned int r = sc.count[j] + rank;
        if (ok && int(r) < cap)
          storeLS(ls, ev.md, innerMD, outerMD, static_cast<uint16_t>(firstModule + j), outerLM, v, base + r);
        __syncwarp();
        if (ok && rank == 0)
          sc.count[j] += __popc(peers);
        __syncwarp();
      }
      __syncwarp();  // the chunk's scratch has been read
    }
    if (nMDsOwn != 0) {
      const unsigned int n = sc.count[lane];
      ls.nSegments[own] = (int(n) < capOwn) ? n : (capOwn > 0 ? unsigned(capOwn) : 0u);
      ls.totOccupancySegments[own] = n;
      if (int(n) > capOwn)
        atomicOr(&ev.sc->status, kStatusCapOverflow);
    }
    __syncwarp();
  }

  __global__ void __launch_bounds__(LST_LB_LS) kCreateLS(DeviceES es, const EventView* evs, unsigned int modulesPerTask) {
    kernelEntry();
    __shared__ LSScratch sScratch[kLSWarps];
    const EventView& ev = evs[blockIdx.y];
    const int wib = threadIdx.x >> 5;
    const unsigned int nTasks = (es.nLowerModules + modulesPerTask - 1u) / modulesPerTask;
    // tasks from the event's counter (zero before the kernel)
    WarpTasks tasks(&ev.sc->lsNext);
    for (unsigned int task = tasks.take(); task < nTasks; task = tasks.take())
      lsTask(es, ev, task * modulesPerTask, modulesPerTask, sScratch[wib]);
  }

  // SDL/Segment.h:1010-1029
  __device__ __forceinline__ void lsRanges(DeviceES const& es, const EventView& ev) {
    for (unsigned int i = blockIdx.x * blockDim.x + threadIdx.x; i < es.nLowerModules; i += gridDim.x * blockDim.x) {
      if (ev.ls.nSegments[i] == 0) {
        ev.rg.segmentRanges[i * 2] = -1;
        ev.rg.segmentRanges[i * 2 + 1] = -1;
      } else {
        ev.rg.segmentRanges[i * 2] = es.lsOffset[i];
        ev.rg.segmentRanges[i * 2 + 1] = es.lsOffset[i] + ev.ls.nSegments[i] - 1;
      }
    }
  }

  // ================================================= MD-keyed indices
  // For one module: the objects [0, n) of the module (segments or triplets,
  // in storage order) grouped by the module-local index of their first
  // mini-doublet, stably, so that each group keeps storage order.  Written:
  // start[md] / count[md] for every MD of the module, perm[] the object
  // indices (module-relative).  One warp; `bins` / `cursor` are warp-private
  // shared arrays of kMaxModuleMDs entries.
  constexpr int kMaxModuleMDs = 128;

  template <typename FirstMD>
  __device__ __forceinline__ void buildByMD(unsigned int n, unsigned int nBins, FirstMD firstMD, uint16_t* start,
                                            uint16_t* count, uint16_t* perm, unsigned int* bins,
                                            unsigned int* cursor) {
    for (unsigned int b = laneId(); b < nBins; b += 32)
      bins[b] = 0;
    __syncwarp();
    for (unsigned int k = laneId(); k < n; k += 32)
      atomicAdd(&bins[firstMD(k)], 1u);
    __syncwarp();
    // exclusive scan of the bins
    unsigned int carry = 0;
    for (unsigned int b0 = 0; b0 < nBins; b0 += 32) {
      unsigned int b = b0 + laneId();
      unsigned int c = b < nBins ? bins[b] : 0u;
      unsigned int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        unsigned int y = __shfl_up_sync(kFullMask, incl, o);
        if (int(laneId()) >= o)
          incl += y;
      }
      if (b < nBins) {
        cursor[b] = carry + incl - c;
        start[b] = static_cast<uint16_t>(carry + incl - c);
        count[b] = static_cast<uint16_t>(c);
      }
      carry += __shfl_sync(kFullMask, incl, 31);
    }
    __syncwarp();
    // stable placement, 32 objects at a time
    for (unsigned int k0 = 0; k0 < n; k0 += 32) {
      unsigned int k = k0 + laneId();
      bool valid = k < n;
      unsigned int b = valid ? firstMD(k) : 0xffffffffu;
      unsigned int active = __ballot_sync(kFullMask, valid);
      unsigned int peers = __match_any_sync(kFullMask, b) & active;
      if (valid) {
        unsigned int rank = __popc(peers & lanesBelowMask());
        perm[cursor[b] + rank] = static_cast<uint16_t>(k);
      }
      __syncwarp();
      if (valid && laneId() == 31u - __clz(peers))
        cursor[b] += __popc(peers);
      __syncwarp();
    }
  }

  // The same grouping for `group` (up to 32) consecutive modules at once (most
  // modules hold a few objects): their bins lie side by side in bins[0, sum of the modules'
  // MDs), each object is counted into its module's bin, and a module-relative
  // start is the running count over all bins minus the objects of the
  // group's earlier modules (each object lies in a bin of its own module).
  // Placement takes the group's objects in storage order, so each group stays
  // stable.  The module of the f-th object or b-th bin is found by a search
  // over the lanes' prefix counts.  Returns false (having written nothing)
  // when the bins do not fit, and the caller groups module by module.
  // nOf(w) = objects of module w (0 for a module past the end), objBase(w) =
  // its first object, firstMD(w, k) = module-relative first MD of object k.
  constexpr unsigned int kByMDGroupBins = 512;
  constexpr int kByMDKeptChunks = 8;  // bins of the first chunks kept in registers between the passes
  __device__ __forceinline__ int laneOwner(unsigned int incl, unsigned int f) {
    int owner = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
      const unsigned int c = __shfl_sync(kFullMask, incl, owner + step - 1);
      if (c <= f)
        owner += step;
    }
    return owner;
  }
  template <typename NOf, typename ObjBase, typename FirstMD>
  __device__ __forceinline__ bool buildByMDGroup(DeviceES const& es, const EventView& ev, unsigned int w0,
                                                 unsigned int group, NOf nOf,
                                                 ObjBase objBase, FirstMD firstMD, uint16_t* start, uint16_t* count,
                                                 uint16_t* perm, unsigned int* bins, unsigned int* cursor) {
    const unsigned int lane = laneId();
    const unsigned int w = w0 + lane;
    const bool inRange = lane < group && w < es.nLowerModules;
    const unsigned int n = inRange ? nOf(w) : 0u;
    const unsigned int nMD = (inRange && n > 0) ? ev.md.nMDs[w] : 0u;
    const unsigned int mdBase = inRange ? static_cast<unsigned int>(es.mdOffset[w]) : 0u;
    const unsigned int base = (inRange && n > 0) ? objBase(w) : 0u;
    const unsigned int objIncl = laneInclusiveSum(n), binIncl = laneInclusiveSum(nMD);
    const unsigned int nObj = __shfl_sync(kFullMask, objIncl, 31), nBins = __shfl_sync(kFullMask, binIncl, 31);
    if (nBins > kByMDGroupBins)
      return false;
    if (nObj == 0)
      return true;
    const unsigned int objExcl = objIncl - n, binExcl = binIncl - nMD;
    for (unsigned int b = lane; b < nBins; b += 32)
      bins[b] = 0;
    __syncwarp();
    unsigned int kept[kByMDKeptChunks];
    for (unsigned int f0 = 0; f0 < nObj; f0 += 32) {
      const unsigned int f = f0 + lane;
      const int o = laneOwner(objIncl, f);
      const unsigned int oObjExcl = __shfl_sync(kFullMask, objExcl, o);
      const unsigned int oBinExcl = __shfl_sync(kFullMask, binExcl, o);
      unsigned int bin = 0xffffffffu;
      if (f < nObj) {
        bin = oBinExcl + firstMD(w0 + o, f - oObjExcl);
        atomicAdd(&bins[bin], 1u);
      }
#pragma unroll
      for (int c = 0; c < kByMDKeptChunks; ++c)
        if (f0 == 32u * c)
          kept[c] = bin;
    }
    __syncwarp();
    // running count over all bins -> module-relative starts
    unsigned int carry = 0;
    for (unsigned int b0 = 0; b0 < nBins; b0 += 32) {
      const unsigned int b = b0 + lane;
      const unsigned int c = b < nBins ? bins[b] : 0u;
      const unsigned int incl = laneInclusiveSum(c);
      const int o = laneOwner(binIncl, b);
      const unsigned int oObjExcl = __shfl_sync(kFullMask, objExcl, o);
      const unsigned int oBinExcl = __shfl_sync(kFullMask, binExcl, o);
      const unsigned int oMdBase = __shfl_sync(kFullMask, mdBase, o);
      if (b < nBins) {
        const unsigned int rel = carry + incl - c - oObjExcl;
        cursor[b] = rel;
        start[oMdBase + (b - oBinExcl)] = static_cast<uint16_t>(rel);
        count[oMdBase + (b - oBinExcl)] = static_cast<uint16_t>(c);
      }
      carry += __shfl_sync(kFullMask, incl, 31);
    }
    __syncwarp();
    // stable placement, 32 objects at a time
    for (unsigned int f0 = 0; f0 < nObj; f0 += 32) {
      const unsigned int f = f0 + lane;
      const int o = laneOwner(objIncl, f);
      const unsigned int oObjExcl = __shfl_sync(kFullMask, objExcl, o);
      const unsigned int oBinExcl = __shfl_sync(kFullMask, binExcl, o);
      const unsigned int oBase = __shfl_sync(kFullMask, base, o);
      const bool valid = f < nObj;
      const unsigned int k = f - oObjExcl;
      unsigned int bin = 0xffffffffu;
      if (f0 < 32u * kByMDKeptChunks) {
#pragma unroll
        for (int c = 0; c < kByMDKeptChunks; ++c)
          if (f0 == 32u * c)
            bin = kept[c];
      } else if (valid) {
        bin = oBinExcl + firstMD(w0 + o, k);
      }
      const unsigned int active = __ballot_sync(kFullMask, valid);
      const unsigned int peers = __match_any_sync(kFullMask, bin) & active;
      if (valid) {
        const unsigned int rank = __popc(peers & lanesBelowMask());
        perm[oBase + cursor[bin] + rank] = static_cast<uint16_t>(k);
      }
      __syncwarp();
      if (valid && lane == 31u - __clz(peers))
        cursor[bin] += __popc(peers);
      __syncwarp();
    }
    return true;
  }

  // Segments of each lower module grouped by inner MD (after kCreateLS): a
  // warp takes `group` modules at a time (32; 8 for a few events), module by
  // module where their bins do not fit (or the fallback paths are forced).  Also sets the modules' segment
  // ranges and clears kCreateLS's counter.
  constexpr int kIdxWarps = 4;
  __global__ void kLSByMD(DeviceES es, const EventView* evs, unsigned int group) {
    kernelEntry();
    __shared__ unsigned int sBins[kIdxWarps][kByMDGroupBins];
    __shared__ unsigned int sCursor[kIdxWarps][kByMDGroupBins];
    const EventView& ev = evs[blockIdx.y];
    lsRanges(es, ev);
    if (blockIdx.x == 0 && threadIdx.x == 0)
      ev.sc->lsNext = 0;
    const int wib = threadIdx.x >> 5;
    const unsigned int* mdIdx = ev.ls.mdIndices;
    const unsigned int nWarps = gridDim.x * kIdxWarps;
    for (unsigned int w0 = (blockIdx.x * kIdxWarps + wib) * group; w0 < es.nLowerModules; w0 += nWarps * group) {
      __syncwarp();
      if (!ev.forceWalk &&
          buildByMDGroup(
              es, ev, w0, group, [&](unsigned int w) { return static_cast<unsigned int>(ev.ls.nSegments[w]); },
              [&](unsigned int w) { return static_cast<unsigned int>(es.lsOffset[w]); },
              [&](unsigned int w, unsigned int k) { return mdIdx[2 * (es.lsOffset[w] + k)] - es.mdOffset[w]; },
              ev.mdLSStart, ev.mdLSCount, ev.lsByMD, sBins[wib], sCursor[wib]))
        continue;
      for (unsigned int w = w0; w < w0 + group && w < es.nLowerModules; ++w) {
        __syncwarp();
        const unsigned int n = ev.ls.nSegments[w];
        if (n == 0)
          continue;
        const unsigned int mdBase = es.mdOffset[w];
        const unsigned int nMD = ev.md.nMDs[w];
        const unsigned int segBase = es.lsOffset[w];
        buildByMD(
            n, nMD, [&](unsigned int k) { return mdIdx[2 * (segBase + k)] - mdBase; }, ev.mdLSStart + mdBase,
            ev.mdLSCount + mdBase, ev.lsByMD + segBase, sBins[wib], sCursor[wib]);
      }
    }
  }

  // SDL/Triplet.h:1104-1122
  __device__ __forceinline__ void t3Ranges(DeviceES const& es, const EventView& ev) {
    for (unsigned int i = blockIdx.x * blockDim.x + threadIdx.x; i < es.nLowerModules; i += gridDim.x * blockDim.x) {
      if (ev.t3.nTriplets[i] == 0) {
        ev.rg.tripletRanges[i * 2] = -1;
        ev.rg.tripletRanges[i * 2 + 1] = -1;
      } else {
        ev.rg.tripletRanges[i * 2] = ev.rg.tripletModuleIndices[i];
        ev.rg.tripletRanges[i * 2 + 1] = ev.rg.tripletModuleIndices[i] + ev.t3.nTriplets[i] - 1;
      }
    }
  }

  // Triplets of each lower module grouped by first MD (after kCreateT3), in
  // the same way, with the modules' triplet ranges and kCreateT3's counter.
  __global__ void kT3ByMD(DeviceES es, const EventView* evs, unsigned int group) {
    kernelEntry();
    __shared__ unsigned int sBins[kIdxWarps][kByMDGroupBins];
    __shared__ unsigned int sCursor[kIdxWarps][kByMDGroupBins];
    const EventView& ev = evs[blockIdx.y];
    t3Ranges(es, ev);
    if (blockIdx.x == 0 && threadIdx.x == 0)
      ev.sc->t3Next = 0;
    const int wib = threadIdx.x >> 5;
    const unsigned int* segIdx = ev.t3.segmentIndices;
    const unsigned int* mdIdx = ev.ls.mdIndices;
    const unsigned int nWarps = gridDim.x * kIdxWarps;
    for (unsigned int w0 = (blockIdx.x * kIdxWarps + wib) * group; w0 < es.nLowerModules; w0 += nWarps * group) {
      __syncwarp();
      if (!ev.forceWalk &&
          buildByMDGroup(
              es, ev, w0, group, [&](unsigned int w) { return static_cast<unsigned int>(ev.t3.nTriplets[w]); },
              [&](unsigned int w) { return static_cast<unsigned int>(ev.rg.tripletModuleIndices[w]); },
              [&](unsigned int w, unsigned int k) {
                return mdIdx[2 * segIdx[2 * (ev.rg.tripletModuleIndices[w] + k)]] - es.mdOffset[w];
              },
              ev.mdT3Start, ev.mdT3Count, ev.t3ByMD, sBins[wib], sCursor[wib]))
        continue;
      for (unsigned int w = w0; w < w0 + group && w < es.nLowerModules; ++w) {
        __syncwarp();
        const unsigned int n = ev.t3.nTriplets[w];
        if (n == 0)
          continue;
        const unsigned int mdBase = es.mdOffset[w];
        const unsigned int nMD = ev.md.nMDs[w];
        const unsigned int t3Base = ev.rg.tripletModuleIndices[w];
        buildByMD(
            n, nMD, [&](unsigned int k) { return mdIdx[2 * segIdx[2 * (t3Base + k)]] - mdBase; },
            ev.mdT3Start + mdBase, ev.mdT3Count + mdBase, ev.t3ByMD + t3Base, sBins[wib], sCursor[wib]);
      }
    }
  }

  // ============================================================ triplets
  // Modules of a one-block-per-event scan over the lower modules: each warp takes
  // a contiguous run of them, kScanSteps x 32 at a time with all loads of a run
  // issued before the first sum, so that the scan costs one round of loads and one
  // block scan of the warps' totals per run (13200 modules: one run).
  constexpr int kScanSteps = 13;
  constexpr unsigned int kScanRun = 32u * 32u * kScanSteps;  // modules of one run of a 1024-thread block

  // Per-module triplet offsets (SDL/Triplet.h:1007-1102); one block per event.
  __global__ void __launch_bounds__(1024) kT3Offsets(DeviceES es, const EventView* evs) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    const unsigned int lane = laneId(), wid = threadIdx.x >> 5;
    unsigned int carry = 0;
    for (unsigned int base = 0; base < es.nLowerModules; base += kScanRun) {
      const unsigned int i0 = base + wid * 32u * kScanSteps + lane;
      unsigned int occ[kScanSteps], ex[kScanSteps], sum = 0;
#pragma unroll
      for (int k = 0; k < kScanSteps; ++k) {
        const unsigned int i = i0 + 32u * k;
        occ[k] = i < es.nLowerModules && ev.ls.nSegments[i] != 0 ? static_cast<unsigned int>(es.t3CapIfUsed[i]) : 0u;
      }
#pragma unroll
      for (int k = 0; k < kScanSteps; ++k) {
        const unsigned int incl = laneInclusiveSum(occ[k]);
        ex[k] = sum + incl - occ[k];
        sum += __shfl_sync(kFullMask, incl, 31);
      }
      unsigned int tot;
      // (the warp's total from its first lane, so that the exclusive sum at that
      // lane is the total of the warps before it)
      const unsigned int before =
          __shfl_sync(kFullMask, blockExclusiveScan(lane == 0 ? sum : 0u, tot), 0);
#pragma unroll
      for (int k = 0; k < kScanSteps; ++k) {
        const unsigned int i = i0 + 32u * k;
        if (i < es.nLowerModules) {
          ev.rg.tripletModuleIndices[i] = static_cast<int>(carry + before + ex[k]);
          ev.rg.tripletModuleOccupancy[i] = static_cast<int>(occ[k]);
        }
      }
      carry += tot;
    }
    if (threadIdx.x == 0)
      *ev.rg.device_nTotalTrips = carry;
  }

  // Triplets (SDL/Triplet.h:874-1005): a block walks (inner segment, outer
  // segment of the middle module) of several inner lower modules in order.
  //
  // Most modules hold a few inner segments and some twenty candidates, the
  // heaviest thousands.  A task is therefore up to kT3TaskModules modules, whose
  // inner segments are dealt out across the module boundaries, a thread each, so
  // that the chain of a dozen dependent loads to a triplet is not spent on one
  // module's few candidates; and a task is a block's rather than a warp's, so that
  // a heavy module does not outlast the rest of the kernel in one warp.  For each
  // inner segment shared memory holds the prefix of its candidates and where its
  // outer segments are listed (the MD-keyed segment index of the middle module),
  // so that a candidate reaches its outer segment with one global load.  Only
  // outer segments whose inner MD is the inner segment's outer MD can pass (the
  // first test of the reference's triplet algorithm), so no others are listed;
  // they come in storage order, and candidates keep the reference's (inner,
  // outer) order.
  //
  // Three quarters of the candidates end at the r-z residual (241k per PU200
  // event: 93k have layers that never pass, 86k a residual too large), so a
  // candidate takes that test first and the ones that pass wait in a queue,
  // in order, until there is one for every thread for the rest of the tests.  A
  // passing triplet's place is its module's running count plus the passing
  // candidates of the same module before it.
  //
  // Bound by the latency of the gathers (long scoreboard and the barriers that
  // wait for them; issue slots half used).  A warp per module, all tests in one
  // pass: 64 PU200 events 1120 us, 8 events 183, one 86; so 520 (with the blocks
  // per SM of the default shape; 760 at the same 16), 115 and 38.  A warp per
  // task of 8 modules: 636 at 16 blocks per SM, but 180 for 8 events and 66 for
  // one, where single warps with heavy modules set the length.
  constexpr int kT3Warps = 4;
  constexpr unsigned int kT3Threads = 32 * kT3Warps;  // threads per block the kernel is launched with (at most)
  constexpr unsigned int kT3TaskModules = 32;         // modules per task (at most, a lane each)
  struct T3Scratch {
    unsigned int pre[kT3Threads + 1];
    unsigned int innerSeg[kT3Threads];
    unsigned int listStart[kT3Threads];  // first entry of the inner segment's outer segments in lsByMD
    unsigned int outerBase[kT3Threads];  // first segment of the middle module
    unsigned int modulePre[kT3TaskModules + 1];  // prefix of the task's inner segments over its modules
    unsigned int segBase[kT3TaskModules], flags[kT3TaskModules], count[kT3TaskModules];
    unsigned int passing[32 * kT3Warps];  // per warp and module, of the candidates in hand
    unsigned int warpCount[kT3Warps];
    uint2 queue[2 * kT3Threads];           // (inner, outer) segments that passed the r-z test
    uint8_t queueModule[2 * kT3Threads];   //   and the number of the module in the task
    uint8_t module[kT3Threads];
  };
  __device__ __forceinline__ void t3Task(DeviceES const& es, const EventView& ev, unsigned int firstModule,
                                         unsigned int nModules, T3Scratch& sc) {
    const Modules& m = es.m;
    const unsigned int lane = laneId(), wid = threadIdx.x >> 5, nThreads = blockDim.x;
    const Segments& ls = ev.ls;
    const MDRec* rec = ev.md.rec;
    // the lane's module (every warp has all of the task's)
    const unsigned int own = firstModule + lane;
    const bool valid = lane < nModules && own < es.nLowerModules && m.nConnectedModules[own] != 0;
    const unsigned int nInnerOwn = valid ? static_cast<unsigned int>(ls.nSegments[own]) : 0u;
    const int capOwn = valid ? ev.rg.tripletModuleOccupancy[own] : 0;
    const unsigned int baseOwn = valid ? static_cast<unsigned int>(ev.rg.tripletModuleIndices[own]) : 0u;
    const unsigned int incl = laneInclusiveSum(nInnerOwn);
    const unsigned int nInner = __shfl_sync(kFullMask, incl, 31);
    if (wid == 0) {
      sc.segBase[lane] = valid ? static_cast<unsigned int>(es.lsOffset[own]) : 0u;
      sc.flags[lane] = valid ? es.lsCuts[own].flags : 0u;
      sc.count[lane] = 0;
      sc.modulePre[lane + 1] = incl;
      if (lane == 0)
        sc.modulePre[0] = 0;
    }
    __syncthreads();
    Triplets t3 = ev.t3;
    unsigned int queued = 0;
    for (unsigned int c0 = 0; c0 < nInner; c0 += nThreads) {
      const int n = int(min(nInner - c0, nThreads));
      const bool lastChunk = c0 + nThreads >= nInner;
      unsigned int nOuter = 0;
      if (int(threadIdx.x) < n) {
        const unsigned int g = c0 + threadIdx.x;
        const int j = findSlot(sc.modulePre, kT3TaskModules, g);
        const unsigned int seg = sc.segBase[j] + (g - sc.modulePre[j]);
        const uint16_t middle = ls.outerLowerModuleIndices[seg];
        const unsigned int mdMid = ls.mdIndices[2 * seg + 1];
        const unsigned int outerBase = es.lsOffset[middle];
        const unsigned int listStart = ev.mdLSStart[mdMid], listed = ev.mdLSCount[mdMid];
        sc.innerSeg[threadIdx.x] = seg;
        sc.module[threadIdx.x] = static_cast<uint8_t>(j);
        sc.outerBase[threadIdx.x] = outerBase;
        if (ls.nSegments[middle] != 0) {  // (the index is written for these only)
          sc.listStart[threadIdx.x] = outerBase + listStart;
          nOuter = listed;
        }
      }
      unsigned int total;
      const unsigned int before = blockExclusiveScan(nOuter, total);
      if (int(threadIdx.x) < n)
        sc.pre[threadIdx.x] = before;
      if (threadIdx.x == 0)
        sc.pre[n] = total;
      __syncthreads();
      for (unsigned int start = 0; start < total || (lastChunk && queued > 0); start += nThreads) {
        const unsigned int f = start + threadIdx.x;
        bool pass = false;
        unsigned int innerSeg = 0, outerSeg = 0, module = 0;
        if (f < total) {
          const int i = findSlot(sc.pre, n, f);
          innerSeg = sc.innerSeg[i];
          module = sc.module[i];
          outerSeg = sc.outerBase[i] + ev.lsByMD[sc.listStart[i] + (f - sc.pre[i])];
          const float cut =
              t3RZCut(cutLayer(sc.flags[module]), cutLayer(es.lsCuts[ls.outerLowerModuleIndices[innerSeg]].flags),
                      cutLayer(es.lsCuts[ls.outerLowerModuleIndices[outerSeg]].flags));
          if (cut > 0) {
            const MDRec& in = rec[ls.mdIndices[2 * innerSeg]];
            const MDRec& mid = rec[ls.mdIndices[2 * innerSeg + 1]];
            const MDRec& out = rec[ls.mdIndices[2 * outerSeg + 1]];
            pass = t3PassRZ(in.rt, in.z, mid.rt, mid.z, out.rt, out.z, cut);
          }
        }
        const unsigned int at = blockQueuePlace(pass, sc.warpCount, queued);
        if (pass) {
          sc.queue[at] = make_uint2(innerSeg, outerSeg);
          sc.queueModule[at] = static_cast<uint8_t>(module);
        }
        __syncthreads();
        const bool flush = lastChunk && start + nThreads >= total;
        while (queued >= nThreads || (flush && queued > 0)) {
          bool ok = false;
          T3Values v;
          uint16_t middle = 0, outerOuter = 0;
          const uint2 segs = sc.queue[threadIdx.x], moved = sc.queue[nThreads + threadIdx.x];
          const unsigned int j = threadIdx.x < queued ? sc.queueModule[threadIdx.x] : 0u;
          const uint8_t movedModule = sc.queueModule[nThreads + threadIdx.x];
          if (threadIdx.x < queued) {
            middle = ls.outerLowerModuleIndices[segs.x];
            outerOuter = ls.outerLowerModuleIndices[segs.y];
            ok = t3Rest(sc.flags[j], es.lsCuts[middle].flags, es.lsCuts[outerOuter].flags, m.ptCut,
                        rec[ls.mdIndices[2 * segs.x]], rec[ls.mdIndices[2 * segs.x + 1]],
                        rec[ls.mdIndices[2 * segs.y + 1]], ls, segs.x, v);
          }
          const int cap = __shfl_sync(kFullMask, capOwn, j);
          const unsigned int base = __shfl_sync(kFullMask, baseOwn, j);
          const unsigned int r = blockModuleRank(ok, j, sc.passing, sc.count);
          if (ok && int(r) < cap)
            storeT3(m, ev.md, ls, t3, segs.x, segs.y, static_cast<uint16_t>(firstModule + j), middle, outerOuter, v,
                    base + r);
          sc.queue[threadIdx.x] = moved;
          sc.queueModule[threadIdx.x] = movedModule;
          queued -= min(queued, nThreads);
          blockRankDone(sc.passing, sc.count);
        }
      }
      __syncthreads();  // the chunk's scratch has been read
    }
    if (wid == 0 && nInnerOwn > 0) {
      const unsigned int n = sc.count[lane];
      t3.nTriplets[own] = (int(n) < capOwn) ? n : (capOwn > 0 ? unsigned(capOwn) : 0u);
      t3.totOccupancyTriplets[own] = n;
      if (int(n) > capOwn)
        atomicOr(&ev.sc->status, kStatusCapOverflow);
    }
  }

  __global__ void __launch_bounds__(LST_LB_T3) kCreateT3(DeviceES es, const EventView* evs, unsigned int modulesPerTask) {
    kernelEntry();
    __shared__ T3Scratch sc;
    const EventView& ev = evs[blockIdx.y];
    const unsigned int nTasks = (es.nLowerModules + modulesPerTask - 1u) / modulesPerTask;
    // tasks from the event's counter (zero before the kernel)
    BlockTasks tasks(&ev.sc->t3Next);
    for (unsigned int task = tasks.take(); task < nTasks; task = tasks.take())
      t3Task(es, ev, task * modulesPerTask, modulesPerTask, sc);
  }

  // ========================================================= quintuplets
  // A quintuplet candidate's key: its module's position in the eligible-module
  // list (12 bits), its inner triplet's number in the module (10) and the outer
  // triplet's position in the list of triplets that start at the shared
  // mini-doublet (10), so that keys ascend in the order of the reference's loops.
  // An event that does not fit (there are 2756 eligible modules in both shipped
  // geometries, and a module holds at most 755 triplets) takes the walk.
  constexpr unsigned int kT5KeyModuleShift = 20, kT5KeyInnerShift = 10;
  constexpr unsigned int kT5KeyModules = 1u << (32 - kT5KeyModuleShift);
  constexpr unsigned int kT5KeyLimit = 1u << kT5KeyInnerShift;  // inner triplets, outer triplets of one
  constexpr unsigned int kT5StagedCap = 1u << 16;  // candidates per event that pass the tracklet tests
  constexpr unsigned int kT5RankCap = 8192;        // passing candidates per event
  constexpr unsigned int kT5SortCap = 1u << 15;    // quintuplets per event listed for the track-candidate stage
  // Eligible T5 seed modules and their offsets (SDL/Quintuplet.h:3117-3213),
  // and the tasks of kT5Eval's warps: innerPerTask (up to 32) inner triplets of one module.
  // One block per event, a run of modules per warp as in kT3Offsets; the three
  // sums (modules, quintuplet places, tasks) are scanned together.
  __global__ void __launch_bounds__(1024) kT5Eligible(DeviceES es, const EventView* evs, unsigned int innerPerTask) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    const unsigned int lane = laneId(), wid = threadIdx.x >> 5;
    unsigned int runN = 0, runQ = 0, runT = 0;
    for (unsigned int base = 0; base < es.nLowerModules; base += kScanRun) {
      const unsigned int i0 = base + wid * 32u * kScanSteps + lane;
      unsigned int nT3[kScanSteps];
      int cap[kScanSteps];
      unsigned int layer12 = 0;  // bit k: module of step k lies in layer 1 or 2
      unsigned int sumN = 0, sumQ = 0, sumT = 0;
#pragma unroll
      for (int k = 0; k < kScanSteps; ++k) {
        const unsigned int i = i0 + 32u * k;
        const bool in = i < es.nLowerModules;
        nT3[k] = in ? static_cast<unsigned int>(ev.t3.nTriplets[i]) : 0u;
        cap[k] = in ? es.t5CapIfEligible[i] : -1;
        const int layer = in ? es.m.layers[i] : 0;
        layer12 |= (layer == 1 || layer == 2) ? 1u << k : 0u;
      }
      auto tasksOf = [&](int k) {
        return (layer12 >> k) & 1u ? (nT3[k] + innerPerTask - 1u) / innerPerTask : 0u;
      };
#pragma unroll
      for (int k = 0; k < kScanSteps; ++k)
        if (nT3[k] != 0 && cap[k] >= 0) {
          ++sumN;
          sumQ += static_cast<unsigned int>(cap[k]);
          sumT += tasksOf(k);
        }
      unsigned int totN, totQ, totT;
      const unsigned int n0 = laneInclusiveSum(sumN), q0 = laneInclusiveSum(sumQ), t0 = laneInclusiveSum(sumT);
      const unsigned int bN = blockExclusiveScan(lane == 31 ? n0 : 0u, totN);
      const unsigned int bQ = blockExclusiveScan(lane == 31 ? q0 : 0u, totQ);
      const unsigned int bT = blockExclusiveScan(lane == 31 ? t0 : 0u, totT);
      // (before lane 31's value is added, every lane of the warp has the total of
      // the warps before it)
      unsigned int posN = runN + bN, posQ = runQ + bQ, posT = runT + bT;
#pragma unroll
      for (int k = 0; k < kScanSteps; ++k) {
        const unsigned int i = i0 + 32u * k;
        const bool on = nT3[k] != 0 && cap[k] >= 0;
        const unsigned int occ = on ? static_cast<unsigned int>(cap[k]) : 0u, nTasks = on ? tasksOf(k) : 0u;
        const unsigned int mask = __ballot_sync(kFullMask, on);
        const unsigned int inclQ = laneInclusiveSum(occ), inclT = laneInclusiveSum(nTasks);
        if (on) {
          const unsigned int pos = posN + __popc(mask & lanesBelowMask());
          const unsigned int first = posT + inclT - nTasks;
          for (unsigned int t = 0; t < nTasks; ++t)
            ev.t5Task[first + t] = (pos << kT5KeyModuleShift) | (t * innerPerTask);
          ev.rg.indicesOfEligibleT5Modules[pos] = static_cast<uint16_t>(i);
          ev.rg.quintupletModuleIndices[i] = static_cast<int>(posQ + inclQ - occ);
          ev.rg.quintupletModuleOccupancy[i] = static_cast<int>(occ);
          // (the modules' counts are written by the kernels that store the T5s, for
          // the modules that have any)
          ev.t5.nQuintuplets[i] = 0;
          ev.t5.totOccupancyQuintuplets[i] = 0;
        }
        posN += __popc(mask);
        posQ += __shfl_sync(kFullMask, inclQ, 31);
        posT += __shfl_sync(kFullMask, inclT, 31);
      }
      runN += totN;
      runQ += totQ;
      runT += totT;
    }
    if (threadIdx.x == 0) {
      *ev.rg.nEligibleT5Modules = static_cast<uint16_t>(runN);
      *ev.rg.device_nTotalQuints = runQ;
      ev.sc->t5Tasks = runT;
      ev.sc->t5InnerPerTask = innerPerTask;
      ev.sc->t5Overflow = runN > kT5KeyModules ? 1u : 0u;
      ev.sc->t5Next = 0;
      ev.sc->t5StagedCount = 0;
      ev.sc->t5PassCount = 0;
      ev.sc->t5ListCount = 0;
    }
  }

  // Appends a stored quintuplet to the event's list (any order), which the
  // kernels of the track-candidate stage share out over their warps.
  __device__ __forceinline__ void t5ListAdd(const EventView& ev, unsigned int q, unsigned int module) {
    const unsigned int k = atomicAdd(&ev.sc->t5ListCount, 1u);
    if (k < kT5SortCap)
      ev.t5List[k] = make_uint2(q, module);
  }

  // One warp per eligible module walking (inner T3, outer T3) in order
  // (SDL/Quintuplet.h:2988-3115).
  constexpr int kT5Warps = 4;
  constexpr int kT5MaxInner = 1024;
  __device__ __forceinline__ void t5Module(
      DeviceES const& es, const EventView& ev, unsigned int module, unsigned int* pre, bool useDnn) {
    const uint16_t lm1 = ev.rg.indicesOfEligibleT5Modules[module];
    const Modules& m = es.m;
    const int layer = m.layers[lm1];
    if (layer != 1 && layer != 2)
      return;
    const unsigned int nInner = ev.t3.nTriplets[lm1];
    const unsigned int t3Base = ev.rg.tripletModuleIndices[lm1];
    const Triplets& t3r = ev.t3;
    // Only outer triplets whose first MD is the inner triplet's third MD can
    // pass (the first test of the reference's quintuplet algorithm); they are
    // enumerated through the MD-keyed triplet index in storage order.
    const unsigned int total = warpPrefix(pre, int(nInner), [&](int i) {
      uint16_t lm3 = t3r.lowerModuleIndices[3 * (t3Base + i) + 2];
      if (t3r.nTriplets[lm3] == 0)
        return 0u;
      const unsigned int seg2 = t3r.segmentIndices[2 * (t3Base + i) + 1];
      return static_cast<unsigned int>(ev.mdT3Count[ev.ls.mdIndices[2 * seg2 + 1]]);
    });
    const int cap = ev.rg.quintupletModuleOccupancy[lm1];
    const unsigned int base = ev.rg.quintupletModuleIndices[lm1];
    Triplets t3 = ev.t3;
    Quintuplets t5 = ev.t5;
    ConstDnn dnn;
    unsigned int count = 0;
    for (unsigned int start = 0; start < total; start += 32) {
      unsigned int f = start + laneId();
      bool ok = false;
      T5Values v;
      unsigned int innerT3 = 0, outerT3 = 0;
      uint16_t lm[5] = {lm1, 0, 0, 0, 0};
      if (f < total) {
        int i = findSlot(pre, int(nInner), f);
        innerT3 = t3Base + i;
        lm[1] = t3.lowerModuleIndices[3 * innerT3 + 1];
        lm[2] = t3.lowerModuleIndices[3 * innerT3 + 2];
        const unsigned int mdMid = ev.ls.mdIndices[2 * t3.segmentIndices[2 * innerT3 + 1] + 1];
        const unsigned int outerBase = ev.rg.tripletModuleIndices[lm[2]];
        outerT3 = outerBase + ev.t3ByMD[outerBase + ev.mdT3Start[mdMid] + (f - pre[i])];
        lm[3] = t3.lowerModuleIndices[3 * outerT3 + 1];
        lm[4] = t3.lowerModuleIndices[3 * outerT3 + 2];
        ok = t5Select(m, ev.md, ev.ls, t3, dnn.get(), useDnn, c_t5dnnWP, lm, innerT3, outerT3, v);
      }
      unsigned int tot;
      unsigned int r = count + warpRank(ok, tot);
      if (ok && int(r) < cap) {
        storeT5(ev.md, ev.ls, t3, t5, innerT3, outerT3, lm, layer, v, base + r);
        t5ListAdd(ev, base + r, module);
      }
      count += tot;
    }
    if (laneId() == 0) {
      t5.nQuintuplets[lm1] = (int(count) < cap) ? count : (cap > 0 ? unsigned(cap) : 0u);
      t5.totOccupancyQuintuplets[lm1] = count;
      if (int(count) > cap)
        atomicOr(&ev.sc->status, kStatusCapOverflow);
    }
  }

  // ------------------------------------------ T5 as a candidate work list
  // The warp-per-module walk above leaves most lanes idle: a few modules own
  // most candidates and the candidates diverge early.  Instead kT5Eval deals out
  // the modules' inner triplets, 32 to a warp task, and runs the selection with
  // full warps, kT5Classify the rest of it on what reaches the classifier, and
  // kT5RankEmit stores the passing candidates in key order, so ranks, caps and
  // stored values are those of the walk.  Events that overflow a list take the
  // walk instead.
  constexpr unsigned int kCandQueueCap = 1u << 18;  // pre-selected pT5 / pT3 candidates per event
  __device__ __forceinline__ bool t5NeedsWalk(const EventView& ev) {
    return ev.forceWalk || ev.sc->t5Overflow || ev.sc->t5StagedCount > kT5StagedCap || ev.sc->t5PassCount > kT5RankCap;
  }

  // Candidate numbering over the event, for the probe: the prefix of the
  // candidates over a module's inner triplets, and of the modules.
  __device__ __forceinline__ unsigned int t5CandidatesOf(const EventView& ev, unsigned int innerT3) {
    const Triplets& t3 = ev.t3;
    uint16_t lm3 = t3.lowerModuleIndices[3 * innerT3 + 2];
    if (t3.nTriplets[lm3] == 0)
      return 0u;
    const unsigned int seg2 = t3.segmentIndices[2 * innerT3 + 1];
    return static_cast<unsigned int>(ev.mdT3Count[ev.ls.mdIndices[2 * seg2 + 1]]);
  }

  // (inner, outer) triplets of candidate f of module lm1.
  __device__ __forceinline__ void t5Candidate(const EventView& ev, unsigned int t3Base, unsigned int nInner, unsigned int f,
                                              unsigned int& innerT3, unsigned int& outerT3) {
    const unsigned int* pre = ev.t5CandPre + t3Base;
    int lo = 0, hi = int(nInner);
    while (hi - lo > 1) {
      int mid = (lo + hi) >> 1;
      if (pre[mid] <= f)
        lo = mid;
      else
        hi = mid;
    }
    innerT3 = t3Base + lo;
    const Triplets& t3 = ev.t3;
    const unsigned int mdMid = ev.ls.mdIndices[2 * t3.segmentIndices[2 * innerT3 + 1] + 1];
    const unsigned int outerBase = ev.rg.tripletModuleIndices[t3.lowerModuleIndices[3 * innerT3 + 2]];
    outerT3 = outerBase + ev.t3ByMD[outerBase + ev.mdT3Start[mdMid] + (f - pre[lo])];
  }

  __global__ void kT5Prefix(DeviceES es, const EventView* evs) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    const int wpb = blockDim.x >> 5;
    const int nE = *ev.rg.nEligibleT5Modules;
    for (int w = blockIdx.x * wpb + (threadIdx.x >> 5); w < nE; w += gridDim.x * wpb) {
      const uint16_t lm1 = ev.rg.indicesOfEligibleT5Modules[w];
      const int layer = es.m.layers[lm1];
      unsigned int carry = 0;
      if (layer == 1 || layer == 2) {
        const unsigned int nInner = ev.t3.nTriplets[lm1];
        const unsigned int t3Base = ev.rg.tripletModuleIndices[lm1];
        for (unsigned int b = 0; b < nInner; b += 32) {
          unsigned int i = b + laneId();
          unsigned int c = i < nInner ? t5CandidatesOf(ev, t3Base + i) : 0u;
          unsigned int incl = c;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            unsigned int y = __shfl_up_sync(kFullMask, incl, o);
            if (int(laneId()) >= o)
              incl += y;
          }
          if (i < nInner)
            ev.t5CandPre[t3Base + i] = carry + incl - c;
          carry += __shfl_sync(kFullMask, incl, 31);
        }
      }
      if (laneId() == 0)
        ev.t5ModCand[w] = carry;
    }
  }

  __global__ void __launch_bounds__(1024) kT5ModScan(DeviceES es, const EventView* evs) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    const unsigned int nE = *ev.rg.nEligibleT5Modules;
    unsigned int carry = 0;
    for (unsigned int base = 0; base < nE; base += blockDim.x) {
      unsigned int i = base + threadIdx.x;
      unsigned int c = i < nE ? ev.t5ModCand[i] : 0u;
      unsigned int tot;
      unsigned int ex = blockExclusiveScan(c, tot);
      if (i < nE)
        ev.t5ModOff[i] = carry + ex;
      carry += tot;
    }
    if (threadIdx.x == 0) {
      ev.t5ModOff[nE] = carry;
      ev.sc->t5CandTotal = carry;
    }
  }

  // The T5 selection up to the classifier (SDL/Quintuplet.h:2508-2920).  A warp
  // takes a task of a few inner triplets (up to 32) of one module: its lanes fetch where
  // their outer triplets are listed (those that start at the inner triplet's
  // third mini-doublet), and the candidates are tested 32 at a time.  Each long
  // test runs when the warp's own queue for it, in shared memory, holds a warp
  // full of candidates: the radius tests leave about a quarter of the candidates
  // of a PU200 event, the first tracklet test 70% of those, the second 45%; what
  // passes goes to the event's list in any order.  The two tracklet tests share
  // one copy of the code.  A candidate's outcome does not depend on which thread
  // evaluates it.
  //
  // Bound by the latency of dependent gathers and of instruction fetches: with
  // three inlined tracklet algorithms and the r-z fit's tables in this kernel it
  // waited mostly for instructions (64 PU200 events: 1019 us, now 510).  Numbering
  // the candidates over the event (a prefix kernel, a scan, a radius kernel that
  // filled a queue in memory) and evaluating the classifier at the end of this
  // kernel's blocks took, with the emission, 1.46 ms for 64 PU200 events and 360
  // us for one; this, kT5Classify and kT5RankEmit take 0.82 ms and 120 us.
  constexpr int kT5EvalWarps = 4;
  struct T5Scratch {
    unsigned int pre[33];
    unsigned int listStart[32];  // per inner triplet: its first entry in t3ByMD
    unsigned int outerBase[32];  //   and the first triplet of that list's module
    unsigned int key[2][64], inner[2][64], outer[2][64];  // candidates waiting for the two tracklet tests
  };
  struct T5Staged {
    unsigned int key, inner, outer;
  };
  struct T5Objects {  // a candidate's segments, mini-doublets and modules
    unsigned int seg1, seg3, seg4;
    unsigned int md[5];
    uint16_t lm[5];
  };
  __device__ __forceinline__ void t5Objects(const EventView& ev, unsigned int inner, unsigned int outer, T5Objects& o) {
    const Triplets& t = ev.t3;
    const unsigned int* mdIdx = ev.ls.mdIndices;
    const unsigned int seg2 = t.segmentIndices[2 * inner + 1];
    o.seg1 = t.segmentIndices[2 * inner];
    o.seg3 = t.segmentIndices[2 * outer];
    o.seg4 = t.segmentIndices[2 * outer + 1];
    o.lm[0] = t.lowerModuleIndices[3 * inner];
    o.lm[1] = t.lowerModuleIndices[3 * inner + 1];
    o.lm[2] = t.lowerModuleIndices[3 * inner + 2];
    o.lm[3] = t.lowerModuleIndices[3 * outer + 1];
    o.lm[4] = t.lowerModuleIndices[3 * outer + 2];
    o.md[0] = mdIdx[2 * o.seg1];
    o.md[1] = mdIdx[2 * seg2];
    o.md[2] = mdIdx[2 * seg2 + 1];
    o.md[3] = mdIdx[2 * o.seg3 + 1];
    o.md[4] = mdIdx[2 * o.seg4 + 1];
  }

  __global__ void __launch_bounds__(LST_LB_T5EVAL) kT5Eval(DeviceES es, const EventView* evs) {
    kernelEntry();
    __shared__ T5Scratch sScratch[kT5EvalWarps];
    const EventView& ev = evs[blockIdx.y];
    if (ev.forceWalk || ev.sc->t5Overflow)
      return;
    T5Scratch& sc = sScratch[threadIdx.x >> 5];
    const Triplets& t3 = ev.t3;
    const unsigned int nTasks = ev.sc->t5Tasks, innerPerTask = ev.sc->t5InnerPerTask;
    WarpTasks tasks(&ev.sc->t5Next);
    const unsigned int lane = laneId();
    bool more = true;                // the event may have tasks left
    unsigned int module = 0, inner0 = 0, t3Base = 0;  // the current task: module position, first inner triplet
    unsigned int f0 = 0, total = 0;  //   and its candidates from f0 on
    int nInner = 0;
    unsigned int n0 = 0, n1 = 0;  // entries in the two queues
    while (true) {
      while (n0 < 32u) {
        if (f0 < total) {
          const unsigned int f = f0 + lane;
          f0 += 32u;
          bool pass = false;
          unsigned int key = 0, inner = 0, outer = 0;
          if (f < total) {
            const int i = findSlot(sc.pre, nInner, f);
            const unsigned int pos = f - sc.pre[i];
            inner = t3Base + inner0 + unsigned(i);
            outer = sc.outerBase[i] + ev.t3ByMD[sc.listStart[i] + pos];
            key = (module << kT5KeyModuleShift) | ((inner0 + unsigned(i)) << kT5KeyInnerShift) | pos;
            if (pos >= kT5KeyLimit || inner0 + unsigned(i) >= kT5KeyLimit) {
              ev.sc->t5Overflow = 1;
            } else {
              const uint16_t lm[5] = {t3.lowerModuleIndices[3 * inner], t3.lowerModuleIndices[3 * inner + 1],
                                      t3.lowerModuleIndices[3 * inner + 2], t3.lowerModuleIndices[3 * outer + 1],
                                      t3.lowerModuleIndices[3 * outer + 2]};
              T5Values v;
              T5Stage st;
              pass = t5RadiusStage(es.m, ev.md, ev.ls, t3, lm, inner, outer, v, st);
            }
          }
          const unsigned int ok = __ballot_sync(kFullMask, pass);
          if (pass) {
            const unsigned int k = n0 + __popc(ok & lanesBelowMask());
            sc.key[0][k] = key;
            sc.inner[0][k] = inner;
            sc.outer[0][k] = outer;
          }
          n0 += __popc(ok);
        } else if (more) {
          const unsigned int task = tasks.take();
          more = task < nTasks;
          if (!more)
            break;
          __syncwarp();  // the previous task's scratch has been read
          module = ev.t5Task[task] >> kT5KeyModuleShift;
          inner0 = ev.t5Task[task] & ((1u << kT5KeyModuleShift) - 1u);
          const uint16_t lm1 = ev.rg.indicesOfEligibleT5Modules[module];
          t3Base = ev.rg.tripletModuleIndices[lm1];
          nInner = int(min(innerPerTask, static_cast<unsigned int>(t3.nTriplets[lm1]) - inner0));
          total = warpPrefix(sc.pre, nInner, [&](int i) {
            const unsigned int in = t3Base + inner0 + unsigned(i);
            const uint16_t lm3 = t3.lowerModuleIndices[3 * in + 2];
            const unsigned int mdMid = ev.ls.mdIndices[2 * t3.segmentIndices[2 * in + 1] + 1];
            if (t3.nTriplets[lm3] == 0)
              return 0u;
            const unsigned int base = ev.rg.tripletModuleIndices[lm3];
            sc.outerBase[i] = base;
            sc.listStart[i] = base + ev.mdT3Start[mdMid];
            return static_cast<unsigned int>(ev.mdT3Count[mdMid]);
          });
          f0 = 0;
        } else {
          break;
        }
      }
      __syncwarp();
      // the second queue if it holds a warp full, or, at the end of the candidates,
      // the first that holds any
      const bool second = n1 >= 32u || n0 == 0;
      const unsigned int have = second ? n1 : n0;
      if (have == 0)
        break;
      const unsigned int take = min(have, 32u), at = have - take;
      bool pass = lane < take;
      unsigned int key = 0, inner = 0, outer = 0;
      if (pass) {
        key = sc.key[second][at + lane];
        inner = sc.inner[second][at + lane];
        outer = sc.outer[second][at + lane];
      }
      (second ? n1 : n0) = at;
      __syncwarp();  // the entries have been read
      if (pass) {
        T5Objects o;
        t5Objects(ev, inner, outer, o);
        pass = t4Select(es.m, ev.md, ev.ls, t5Tracklet(o.lm, o.seg1, second ? o.seg4 : o.seg3, o.md, second ? 1 : 0));
      }
      const unsigned int ok = __ballot_sync(kFullMask, pass);
      if (ok == 0u)
        continue;
      if (!second) {
        if (pass) {
          const unsigned int k = n1 + __popc(ok & lanesBelowMask());
          sc.key[1][k] = key;
          sc.inner[1][k] = inner;
          sc.outer[1][k] = outer;
        }
        n1 += __popc(ok);
        __syncwarp();
        continue;
      }
      unsigned int start = 0;
      if (lane == 0)
        start = atomicAdd(&ev.sc->t5StagedCount, __popc(ok));
      start = __shfl_sync(kFullMask, start, 0);
      const unsigned int k = start + __popc(ok & lanesBelowMask());
      if (pass && k < kT5StagedCap)
        ev.t5Staged[k] = T5Staged{key, inner, outer};
    }
  }

  // The forward pass of the classifier for a warp's candidates, accumulating in
  // the reference's order (SDL/NeuralNetwork.h:116-164; t5DnnForward is the same
  // sums one column at a time).  act: this thread's column of the block's
  // activations in shared memory, row stride kT5ClassifyThreads.
  constexpr int kT5ClassifyThreads = 64;
  template <int kRows>
  __device__ __forceinline__ void t5DnnLayer(const float* w, const float* b, float* act) {
    float acc[32];
#pragma unroll
    for (int c = 0; c < 32; ++c)
      acc[c] = 0;
#pragma unroll 2
    for (int in = 0; in < kRows; ++in) {
      const float x = act[in * kT5ClassifyThreads];
      const float4* row = reinterpret_cast<const float4*>(w + in * 32);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float4 q = row[c];
        acc[4 * c] += x * q.x;
        acc[4 * c + 1] += x * q.y;
        acc[4 * c + 2] += x * q.z;
        acc[4 * c + 3] += x * q.w;
      }
    }
#pragma unroll
    for (int c = 0; c < 32; ++c) {
      const float v = acc[c] + b[c];
      act[c * kT5ClassifyThreads] = v > 0.f ? v : 0.f;
    }
  }

  // The rest of the T5 selection (SDL/Quintuplet.h:2715-2984) on the candidates
  // that pass the tracklet tests, a thread each: the r-z fit, and on those that
  // pass it (about half, gathered in shared memory so that the threads are filled
  // again) the circle regression, the DNN (or the cut-only method's chi-squared
  // table) and the chi-squared of the non-anchor hits.  The weights come from
  // memory (a copy beside the constant one, whose reads at 32 addresses a warp are
  // served one by one), only in blocks that have a candidate.
  __global__ void __launch_bounds__(kT5ClassifyThreads) kT5Classify(DeviceES es, const EventView* evs, bool useDnn) {
    kernelEntry();
    __shared__ __align__(16) float sW[kT5DnnParams + 3];
    __shared__ float sAct[38 * kT5ClassifyThreads];
    __shared__ T5Staged sFit[2 * kT5ClassifyThreads];  // candidates that pass the r-z fit
    __shared__ float sRz[2 * kT5ClassifyThreads];
    __shared__ bool sTight[2 * kT5ClassifyThreads];
    __shared__ unsigned int sCount;
    const EventView& ev = evs[blockIdx.y];
    const unsigned int n = ev.sc->t5StagedCount;
    if (ev.forceWalk || ev.sc->t5Overflow || n > kT5StagedCap || blockIdx.x * kT5ClassifyThreads >= n)
      return;
    const T5DnnWeights& w = *reinterpret_cast<const T5DnnWeights*>(sW);
    if (useDnn) {
      const float* src = reinterpret_cast<const float*>(&g_t5dnn);
      for (int i = threadIdx.x; i < kT5DnnParams; i += kT5ClassifyThreads)
        sW[i] = src[i];
    }
    if (threadIdx.x == 0)
      sCount = 0;
    __syncthreads();
    const float wp = c_t5dnnWP;
    const MiniDoublets& md = ev.md;
    for (unsigned int base = blockIdx.x * kT5ClassifyThreads;; base += gridDim.x * kT5ClassifyThreads) {
      const bool more = base < n;
      const unsigned int q = base + threadIdx.x;
      if (more && q < n) {
        const T5Staged st = ev.t5Staged[q];
        T5Objects o;
        t5Objects(ev, st.inner, st.outer, o);
        const float radius = ev.t3.circleRadius[st.inner];
        float rz = 0;
        bool tight = false;
        if (t5PassRZ(es.m, md, o.md, o.lm, rz, 2 * k2Rinv1GeVf * radius, radius, ev.t3.circleCenterX[st.inner],
                     ev.t3.circleCenterY[st.inner], tight)) {
          const unsigned int k = atomicAdd(&sCount, 1u);  // at most 63 left over and 64 new ones
          sFit[k] = st;
          sRz[k] = rz;
          sTight[k] = tight;
        }
      }
      __syncthreads();
      const unsigned int have = sCount;
      __syncthreads();  // everyone has read the count before anyone adds to it again
      if (have < kT5ClassifyThreads && more)
        continue;
      const unsigned int take = min(have, unsigned(kT5ClassifyThreads)), at = have - take + threadIdx.x;
      bool mine = threadIdx.x < take;
      T5Staged st{};
      T5Values v;
      bool tight = false;
      if (mine) {
        st = sFit[at];
        v.rzChiSquared = sRz[at];
        tight = sTight[at];
      }
      if (threadIdx.x == 0)
        sCount = have - take;
      __syncthreads();  // the entries have been read, the count is set
      if (mine) {
        T5Objects o;
        t5Objects(ev, st.inner, st.outer, o);
        v.innerRadius = ev.t3.circleRadius[st.inner];
        v.outerRadius = ev.t3.circleRadius[st.outer];
        float xs[5], ys[5];
#pragma unroll
        for (int i = 0; i < 5; ++i) {
          xs[i] = md.rec[o.md[i]].x;
          ys[i] = md.rec[o.md[i]].y;
        }
        float g, f;
        v.bridgeRadius = circleFrom3(xs[1], ys[1], xs[2], ys[2], xs[3], ys[3], g, f);
        t5Regression(es.m, o.lm, xs, ys, v);
        if (useDnn) {
          float feat[38];
          t5DnnFeatures(es.m, md, ev.ls, ev.t3, xs, ys, o.md, o.lm, st.inner, v.innerRadius, v.outerRadius,
                        v.bridgeRadius, feat);
          float* act = sAct + threadIdx.x;
#pragma unroll
          for (int i = 0; i < 38; ++i)
            act[i * kT5ClassifyThreads] = feat[i];
          t5DnnLayer<38>(w.w0, w.b0, act);
          t5DnnLayer<32>(w.w2, w.b2, act);
          float out = 0;
#pragma unroll 8
          for (int in = 0; in < 32; ++in)
            out += act[in * kT5ClassifyThreads] * w.w4[in];
          out += w.b4[0];
          const float inference = fexp(out) / (fexp(out) + 1);
          mine = inference > wp;
          tight = tight and (inference > wp);
        } else if (v.regressionRadius < 5.0f / (2.f * k2Rinv1GeVf)) {
          mine = t5PassRPhiChi2(es.m, o.lm, v.chiSquared);
        }
        if (mine) {
          t5NonAnchor(es.m, md, o.lm, o.md, v);
          v.tightCutFlag = tight;
          const unsigned int slot = atomicAdd(&ev.sc->t5PassCount, 1u);
          if (slot < kT5RankCap) {
            ev.t5PassValues[slot] = v;
            ev.t5PassC[slot] = st.key;
            ev.t5PassT3[slot] = make_uint2(st.inner, st.outer);
          }
        }
      }
      if (!more && have <= kT5ClassifyThreads)
        break;
    }
  }

  // The warp-per-module walk, for events that overflow a list (a no-op for the
  // others).
  // Register budget: this fallback does work only for events whose candidates
  // overflow the lists; for the others its blocks return at once, and the
  // budget lets more of them be resident, so the launch drains in fewer waves.
  __global__ void __launch_bounds__(128, 8) kT5Walk(DeviceES es, const EventView* evs, bool useDnn) {
    kernelEntry();
    __shared__ unsigned int sPre[kT5Warps][kT5MaxInner + 1];
    const EventView& ev = evs[blockIdx.y];
    if (!t5NeedsWalk(ev))
      return;
    const int wib = threadIdx.x >> 5;
    const int nE = *ev.rg.nEligibleT5Modules;
    for (int w = blockIdx.x * kT5Warps + wib; w < nE; w += gridDim.x * kT5Warps) {
      __syncwarp();
      t5Module(es, ev, unsigned(w), sPre[wib], useDnn);
    }
  }

  // The passing quintuplet candidates stored in key order: a thread per candidate
  // counts the candidates of its module with a smaller key -- the reference's
  // occupancy rank -- and all of the module's, over the event's keys in shared
  // memory; the one with the largest key writes the module's counts.  Bound by
  // the scattered stores; one block per event with a bitonic sort of the keys took
  // 76 us for 8 PU200 events, up to 16 blocks 29.
  constexpr int kT5RankThreads = 128;
  __global__ void __launch_bounds__(kT5RankThreads) kT5RankEmit(DeviceES es, const EventView* evs) {
    kernelEntry();
    __shared__ __align__(16) unsigned int sKey[kT5RankCap];
    const EventView& ev = evs[blockIdx.y];
    const unsigned int n = ev.sc->t5PassCount;
    if (t5NeedsWalk(ev) || blockIdx.x * kT5RankThreads >= n)
      return;
    const unsigned int n4 = n & ~3u;  // four keys a read
    for (unsigned int j = threadIdx.x; j < n; j += kT5RankThreads)
      sKey[j] = ev.t5PassC[j];
    __syncthreads();
    Triplets t3 = ev.t3;
    Quintuplets t5 = ev.t5;
    for (unsigned int q = blockIdx.x * kT5RankThreads + threadIdx.x; q < n; q += gridDim.x * kT5RankThreads) {
      const unsigned int key = sKey[q], w = key >> kT5KeyModuleShift, base = w << kT5KeyModuleShift;
      unsigned int r = 0, count = 0;
      auto add = [&](unsigned int k) {
        const unsigned int d = k - base;  // wraps to a large value below the module's keys
        r += d < key - base ? 1u : 0u;
        count += d < (1u << kT5KeyModuleShift) ? 1u : 0u;
      };
#pragma unroll 2
      for (unsigned int j = 0; j < n4; j += 4) {
        const uint4 k = *reinterpret_cast<const uint4*>(sKey + j);
        add(k.x);
        add(k.y);
        add(k.z);
        add(k.w);
      }
      for (unsigned int j = n4; j < n; ++j)
        add(sKey[j]);
      const uint16_t lm1 = ev.rg.indicesOfEligibleT5Modules[w];
      const int cap = ev.rg.quintupletModuleOccupancy[lm1];
      if (int(r) < cap) {
        const uint2 t = ev.t5PassT3[q];
        uint16_t lm[5] = {lm1, t3.lowerModuleIndices[3 * t.x + 1], t3.lowerModuleIndices[3 * t.x + 2],
                          t3.lowerModuleIndices[3 * t.y + 1], t3.lowerModuleIndices[3 * t.y + 2]};
        storeT5(ev.md, ev.ls, t3, t5, t.x, t.y, lm, es.m.layers[lm1], ev.t5PassValues[q],
                ev.rg.quintupletModuleIndices[lm1] + r);
        t5ListAdd(ev, ev.rg.quintupletModuleIndices[lm1] + r, w);
      }
      if (r + 1 == count) {
        t5.nQuintuplets[lm1] = (int(count) < cap) ? count : (cap > 0 ? unsigned(cap) : 0u);
        t5.totOccupancyQuintuplets[lm1] = count;
        if (int(count) > cap)
          atomicOr(&ev.sc->status, kStatusCapOverflow);
      }
    }
  }

  // Classifier-stage probe: every T5 candidate that reaches the DNN decision,
  // with its features, the loaded weights' score, the cut-only decision and
  // its 10 hits, appended to the caller's buffers (order not fixed).
  struct T5ProbeOut {
    float* feat;      // capacity x 38
    float* score;     // capacity
    uint8_t* cutPass; // capacity
    uint8_t* rzTight; // capacity
    unsigned int* hits;  // capacity x 10 (event-local hit indices)
    int* eventIndex;     // capacity (slot)
    unsigned int capacity;
    unsigned int* count;
  };

  __global__ void kT5Probe(DeviceES es, const EventView* evs, int firstSlot, T5ProbeOut out) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    const unsigned int total = ev.sc->t5CandTotal;
    const int nE = *ev.rg.nEligibleT5Modules;
    const unsigned int* off = ev.t5ModOff;
    ConstDnn dnn;
    for (unsigned int c = blockIdx.x * blockDim.x + threadIdx.x; c < total; c += gridDim.x * blockDim.x) {
      int lo = 0, hi = nE;
      while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (off[mid] <= c)
          lo = mid;
        else
          hi = mid;
      }
      const uint16_t lm1 = ev.rg.indicesOfEligibleT5Modules[lo];
      unsigned int innerT3, outerT3;
      t5Candidate(ev, ev.rg.tripletModuleIndices[lm1], ev.t3.nTriplets[lm1], c - off[lo], innerT3, outerT3);
      uint16_t lm[5] = {lm1,
                        ev.t3.lowerModuleIndices[3 * innerT3 + 1],
                        ev.t3.lowerModuleIndices[3 * innerT3 + 2],
                        ev.t3.lowerModuleIndices[3 * outerT3 + 1],
                        ev.t3.lowerModuleIndices[3 * outerT3 + 2]};
      T5Values v;
      T5Probe p;
      if (!t5Select(es.m, ev.md, ev.ls, ev.t3, dnn.get(), true, c_t5dnnWP, lm, innerT3, outerT3, v, &p))
        continue;
      const unsigned int slot = atomicAdd(out.count, 1u);
      if (slot >= out.capacity)
        continue;
      for (int k = 0; k < 38; ++k)
        out.feat[38 * size_t(slot) + k] = p.feat[k];
      out.score[slot] = p.dnnScore;
      out.cutPass[slot] = p.cutPass ? 1 : 0;
      out.rzTight[slot] = p.rzTight ? 1 : 0;
      for (int k = 0; k < 6; ++k)
        out.hits[10 * size_t(slot) + k] = ev.t3.hitIndices[6 * innerT3 + k];
      for (int k = 0; k < 4; ++k)
        out.hits[10 * size_t(slot) + 6 + k] = ev.t3.hitIndices[6 * outerT3 + 2 + k];
      out.eventIndex[slot] = firstSlot + int(blockIdx.y);
    }
  }

  // Number of hits two T5s share (SDL/Kernels.h:42-84).
  LST_DEV int sharedHitsT5(const Quintuplets& q, unsigned int ix, unsigned int jx) {
    int nMatched = 0;
    for (int i = 0; i < 10; i++) {
      unsigned int a = q.hitIndices[10 * ix + i];
      bool matched = false;
      for (int j = 0; j < 10; j++)
        if (a == q.hitIndices[10 * jx + j]) {
          matched = true;
          break;
        }
      if (matched)
        nMatched++;
    }
    return nMatched;
  }

  // SDL/Quintuplet.h:3215-3235
  __device__ __forceinline__ void t5Ranges(DeviceES const& es, const EventView& ev) {
    for (unsigned int i = blockIdx.x * blockDim.x + threadIdx.x; i < es.nLowerModules; i += gridDim.x * blockDim.x) {
      if (ev.t5.nQuintuplets[i] == 0 or ev.rg.quintupletModuleIndices[i] == -1) {
        ev.rg.quintupletRanges[i * 2] = -1;
        ev.rg.quintupletRanges[i * 2 + 1] = -1;
      } else {
        ev.rg.quintupletRanges[i * 2] = ev.rg.quintupletModuleIndices[i];
        ev.rg.quintupletRanges[i * 2 + 1] = ev.rg.quintupletModuleIndices[i] + ev.t5.nQuintuplets[i] - 1;
      }
    }
  }

  // Duplicate removal among the T5s of one module (SDL/Kernels.h:202-249).
  // Every pair (i < j) of a module is independent and only ever sets isDup
  // bit 1, so the pairs are dealt out in tiles of 32 x 32 to all warps of the
  // event: a module may hold a few hundred T5s (of about 1300 in the event),
  // nearly all of them within the eta / phi windows of one another, and one
  // block working through such a module's pairs took 1.3 ms.  Each block scans
  // the eligible modules' counts itself (a few microseconds, in place of a
  // list made by another launch), numbers the tile pairs (ti <= tj) of the
  // modules with two or more T5s, and takes the tile pairs of its warps: a
  // lane holds one T5 of tile tj in registers, and the T5s of tile ti, one per
  // lane, are broadcast in turn, so that the ten-by-ten hit comparison reads
  // no memory.  Bound by the comparisons' issue slots.
  constexpr int kT5DedupThreads = 256;
  constexpr unsigned int kT5DedupPerThread = 8;
  constexpr unsigned int kT5DedupChunk = kT5DedupThreads * kT5DedupPerThread;  // eligible modules scanned at a time
  __global__ void __launch_bounds__(kT5DedupThreads) kT5DedupAfterBuild(DeviceES es, const EventView* evs) {
    kernelEntry();
    __shared__ unsigned int sPre[kT5DedupChunk + 1];  // first tile pair of each listed module
    __shared__ uint16_t sMods[kT5DedupChunk];
    const EventView& ev = evs[blockIdx.y];
    t5Ranges(es, ev);
    const unsigned int nElig = *ev.rg.nEligibleT5Modules;
    const unsigned int lane = laneId();
    Quintuplets q = ev.t5;
    for (unsigned int c0 = 0; c0 < nElig; c0 += kT5DedupChunk) {
      uint16_t mods[kT5DedupPerThread];
      unsigned int pairs[kT5DedupPerThread];
      unsigned int myMods = 0, myPairs = 0;
#pragma unroll
      for (unsigned int k = 0; k < kT5DedupPerThread; ++k) {
        const unsigned int e = c0 + threadIdx.x * kT5DedupPerThread + k;
        mods[k] = e < nElig ? ev.rg.indicesOfEligibleT5Modules[e] : 0;
      }
#pragma unroll
      for (unsigned int k = 0; k < kT5DedupPerThread; ++k) {
        const unsigned int e = c0 + threadIdx.x * kT5DedupPerThread + k;
        const unsigned int n = e < nElig ? q.nQuintuplets[mods[k]] : 0u;
        const unsigned int tiles = (n + 31u) >> 5;
        pairs[k] = n >= 2 ? tiles * (tiles + 1) / 2 : 0u;
        myMods += pairs[k] ? 1u : 0u;
        myPairs += pairs[k];
      }
      unsigned int nMods, nPairs;
      unsigned int slot = blockExclusiveScan(myMods, nMods);
      unsigned int first = blockExclusiveScan(myPairs, nPairs);
#pragma unroll
      for (unsigned int k = 0; k < kT5DedupPerThread; ++k) {
        if (pairs[k] == 0)
          continue;
        sMods[slot] = mods[k];
        sPre[slot++] = first;
        first += pairs[k];
      }
      if (threadIdx.x == 0)
        sPre[nMods] = nPairs;
      __syncthreads();
      const unsigned int wpb = kT5DedupThreads / 32;
      for (unsigned int t = blockIdx.x * wpb + (threadIdx.x >> 5); t < nPairs; t += gridDim.x * wpb) {
        const int k = findSlot(sPre, int(nMods), t);
        const uint16_t lm = sMods[k];
        const unsigned int n = q.nQuintuplets[lm];
        const unsigned int base = ev.rg.quintupletModuleIndices[lm];
        const unsigned int local = t - sPre[k];
        unsigned int tj = 0;
        while ((tj + 1) * (tj + 2) / 2 <= local)
          ++tj;
        const unsigned int ti = local - tj * (tj + 1) / 2;
        const unsigned int i = 32 * ti + lane, j = 32 * tj + lane;
        const unsigned int ix = base + min(i, n - 1), jx = base + min(j, n - 1);
        const float etaI = q.eta[ix], phiI = q.phi[ix], scoreI = q.score_rphisum[ix];
        const float etaJ = q.eta[jx], phiJ = q.phi[jx], scoreJ = q.score_rphisum[jx];
        unsigned int hitI[10], hitJ[10];
        // (40 bytes per T5: the ten indices lie on an 8-byte boundary)
        const uint2* hI = reinterpret_cast<const uint2*>(q.hitIndices + 10 * size_t(ix));
        const uint2* hJ = reinterpret_cast<const uint2*>(q.hitIndices + 10 * size_t(jx));
#pragma unroll
        for (int a = 0; a < 5; ++a) {
          const uint2 u = hI[a], v = hJ[a];
          hitI[2 * a] = u.x;
          hitI[2 * a + 1] = u.y;
          hitJ[2 * a] = v.x;
          hitJ[2 * a + 1] = v.y;
        }
        const unsigned int rows = min(n - 32 * ti, 32u);
        for (unsigned int r = 0; r < rows; ++r) {
          const float eta1 = __shfl_sync(kFullMask, etaI, r), phi1 = __shfl_sync(kFullMask, phiI, r);
          const float dEta = fabs_(eta1 - etaJ);
          const float dPhi = wrapDPhi(phi1, phiJ);
          const bool near = j < n && j > 32 * ti + r && !(dEta > 0.1f) && !(fabs_(dPhi) > 0.1f);
          if (!__any_sync(kFullMask, near))
            continue;
          int nMatched = 0;
#pragma unroll
          for (int a = 0; a < 10; ++a) {
            const unsigned int h = __shfl_sync(kFullMask, hitI[a], r);
            bool matched = false;
#pragma unroll
            for (int b = 0; b < 10; ++b)
              matched |= h == hitJ[b];
            nMatched += matched ? 1 : 0;
          }
          const float score1 = __shfl_sync(kFullMask, scoreI, r);
          if (near && nMatched >= 7) {
            if (score1 >= scoreJ)
              q.isDup[base + 32 * ti + r] = 1;
            else
              q.isDup[jx] = 1;
          }
        }
      }
      __syncthreads();  // sMods / sPre are rewritten for the next chunk
    }
  }

  // ==================================================== pLS cleaning
  // SDL/Kernels.h:384-473.  Pass 1 sets bit 1 of isDup directly; pass 2 marks
  // plsFlag and kCrossCleanPLS folds it into bit 2 afterwards, so that pass 2
  // reads the pass-1 bit while other threads mark removals.
  // pLS binned by eta: bins of width 0.02 over [-6, 6) (clamped at both ends)
  // plus a last bin for non-finite eta, which must meet every pLS because a
  // NaN never satisfies the reference's |deta| > 0.1 skip.  Two etas within
  // 0.1 of each other land at most kPLSBinReach bins apart (5 bin widths plus
  // the rounding of the bin coordinate).
  constexpr int kPLSBins = 600;
  constexpr int kPLSBinReach = 6;
  LST_DEV int plsEtaBin(float eta) {
    if (!(fabsf(eta) <= 3.0e38f))
      return kPLSBins;
    float t = (eta + 6.0f) * 50.0f;
    if (t < 0.f)
      return 0;
    if (t >= float(kPLSBins))
      return kPLSBins - 1;
    return static_cast<int>(t);
  }

  // The removal of one tested pLS pair (SDL/Kernels.h:384-473): ix the lower
  // index (the reference's outer loop), jx the higher; marks the one to go.
  LST_DEV void plsRemoveOf(const EventView& ev, unsigned int ix, unsigned int jx, bool secondpass) {
    const Segments& s = ev.ls;
    const int8_t quad_diff = s.isQuad[ix] - s.isQuad[jx];
    const float score_diff = s.score[ix] - s.score[jx];
    unsigned int idxToRemove;
    if (quad_diff > 0)
      idxToRemove = jx;
    else if (quad_diff < 0)
      idxToRemove = ix;
    else if (score_diff < 0)
      idxToRemove = jx;
    else if (score_diff > 0)
      idxToRemove = ix;
    else
      idxToRemove = ix;
    if (secondpass)
      ev.plsFlag[idxToRemove] = 1;
    else
      s.isDup[idxToRemove] = 1;
  }

  LST_DEV bool plsCleanEligible(const Segments& s, unsigned int i, bool secondpass) {
    return !secondpass || (s.isQuad[i] && !(s.isDup[i] & 1));
  }

  // pLS duplicate removal (SDL/Kernels.h:384-473).  Pass 1 sets bit 1 of
  // isDup directly; pass 2 marks plsFlag and kCrossCleanPLS folds it into bit 2
  // afterwards, so that pass 2 reads the pass-1 bit while other threads mark
  // removals.  The outcome of a pair (ix < jx) depends only on the two pLS, and
  // marks are only ever set, so any visiting order and any repeat visit give
  // the reference's result.  A pair removes a pLS
  //   pass 1: if ix has at least 3 of its 4 hits among jx's (npMatched >= 3),
  //   pass 2: if they have a hit in common (npMatched >= 1) or dR2 < 1e-5,
  // in both cases unless |deta| > 0.1 (a NaN never satisfies that skip), and
  // in pass 2 only between quads without a pass-1 mark.
  //
  // kPLSCleanHits finds every pair of the hit conditions: one thread per pLS
  // ix walks the hit index for its hits (pass 1: hits 0 and 1, one of which
  // is among jx's when three of the four are; pass 2: all four) and tests the
  // higher-index pLS jx found there.  A pair met through several hits is
  // tested again, which changes nothing.
  __global__ void kPLSCleanHits(DeviceES es, const EventView* evs, bool secondpass) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    const Segments& s = ev.ls;
    unsigned int nPix = s.nSegments[es.pixelModule];
    if (nPix > kMaxPixelSegments)
      nPix = kMaxPixelSegments;
    const unsigned int maxSteps = 4 * nPix;  // a chain holds each entry once: no walk takes more
    const uint4* hits = reinterpret_cast<const uint4*>(s.pLSHitsIdxs);
    for (unsigned int ix = blockIdx.x * blockDim.x + threadIdx.x; ix < nPix; ix += gridDim.x * blockDim.x) {
      if (!plsCleanEligible(s, ix, secondpass))
        continue;
      const uint4 h1 = hits[ix];
      const unsigned int h1a[4] = {h1.x, h1.y, h1.z, h1.w};
      const float eta1 = s.eta[ix];
      const int nSlots = secondpass ? 4 : 2;
      for (int slot = 0; slot < nSlots; ++slot) {
        const unsigned int h = h1a[slot];
        unsigned int steps = 0;
        for (unsigned int e = ev.plsHitHead[plsHitBucket(h)]; e != kPLSHitNone; e = ev.plsHitNext[e]) {
          if (++steps > maxSteps) {
            atomicOr(&ev.sc->status, kStatusInvalidInput);
            break;
          }
          const unsigned int jx = e >> 2;
          if (jx <= ix || jx >= nPix || s.pLSHitsIdxs[e] != h)
            continue;
          if (fabs_(s.eta[jx] - eta1) > 0.1f)
            continue;
          if (!plsCleanEligible(s, jx, secondpass))
            continue;
          bool remove = true;  // pass 2: a hit in common
          if (!secondpass) {
            const uint4 h2 = hits[jx];
            int npMatched = 0;
            for (int k = 0; k < 4; k++)
              if (h1a[k] == h2.x || h1a[k] == h2.y || h1a[k] == h2.z || h1a[k] == h2.w)
                npMatched++;
            remove = npMatched >= 3;
          }
          if (remove)
            plsRemoveOf(ev, ix, jx, secondpass);
        }
      }
    }
  }

  // One pass-2 pLS as kPLSCleanNear reads it, stored in eta-bin order so that
  // a tile of candidates is one coalesced read.
  struct __align__(16) PLSRec {
    float eta, phi;
    unsigned int index, pad;
  };

  // Counting sort, by eta bin, of the pLS that pass 2 tests (the quads
  // without a pass-1 mark), one block per event; writes the bin starts (the
  // last entry being the number of records) and the sorted records.
  __global__ void __launch_bounds__(1024) kPLSBin(DeviceES es, const EventView* evs) {
    kernelEntry();
    __shared__ unsigned int sCount[kPLSBins + 1];
    __shared__ unsigned int sCursor[kPLSBins + 1];
    const EventView& ev = evs[blockIdx.y];
    const Segments& s = ev.ls;
    unsigned int nPix = s.nSegments[es.pixelModule];
    if (nPix > kMaxPixelSegments)
      nPix = kMaxPixelSegments;
    for (int b = threadIdx.x; b <= kPLSBins; b += blockDim.x)
      sCount[b] = 0;
    __syncthreads();
    // The eligible pLS among 8 of this thread's at a time, all loads of a round
    // issued together (a round of one pLS per thread waited for each load).
    constexpr int kRound = 8;
    auto round = [&](unsigned int i0, float* eta, float* phi) {
      unsigned int on = 0;
      int8_t quad[kRound], dup[kRound];
#pragma unroll
      for (int k = 0; k < kRound; ++k) {
        const unsigned int i = i0 + k * 1024u;
        const bool in = i < nPix;
        quad[k] = in ? s.isQuad[i] : 0;
        dup[k] = in ? s.isDup[i] : 1;
        eta[k] = in ? s.eta[i] : 0.f;
        if (phi)
          phi[k] = in ? s.phi[i] : 0.f;
      }
#pragma unroll
      for (int k = 0; k < kRound; ++k)
        on |= quad[k] && !(dup[k] & 1) ? 1u << k : 0u;
      return on;
    };
    for (unsigned int i0 = threadIdx.x; i0 < nPix; i0 += kRound * 1024u) {
      float eta[kRound];
      const unsigned int on = round(i0, eta, nullptr);
#pragma unroll
      for (int k = 0; k < kRound; ++k)
        if ((on >> k) & 1u)
          atomicAdd(&sCount[plsEtaBin(eta[k])], 1u);
    }
    __syncthreads();
    unsigned int c = threadIdx.x <= kPLSBins ? sCount[threadIdx.x] : 0u;
    unsigned int tot;
    unsigned int ex = blockExclusiveScan(c, tot);
    if (threadIdx.x <= kPLSBins) {
      sCursor[threadIdx.x] = ex;
      ev.plsBinStart[threadIdx.x] = ex;
    }
    if (threadIdx.x == 0)
      ev.plsBinStart[kPLSBins + 1] = tot;
    __syncthreads();
    for (unsigned int i0 = threadIdx.x; i0 < nPix; i0 += kRound * 1024u) {
      float eta[kRound], phi[kRound];
      const unsigned int on = round(i0, eta, phi);
#pragma unroll
      for (int k = 0; k < kRound; ++k)
        if ((on >> k) & 1u) {
          PLSRec r;
          r.eta = eta[k];
          r.phi = phi[k];
          r.index = i0 + k * 1024u;
          r.pad = 0;
          ev.plsRec[atomicAdd(&sCursor[plsEtaBin(r.eta)], 1u)] = r;
        }
    }
  }

  // kPLSCleanNear finds the pass-2 pairs of the dR2 condition.  dR2 < 1e-5
  // needs |deta| < 0.0032, so both lie in the same or adjacent eta bins, and
  // a NaN or infinite eta never passes (the non-finite bin is left out).  Each
  // pair is tested once, by the record that comes first in the eta-sorted
  // order: each block takes kPLSCleanTile consecutive finite records (one per
  // thread) and streams, through shared memory, the later records up to one
  // bin above its last record's bin; each warp tests only the part its own
  // records can reach.  dEta and dPhi are taken with the lower index first,
  // as in the reference.
  constexpr int kPLSCleanTile = 128;

  __global__ void __launch_bounds__(kPLSCleanTile) kPLSCleanNear(DeviceES es, const EventView* evs) {
    kernelEntry();
    __shared__ PLSRec sT[kPLSCleanTile];
    const EventView& ev = evs[blockIdx.y];
    const PLSRec* rec = ev.plsRec;
    const unsigned int* binStart = ev.plsBinStart;
    const unsigned int nFinite = binStart[kPLSBins];
    const unsigned int warp = threadIdx.x >> 5;
    for (unsigned int k0 = blockIdx.x * kPLSCleanTile; k0 < nFinite; k0 += gridDim.x * kPLSCleanTile) {
      const unsigned int k = k0 + threadIdx.x;
      const bool active = k < nFinite;
      PLSRec me{};
      if (active)
        me = rec[k];
      const unsigned int kLast = min(k0 + kPLSCleanTile, nFinite) - 1;
      const unsigned int span = binStart[min(plsEtaBin(rec[kLast].eta) + 1, kPLSBins - 1) + 1] - k0;
      // this warp's part of the stream: offsets [tW0, tW1)
      const unsigned int kW0 = k0 + warp * 32;
      const unsigned int tW0 = warp * 32;
      unsigned int tW1 = 0;
      if (kW0 < nFinite) {
        const unsigned int kW1 = min(kW0 + 32, nFinite) - 1;
        tW1 = binStart[min(plsEtaBin(rec[kW1].eta) + 1, kPLSBins - 1) + 1] - k0;
      }
      for (unsigned int t0 = 0; t0 < span; t0 += kPLSCleanTile) {
        __syncthreads();
        const unsigned int t = t0 + threadIdx.x;
        if (t < span)
          sT[threadIdx.x] = rec[k0 + t];
        __syncthreads();
        if (!active)
          continue;
        const unsigned int nt = min(span - t0, unsigned(kPLSCleanTile));
        const unsigned int uEnd = tW1 > t0 ? min(tW1 - t0, nt) : 0u;
        for (unsigned int u = tW0 > t0 ? tW0 - t0 : 0u; u < uEnd; ++u) {
          if (t0 + u <= threadIdx.x)
            continue;
          const PLSRec o = sT[u];
          const bool meLow = me.index < o.index;
          const float eta1 = meLow ? me.eta : o.eta, eta2 = meLow ? o.eta : me.eta;
          const float phi1 = meLow ? me.phi : o.phi, phi2 = meLow ? o.phi : me.phi;
          const float dEta = fabs_(eta1 - eta2);
          const float dPhi = wrapDPhi(phi1, phi2);
          const float dR2 = dEta * dEta + dPhi * dPhi;
          if (dR2 < 1e-5f)
            plsRemoveOf(ev, meLow ? me.index : o.index, meLow ? o.index : me.index, true);
        }
      }
    }
  }

  // ============================================ pixel-map slices per pLS
  // The connected modules of pLS i: es.m.connectedPixels[index .. index + size)
  // (SDL/Event.cc:1055-1080).
  __device__ __forceinline__ void pixelSlice(DeviceES const& es, const EventView& ev, unsigned int i, unsigned int& size,
                                             unsigned int& index) {
    const int8_t pixelType = ev.ls.pixelType[i];
    const int superbin = ev.ls.superbin[i];
    size = 0;
    index = 0;
    if ((superbin < 0) or (superbin >= int(kSizeSuperbins)) or (pixelType > 2) or (pixelType < 0))
      return;
    if (pixelType == 0) {
      size = es.cpSizes[superbin];
      index = es.cpIndex[superbin];
    } else if (pixelType == 1) {
      size = es.cpSizesPos[superbin];
      index = es.cpIndexPos[superbin] + es.pixelIndexOffsetPos;
    } else {
      size = es.cpSizesNeg[superbin];
      index = es.cpIndexNeg[superbin] + es.pixelIndexOffsetNeg;
    }
  }

  // ============================================================== pT5
  // Candidate modules of a pLS for pT5 (SDL/PixelTriplet.h:2697-2716).
  __device__ __forceinline__ unsigned int pt5ModuleCount(DeviceES const& es, const EventView& ev, uint16_t mod) {
    if (mod >= es.nLowerModules)
      return 0;
    if (es.m.moduleType[mod] == TwoS)
      return 0;
    return ev.t5.nQuintuplets[mod];
  }

  // Ends a count kernel of the fallback walk: the last block of the event to get
  // here scans the per-pLS pass counts (the others' writes are visible: each block
  // fences its own before it is counted).
  // which = 0: pT5 (cap 15000), 1: pT3 (cap 5000).
  __device__ __forceinline__ void plsScanByLast(DeviceES const& es, const EventView& ev, int which) {
    __shared__ bool sLast;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
      sLast = atomicAdd(&ev.sc->walkDone, 1u) + 1u == gridDim.x;
    __syncthreads();
    if (!sLast)
      return;
    __threadfence();
    const unsigned int n = ev.ls.nSegments[es.pixelModule];
    const volatile unsigned int* counts = ev.plsCount;
    unsigned int carry = 0;
    for (unsigned int base = 0; base < n; base += blockDim.x) {
      unsigned int i = base + threadIdx.x;
      unsigned int c = (i < n) ? counts[i] : 0u;
      unsigned int tot;
      unsigned int ex = blockExclusiveScan(c, tot);
      if (i < n)
        ev.plsOffset[i] = carry + ex;
      carry += tot;
    }
    if (threadIdx.x == 0) {
      ev.sc->walkDone = 0;
      if (which == 0) {
        ev.sc->nPT5Total = carry;
        *ev.pt5.totOccupancyPixelQuintuplets = carry;
        *ev.pt5.nPixelQuintuplets = carry < kMaxPixelQuintuplets ? carry : kMaxPixelQuintuplets;
      } else {
        ev.sc->nPT3Total = carry;
        *ev.pt3.totOccupancyPixelTriplets = carry;
        *ev.pt3.nPixelTriplets = carry < kMaxPixelTriplets ? carry : kMaxPixelTriplets;
      }
      if ((which == 0 && carry > kMaxPixelQuintuplets) || (which == 1 && carry > kMaxPixelTriplets))
        atomicOr(&ev.sc->status, kStatusCapOverflow);
    }
  }

  // Walks the pT5 candidates of one pLS in order; emit selects the pass:
  // count passing candidates, or store those with global rank < cap.
  constexpr int kPixWarps = 4;
  template <bool kEmit>
  __device__ __forceinline__ void pt5Walk(DeviceES const& es, const EventView& ev, unsigned int iPLS, unsigned int* pre,
                                          uint16_t* mods) {
    if (ev.ls.isDup[iPLS])
      return;
    unsigned int nConn, cidx;
    pixelSlice(es, ev, iPLS, nConn, cidx);
    for (unsigned int k = laneId(); k < nConn; k += 32)
      mods[k] = static_cast<uint16_t>(es.m.connectedPixels[cidx + k]);
    __syncwarp();
    const unsigned int total = warpPrefix(pre, int(nConn), [&](int k) { return pt5ModuleCount(es, ev, mods[k]); });
    const unsigned int plsIndex = es.lsOffset[es.nLowerModules] + iPLS;
    unsigned int count = 0;
    unsigned int rankBase = kEmit ? ev.plsOffset[iPLS] : 0u;
    Segments ls = ev.ls;
    Triplets t3 = ev.t3;
    Quintuplets t5 = ev.t5;
    PixelQuintuplets pt5 = ev.pt5;
    for (unsigned int start = 0; start < total; start += 32) {
      unsigned int f = start + laneId();
      bool ok = false;
      PT5Values v;
      unsigned int t5i = 0;
      if (f < total) {
        int k = findSlot(pre, int(nConn), f);
        t5i = ev.rg.quintupletModuleIndices[mods[k]] + (f - pre[k]);
        if (!t5.isDup[t5i])
          ok = pt5Select(es.m, ev.rg, ev.md, ls, t3, t5, plsIndex, t5i, iPLS, v);
      }
      unsigned int tot;
      unsigned int r = rankBase + count + warpRank(ok, tot);
      if (kEmit && ok && r < kMaxPixelQuintuplets)
        storePT5(ev.md, ls, t3, t5, pt5, plsIndex, iPLS, t5i, v, r);
      count += tot;
    }
    if (!kEmit && laneId() == 0)
      ev.plsCount[iPLS] = count;
  }

  // Register budget: this fallback does work only for events whose candidates
  // overflow the lists; for the others its blocks return at once, and the
  // budget lets more of them be resident, so the launch drains in fewer waves.
  __global__ void __launch_bounds__(128, 8) kPT5Count(DeviceES es, const EventView* evs) {
    kernelEntry();
    __shared__ unsigned int sPre[kPixWarps][kMaxConnectedModules + 1];
    __shared__ uint16_t sMods[kPixWarps][kMaxConnectedModules];
    const EventView& ev = evs[blockIdx.y];
    if (!ev.sc->pixFallback)
      return;
    const int wib = threadIdx.x >> 5;
    const unsigned int nPLS = ev.ls.nSegments[es.pixelModule];
    for (unsigned int i = blockIdx.x * kPixWarps + wib; i < nPLS; i += gridDim.x * kPixWarps) {
      __syncwarp();
      if (laneId() == 0)
        ev.plsCount[i] = 0;
      pt5Walk<false>(es, ev, i, sPre[wib], sMods[wib]);
    }
    plsScanByLast(es, ev, 0);
  }

  // Register budget: this fallback does work only for events whose candidates
  // overflow the lists; for the others its blocks return at once, and the
  // budget lets more of them be resident, so the launch drains in fewer waves.
  __global__ void __launch_bounds__(128, 8) kPT5Emit(DeviceES es, const EventView* evs) {
    kernelEntry();
    __shared__ unsigned int sPre[kPixWarps][kMaxConnectedModules + 1];
    __shared__ uint16_t sMods[kPixWarps][kMaxConnectedModules];
    const EventView& ev = evs[blockIdx.y];
    if (!ev.sc->pixFallback)
      return;
    const int wib = threadIdx.x >> 5;
    const unsigned int nPLS = ev.ls.nSegments[es.pixelModule];
    for (unsigned int i = blockIdx.x * kPixWarps + wib; i < nPLS; i += gridDim.x * kPixWarps) {
      __syncwarp();
      if (ev.plsCount[i] == 0 || ev.plsOffset[i] >= kMaxPixelQuintuplets)
        continue;
      pt5Walk<true>(es, ev, i, sPre[wib], sMods[wib]);
    }
  }

  // pT5 duplicate removal (SDL/Kernels.h:356-382): pT5 ix is removed if some
  // jx shares at least 7 of its 14 hit slots and has a lower score (ties: the
  // higher index goes).  The outcome is an OR over jx, and a pair sharing 7
  // slots shares one of any 8 of them, so only pairs that meet in one of ix's
  // first 8 slots need the full test.  kPixRankEmit<5> chains the event's (slot,
  // pT5) entries e = 14 pT5 + slot by hit as it stores the pT5s, in a hash table
  // in memory (a head per bucket, emptied by kPixEval<5>, and a next index per
  // entry), and kPT5DedupHits gives each of the first 8 slots of each pT5 a
  // thread that walks its hit's chain.  Bound by the latency of the walks.
  // Tables in shared memory, built by each of two blocks per event, held 1170
  // pT5s, and a denser event of a batch (PU250, pt0.6) took the tiles below:
  // 738 + 71 us for 13 PU250 events, now 22 here and 28 more in kPixRankEmit<5>.
  // Events whose pT5s the walk stored take the tiles.
  constexpr unsigned int kPT5HitBucketBits = 15;
  constexpr unsigned int kPT5HitBuckets = 1u << kPT5HitBucketBits;
  constexpr unsigned int kPT5HitNone = 0xffffffffu;
  constexpr unsigned int kPT5DedupSlots = 8;
  LST_DEV unsigned int pt5HitBucket(unsigned int h) { return (h * 2654435761u) >> (32 - kPT5HitBucketBits); }

  // Every pair, in tiles staged in shared memory (a block of kDedupTile threads).
  constexpr int kDedupTile = 128;
  __device__ __forceinline__ void pt5DedupTiles(const EventView& ev) {
    __shared__ unsigned int sHits[kDedupTile * 14];
    __shared__ float sScore[kDedupTile];
    const unsigned int n = *ev.pt5.nPixelQuintuplets;
    PixelQuintuplets p = ev.pt5;
    for (unsigned int ixBase = blockIdx.x * kDedupTile; ixBase < n; ixBase += gridDim.x * kDedupTile) {
      const unsigned int ix = ixBase + threadIdx.x;
      const bool valid = ix < n;
      unsigned int mine[14];
      float score1 = 0.f;
      if (valid) {
#pragma unroll
        for (int i = 0; i < 14; ++i)
          mine[i] = p.hitIndices[14 * ix + i];
        score1 = p.score[ix];
      }
      bool dup = false;
      for (unsigned int jBase = 0; jBase < n; jBase += kDedupTile) {
        const unsigned int tile = (n - jBase < kDedupTile) ? n - jBase : kDedupTile;
        __syncthreads();
        for (unsigned int t = threadIdx.x; t < tile * 14; t += blockDim.x)
          sHits[t] = p.hitIndices[14 * jBase + t];
        for (unsigned int t = threadIdx.x; t < tile; t += blockDim.x)
          sScore[t] = p.score[jBase + t];
        __syncthreads();
        if (!valid || dup)
          continue;
        for (unsigned int jj = 0; jj < tile; ++jj) {
          const unsigned int jx = jBase + jj;
          if (jx == ix)
            continue;
          const unsigned int* other = sHits + 14 * jj;
          int nMatched = 0;
#pragma unroll
          for (int i = 0; i < 14; ++i) {
            bool matched = false;
#pragma unroll
            for (int j = 0; j < 14; ++j)
              matched |= (mine[i] == other[j]);
            nMatched += matched ? 1 : 0;
          }
          const float score2 = sScore[jj];
          if (nMatched >= 7) {
            if (score1 > score2 or ((score1 == score2) and (ix > jx))) {
              dup = true;
              break;
            }
          }
        }
      }
      if (valid && dup)
        p.isDup[ix] = 1;
    }
  }

  __global__ void __launch_bounds__(kDedupTile) kPT5DedupHits(DeviceES es, const EventView* evs) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    const unsigned int n = *ev.pt5.nPixelQuintuplets;
    if (blockIdx.x == 0 && threadIdx.x == 0)
      pixCountersClear(ev);  // the pixel lists have been read
    if (ev.sc->pixFallback) {
      pt5DedupTiles(ev);
      return;
    }
    PixelQuintuplets p = ev.pt5;
    for (unsigned int t = blockIdx.x * blockDim.x + threadIdx.x; t < kPT5DedupSlots * n;
         t += gridDim.x * blockDim.x) {
      const unsigned int a = t / kPT5DedupSlots;
      const unsigned int h = p.hitIndices[14 * a + t % kPT5DedupSlots];
      const float score1 = p.score[a];
      for (unsigned int q = ev.pt5HitHead[pt5HitBucket(h)]; q != kPT5HitNone; q = ev.pt5HitNext[q]) {
        const unsigned int b = q / 14;
        if (p.hitIndices[q] != h || b == a)
          continue;
        const float score2 = p.score[b];
        if (!(score1 > score2 or ((score1 == score2) and (a > b))))
          continue;
        // (56 bytes per pT5: the fourteen indices lie on an 8-byte boundary)
        const uint2* mine = reinterpret_cast<const uint2*>(p.hitIndices + 14 * size_t(a));
        const uint2* other = reinterpret_cast<const uint2*>(p.hitIndices + 14 * size_t(b));
        uint2 o[7];
#pragma unroll
        for (int j = 0; j < 7; ++j)
          o[j] = other[j];
        int nMatched = 0;
#pragma unroll
        for (int i = 0; i < 7; ++i) {
          const uint2 m = mine[i];
          bool mx = false, my = false;
#pragma unroll
          for (int j = 0; j < 7; ++j) {
            mx |= m.x == o[j].x || m.x == o[j].y;
            my |= m.y == o[j].x || m.y == o[j].y;
          }
          nMatched += (mx ? 1 : 0) + (my ? 1 : 0);
        }
        if (nMatched >= 7) {
          p.isDup[a] = 1;
          break;
        }
      }
    }
  }

  // Writes a track candidate built from a pT3 / T5 / pT5 record
  // (SDL/TrackCandidate.h:130-163); unused slots are zeroed.
  LST_DEV void storeTC(TrackCandidates& tc,
                       short type,
                       unsigned int innerIdx,
                       unsigned int outerIdx,
                       const uint8_t* logicalLayers,
                       const uint16_t* lowerModules,
                       const unsigned int* hitIndices,
                       int pixelSeedIndex,
                       float centerX,
                       float centerY,
                       float radius,
                       unsigned int idx,
                       unsigned int directIdx) {
    // (loads before stores, as in storeMD)
    const bool seven = type == 7;
    uint8_t layers[7];
    uint16_t modules[7];
    unsigned int hits[14];
#pragma unroll
    for (int i = 0; i < 7; i++) {
      const bool has = i < 5 || seven;
      layers[i] = has ? logicalLayers[i] : 0;
      modules[i] = has ? lowerModules[i] : 0;
      hits[2 * i] = has ? hitIndices[2 * i] : 0;
      hits[2 * i + 1] = has ? hitIndices[2 * i + 1] : 0;
    }
    tc.trackCandidateType[idx] = type;
    tc.directObjectIndices[idx] = directIdx;
    tc.pixelSeedIndex[idx] = pixelSeedIndex;
    tc.objectIndices[2 * idx] = innerIdx;
    tc.objectIndices[2 * idx + 1] = outerIdx;
#pragma unroll
    for (int i = 0; i < 7; i++) {
      tc.logicalLayers[7 * idx + i] = layers[i];
      tc.lowerModuleIndices[7 * idx + i] = modules[i];
    }
#pragma unroll
    for (int i = 0; i < 14; i++)
      tc.hitIndices[14 * idx + i] = hits[i];
    tc.centerX[idx] = centerX;
    tc.centerY[idx] = centerY;
    tc.radius[idx] = radius;
  }

  // pT5 -> TC (SDL/TrackCandidate.h:531-581); one block per event.
  __global__ void __launch_bounds__(1024) kAddPT5TC(DeviceES es, const EventView* evs) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    const unsigned int n = *ev.pt5.nPixelQuintuplets;
    const unsigned int pLS_offset = es.lsOffset[es.nLowerModules];
    const unsigned int start = *ev.tc.nTrackCandidates;
    TrackCandidates tc = ev.tc;
    PixelQuintuplets p = ev.pt5;
    unsigned int carry = 0;
    for (unsigned int base = 0; base < n; base += blockDim.x) {
      unsigned int i = base + threadIdx.x;
      bool f = i < n && !p.isDup[i];
      unsigned int tot;
      unsigned int ex = blockExclusiveScan(f ? 1u : 0u, tot);
      unsigned int idx = start + carry + ex;
      if (f && idx < kMaxPixelTrackCandidates) {
        float radius = 0.5f * (p.pixelRadius[i] + p.quintupletRadius[i]);
        unsigned int pix = p.pixelIndices[i];
        storeTC(tc, 7, pix, p.T5Indices[i], &p.logicalLayers[7 * i], &p.lowerModuleIndices[7 * i], &p.hitIndices[14 * i],
                static_cast<int>(ev.ls.seedIdx[pix - pLS_offset]), p.centerX[i], p.centerY[i], radius, idx, i);
      }
      carry += tot;
    }
    if (threadIdx.x == 0) {
      unsigned int accepted = (start + carry <= kMaxPixelTrackCandidates) ? carry
                              : (start < kMaxPixelTrackCandidates ? kMaxPixelTrackCandidates - start : 0u);
      if (accepted < carry)
        atomicOr(&ev.sc->status, kStatusTCTruncated);
      *tc.nTrackCandidates = start + accepted;
      *tc.nTrackCandidatespT5 += accepted;
    }
  }

  // ============================================================== pT3
  // Candidate modules of a pLS for pT3 (SDL/PixelTriplet.h:1046-1081).
  __device__ __forceinline__ unsigned int pt3ModuleCount(DeviceES const& es, const EventView& ev, uint16_t mod) {
    if (mod >= es.nLowerModules)
      return 0;
    if (es.m.moduleType[mod] == TwoS)
      return 0;
    int layer = es.m.layers[mod];
    if (layer != 1 && layer != 2)
      return 0;
    return ev.t3.nTriplets[mod];
  }

  template <bool kEmit>
  __device__ __forceinline__ void pt3Walk(DeviceES const& es, const EventView& ev, unsigned int iPLS, unsigned int* pre,
                                          uint16_t* mods) {
    if (ev.ls.isDup[iPLS] || ev.ls.partOfPT5[iPLS])
      return;
    unsigned int nConn, cidx;
    pixelSlice(es, ev, iPLS, nConn, cidx);
    for (unsigned int k = laneId(); k < nConn; k += 32)
      mods[k] = static_cast<uint16_t>(es.m.connectedPixels[cidx + k]);
    __syncwarp();
    const unsigned int total = warpPrefix(pre, int(nConn), [&](int k) { return pt3ModuleCount(es, ev, mods[k]); });
    const unsigned int plsIndex = es.lsOffset[es.nLowerModules] + iPLS;
    unsigned int count = 0;
    unsigned int rankBase = kEmit ? ev.plsOffset[iPLS] : 0u;
    Triplets t3 = ev.t3;
    PixelTriplets pt3 = ev.pt3;
    for (unsigned int start = 0; start < total; start += 32) {
      unsigned int f = start + laneId();
      bool ok = false;
      PT3Values v;
      unsigned int t3i = 0;
      short adj = 0;
      if (f < total) {
        int k = findSlot(pre, int(nConn), f);
        uint16_t mod = mods[k];
        adj = es.m.layers[mod] == 1 ? 1 : 0;
        t3i = ev.rg.tripletModuleIndices[mod] + (f - pre[k]);
        if (es.m.moduleType[t3.lowerModuleIndices[3 * t3i + 1]] != TwoS && !t3.partOfPT5[t3i])
          ok = pt3Select(es.m, ev.rg, ev.md, ev.ls, t3, plsIndex, t3i, true, v);
      }
      unsigned int tot;
      unsigned int r = rankBase + count + warpRank(ok, tot);
      if (kEmit && ok && r < kMaxPixelTriplets) {
        storePT3(es.m, ev.md, ev.ls, t3, pt3, plsIndex, iPLS, t3i, adj, v, r);
        t3.partOfPT3[t3i] = 1;
      }
      count += tot;
    }
    if (!kEmit && laneId() == 0)
      ev.plsCount[iPLS] = count;
  }

  // Register budget: this fallback does work only for events whose candidates
  // overflow the lists; for the others its blocks return at once, and the
  // budget lets more of them be resident, so the launch drains in fewer waves.
  __global__ void __launch_bounds__(128, 8) kPT3Count(DeviceES es, const EventView* evs) {
    kernelEntry();
    __shared__ unsigned int sPre[kPixWarps][kMaxConnectedModules + 1];
    __shared__ uint16_t sMods[kPixWarps][kMaxConnectedModules];
    const EventView& ev = evs[blockIdx.y];
    if (!ev.sc->pixFallback)
      return;
    const int wib = threadIdx.x >> 5;
    const unsigned int nPLS = ev.ls.nSegments[es.pixelModule];
    for (unsigned int i = blockIdx.x * kPixWarps + wib; i < nPLS; i += gridDim.x * kPixWarps) {
      __syncwarp();
      if (laneId() == 0)
        ev.plsCount[i] = 0;
      pt3Walk<false>(es, ev, i, sPre[wib], sMods[wib]);
    }
    plsScanByLast(es, ev, 1);
  }

  // Register budget: this fallback does work only for events whose candidates
  // overflow the lists; for the others its blocks return at once, and the
  // budget lets more of them be resident, so the launch drains in fewer waves.
  __global__ void __launch_bounds__(128, 8) kPT3Emit(DeviceES es, const EventView* evs) {
    kernelEntry();
    __shared__ unsigned int sPre[kPixWarps][kMaxConnectedModules + 1];
    __shared__ uint16_t sMods[kPixWarps][kMaxConnectedModules];
    const EventView& ev = evs[blockIdx.y];
    if (!ev.sc->pixFallback)
      return;
    const int wib = threadIdx.x >> 5;
    const unsigned int nPLS = ev.ls.nSegments[es.pixelModule];
    for (unsigned int i = blockIdx.x * kPixWarps + wib; i < nPLS; i += gridDim.x * kPixWarps) {
      __syncwarp();
      if (ev.plsCount[i] == 0 || ev.plsOffset[i] >= kMaxPixelTriplets)
        continue;
      pt3Walk<true>(es, ev, i, sPre[wib], sMods[wib]);
    }
  }

  // ------------------------------------- pT5 / pT3 as candidate lists
  // The candidates of a pLS are its (connected module, object) pairs in the
  // reference's loop order (SDL/PixelTriplet.h:1043-1158, :2697-2786).  A
  // candidate's key is its pLS (16 bits) and its number f within the pLS (16
  // bits), so that keys ascend in the order of the reference's loop nest, and
  // the global rank of a passing candidate is the number of passing candidates
  // with a smaller key.  kPixMid walks all candidates and queues those that
  // pass the opening tests, kPixEval runs the rest of the selection on them,
  // and kPixRankEmit ranks the passing ones and stores the first 15000 (pT5) /
  // 5000 (pT3).  Events that overflow the lists (or a pLS with more
  // than 2^16 candidates) take the per-pLS count/emit walk instead.
  constexpr unsigned int kPixPassCap = 8192;
  constexpr unsigned int kPixKeyCandidates = 1u << 16;  // candidates of one pLS that a key can number
  static_assert(kMaxPixelSegments <= (1u << 16), "a key holds a pLS in 16 bits");

  template <int K>
  __device__ __forceinline__ unsigned int pixModuleCount(DeviceES const& es, const EventView& ev, uint16_t mod) {
    return K == 5 ? pt5ModuleCount(es, ev, mod) : pt3ModuleCount(es, ev, mod);
  }

  template <int K>
  __device__ __forceinline__ bool pixSkipPLS(const EventView& ev, unsigned int i) {
    return K == 5 ? (ev.ls.isDup[i] != 0) : (ev.ls.isDup[i] || ev.ls.partOfPT5[i]);
  }

  // The opening tests of the pT5 / pT3 selection: the object's flags and the
  // pLS-triplet radius criterion, which most candidates fail, then the first
  // pixel tracklet algorithm (of the pLS with the triplet's, or the
  // quintuplet's inner triplet's, inner segment), a long test that few of the
  // others pass.  A warp takes a few consecutive pLS (their flags and pixel-map
  // slices fetched by its lanes together), deals their (pLS, connected module)
  // pairs to its lanes and keeps the pairs that have candidates in shared memory,
  // with their running count, so that a candidate finds its pLS and object there
  // and the lanes are filled across pLS.  Survivors of the flags and the radius
  // criterion wait in the warp's own queue in shared memory until there is a warp
  // full of them for the tracklet's opening windows; those of the windows (half)
  // wait likewise for the rest of it, and what passes that goes to the event's
  // queue in any order.
  // A candidate's outcome does not depend on which thread evaluates it, and the
  // passing ones are ranked by key afterwards.
  //
  // Bound by the latency of dependent gathers.  A list of candidates numbered
  // over the event (a prefix kernel, a scan, and per candidate a chunk table,
  // a walk over the pLS offsets and a binary search in the pLS's prefix: about
  // 16 dependent loads), with the radius survivors in a queue in memory between
  // two kernels, took 1.59 ms (pT3) and 0.56 ms (pT5) for 64 PU200 events, this
  // with kPixEval 1.40 and 0.45 ms.  PU250 and pt0.6 events also
  // overflowed that queue's 2^18 entries, and every candidate took the whole
  // selection (3.5 ms for the pT3s of 16 pt0.6 events, now 0.97); here only
  // candidates that pass the tracklet are queued, a thirtieth of them.  The
  // scratch is kept at 9 KB a block: with 18 KB too little of the L1 was left
  // (pT3 1.57 ms).
  constexpr int kPixMidWarps = 4;
  constexpr unsigned int kPixPairs = 128;  // (pLS, connected module) pairs of one group, at least a row of the pixel map
  static_assert(kPixPairs >= kMaxConnectedModules, "a pLS's connected modules fit a group");
  struct PixScratch {
    unsigned int pre[kPixPairs + 1];  // per pair with candidates: its first candidate within the group
    unsigned int obj[kPixPairs];      //   its first object
    uint8_t owner[kPixPairs];         //   and the lane of its pLS
    unsigned int first[32];           // per lane's pLS: its first candidate within the group
    // candidates waiting for the tracklet's windows [0] and its long part [1]
    unsigned int qKey[2][64], qObj[2][64];
  };
  template <int K>
  __global__ void __launch_bounds__(LST_LB_PIXMID) kPixMid(DeviceES es, const EventView* evs) {
    kernelEntry();
    __shared__ PixScratch sScratch[kPixMidWarps];
    const EventView& ev = evs[blockIdx.y];
    PixScratch& sc = sScratch[threadIdx.x >> 5];
    const unsigned int nPLS = ev.ls.nSegments[es.pixelModule];
    const unsigned int plsBase = es.lsOffset[es.nLowerModules];
    const unsigned int lane = laneId();
    const unsigned int nWarps = gridDim.x * (blockDim.x >> 5);
    const unsigned int perTask = min(32u, max(1u, nPLS / (2u * nWarps)));
    WarpTasks tasks(&ev.sc->pixNext);
    bool more = true;                  // the event may have tasks left
    unsigned int task = 0, left = 0;   // the current task's first pLS and the lanes of those not yet grouped
    unsigned int size = 0, index = 0;  // this lane's pLS of the task: its pixel-map slice
    unsigned int f0 = 0, total = 0;    // the current group's candidates from f0 on
    int nPairs = 0;                    //   and its pairs that have any
    unsigned int fill[2] = {0, 0};
    // the triplet (a quintuplet's inner one) that the opening tests take
    auto tripletOf = [&](unsigned int obj) { return K == 5 ? ev.t5.tripletIndices[2 * obj] : obj; };
    auto push = [&](int level, bool pass, unsigned int key, unsigned int obj) {
      const unsigned int ok = __ballot_sync(kFullMask, pass);
      if (pass) {
        const unsigned int k = fill[level] + __popc(ok & lanesBelowMask());
        sc.qKey[level][k] = key;
        sc.qObj[level][k] = obj;
      }
      fill[level] += __popc(ok);
      __syncwarp();
    };
    // up to 32 entries off the queue; false on the lanes without one
    auto pop = [&](int level, unsigned int& key, unsigned int& obj) {
      const unsigned int take = min(fill[level], 32u);
      fill[level] -= take;
      const bool have = lane < take;
      if (have) {
        key = sc.qKey[level][fill[level] + lane];
        obj = sc.qObj[level][fill[level] + lane];
      }
      __syncwarp();  // the entries have been read
      return have;
    };
    while (true) {
      while (fill[1] < 32u) {
        while (fill[0] < 32u) {
          if (f0 < total) {
            const unsigned int f = f0 + lane;
            f0 += 32u;
            bool pass = false;
            unsigned int obj = 0, key = 0;
            if (f < total) {
              const int k = findSlot(sc.pre, nPairs, f);
              const unsigned int iPLS = task + sc.owner[k], number = f - sc.first[sc.owner[k]];
              obj = sc.obj[k] + (f - sc.pre[k]);
              key = (iPLS << 16) | number;
              if (number >= kPixKeyCandidates)
                ev.sc->pixOverflow = 1;
              else if (K == 5)
                pass = !ev.t5.isDup[obj];
              else
                pass = es.m.moduleType[ev.t3.lowerModuleIndices[3 * obj + 1]] != TwoS && !ev.t3.partOfPT5[obj];
              if (pass)
                pass = pt3RadiusPass(es.m, ev.rg, ev.ls, ev.t3, plsBase + iPLS, tripletOf(obj));
            }
            push(0, pass, key, obj);
          } else if (left != 0) {
            // the next group: the pLS left, as long as their pairs fit
            const unsigned int mine = (left >> lane) & 1u ? size : 0u;
            const unsigned int incl = laneInclusiveSum(mine);
            const unsigned int fits = __ballot_sync(kFullMask, mine != 0 && incl <= kPixPairs);
            const unsigned int pairs = __shfl_sync(kFullMask, incl, 31 - __clz(fits));
            left &= ~fits;
            __syncwarp();  // the previous group's scratch has been read
            nPairs = 0;
            total = 0;
            for (unsigned int p0 = 0; p0 < pairs; p0 += 32) {
              const unsigned int p = p0 + lane;
              const int o = laneOwner(incl, p);
              const unsigned int k = p - (__shfl_sync(kFullMask, incl, o) - __shfl_sync(kFullMask, size, o));
              const unsigned int slice = __shfl_sync(kFullMask, index, o);
              unsigned int n = 0, obj = 0;
              if (p < pairs) {
                const uint16_t mod = static_cast<uint16_t>(es.m.connectedPixels[slice + k]);
                n = pixModuleCount<K>(es, ev, mod);
                if (n != 0)
                  obj = static_cast<unsigned int>(K == 5 ? ev.rg.quintupletModuleIndices[mod]
                                                         : ev.rg.tripletModuleIndices[mod]);
              }
              const unsigned int upTo = total + laneInclusiveSum(n);
              const unsigned int has = __ballot_sync(kFullMask, n != 0);
              if (p < pairs && k == 0)
                sc.first[o] = upTo - n;
              if (n != 0) {
                const int e = nPairs + __popc(has & lanesBelowMask());
                sc.pre[e] = upTo - n;
                sc.obj[e] = obj;
                sc.owner[e] = static_cast<uint8_t>(o);
              }
              nPairs += __popc(has);
              total = __shfl_sync(kFullMask, upTo, 31);
            }
            __syncwarp();
            f0 = 0;
          } else if (more) {
            task = tasks.take() * perTask;
            more = task < nPLS;
            const unsigned int i = task + lane;
            size = 0;
            if (lane < perTask && i < nPLS && !pixSkipPLS<K>(ev, i))
              pixelSlice(es, ev, i, size, index);
            left = __ballot_sync(kFullMask, size != 0);
          } else {
            break;
          }
        }
        if (fill[0] == 0)
          break;
        unsigned int key = 0, obj = 0;
        bool pass = pop(0, key, obj);
        if (pass)
          pass = pt3FirstWindows(es.m, ev.rg, ev.md, ev.ls, ev.t3, plsBase + (key >> 16), tripletOf(obj));
        push(1, pass, key, obj);
      }
      if (fill[1] == 0)
        break;
      unsigned int key = 0, obj = 0;
      bool pass = pop(1, key, obj);
      if (pass)
        pass = pt3FirstBeta(es.m, ev.rg, ev.md, ev.ls, ev.t3, plsBase + (key >> 16), tripletOf(obj),
                            ev.plsPhiP[key >> 16]);
      const unsigned int ok = __ballot_sync(kFullMask, pass);
      if (ok == 0u)
        continue;
      unsigned int start = 0;
      if (lane == 0)
        start = atomicAdd(&ev.sc->pixQueueCount, __popc(ok));
      start = __shfl_sync(kFullMask, start, 0);
      const unsigned int k = start + __popc(ok & lanesBelowMask());
      if (pass && k < kCandQueueCap) {
        ev.candQueue[k] = key;
        ev.candQueueObj[k] = obj;
      }
    }
  }

  // The rest of the selection for the queued candidates.
  // (blocks per SM 6 / 7 / 8 / 10: 64 PU200 events, pT5 + pT3, 241 / 209 / 217 / 238 us;
  // 8 events 78 / 82 / 84 / 102; 16 pt0.6 events 117 / 124 / 132 / 156)
  template <int K>
  __global__ void __launch_bounds__(LST_LB_EVAL) kPixEval(DeviceES es, const EventView* evs) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    if (K == 5)
      for (unsigned int i = blockIdx.x * blockDim.x + threadIdx.x; i < kPT5HitBuckets; i += gridDim.x * blockDim.x)
        ev.pt5HitHead[i] = kPT5HitNone;
    const unsigned int n = ev.sc->pixQueueCount;
    if (n > kCandQueueCap)
      return;  // the event takes the walk (kPixRankEmit)
    const unsigned int plsBase = es.lsOffset[es.nLowerModules];
    for (unsigned int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
      const unsigned int c = ev.candQueue[q], iPLS = c >> 16, obj = ev.candQueueObj[q];
      float vals[8];
      bool ok;
      if (K == 5) {
        PT5Values v;
        ok = pt5Select(es.m, ev.rg, ev.md, ev.ls, ev.t3, ev.t5, plsBase + iPLS, obj, iPLS, v, true);
        vals[0] = v.rzChiSquared;
        vals[1] = v.rPhiChiSquared;
        vals[2] = v.rPhiChiSquaredInwards;
        vals[3] = v.pixelRadius;
        vals[4] = v.quintupletRadius;
        vals[5] = v.centerX;
        vals[6] = v.centerY;
        vals[7] = 0.f;
      } else {
        PT3Values v;
        ok = pt3Select(es.m, ev.rg, ev.md, ev.ls, ev.t3, plsBase + iPLS, obj, true, v, true);
        vals[0] = v.pixelRadius;
        vals[1] = v.pixelRadiusError;
        vals[2] = v.tripletRadius;
        vals[3] = v.centerX;
        vals[4] = v.centerY;
        vals[5] = v.rzChiSquared;
        vals[6] = v.rPhiChiSquared;
        vals[7] = v.rPhiChiSquaredInwards;
      }
      if (ok) {
        const unsigned int slot = atomicAdd(&ev.sc->pixPassCount, 1u);
        if (slot < kPixPassCap) {
          ev.pixPassC[slot] = c;
          ev.pixPassObj[slot] = obj;
#pragma unroll
          for (int k = 0; k < 8; ++k)
            ev.pixPassV[8 * slot + k] = vals[k];
        }
      }
    }
  }

  // Ranks the passing candidates by key and stores them: a thread per candidate
  // counts the smaller keys, which every block of the event keeps in shared
  // memory.  Bound by the scattered stores of the pT5s / pT3s; for 13 PU250
  // events one block each took 113 us (pT5), up to 16 blocks 51.
  constexpr int kPixRankThreads = 128;
  template <int K>
  __global__ void __launch_bounds__(kPixRankThreads) kPixRankEmit(DeviceES es, const EventView* evs) {
    kernelEntry();
    __shared__ __align__(16) unsigned int sKey[kPixPassCap];
    const EventView& ev = evs[blockIdx.y];
    const unsigned int n = ev.sc->pixPassCount;
    const unsigned int capOut = K == 5 ? kMaxPixelQuintuplets : kMaxPixelTriplets;
    if (n > kPixPassCap || ev.sc->pixQueueCount > kCandQueueCap || ev.sc->pixOverflow || ev.forceWalk) {
      if (blockIdx.x == 0 && threadIdx.x == 0)
        ev.sc->pixFallback = 1;
      return;
    }
    if (blockIdx.x != 0 && blockIdx.x * blockDim.x >= n)
      return;
    const unsigned int n4 = (n + 3u) & ~3u;  // (four keys a read; the last ones never rank below)
    for (unsigned int j = threadIdx.x; j < n4; j += blockDim.x)
      sKey[j] = j < n ? ev.pixPassC[j] : 0xffffffffu;
    __syncthreads();
    const unsigned int plsBase = es.lsOffset[es.nLowerModules];
    Segments ls = ev.ls;
    Triplets t3 = ev.t3;
    Quintuplets t5 = ev.t5;
    for (unsigned int sIdx = blockIdx.x * blockDim.x + threadIdx.x; sIdx < n; sIdx += gridDim.x * blockDim.x) {
      const unsigned int key = sKey[sIdx];
      unsigned int rank = 0;
#pragma unroll 4
      for (unsigned int j = 0; j < n4; j += 4) {
        const uint4 k = *reinterpret_cast<const uint4*>(sKey + j);
        rank += (k.x < key ? 1u : 0u) + (k.y < key ? 1u : 0u) + (k.z < key ? 1u : 0u) + (k.w < key ? 1u : 0u);
      }
      if (rank >= capOut)
        continue;
      const unsigned int obj = ev.pixPassObj[sIdx];
      const unsigned int iPLS = key >> 16;
      const float* vals = ev.pixPassV + 8 * sIdx;
      if (K == 5) {
        PT5Values v;
        v.rzChiSquared = vals[0];
        v.rPhiChiSquared = vals[1];
        v.rPhiChiSquaredInwards = vals[2];
        v.pixelRadius = vals[3];
        v.quintupletRadius = vals[4];
        v.centerX = vals[5];
        v.centerY = vals[6];
        PixelQuintuplets pt5 = ev.pt5;
        storePT5(ev.md, ls, t3, t5, pt5, plsBase + iPLS, iPLS, obj, v, rank);
        // all exchanges in flight at once: reads first, next indices last
        unsigned int link[14];
#pragma unroll
        for (unsigned int k = 0; k < 14; ++k)
          link[k] = pt5.hitIndices[14 * rank + k];
#pragma unroll
        for (unsigned int k = 0; k < 14; ++k)
          link[k] = atomicExch(&ev.pt5HitHead[pt5HitBucket(link[k])], 14 * rank + k);
#pragma unroll
        for (unsigned int k = 0; k < 14; ++k)
          ev.pt5HitNext[14 * rank + k] = link[k];
      } else {
        PT3Values v;
        v.pixelRadius = vals[0];
        v.pixelRadiusError = vals[1];
        v.tripletRadius = vals[2];
        v.centerX = vals[3];
        v.centerY = vals[4];
        v.rzChiSquared = vals[5];
        v.rPhiChiSquared = vals[6];
        v.rPhiChiSquaredInwards = vals[7];
        PixelTriplets pt3 = ev.pt3;
        const short adj = es.m.layers[t3.lowerModuleIndices[3 * obj]] == 1 ? 1 : 0;
        storePT3(es.m, ev.md, ls, t3, pt3, plsBase + iPLS, iPLS, obj, adj, v, rank);
        t3.partOfPT3[obj] = 1;
      }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      ev.sc->pixFallback = 0;
      const unsigned int stored = n < capOut ? n : capOut;
      if (K == 5) {
        ev.sc->nPT5Total = n;
        *ev.pt5.totOccupancyPixelQuintuplets = n;
        *ev.pt5.nPixelQuintuplets = stored;
      } else {
        ev.sc->nPT3Total = n;
        *ev.pt3.totOccupancyPixelTriplets = n;
        *ev.pt3.nPixelTriplets = stored;
      }
      if (n > capOut)
        atomicOr(&ev.sc->status, kStatusCapOverflow);
    }
  }

  // Shared pixel and outer hits of two pT3s (SDL/Kernels.h:138-200).
  // SDL/Kernels.h:325-356.  pT3 ix is removed as soon as one jx meets the
  // condition (the reference's loop breaks there), so the outcome is the OR of
  // the condition over jx: one warp per ix, its lanes over jx.
  __global__ void kPT3Dedup(DeviceES es, const EventView* evs) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    if (blockIdx.x == 0 && threadIdx.x == 0)
      pixCountersClear(ev);  // the pixel lists have been read
    const unsigned int n = *ev.pt3.nPixelTriplets;
    PixelTriplets p = ev.pt3;
    const unsigned int wpb = blockDim.x >> 5;
    for (unsigned int ix = blockIdx.x * wpb + (threadIdx.x >> 5); ix < n; ix += gridDim.x * wpb) {
      unsigned int mine[10];
#pragma unroll
      for (int i = 0; i < 10; ++i)
        mine[i] = p.hitIndices[10 * ix + i];
      const uint8_t li = p.logicalLayers[5 * ix + 2];
      const float scoreI = p.score[ix];
      bool dup = false;
      for (unsigned int j0 = 0; j0 < n && !dup; j0 += 32) {
        const unsigned int jx = j0 + laneId();
        bool c = false;
        if (jx < n && jx != ix) {
          unsigned int other[10];
#pragma unroll
          for (int i = 0; i < 10; ++i)
            other[i] = p.hitIndices[10 * jx + i];
          int np = 0, nm = 0;
#pragma unroll
          for (int a = 0; a < 4; ++a) {
            bool m = false;
#pragma unroll
            for (int b = 0; b < 4; ++b)
              m |= mine[a] == other[b];
            np += m ? 1 : 0;
          }
#pragma unroll
          for (int a = 4; a < 10; ++a) {
            bool m = false;
#pragma unroll
            for (int b = 4; b < 10; ++b)
              m |= mine[a] == other[b];
            nm += m ? 1 : 0;
          }
          if (np + nm >= 5) {
            const uint8_t lj = p.logicalLayers[5 * jx + 2];
            const float scoreJ = p.score[jx];
            c = lj < li || (li == lj && scoreI > scoreJ) || (li == lj && scoreI == scoreJ && ix < jx);
          }
        }
        dup = __any_sync(kFullMask, c);
      }
      if (dup && laneId() == 0)
        p.isDup[ix] = 1;
    }
  }

  // ================================================== track candidates
  // pT3 vs pT5 pixel eta/phi (SDL/TrackCandidate.h:204-243).  One warp per
  // pT3, its lanes splitting the pT5 loop; the outcome is an "any" over it.
  __global__ void kCrossCleanPT3(DeviceES es, const EventView* evs) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    const unsigned int nPT3 = *ev.pt3.nPixelTriplets;
    const unsigned int nPT5 = *ev.pt5.nPixelQuintuplets;
    const unsigned int prefix = es.lsOffset[es.nLowerModules];
    const unsigned int nWarps = gridDim.x * (blockDim.x >> 5);
    for (unsigned int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < nPT3; i += nWarps) {
      if (ev.pt3.isDup[i])
        continue;
      const float eta1 = ev.pt3.eta_pix[i], phi1 = ev.pt3.phi_pix[i];
      bool dup = false;
      for (unsigned int j = laneId(); j < nPT5; j += 32) {
        unsigned int pLS_jx = ev.pt5.pixelIndices[j];
        float eta2 = ev.ls.eta[pLS_jx - prefix];
        float phi2 = ev.ls.phi[pLS_jx - prefix];
        float dEta = fabs_(eta1 - eta2);
        float dPhi = wrapDPhi(phi1, phi2);
        float dR2 = dEta * dEta + dPhi * dPhi;
        if (dR2 < 1e-5f)
          dup = true;
      }
      if (__any_sync(kFullMask, dup) && laneId() == 0)
        ev.pt3.isDup[i] = 1;
    }
  }

  // pT3 -> TC (SDL/TrackCandidate.h:383-433); one block per event.
  __global__ void __launch_bounds__(1024) kAddPT3TC(DeviceES es, const EventView* evs) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    const unsigned int n = *ev.pt3.nPixelTriplets;
    const unsigned int pLS_offset = es.lsOffset[es.nLowerModules];
    const unsigned int start = *ev.tc.nTrackCandidates;
    TrackCandidates tc = ev.tc;
    PixelTriplets p = ev.pt3;
    unsigned int carry = 0;
    for (unsigned int base = 0; base < n; base += blockDim.x) {
      unsigned int i = base + threadIdx.x;
      bool f = i < n && !p.isDup[i];
      unsigned int tot;
      unsigned int ex = blockExclusiveScan(f ? 1u : 0u, tot);
      unsigned int idx = start + carry + ex;
      if (f && idx < kMaxPixelTrackCandidates) {
        float radius = 0.5f * (p.pixelRadius[i] + p.tripletRadius[i]);
        unsigned int pix = p.pixelSegmentIndices[i];
        storeTC(tc, 5, i, i, &p.logicalLayers[5 * i], &p.lowerModuleIndices[5 * i], &p.hitIndices[10 * i],
                static_cast<int>(ev.ls.seedIdx[pix - pLS_offset]), p.centerX[i], p.centerY[i], radius, idx, i);
      }
      carry += tot;
    }
    if (threadIdx.x == 0) {
      unsigned int accepted = (start + carry <= kMaxPixelTrackCandidates) ? carry
                              : (start < kMaxPixelTrackCandidates ? kMaxPixelTrackCandidates - start : 0u);
      if (accepted < carry)
        atomicOr(&ev.sc->status, kStatusTCTruncated);
      *tc.nTrackCandidates = start + accepted;
      *tc.nTrackCandidatespT3 += accepted;
    }
  }

  // Cross-module T5 duplicate removal before TC building
  // (SDL/Kernels.h:251-323), which marks t5Flag.  The reference visits
  // the ordered pairs (ix in module A, jx in module B) with A's position in
  // the eligible-module list not after B's and ix != jx; a pair whose
  // |deta| > 0.1 is skipped at the first test, and marks are only ever set.
  // kT5Bin counting-sorts the event's quintuplets into the pLS-cleaning eta bins
  // (one block per event), and kT5DedupBinned gives each quintuplet a warp that
  // visits the same ordered pairs among the bins within reach (and the non-finite
  // bin, which meets every quintuplet, as does a quintuplet of non-finite eta).
  // Events with more quintuplets than kT5SortCap keep the module-pair walk.
  __global__ void __launch_bounds__(1024) kT5Bin(DeviceES es, const EventView* evs) {
    kernelEntry();
    __shared__ unsigned int sCount[kPLSBins + 1];
    const EventView& ev = evs[blockIdx.y];
    const unsigned int nE = *ev.rg.nEligibleT5Modules;
    const unsigned int total = ev.sc->t5ListCount;
    const Quintuplets& q = ev.t5;
    // (the counts that kCrossCleanT5 adds to, and the marks of the cleaning)
    for (unsigned int e = threadIdx.x; e < nE; e += blockDim.x)
      ev.moduleCount[e] = 0;
    if (total > kT5SortCap || ev.forceWalk) {
      for (unsigned int e = threadIdx.x; e < nE; e += blockDim.x) {
        const uint16_t lm = ev.rg.indicesOfEligibleT5Modules[e];
        const unsigned int n = q.nQuintuplets[lm], base = ev.rg.quintupletModuleIndices[lm];
        for (unsigned int j = 0; j < n; ++j)
          ev.t5Flag[base + j] = 0;
      }
      return;
    }
    for (int b = threadIdx.x; b <= kPLSBins; b += blockDim.x)
      sCount[b] = 0;
    __syncthreads();
    for (unsigned int k = threadIdx.x; k < total; k += blockDim.x) {
      const unsigned int ix = ev.t5List[k].x;
      ev.t5Flag[ix] = 0;
      atomicAdd(&sCount[plsEtaBin(q.eta[ix])], 1u);
    }
    __syncthreads();
    const unsigned int c = threadIdx.x <= kPLSBins ? sCount[threadIdx.x] : 0u;
    unsigned int tot;
    const unsigned int ex = blockExclusiveScan(c, tot);
    if (threadIdx.x <= kPLSBins) {
      sCount[threadIdx.x] = ex;
      ev.t5BinStart[threadIdx.x] = ex;
    }
    if (threadIdx.x == 0)
      ev.t5BinStart[kPLSBins + 1] = tot;
    __syncthreads();
    for (unsigned int k = threadIdx.x; k < total; k += blockDim.x) {
      const uint2 t = ev.t5List[k];
      const unsigned int pos = atomicAdd(&sCount[plsEtaBin(q.eta[t.x])], 1u);
      ev.t5Order[pos] = t.x;
      ev.t5OrderPos[pos] = static_cast<uint16_t>(t.y);
    }
  }

  // The reference's test of one ordered pair (ix, jx), marking the loser.
  LST_DEV void t5CrossPair(const EventView& ev, unsigned int ix, unsigned int jx, float eta1, float phi1,
                           float score1) {
    const Quintuplets& q = ev.t5;
    if (q.partOfPT5[jx] || (q.isDup[jx] & 1))
      return;
    float eta2 = q.eta[jx], phi2 = q.phi[jx], score2 = q.score_rphisum[jx];
    float dEta = fabs_(eta1 - eta2);
    float dPhi = wrapDPhi(phi1, phi2);
    if (dEta > 0.1f)
      return;
    if (fabs_(dPhi) > 0.1f)
      return;
    float dR2 = dEta * dEta + dPhi * dPhi;
    int nMatched = sharedHitsT5(q, ix, jx);
    if (dR2 < 0.001f || nMatched >= 5) {
      if (score1 > score2)
        ev.t5Flag[ix] = 1;
      else if (score1 < score2)
        ev.t5Flag[jx] = 1;
      else
        ev.t5Flag[ix < jx ? ix : jx] = 1;
    }
  }

  // A warp per quintuplet, its lanes over the partners within reach (one thread
  // per quintuplet walked some 65 partners one after the other: 97 us for one
  // PU200 event, now 25).  Events with more quintuplets than the list holds
  // visit the module pairs, a warp per module.
  __global__ void kT5DedupBinned(DeviceES es, const EventView* evs) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    const unsigned int n = ev.sc->t5ListCount;
    const Quintuplets& q = ev.t5;
    if (n > kT5SortCap || ev.forceWalk) {
      const int nE = *ev.rg.nEligibleT5Modules;
      const int nWarps = static_cast<int>((gridDim.x * blockDim.x) >> 5);
      for (int warp = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5); warp < nE; warp += nWarps) {
        uint16_t lowmod1 = ev.rg.indicesOfEligibleT5Modules[warp];
        unsigned int n1 = q.nQuintuplets[lowmod1];
        unsigned int base1 = ev.rg.quintupletModuleIndices[lowmod1];
        for (unsigned int ix1 = laneId(); ix1 < n1; ix1 += 32) {
          unsigned int ix = base1 + ix1;
          if (q.partOfPT5[ix] || (q.isDup[ix] & 1))
            continue;
          float eta1 = q.eta[ix], phi1 = q.phi[ix], score1 = q.score_rphisum[ix];
          for (int idx2 = warp; idx2 < nE; idx2++) {
            uint16_t lowmod2 = ev.rg.indicesOfEligibleT5Modules[idx2];
            unsigned int n2 = q.nQuintuplets[lowmod2];
            unsigned int base2 = ev.rg.quintupletModuleIndices[lowmod2];
            for (unsigned int jx1 = 0; jx1 < n2; jx1++) {
              unsigned int jx = base2 + jx1;
              if (ix != jx)
                t5CrossPair(ev, ix, jx, eta1, phi1, score1);
            }
          }
        }
      }
      return;
    }
    const unsigned int* binStart = ev.t5BinStart;
    const unsigned int nFinite = binStart[kPLSBins];
    const unsigned int wpb = blockDim.x >> 5;
    for (unsigned int k = blockIdx.x * wpb + (threadIdx.x >> 5); k < n; k += gridDim.x * wpb) {
      const unsigned int ix = ev.t5Order[k];
      if (q.partOfPT5[ix] || (q.isDup[ix] & 1))
        continue;
      const unsigned int posI = ev.t5OrderPos[k];
      const float eta1 = q.eta[ix], phi1 = q.phi[ix], score1 = q.score_rphisum[ix];
      const int b = plsEtaBin(eta1);
      unsigned int lo = 0, hi = n, lo2 = n;  // positions [lo, hi) then [lo2, n)
      if (b < kPLSBins) {
        lo = binStart[b >= kPLSBinReach ? b - kPLSBinReach : 0];
        hi = binStart[(b + kPLSBinReach < kPLSBins ? b + kPLSBinReach : kPLSBins - 1) + 1];
        lo2 = nFinite;
      }
      for (int part = 0; part < 2; ++part) {
        const unsigned int p0 = part == 0 ? lo : lo2, p1 = part == 0 ? hi : n;
        for (unsigned int p = p0 + laneId(); p < p1; p += 32) {
          const unsigned int jx = ev.t5Order[p];
          const unsigned int posJ = ev.t5OrderPos[p];
          if (jx == ix || posJ < posI)
            continue;
          t5CrossPair(ev, ix, jx, eta1, phi1, score1);
        }
      }
    }
  }

  // T5 vs pT5/pT3 eta/phi (SDL/TrackCandidate.h:245-300), after folding the mark
  // of the cross-module cleaning into isDup; and the count, per eligible module,
  // of the T5s that become track candidates (SDL/TrackCandidate.h:435-487).  A
  // warp per T5, its lanes over the pT5s and pT3s (the outcome is an "any").
  __device__ __forceinline__ void t5CrossClean(const EventView& ev, unsigned int q, unsigned int module) {
    const Quintuplets& t5 = ev.t5;
    const unsigned int nPT5 = *ev.pt5.nPixelQuintuplets;
    const unsigned int loop_bound = nPT5 + *ev.pt3.nPixelTriplets;
    const float eta1 = t5.eta[q], phi1 = t5.phi[q];
    const bool marked = ev.t5Flag[q] != 0;
    const bool kept = t5.isDup[q] == 0 && !marked && !t5.partOfPT5[q];
    bool dup = false;
    if (kept)
      for (unsigned int jx = laneId(); jx < loop_bound; jx += 32) {
        const float eta2 = jx < nPT5 ? ev.pt5.eta[jx] : ev.pt3.eta[jx - nPT5];
        const float phi2 = jx < nPT5 ? ev.pt5.phi[jx] : ev.pt3.phi[jx - nPT5];
        float dEta = fabs_(eta1 - eta2);
        float dPhi = wrapDPhi(phi1, phi2);
        float dR2 = dEta * dEta + dPhi * dPhi;
        if (dR2 < 1e-3f)
          dup = true;
      }
    dup = __any_sync(kFullMask, dup);
    if (laneId() == 0) {
      if (marked)
        t5.isDup[q] |= 2;
      else if (dup)
        t5.isDup[q] = 1;
      else if (kept && t5.TightCutFlag[q])
        atomicAdd(&ev.moduleCount[module], 1u);
    }
  }
  __global__ void kCrossCleanT5(DeviceES es, const EventView* evs) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    const unsigned int wpb = blockDim.x >> 5;
    const unsigned int warp = blockIdx.x * wpb + (threadIdx.x >> 5), nWarps = gridDim.x * wpb;
    const unsigned int n = ev.sc->t5ListCount;
    if (n <= kT5SortCap && !ev.forceWalk) {
      for (unsigned int k = warp; k < n; k += nWarps) {
        const uint2 t = ev.t5List[k];
        t5CrossClean(ev, t.x, t.y);
      }
      return;
    }
    const unsigned int nE = *ev.rg.nEligibleT5Modules;
    for (unsigned int e = warp; e < nE; e += nWarps) {
      const uint16_t lm = ev.rg.indicesOfEligibleT5Modules[e];
      const unsigned int nT5 = ev.t5.nQuintuplets[lm], base = ev.rg.quintupletModuleIndices[lm];
      for (unsigned int j = 0; j < nT5; ++j)
        t5CrossClean(ev, base + j, e);
    }
  }

  // T5 -> TC (SDL/TrackCandidate.h:435-487): scan of the modules' counts, then
  // emit in (module, T5) order.
  __global__ void __launch_bounds__(1024) kT5TCScan(DeviceES es, const EventView* evs) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    const unsigned int n = *ev.rg.nEligibleT5Modules;
    unsigned int carry = 0;
    for (unsigned int base = 0; base < n; base += blockDim.x) {
      unsigned int i = base + threadIdx.x;
      unsigned int c = (i < n) ? ev.moduleCount[i] : 0u;
      unsigned int tot;
      unsigned int ex = blockExclusiveScan(c, tot);
      if (i < n)
        ev.moduleOffset[i] = carry + ex;
      carry += tot;
    }
    if (threadIdx.x == 0) {
      // (the store's end bounds a stage that is run again on the same event, which
      // appends to its candidates)
      const unsigned int begin = *ev.tc.nTrackCandidates;
      const unsigned int room = begin < kMaxTrackCandidates ? kMaxTrackCandidates - begin : 0u;
      const unsigned int accepted = min(carry, min(kMaxNonPixelTrackCandidates, room));
      if (accepted < carry)
        atomicOr(&ev.sc->status, kStatusTCTruncated);
      ev.sc->t5TCStart = begin;
      *ev.tc.nTrackCandidates += accepted;
      *ev.tc.nTrackCandidatesT5 += accepted;
    }
  }

  __global__ void kT5TCEmit(DeviceES es, const EventView* evs) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nE = *ev.rg.nEligibleT5Modules;
    if (warp >= nE)
      return;
    const unsigned int start = ev.sc->t5TCStart;
    uint16_t lm = ev.rg.indicesOfEligibleT5Modules[warp];
    unsigned int n = ev.t5.nQuintuplets[lm];
    unsigned int base = ev.rg.quintupletModuleIndices[lm];
    unsigned int rank = ev.moduleOffset[warp];
    TrackCandidates tc = ev.tc;
    const Quintuplets& q = ev.t5;
    for (unsigned int s0 = 0; s0 < n; s0 += 32) {
      unsigned int j = s0 + laneId();
      bool f = false;
      unsigned int qi = base + j;
      if (j < n)
        f = !(q.isDup[qi] or q.partOfPT5[qi]) && q.TightCutFlag[qi];
      unsigned int tot;
      unsigned int r = rank + warpRank(f, tot);
      if (f && r < kMaxNonPixelTrackCandidates && start + r < kMaxTrackCandidates)
        storeTC(tc, 4, qi, qi, &q.logicalLayers[5 * qi], &q.lowerModuleIndices[5 * qi], &q.hitIndices[10 * qi], -1,
                q.regressionG[qi], q.regressionF[qi], q.regressionRadius[qi], start + r, qi);
      rank += tot;
    }
  }

  // Per-TC record for the pLS cross-cleaning (SDL/TrackCandidate.h:302-381):
  // the candidate's type, the (eta, phi) a pLS is compared with, and the
  // four pixel hits of its pLS (pT3, pT5).
  struct TCCleanInfo {
    float eta, phi;
    int type;
    int hits[4];
  };

  LST_DEV void pixelHitsOf(const Segments& s, const MiniDoublets& md, const Hits& h, unsigned int plsIndex, int* out) {
    out[0] = static_cast<int>(h.idxs[md.anchorHitIndices[s.mdIndices[2 * plsIndex]]]);
    out[1] = static_cast<int>(h.idxs[md.anchorHitIndices[s.mdIndices[2 * plsIndex + 1]]]);
    out[2] = static_cast<int>(h.idxs[md.outerHitIndices[s.mdIndices[2 * plsIndex]]]);
    out[3] = static_cast<int>(h.idxs[md.outerHitIndices[s.mdIndices[2 * plsIndex + 1]]]);
  }

  // Shared pixel hits of two pLS (SDL/TrackCandidate.h:165-202), -1 entries skipped.
  LST_DEV int sharedPixelHits(const int* phits1, const int* phits2) {
    int npMatched = 0;
    for (int i = 0; i < 4; i++) {
      bool pmatched = false;
      if (phits1[i] == -1)
        continue;
      for (int j = 0; j < 4; j++) {
        if (phits2[j] == -1)
          continue;
        if (phits1[i] == phits2[j]) {
          pmatched = true;
          break;
        }
      }
      if (pmatched)
        npMatched++;
    }
    return npMatched;
  }

  __global__ void kTCCleanInfo(DeviceES es, const EventView* evs) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    const unsigned int nTC = *ev.tc.nTrackCandidates;
    const unsigned int prefix = es.lsOffset[es.nLowerModules];
    for (unsigned int t = blockIdx.x * blockDim.x + threadIdx.x; t < nTC; t += gridDim.x * blockDim.x) {
      TCCleanInfo info;
      info.type = ev.tc.trackCandidateType[t];
      const unsigned int innerIdx = ev.tc.objectIndices[2 * t];
      info.eta = 0.f;
      info.phi = 0.f;
      info.hits[0] = info.hits[1] = info.hits[2] = info.hits[3] = -1;
      if (info.type == 4) {
        info.eta = ev.t5.eta[innerIdx];
        info.phi = ev.t5.phi[innerIdx];
      } else if (info.type == 5) {
        info.eta = ev.pt3.eta_pix[innerIdx];
        info.phi = ev.pt3.phi_pix[innerIdx];
        pixelHitsOf(ev.ls, ev.md, ev.hits, ev.pt3.pixelSegmentIndices[innerIdx], info.hits);
      } else if (info.type == 7) {
        info.eta = ev.ls.eta[innerIdx - prefix];
        info.phi = ev.ls.phi[innerIdx - prefix];
        pixelHitsOf(ev.ls, ev.md, ev.hits, innerIdx, info.hits);
      }
      ev.tcCleanInfo[t] = info;
    }
  }

  // pLS vs existing TCs (SDL/TrackCandidate.h:302-381).  A quadruplet pLS
  // that is not yet a duplicate becomes one if some TC of type 5 or 7 shares a
  // pixel hit with it, if some T5 TC (type 4) lies within dR^2 < 1e-3, or if
  // some type 5 / 7 TC lies within dR^2 < 1e-6; the outcome is an OR over the
  // TCs, so it is evaluated per pLS without walking every TC:
  //  - the pixel hits of all type 5 / 7 TCs go into a shared-memory hash set,
  //    and a pLS shares a hit with one of them iff one of its hits is in it;
  //  - the TCs are counting-sorted by eta into the pLS-cleaning bins (width
  //    0.02), and only bins within kXCleanReach of the pLS's bin are read:
  //    dR^2 < 1e-3 needs |deta| < 0.0317 (two bin widths plus rounding), and a
  //    non-finite eta or dR^2 never passes the test.
  // A set with more TCs than kXCleanMaxTC, or more hits than the hash holds,
  // is checked pair by pair instead.
  constexpr unsigned int kXCleanHashSlots = 1u << 14;
  constexpr unsigned int kXCleanMaxTC = 4096;
  constexpr int kXCleanReach = 3;
  constexpr int kXCleanBlocksPerEvent = 4;
  constexpr size_t kXCleanSmem =
      kXCleanHashSlots * 4 + 2 * (kPLSBins + 2) * 4 + kXCleanMaxTC * (sizeof(float) * 2 + sizeof(int));

  LST_DEV unsigned int xcleanSlot(unsigned int key) { return (key * 2654435761u) >> 18; }

  LST_DEV bool xcleanPairDup(const TCCleanInfo& info, const int* phits1, float eta1, float phi1) {
    if (info.type == 4) {
      float dEta = fabs_(eta1 - info.eta);
      float dPhi = wrapDPhi(phi1, info.phi);
      return dEta * dEta + dPhi * dPhi < 1e-3f;
    }
    if (info.type == 5 || info.type == 7) {
      if (sharedPixelHits(phits1, info.hits) > 0)
        return true;
      float dEta = fabs_(eta1 - info.eta);
      float dPhi = wrapDPhi(phi1, info.phi);
      return dEta * dEta + dPhi * dPhi < 0.000001f;
    }
    return false;
  }

  __global__ void __launch_bounds__(1024) kCrossCleanPLS(DeviceES es, const EventView* evs) {
    kernelEntry();
    extern __shared__ __align__(16) unsigned char xsm[];
    unsigned int* sHash = reinterpret_cast<unsigned int*>(xsm);
    unsigned int* sBinStart = sHash + kXCleanHashSlots;
    unsigned int* sCursor = sBinStart + kPLSBins + 2;
    float* sEta = reinterpret_cast<float*>(sCursor + kPLSBins + 2);
    float* sPhi = sEta + kXCleanMaxTC;
    int* sType = reinterpret_cast<int*>(sPhi + kXCleanMaxTC);
    __shared__ unsigned int sOverflow;
    const EventView& ev = evs[blockIdx.y];
    const unsigned int nPix = ev.ls.nSegments[es.pixelModule];
    const unsigned int prefix = es.lsOffset[es.nLowerModules];
    const unsigned int nTC = *ev.tc.nTrackCandidates;
    const TCCleanInfo* infos = ev.tcCleanInfo;
    Segments s = ev.ls;

    if (threadIdx.x == 0)
      sOverflow = (nTC > kXCleanMaxTC || ev.forceWalk) ? 1u : 0u;
    for (unsigned int t = threadIdx.x; t < kXCleanHashSlots; t += blockDim.x)
      sHash[t] = 0;
    for (unsigned int t = threadIdx.x; t < kPLSBins + 2; t += blockDim.x)
      sCursor[t] = 0;
    __syncthreads();
    const bool fits = nTC <= kXCleanMaxTC;
    if (fits) {
      for (unsigned int t = threadIdx.x; t < nTC; t += blockDim.x) {
        const TCCleanInfo info = infos[t];
        if (info.type == 5 || info.type == 7) {
          for (int a = 0; a < 4; ++a) {
            if (info.hits[a] == -1)
              continue;
            const unsigned int key = static_cast<unsigned int>(info.hits[a]) + 1u;
            unsigned int slot = xcleanSlot(key), probes = 0;
            while (true) {
              const unsigned int old = atomicCAS(&sHash[slot], 0u, key);
              if (old == 0u || old == key)
                break;
              if (++probes == kXCleanHashSlots) {
                sOverflow = 1;
                break;
              }
              slot = (slot + 1) & (kXCleanHashSlots - 1);
            }
          }
        }
        if (info.type == 4 || info.type == 5 || info.type == 7)
          atomicAdd(&sCursor[plsEtaBin(info.eta)], 1u);
      }
    }
    __syncthreads();
    const bool fast = sOverflow == 0;
    if (fast) {
      unsigned int tot;
      const unsigned int c = threadIdx.x <= kPLSBins ? sCursor[threadIdx.x] : 0u;
      const unsigned int ex = blockExclusiveScan(c, tot);
      if (threadIdx.x <= kPLSBins) {
        sBinStart[threadIdx.x] = ex;
        sCursor[threadIdx.x] = ex;
      }
      if (threadIdx.x == 0)
        sBinStart[kPLSBins + 1] = tot;
      __syncthreads();
      for (unsigned int t = threadIdx.x; t < nTC; t += blockDim.x) {
        const TCCleanInfo& info = infos[t];
        if (info.type == 4 || info.type == 5 || info.type == 7) {
          const unsigned int pos = atomicAdd(&sCursor[plsEtaBin(info.eta)], 1u);
          sEta[pos] = info.eta;
          sPhi[pos] = info.phi;
          sType[pos] = info.type;
        }
      }
      __syncthreads();
    }

    for (unsigned int i = blockIdx.x * blockDim.x + threadIdx.x; i < nPix; i += gridDim.x * blockDim.x) {
      // the mark of the second cleaning pass (SDL/Kernels.h:384-473), set between
      // quads without a pass-1 mark only
      if (i < kMaxPixelSegments && ev.plsFlag[i]) {
        s.isDup[i] |= 2;
        ev.plsFlag[i] = 0;
        continue;
      }
      if (!s.isQuad[i] || s.isDup[i])
        continue;
      int phits1[4];
      pixelHitsOf(s, ev.md, ev.hits, prefix + i, phits1);
      const float eta1 = s.eta[i], phi1 = s.phi[i];
      bool dup = false;
      if (fast) {
        for (int a = 0; a < 4 && !dup; ++a) {
          if (phits1[a] == -1)
            continue;
          const unsigned int key = static_cast<unsigned int>(phits1[a]) + 1u;
          unsigned int slot = xcleanSlot(key);
          for (unsigned int probes = 0; probes < kXCleanHashSlots; ++probes) {
            const unsigned int h = sHash[slot];
            if (h == key) {
              dup = true;
              break;
            }
            if (h == 0u)
              break;
            slot = (slot + 1) & (kXCleanHashSlots - 1);
          }
        }
        const int b = plsEtaBin(eta1);
        if (!dup && b < kPLSBins) {
          const int b0 = b >= kXCleanReach ? b - kXCleanReach : 0;
          const int b1 = b + kXCleanReach < kPLSBins ? b + kXCleanReach : kPLSBins - 1;
          for (unsigned int k = sBinStart[b0]; k < sBinStart[b1 + 1] && !dup; ++k) {
            float dEta = fabs_(eta1 - sEta[k]);
            float dPhi = wrapDPhi(phi1, sPhi[k]);
            const float dR2 = dEta * dEta + dPhi * dPhi;
            dup = sType[k] == 4 ? dR2 < 1e-3f : dR2 < 0.000001f;
          }
        }
      } else {
        for (unsigned int t = 0; t < nTC && !dup; ++t)
          dup = xcleanPairDup(infos[t], phits1, eta1, phi1);
      }
      if (dup)
        s.isDup[i] = 1;
    }
  }

  // pLS -> TC (SDL/TrackCandidate.h:489-529): the quads without a duplicate mark,
  // in order.  Each block takes chunks of 256 pLS, counts the candidates before
  // its chunk itself (their flags are two bytes a pLS), lists its own in shared
  // memory and writes their rows, which lie side by side, as whole lines.  The
  // last block to finish sets the counts, which all blocks have read by then.
  // Bound by the row stores; one block per event with a store per word took 78 us
  // for one PU200 event, now under 19 (64 events: 93, now 56).
  constexpr int kAddPLSThreads = 256;
  __global__ void __launch_bounds__(kAddPLSThreads) kAddPLSTC(DeviceES es, const EventView* evs) {
    kernelEntry();
    __shared__ unsigned int sList[kAddPLSThreads];
    const EventView& ev = evs[blockIdx.y];
    const unsigned int n = ev.ls.nSegments[es.pixelModule];
    const unsigned int start = *ev.tc.nTrackCandidates;
    const unsigned int nT5TC = *ev.tc.nTrackCandidatesT5;
    const unsigned int nChunks = (n + kAddPLSThreads - 1) / kAddPLSThreads;
    TrackCandidates tc = ev.tc;
    const Segments& s = ev.ls;
    // candidates with idx - nT5TC < kMaxPixelTrackCandidates are stored: `room` of them
    // (and none past the store's end)
    const unsigned int room =
        (start - nT5TC < kMaxPixelTrackCandidates && start < kMaxTrackCandidates)
            ? min(kMaxPixelTrackCandidates - (start - nT5TC), kMaxTrackCandidates - start)
            : 0u;
    auto chosen = [&](unsigned int i) { return i < n && s.isQuad[i] && !s.isDup[i]; };
    unsigned int before = 0, counted = 0;  // candidates in the pLS [0, counted)
    for (unsigned int c = blockIdx.x; c < nChunks; c += gridDim.x) {
      const unsigned int base = c * kAddPLSThreads;
      // four pLS a word (the flag arrays start 256-byte aligned, the chunks are
      // multiples of 256)
      unsigned int mine = 0;
      const unsigned int* quads = reinterpret_cast<const unsigned int*>(s.isQuad);
      const unsigned int* dups = reinterpret_cast<const unsigned int*>(s.isDup);
#pragma unroll 4
      for (unsigned int w = counted / 4 + threadIdx.x; w < base / 4; w += kAddPLSThreads)
        mine += __popc(__vcmpne4(quads[w], 0u) & __vcmpeq4(dups[w], 0u) & 0x01010101u);
      unsigned int add;
      blockExclusiveScan(mine, add);
      before += add;
      const unsigned int i = base + threadIdx.x;
      const bool f = chosen(i);
      unsigned int tot;
      const unsigned int ex = blockExclusiveScan(f ? 1u : 0u, tot);
      if (f)
        sList[ex] = i;
      __syncthreads();
      const unsigned int rows = before < room ? min(tot, room - before) : 0u;
      const unsigned int idx0 = start + before;
      for (unsigned int r = threadIdx.x; r < rows; r += kAddPLSThreads) {
        const unsigned int pls = sList[r];
        const int seed = static_cast<int>(s.seedIdx[pls]);
        tc.trackCandidateType[idx0 + r] = 8;
        tc.directObjectIndices[idx0 + r] = pls;
        tc.pixelSeedIndex[idx0 + r] = seed;
        tc.objectIndices[2 * (idx0 + r)] = pls;
        tc.objectIndices[2 * (idx0 + r) + 1] = pls;
        tc.centerX[idx0 + r] = 0;
        tc.centerY[idx0 + r] = 0;
        tc.radius[idx0 + r] = 0;
      }
      for (unsigned int w = threadIdx.x; w < 14 * rows; w += kAddPLSThreads) {
        const unsigned int r = w / 14, k = w % 14;
        // hits 0, 2, 1, 3 of the pLS, then zeros
        tc.hitIndices[14 * idx0 + w] =
            k < 4 ? s.pLSHitsIdxs[4 * sList[r] + (k == 1 ? 2u : k == 2 ? 1u : k)] : 0u;
      }
      for (unsigned int w = threadIdx.x; w < 7 * rows; w += kAddPLSThreads) {
        tc.logicalLayers[7 * idx0 + w] = 0;
        tc.lowerModuleIndices[7 * idx0 + w] = 0;
      }
      before += tot;
      counted = base + kAddPLSThreads;
      __syncthreads();  // sList is rewritten for the next chunk
    }
    // (the block with the last chunk knows the event's total)
    if (threadIdx.x != 0)
      return;
    if (nChunks == 0 ? blockIdx.x == 0 : (nChunks - 1) % gridDim.x == blockIdx.x)
      ev.sc->plsTCTotal = before;
    __threadfence();
    if (atomicAdd(&ev.sc->plsTCDone, 1u) + 1u != gridDim.x)
      return;
    __threadfence();
    ev.sc->plsTCDone = 0;
    const unsigned int total = *static_cast<volatile unsigned int*>(&ev.sc->plsTCTotal);
    const unsigned int accepted = total < room ? total : room;
    if (accepted < total)
      atomicOr(&ev.sc->status, kStatusTCTruncated);
    *tc.nTrackCandidates = start + accepted;
    *tc.nTrackCandidatespLS += accepted;
  }


  // ============================================================== counts
  // Object counts of one event, as the reference's getNumberOf* members
  // (SDL/Event.cc:1148-1487): per-layer sums over lower modules with the
  // same inclusion rules as add*ToEventExplicit.  One block per event.
  __global__ void kCounts(DeviceES es, const EventView* evs) {
    kernelEntry();
    __shared__ unsigned int sBins[4][11];
    const EventView& ev = evs[blockIdx.y];
    for (int i = threadIdx.x; i < 44; i += blockDim.x)
      (&sBins[0][0])[i] = 0;
    __syncthreads();
    const Modules& m = es.m;
    for (unsigned int i = threadIdx.x; i < es.nLowerModules; i += blockDim.x) {
      int bin = (m.subdets[i] == Barrel) ? (m.layers[i] - 1) : (6 + m.layers[i] - 1);
      if (bin < 0 || bin >= 11)
        continue;
      unsigned int nmd = ev.md.nMDs[i];
      if (!(nmd == 0 or ev.hits.hitRanges[i * 2] == -1))
        atomicAdd(&sBins[0][bin], nmd);
      unsigned int nls = ev.ls.nSegments[i];
      if (nls != 0)
        atomicAdd(&sBins[1][bin], nls);
      unsigned int nt3 = ev.t3.nTriplets[i];
      if (nt3 != 0)
        atomicAdd(&sBins[2][bin], nt3);
      unsigned int nt5 = ev.t5.nQuintuplets[i];
      if (!(nt5 == 0 or ev.rg.quintupletModuleIndices[i] == -1))
        atomicAdd(&sBins[3][bin], nt5);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      lst_counts* c = ev.counts;
      c->nHits = ev.sc->nHits;
      c->nPixelSegments = ev.ls.nSegments[es.pixelModule];
      c->status = ev.sc->status;
      unsigned int tot[4] = {0, 0, 0, 0};
      for (int k = 0; k < 4; ++k)
        for (int b = 0; b < 11; ++b)
          tot[k] += sBins[k][b];
      for (int b = 0; b < 6; ++b) {
        c->mdBarrel[b] = sBins[0][b];
        c->lsBarrel[b] = sBins[1][b];
        c->t3Barrel[b] = sBins[2][b];
        c->t5Barrel[b] = sBins[3][b];
      }
      for (int b = 0; b < 5; ++b) {
        c->mdEndcap[b] = sBins[0][6 + b];
        c->lsEndcap[b] = sBins[1][6 + b];
        c->t3Endcap[b] = sBins[2][6 + b];
        c->t5Endcap[b] = sBins[3][6 + b];
      }
      c->nMiniDoublets = tot[0];
      c->nSegments = tot[1];
      c->nTriplets = tot[2];
      c->nQuintuplets = tot[3];
      c->nPixelTriplets = *ev.pt3.nPixelTriplets;
      c->nPixelQuintuplets = *ev.pt5.nPixelQuintuplets;
      c->nTrackCandidates = *ev.tc.nTrackCandidates;
      c->nTrackCandidatesPT5 = *ev.tc.nTrackCandidatespT5;
      c->nTrackCandidatesPT3 = *ev.tc.nTrackCandidatespT3;
      c->nTrackCandidatesPLS = *ev.tc.nTrackCandidatespLS;
      c->nTrackCandidatesT5 = *ev.tc.nTrackCandidatesT5;
      c->nPixelTripletsFound = ev.sc->nPT3Total;
      c->nPixelQuintupletsFound = ev.sc->nPT5Total;
      for (int k = 0; k < 4; ++k)
        c->reserved[k] = 0;
    }
  }

  // ============================================================ inputs
  // Sets the hit and pLS counts of one event (per-event input path).
  __global__ void kSetInputCounts(const EventView* evs, int slot, int setHits, unsigned int nHits, int setPLS,
                                  unsigned int nPLS, unsigned int statusBits) {
    kernelEntry();
    const EventView& ev = evs[slot];
    if (setHits)
      ev.sc->nHits = nHits;
    if (setPLS)
      ev.sc->nPLS = nPLS;
    ev.sc->status |= statusBits;
  }

  // Byte layout of one packed input event (see lst_packed_size).
  struct PackedLayout {
    size_t x, y, z, detId, idx, h0, h1, h2, h3, dPhiChange, ptIn, ptErr, px, py, pz, eta, etaErr, phi, charge,
        seedIdx, superbin, pixelType, isQuad, end;
  };
  LST_HD PackedLayout packedLayout(unsigned int nHits, unsigned int nPLS) {
    PackedLayout L;
    size_t o = 16;
    size_t h4 = 4 * size_t(nHits), p4 = 4 * size_t(nPLS);
    L.x = o; o += h4;
    L.y = o; o += h4;
    L.z = o; o += h4;
    L.detId = o; o += h4;
    L.idx = o; o += h4;
    L.h0 = o; o += p4;
    L.h1 = o; o += p4;
    L.h2 = o; o += p4;
    L.h3 = o; o += p4;
    L.dPhiChange = o; o += p4;
    L.ptIn = o; o += p4;
    L.ptErr = o; o += p4;
    L.px = o; o += p4;
    L.py = o; o += p4;
    L.pz = o; o += p4;
    L.eta = o; o += p4;
    L.etaErr = o; o += p4;
    L.phi = o; o += p4;
    L.charge = o; o += p4;
    L.seedIdx = o; o += p4;
    L.superbin = o; o += p4;
    L.pixelType = o; o += nPLS;
    L.isQuad = o; o += nPLS;
    L.end = (o + 15) & ~size_t(15);
    return L;
  }

  // Unpacks the packed inputs of a batch into the event stores: the hits
  // (addHitToEvent's copies) and the pixel-segment fields
  // (addPixelSegmentToEvent's copies).  blockIdx.y = event within the batch.
  __global__ void kUnpack(const EventView* evs, const unsigned char* blobs, const unsigned long long* offsets,
                          unsigned long long totalBytes) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    const unsigned char* b = blobs + offsets[blockIdx.y];
    const unsigned int* hdr = reinterpret_cast<const unsigned int*>(b);
    unsigned int nHits = hdr[0], nPLSIn = hdr[1];
    unsigned int status = 0;
    // A blob whose arrays would end beyond the uploaded bytes is dropped.
    const bool truncated = offsets[blockIdx.y] + packedLayout(nHits, nPLSIn).end > totalBytes;
    if (truncated) {
      status |= kStatusInvalidInput;
      nHits = 0;
      nPLSIn = 0;
    }
    bool reject = nHits > ev.maxHits;
    unsigned int nPLS = nPLSIn;
    if (reject) {
      status |= kStatusHitCapacity;
      nHits = 0;
      nPLS = 0;
    }
    if (nPLS > kMaxPixelSegments) {
      status |= kStatusPLSTruncated;
      nPLS = kMaxPixelSegments;
    }
    if (nHits == 0 && nPLS > 0) {
      status |= kStatusInvalidInput;
      nPLS = 0;
    }
    const PackedLayout L = packedLayout(reject ? 0u : nHits, reject ? 0u : nPLSIn);
    const unsigned int stride = gridDim.x * blockDim.x;
    const unsigned int t0 = blockIdx.x * blockDim.x + threadIdx.x;
    // Two hits per thread and step: ten loads in flight before the stores.
    for (unsigned int i = t0; i < nHits; i += 2 * stride) {
      const unsigned int j = i + stride;
      const bool two = j < nHits;
      const float x0 = reinterpret_cast<const float*>(b + L.x)[i];
      const float y0 = reinterpret_cast<const float*>(b + L.y)[i];
      const float z0 = reinterpret_cast<const float*>(b + L.z)[i];
      const unsigned int d0 = reinterpret_cast<const unsigned int*>(b + L.detId)[i];
      const unsigned int n0 = reinterpret_cast<const unsigned int*>(b + L.idx)[i];
      float x1 = 0.f, y1 = 0.f, z1 = 0.f;
      unsigned int d1 = 0, n1 = 0;
      if (two) {
        x1 = reinterpret_cast<const float*>(b + L.x)[j];
        y1 = reinterpret_cast<const float*>(b + L.y)[j];
        z1 = reinterpret_cast<const float*>(b + L.z)[j];
        d1 = reinterpret_cast<const unsigned int*>(b + L.detId)[j];
        n1 = reinterpret_cast<const unsigned int*>(b + L.idx)[j];
      }
      ev.hits.xs[i] = x0;
      ev.hits.ys[i] = y0;
      ev.hits.zs[i] = z0;
      ev.hits.detid[i] = d0;
      ev.hits.idxs[i] = n0;
      if (two) {
        ev.hits.xs[j] = x1;
        ev.hits.ys[j] = y1;
        ev.hits.zs[j] = z1;
        ev.hits.detid[j] = d1;
        ev.hits.idxs[j] = n1;
      }
    }
    for (unsigned int i = t0; i < nPLS; i += stride) {
      ev.plsHit0[i] = reinterpret_cast<const unsigned int*>(b + L.h0)[i];
      ev.plsHit1[i] = reinterpret_cast<const unsigned int*>(b + L.h1)[i];
      ev.plsHit2[i] = reinterpret_cast<const unsigned int*>(b + L.h2)[i];
      ev.plsHit3[i] = reinterpret_cast<const unsigned int*>(b + L.h3)[i];
      ev.plsDPhiChange[i] = reinterpret_cast<const float*>(b + L.dPhiChange)[i];
      ev.ls.ptIn[i] = reinterpret_cast<const float*>(b + L.ptIn)[i];
      ev.ls.ptErr[i] = reinterpret_cast<const float*>(b + L.ptErr)[i];
      ev.ls.px[i] = reinterpret_cast<const float*>(b + L.px)[i];
      ev.ls.py[i] = reinterpret_cast<const float*>(b + L.py)[i];
      ev.ls.pz[i] = reinterpret_cast<const float*>(b + L.pz)[i];
      ev.ls.eta[i] = reinterpret_cast<const float*>(b + L.eta)[i];
      ev.ls.etaErr[i] = reinterpret_cast<const float*>(b + L.etaErr)[i];
      ev.ls.phi[i] = reinterpret_cast<const float*>(b + L.phi)[i];
      ev.ls.charge[i] = reinterpret_cast<const int*>(b + L.charge)[i];
      ev.ls.seedIdx[i] = reinterpret_cast<const unsigned int*>(b + L.seedIdx)[i];
      ev.ls.superbin[i] = reinterpret_cast<const int*>(b + L.superbin)[i];
      ev.ls.pixelType[i] = reinterpret_cast<const int8_t*>(b + L.pixelType)[i];
      ev.ls.isQuad[i] = reinterpret_cast<const int8_t*>(b + L.isQuad)[i];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      ev.sc->nHits = nHits;
      ev.sc->nPLS = nPLS;
      ev.sc->status |= status;
    }
  }


  // ============================================================ output
  // Track-candidate output in the form of LST::getOutput
  // (SDL/LST.cc:367-427): per candidate its type, pixel seed index and the
  // list of input-ntuple hit indices (14 / 10 / 10 / 4 slots for pT5 / pT3 /
  // T5 / pLS, a repeated 4th hit of pixel objects dropped).
  __device__ __forceinline__ int tcOutputHits(const EventView& ev, unsigned int idx, unsigned int* out) {
    const short type = ev.tc.trackCandidateType[idx];
    const int maxN = type == 7 ? 14 : (type == 5 ? 10 : (type == 4 ? 10 : (type == 8 ? 4 : 0)));
    int n = 0;
    unsigned int last = 0;
    for (int i = 0; i < maxN; ++i) {
      unsigned int g = ev.tc.hitIndices[14 * idx + i];
      unsigned int h = (type == 8) ? g : ev.hits.idxs[g];
      if (type != 4 && n == 3 && last == h)
        continue;
      if (out)
        out[n] = h;
      ++n;
      last = h;
    }
    return n;
  }

  // Per event: output length of every candidate and their offsets; one block
  // per event.
  __global__ void __launch_bounds__(1024) kOutputSizes(const EventView* evs) {
    kernelEntry();
    const EventView& ev = evs[blockIdx.y];
    const unsigned int n = *ev.tc.nTrackCandidates;
    unsigned int carry = 0;
    for (unsigned int base = 0; base < n; base += blockDim.x) {
      unsigned int i = base + threadIdx.x;
      unsigned int len = (i < n) ? static_cast<unsigned int>(tcOutputHits(ev, i, nullptr)) : 0u;
      unsigned int tot;
      unsigned int ex = blockExclusiveScan(len, tot);
      if (i < n) {
        ev.tcOutLen[i] = len;
        ev.tcOutOffset[i] = carry + ex;
      }
      carry += tot;
    }
    if (threadIdx.x == 0)
      ev.sc->nOutHits = carry;
  }

  // Offsets of each event's candidates and hits inside the batch output
  // (exclusive scans over the events); one block.
  __global__ void __launch_bounds__(1024) kOutputEventOffsets(const EventView* evs, int count,
                                                              unsigned long long* offsets) {
    kernelEntry();
    unsigned long long carryTC = 0, carryHits = 0;
    for (int base = 0; base < count; base += blockDim.x) {
      int i = base + threadIdx.x;
      unsigned int ntc = (i < count) ? *evs[i].tc.nTrackCandidates : 0u;
      unsigned int nh = (i < count) ? evs[i].sc->nOutHits : 0u;
      unsigned int totTC, totH;
      unsigned int exTC = blockExclusiveScan(ntc, totTC);
      unsigned int exH = blockExclusiveScan(nh, totH);
      if (i < count) {
        offsets[i] = carryTC + exTC;
        offsets[count + 1 + i] = carryHits + exH;
      }
      carryTC += totTC;
      carryHits += totH;
    }
    if (threadIdx.x == 0) {
      offsets[count] = carryTC;
      offsets[2 * count + 1] = carryHits;
    }
  }

  // The batch output: hits, len, seedIdx and type, each 256-byte aligned.
  struct OutputLayout {
    size_t len, seed, type, end;
  };
  LST_HD OutputLayout outputLayout(size_t nHits, size_t nTC) {
    auto up = [](size_t n) { return (n + 255) & ~size_t(255); };
    OutputLayout l;
    l.len = up(4 * nHits);
    l.seed = up(l.len + 4 * nTC);
    l.type = up(l.seed + 4 * nTC);
    l.end = l.type + 2 * nTC;
    return l;
  }

  // Writes the batch output, if it fits in `room` bytes.
  __global__ void kOutputGather(const EventView* evs, int count, const unsigned long long* offsets,
                                unsigned char* out, size_t room) {
    kernelEntry();
    const OutputLayout l = outputLayout(offsets[2 * count + 1], offsets[count]);
    if (l.end > room)
      return;
    unsigned int* outHits = reinterpret_cast<unsigned int*>(out);
    unsigned int* outLen = reinterpret_cast<unsigned int*>(out + l.len);
    int* outSeed = reinterpret_cast<int*>(out + l.seed);
    short* outType = reinterpret_cast<short*>(out + l.type);
    const EventView& ev = evs[blockIdx.y];
    const unsigned int n = *ev.tc.nTrackCandidates;
    const unsigned long long tc0 = offsets[blockIdx.y];
    const unsigned long long h0 = offsets[count + 1 + blockIdx.y];
    for (unsigned int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
      tcOutputHits(ev, i, outHits + h0 + ev.tcOutOffset[i]);
      outLen[tc0 + i] = ev.tcOutLen[i];
      outSeed[tc0 + i] = ev.tc.pixelSeedIndex[i];
      outType[tc0 + i] = ev.tc.trackCandidateType[i];
    }
  }

  // The events' offsets, and the batch output if it fits in `room` bytes, to
  // pinned host memory, 16 bytes a thread.
  __global__ void kOutputToHost(int count, const unsigned long long* offsets, const unsigned char* out, size_t room,
                                unsigned long long* hostOffsets, unsigned char* host) {
    kernelEntry();
    const unsigned int t = blockIdx.x * blockDim.x + threadIdx.x, nThreads = gridDim.x * blockDim.x;
    for (unsigned int i = t; i < 2u * (count + 1u); i += nThreads)
      hostOffsets[i] = offsets[i];
    const OutputLayout l = outputLayout(offsets[2 * count + 1], offsets[count]);
    if (l.end > room)
      return;
    // (room is a multiple of 16, and so both buffers hold the last part)
    for (size_t i = t; 16 * i < l.end; i += nThreads)
      reinterpret_cast<uint4*>(host)[i] = reinterpret_cast<const uint4*>(out)[i];
  }

}  // namespace lst

#include "lst_seed.h"

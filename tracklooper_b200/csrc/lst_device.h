// Device-side views of the event setup and of one event's object stores.
#pragma once

#include "lst_b200.h"
#include "lst_pixel.h"

namespace lst {

  struct TCCleanInfo;
  struct PLSRec;

  // Event setup resident on the device (read-only during an event).
  struct DeviceES {
    Modules m;
    const unsigned int* cpIndex;
    const unsigned int* cpSizes;
    const unsigned int* cpIndexPos;
    const unsigned int* cpSizesPos;
    const unsigned int* cpIndexNeg;
    const unsigned int* cpSizesNeg;
    unsigned int pixelIndexOffsetPos;
    unsigned int pixelIndexOffsetNeg;
    const int* mdOffset;
    const int* mdCap;
    const int* lsOffset;
    const int* lsCap;
    const int* t3CapIfUsed;
    const int* t5CapIfEligible;
    unsigned int nTotalMDs;
    unsigned int nTotalSegments;
    unsigned int maxTriplets;
    unsigned int maxQuintuplets;
    const MDCut* mdCuts;  // per module: what the mini-doublet and segment cuts take from it
    const LSCut* lsCuts;
    const unsigned int* detHashKey;
    const uint16_t* detHashVal;
    unsigned int detHashBits;
    uint16_t nModules;
    uint16_t nLowerModules;
    uint16_t pixelModule;
  };

  // Status bits reported per event.
  enum StatusBits : unsigned int {
    kStatusUnknownDetId = 1u << 0,       // a hit's detId is not in the geometry
    kStatusUnknownEndcapDetId = 1u << 1,  // a 2S endcap hit without strip orientation
    kStatusHitCapacity = 1u << 2,        // more hits than the event store holds
    kStatusPLSTruncated = 1u << 3,       // more than 50000 pLS: the rest were dropped (as the reference does)
    kStatusTCTruncated = 1u << 4,        // a track-candidate cap was reached
    kStatusCapOverflow = 1u << 5,        // an occupancy cap dropped objects (as the reference does)
    kStatusInvalidInput = 1u << 6,       // a pLS hit index beyond the event's hits (replaced by hit 0)
  };

  // Per-event scalars in device memory.
  struct EventScalars {
    unsigned int nHits;
    unsigned int nPLS;
    unsigned int status;
    unsigned int nPT5Total;
    unsigned int nPT3Total;
    unsigned int nOutHits;  // output hit-list length of the event's track candidates
    unsigned int t5CandTotal;     // quintuplet candidates of the event (probe)
    unsigned int t5Overflow;      // a quintuplet candidate's key does not fit: walk instead
    unsigned int t5Tasks;         // tasks of kT5Eval's warps
    unsigned int t5InnerPerTask;  //   inner triplets of a task, at most 32
    unsigned int t5Next;          //   and the next one
    unsigned int t5StagedCount;   // quintuplet candidates that pass the tracklet tests
    unsigned int t5PassCount;     // passing quintuplet candidates
    unsigned int pixPassCount;    // passing candidates found by kPixEval
    unsigned int pixOverflow;     // a pLS has more candidates than a key can number
    unsigned int pixFallback;     // the pixel stage overflowed the staging: walk instead
    unsigned int pixQueueCount;   // pixel candidates passing the radius criterion and the first tracklet
    unsigned int t5ListCount;     // stored quintuplets (listed in t5List)
    unsigned int t5TCStart;       // first track candidate that is a quintuplet
    unsigned int plsTCTotal;      // pLS that become track candidates, before the cap
    unsigned int walkDone;        // blocks of a fallback count kernel that have finished
    unsigned int plsTCDone;       // blocks of kAddPLSTC that have finished
    unsigned int mdNext;          // next task for kCreateMD's warps
    unsigned int lsNext;          // next task for kCreateLS's warps
    unsigned int pixNext; // next task (a few pLS) for kPixMid's warps
    unsigned int t3Next;          // next task for kCreateT3's blocks
  };

  // All device pointers of one event.
  struct EventView {
    Hits hits;
    Ranges rg;
    MiniDoublets md;
    Segments ls;
    Triplets t3;
    Quintuplets t5;
    PixelTriplets pt3;
    PixelQuintuplets pt5;
    TrackCandidates tc;
    EventScalars* sc;
    lst_counts* counts;
    // pLS inputs that are not stored in the segment store
    unsigned int* plsHit0;
    unsigned int* plsHit1;
    unsigned int* plsHit2;
    unsigned int* plsHit3;
    float* plsDPhiChange;
    float* plsPhiP;  // phi of the pLS momentum (px, py), for the pixel tracklets
    // scratch
    unsigned int* plsCount;
    unsigned int* plsOffset;
    unsigned int* moduleCount;
    unsigned int* moduleOffset;
    uint8_t* t5Flag;   // removal marks of the cross-module T5 cleaning
    uint8_t* plsFlag;  // removal marks of the second pLS cleaning pass
    unsigned int* tcOutLen;     // output hits per track candidate
    unsigned int* tcOutOffset;  // offset of a candidate's hits in the event's output
    // MD-keyed indices: per module, segments / triplets grouped by their first
    // MD (module-relative indices), with per-MD start and count
    uint16_t* lsByMD;
    uint16_t* mdLSStart;
    uint16_t* mdLSCount;
    uint16_t* t3ByMD;
    uint16_t* mdT3Start;
    uint16_t* mdT3Count;
    unsigned int* t5CandPre;    // per inner triplet: its first candidate within the module
    unsigned int* t5ModCand;    // per eligible module: candidates
    unsigned int* t5ModOff;     // per eligible module: first candidate of the event
    unsigned int* t5Task;       // tasks of kT5Eval's warps: module position and first inner triplet
    struct T5Staged* t5Staged;  // quintuplet candidates that pass the tracklet tests
    T5Values* t5PassValues;     // selection values of passing candidates
    unsigned int* t5PassC;      //   their key
    uint2* t5PassT3;            //   and their triplets
    unsigned int* pixPassC;     // passing candidates: key
    unsigned int* pixPassObj;   //   the T5 / T3 index
    float* pixPassV;            //   the selection values (8 per candidate)
    float* hitMiniSlope;        // per hit: the slope term of the mini-doublet dphi threshold
    float* hitShiftXa;          // per hit moved by the strip shift: its moved point and z
    float* hitShiftYa;
    float* hitShiftZn;
    uint2* t5List;              // stored quintuplets: index and module position, any order
    unsigned int* t5Order;      // quintuplets sorted by eta bin (their index)
    uint16_t* t5OrderPos;       //   and their module's position in the eligible-module list
    unsigned int* t5BinStart;   // start of each eta bin in t5Order (bins + 2 entries)
    unsigned int* candQueue;    // keys of the pT5 / pT3 candidates that pass the opening tests, any order
    unsigned int* candQueueObj; //   and their object
    struct TCCleanInfo* tcCleanInfo;  // per track candidate: the pLS cross-cleaning record
    struct PLSRec* plsRec;      // pass-2 pLS records sorted by eta bin
    uint2* seedChunk;           // per chunk of seeds: kept seeds and their pseudo-hits
    unsigned int* plsHitHead;   // hit -> pLS index of the pLS cleaning: chain head per bucket
    unsigned int* plsHitNext;   //   and the next entry (4 pLS + hit slot) per entry
    unsigned int* pt5HitHead;   // hit -> (pT5, slot) chains of the pT5 duplicate removal
    unsigned int* pt5HitNext;
    unsigned int* plsBinStart;  // start of each eta bin in plsRec (bins + 2 entries)
    unsigned int maxHits;
    unsigned int forceWalk;  // take the fallback paths (walks, pair-by-pair tests) for testing them
  };

}  // namespace lst

// Line-segment (LS) selection: a pair of mini-doublets on module-map-connected
// modules; plus the pixel line segments (pLS) built from pixel seeds.  Cut
// arithmetic follows SDL/Segment.h:264-796 and SDL/Segment.h:392-453,1031-1117.
#pragma once

#include "lst_md.h"

namespace lst {

  // What the segment cuts take from a module, formed once per module when the
  // event setup is loaded (kModuleCuts) instead of for every pair: a dozen
  // module look-ups and some ten divisions and square roots per pair less
  // (kCreateLS, 64 PU200 events: 1.74 -> 1.36 ms; kCreateMD with MDCut 1.19 ->
  // 1.16).
  struct alignas(16) LSCut {
    float sdMuls;        // multiple-scattering term
    float tilt;          // r-z tilt term of a tilted barrel module
    float res;           // 0.02 / sensor separation
    unsigned int flags;  // MDCutFlags
  };

  LST_HD LSCut lsCut(const Modules& m, uint16_t mi) {
    const bool barrel = m.subdets[mi] == Barrel;
    LSCut c;
    c.sdMuls = barrel ? miniMulsPtScaleBarrel(m.layers[mi] - 1) * 3.f / m.ptCut
                      : miniMulsPtScaleEndcap(m.layers[mi] - 1) * 3.f / m.ptCut;
    const bool tilted = barrel and m.sides[mi] != Center;
    const float drdz = m.drdzs[mi];
    const float gap = moduleGap(m, mi);
    c.tilt = tilted ? (0.5f * kPixelPSZpitch * drdz / fsqrt(1.f + drdz * drdz) / gap) : 0;
    c.res = 0.02f / gap;
    c.flags = cutFlags(m, mi);
    return c;
  }

  // Thresholds of the three alpha (direction) differences
  // (SDL/Segment.h:264-356).
  LST_HD void lsDAlphaThresholds(const LSCut& in, const LSCut& out, float ptCut, const MDRec& rIn, const MDRec& rOut,
                                 float* thr) {
    const float xIn = rIn.x, yIn = rIn.y, xOut = rOut.x, yOut = rOut.y;
    const bool innerBarrel = (in.flags & kCutBarrel) != 0;
    const bool outerBarrel = (out.flags & kCutBarrel) != 0;
    const float sdMuls = in.sdMuls;
    float segmentDr = fsqrt((yOut - yIn) * (yOut - yIn) + (xOut - xIn) * (xOut - xIn));
    const float dAlpha_Bfield = fasin(fmin_(segmentDr * k2Rinv1GeVf / ptCut, kSinAlphaMax));
    float sdLumForInnerMini, sdLumForOuterMini;
    if (innerBarrel)
      sdLumForInnerMini = in.tilt * dAlpha_Bfield;
    else
      sdLumForInnerMini = rIn.lum;
    if (outerBarrel)
      sdLumForOuterMini = out.tilt * dAlpha_Bfield;
    else
      sdLumForOuterMini = rOut.lum;

    // (both resolutions are taken with the inner module's separation)
    float dAlpha_res_inner = in.res * (innerBarrel ? 1.0f : fabs_(rIn.z) / rIn.rt);
    float dAlpha_res_outer = in.res * (outerBarrel ? 1.0f : fabs_(rOut.z) / rOut.rt);
    float dAlpha_res = dAlpha_res_inner + dAlpha_res_outer;

    if (in.flags & kCutCenter)
      thr[0] = dAlpha_Bfield + fsqrt(dAlpha_res * dAlpha_res + sdMuls * sdMuls);
    else
      thr[0] = dAlpha_Bfield +
               fsqrt(dAlpha_res * dAlpha_res + sdMuls * sdMuls + sdLumForInnerMini * sdLumForInnerMini);
    if (out.flags & kCutCenter)
      thr[1] = dAlpha_Bfield + fsqrt(dAlpha_res * dAlpha_res + sdMuls * sdMuls);
    else
      thr[1] = dAlpha_Bfield +
               fsqrt(dAlpha_res * dAlpha_res + sdMuls * sdMuls + sdLumForOuterMini * sdLumForOuterMini);
    thr[2] = dAlpha_Bfield + fsqrt(dAlpha_res * dAlpha_res + sdMuls * sdMuls);
  }

  struct LSValues {
    float dPhi, dPhiMin, dPhiMax, dPhiChange, dPhiChangeMin, dPhiChangeMax;
  };

  // Barrel-barrel segment (SDL/Segment.h:455-565).  dPhiMin/Max and
  // dPhiChangeMin/Max keep their initial value 0.
  LST_HD_BIG bool lsBarrel(const LSCut& in,
                       const LSCut& out,
                       float ptCut,
                       const MDRec& rIn,
                       const MDRec& rOut,
                       LSValues& v) {
    const float sdMuls = in.sdMuls;
    float xIn = rIn.x, yIn = rIn.y, zIn = rIn.z, rtIn = rIn.rt;
    float xOut = rOut.x, yOut = rOut.y, zOut = rOut.z, rtOut = rOut.rt;

    float sdSlope = rOut.slope;
    float sdPVoff = rOut.pvOff;
    float dzDrtScale = rOut.dzDrtScale;
    const float zGeom = (in.flags & kCutInnerLayers) ? 2.f * kPixelPSZpitch : 2.f * kStrip2SZpitch;
    float zLo = zIn + (zIn - kDeltaZLum) * (rtOut / rtIn - 1.f) * (zIn > 0.f ? 1.f : dzDrtScale) - zGeom;
    float zHi = zIn + (zIn + kDeltaZLum) * (rtOut / rtIn - 1.f) * (zIn < 0.f ? 1.f : dzDrtScale) + zGeom;
    if (!((zOut >= zLo) && (zOut <= zHi)))
      return false;

    float sdCut = sdSlope + fsqrt(sdMuls * sdMuls + sdPVoff * sdPVoff);
    v.dPhi = phiMpiPi(rOut.phi - rIn.phi);
    if (!(fabs_(v.dPhi) <= sdCut))
      return false;
    v.dPhiChange = phiMpiPi(phiOf(xOut - xIn, yOut - yIn) - rIn.phi);
    if (!(fabs_(v.dPhiChange) <= sdCut))
      return false;

    float thr[3];
    lsDAlphaThresholds(in, out, ptCut, rIn, rOut, thr);
    float innerMDAlpha = rIn.dphichange;
    float outerMDAlpha = rOut.dphichange;
    float dAlphaInnerMDSegment = innerMDAlpha - v.dPhiChange;
    float dAlphaOuterMDSegment = outerMDAlpha - v.dPhiChange;
    float dAlphaInnerMDOuterMD = innerMDAlpha - outerMDAlpha;
    if (!(fabs_(dAlphaInnerMDSegment) < thr[0]))
      return false;
    if (!(fabs_(dAlphaOuterMDSegment) < thr[1]))
      return false;
    return fabs_(dAlphaInnerMDOuterMD) < thr[2];
  }

  // Segment with at least one endcap module (SDL/Segment.h:567-705).
  LST_HD_BIG bool lsEndcap(const LSCut& in,
                       const LSCut& out,
                       float ptCut,
                       const MDRec& rIn,
                       const MDRec& rOut,
                       LSValues& v) {
    float zIn = rIn.z, rtIn = rIn.rt;
    float zOut = rOut.z, rtOut = rOut.rt;
    bool outerLayerEndcapTwoS = (out.flags & kCutEndcapTwoS) != 0;
    float sdSlope = rOut.slope;
    float disks2SMinRadius = 60.f;
    float rtGeom = ((rtIn < disks2SMinRadius && rtOut < disks2SMinRadius)
                        ? (2.f * kPixelPSZpitch)
                        : ((rtIn < disks2SMinRadius || rtOut < disks2SMinRadius) ? (kPixelPSZpitch + kStrip2SZpitch)
                                                                                 : (2.f * kStrip2SZpitch)));
    if (!(zIn * zOut >= 0))
      return false;
    float dz = zOut - zIn;
    float dLum = signTransfer(kDeltaZLum, zIn);
    float drtDzScale = rOut.drtDzScale;
    float rtLo = fmax_(rtIn * (1.f + dz / (zIn + dLum) * drtDzScale) - rtGeom, rtIn - 0.5f * rtGeom);
    float rtHi = rtIn * (zOut - dLum) / (zIn - dLum) + rtGeom;
    if (!((rtOut >= rtLo) && (rtOut <= rtHi)))
      return false;

    v.dPhi = phiMpiPi(rOut.phi - rIn.phi);
    float sdCut = sdSlope;
    if (outerLayerEndcapTwoS) {
      float dPhiPos_high = phiMpiPi(rOut.highEdgePhi - rIn.phi);
      float dPhiPos_low = phiMpiPi(rOut.lowEdgePhi - rIn.phi);
      v.dPhiMax = fabs_(dPhiPos_high) > fabs_(dPhiPos_low) ? dPhiPos_high : dPhiPos_low;
      v.dPhiMin = fabs_(dPhiPos_high) > fabs_(dPhiPos_low) ? dPhiPos_low : dPhiPos_high;
    } else {
      v.dPhiMax = v.dPhi;
      v.dPhiMin = v.dPhi;
    }
    if (!(fabs_(v.dPhi) <= sdCut))
      return false;

    float dzFrac = dz / zIn;
    v.dPhiChange = v.dPhi / dzFrac * (1.f + dzFrac);
    v.dPhiChangeMin = v.dPhiMin / dzFrac * (1.f + dzFrac);
    v.dPhiChangeMax = v.dPhiMax / dzFrac * (1.f + dzFrac);
    if (!(fabs_(v.dPhiChange) <= sdCut))
      return false;

    float thr[3];
    lsDAlphaThresholds(in, out, ptCut, rIn, rOut, thr);
    float innerMDAlpha = rIn.dphichange;
    float outerMDAlpha = rOut.dphichange;
    float dAlphaInnerMDSegment = innerMDAlpha - v.dPhiChange;
    float dAlphaOuterMDSegment = outerMDAlpha - v.dPhiChange;
    float dAlphaInnerMDOuterMD = innerMDAlpha - outerMDAlpha;
    if (!(fabs_(dAlphaInnerMDSegment) < thr[0]))
      return false;
    if (!(fabs_(dAlphaOuterMDSegment) < thr[1]))
      return false;
    return fabs_(dAlphaInnerMDOuterMD) < thr[2];
  }

  LST_HD bool lsSelect(const LSCut& in, const LSCut& out, float ptCut, const MDRec& rIn, const MDRec& rOut,
                       LSValues& v) {
    v.dPhiMin = 0;
    v.dPhiMax = 0;
    v.dPhiChangeMin = 0;
    v.dPhiChangeMax = 0;
    if ((in.flags & kCutBarrel) and (out.flags & kCutBarrel))
      return lsBarrel(in, out, ptCut, rIn, rOut, v);
    return lsEndcap(in, out, ptCut, rIn, rOut, v);
  }
  LST_HD bool lsSelect(const Modules& m,
                       const MiniDoublets& md,
                       uint16_t innerLM,
                       uint16_t outerLM,
                       unsigned int innerMD,
                       unsigned int outerMD,
                       LSValues& v) {
    return lsSelect(lsCut(m, innerLM), lsCut(m, outerLM), m.ptCut, md.rec[innerMD], md.rec[outerMD], v);
  }

  // SDL/Segment.h:358-390
  LST_HD void storeLS(Segments& s,
                      const MiniDoublets& md,
                      unsigned int innerMD,
                      unsigned int outerMD,
                      uint16_t innerLM,
                      uint16_t outerLM,
                      const LSValues& v,
                      unsigned int idx) {
    // (loads before stores, as in storeMD)
    const unsigned int innerHit = md.anchorHitIndices[innerMD], outerHit = md.anchorHitIndices[outerMD];
    s.mdIndices[idx * 2] = innerMD;
    s.mdIndices[idx * 2 + 1] = outerMD;
    s.innerLowerModuleIndices[idx] = innerLM;
    s.outerLowerModuleIndices[idx] = outerLM;
    s.innerMiniDoubletAnchorHitIndices[idx] = innerHit;
    s.outerMiniDoubletAnchorHitIndices[idx] = outerHit;
    s.dPhis[idx] = v.dPhi;
    s.dPhiMins[idx] = v.dPhiMin;
    s.dPhiMaxs[idx] = v.dPhiMax;
    s.dPhiChanges[idx] = v.dPhiChange;
    s.dPhiChangeMins[idx] = v.dPhiChangeMin;
    s.dPhiChangeMaxs[idx] = v.dPhiChangeMax;
  }

  // One pixel line segment: two pixel mini-doublets from the seed's four
  // pseudo-hits (storePixelMD, with their records: the segments may be added
  // after the mini-doublet stage), the rz least-squares score and the seed's circle
  // (storePixelLS) (SDL/Segment.h:1031-1117 with SDL/Segment.h:392-453).
  LST_HD void storePixelMD(const Modules& m,
                           const Hits& h,
                           MiniDoublets& md,
                           uint16_t pixelModule,
                           unsigned int idx,
                           unsigned int lowerHit,
                           unsigned int upperHit) {
    const MDValues zero{0, 0, 0, 0, 0, 0, 0, 0, 0};
    const bool swap = m.moduleType[pixelModule] == PS and m.moduleLayerType[pixelModule] == Strip;
    const unsigned int anchor = swap ? upperHit : lowerHit, outer = swap ? lowerHit : upperHit;
    const MDAnchor a = storeMDHits(m, h, md, anchor, outer, pixelModule, idx);
    storeMDPair(m, md, lowerHit, upperHit, pixelModule, zero, idx);
    // (the pixel tracklets read the anchor alone; the other values are those of the
    // cuts between outer-tracker modules)
    md.rec[idx] = MDRec{a.pos.x, a.pos.y, a.pos.z, a.pos.rt, a.phi, 0, 0, 0, 0, 0, a.highEdgePhi, a.lowEdgePhi, 0, 0,
                        anchor, outer};
  }
  LST_HD void storePixelLS(const Modules& m,
                           const Hits& h,
                           Segments& s,
                           uint16_t pixelModule,
                           unsigned int mdBase,
                           unsigned int lsBase,
                           unsigned int tid,
                           unsigned int hit0,
                           unsigned int hit1,
                           unsigned int hit2,
                           unsigned int hit3,
                           float dPhiChange) {
    unsigned int innerMD = mdBase + 2 * tid;
    unsigned int outerMD = mdBase + 2 * tid + 1;
    unsigned int pls = lsBase + tid;
    // The anchor and outer hits of the two mini-doublets (storeMD's rule), so
    // that the values below are read from the hits directly, and before the
    // stores (as in storeMD).
    const bool swap = m.moduleType[pixelModule] == PS and m.moduleLayerType[pixelModule] == Strip;
    const unsigned int inAnchor = swap ? hit1 : hit0, inOuter = swap ? hit0 : hit1;
    const unsigned int outAnchor = swap ? hit3 : hit2, outOuter = swap ? hit2 : hit3;

    float slope = fsinh(h.ys[inOuter]);
    float intercept = h.zs[inAnchor] - slope * h.rts[inAnchor];
    float score_lsq = (h.rts[outAnchor] * slope + intercept) - (h.zs[outAnchor]);
    score_lsq = score_lsq * score_lsq;

    const unsigned int idxInAnchor = h.idxs[inAnchor], idxOutAnchor = h.idxs[outAnchor];
    const unsigned int idxInOuter = h.idxs[inOuter], idxOutOuter = h.idxs[outOuter];
    float circleRadius = h.xs[inOuter] / (2 * k2Rinv1GeVf);
    float circlePhi = h.zs[inOuter];
    const float inAnchorX = h.xs[inAnchor], inAnchorY = h.ys[inAnchor];
    const float outAnchorX = h.xs[outAnchor], outAnchorY = h.ys[outAnchor];
    float candidateCenterXs[2] = {inAnchorX + circleRadius * fsin(circlePhi), inAnchorX - circleRadius * fsin(circlePhi)};
    float candidateCenterYs[2] = {inAnchorY - circleRadius * fcos(circlePhi), inAnchorY + circleRadius * fcos(circlePhi)};
    float bestChiSquared = kInf;
    int bestIndex = 0;
    for (int i = 0; i < 2; i++) {
      float chiSquared = fabs_(fsqrt((outAnchorX - candidateCenterXs[i]) * (outAnchorX - candidateCenterXs[i]) +
                                     (outAnchorY - candidateCenterYs[i]) * (outAnchorY - candidateCenterYs[i])) -
                               circleRadius);
      if (chiSquared < bestChiSquared) {
        bestChiSquared = chiSquared;
        bestIndex = i;
      }
    }
    s.mdIndices[pls * 2] = innerMD;
    s.mdIndices[pls * 2 + 1] = outerMD;
    s.innerLowerModuleIndices[pls] = pixelModule;
    s.outerLowerModuleIndices[pls] = pixelModule;
    s.innerMiniDoubletAnchorHitIndices[pls] = hit0;
    s.outerMiniDoubletAnchorHitIndices[pls] = hit2;
    s.dPhiChanges[pls] = dPhiChange;
    s.isDup[tid] = 0;
    s.score[tid] = score_lsq;
    s.pLSHitsIdxs[4 * tid + 0] = idxInAnchor;
    s.pLSHitsIdxs[4 * tid + 1] = idxOutAnchor;
    s.pLSHitsIdxs[4 * tid + 2] = idxInOuter;
    s.pLSHitsIdxs[4 * tid + 3] = idxOutOuter;
    s.circleCenterX[tid] = candidateCenterXs[bestIndex];
    s.circleCenterY[tid] = candidateCenterYs[bestIndex];
    s.circleRadius[tid] = circleRadius;
  }
  LST_HD void storePixelSegment(const Modules& m,
                                const Hits& h,
                                MiniDoublets& md,
                                Segments& s,
                                uint16_t pixelModule,
                                unsigned int mdBase,
                                unsigned int lsBase,
                                unsigned int tid,
                                unsigned int hit0,
                                unsigned int hit1,
                                unsigned int hit2,
                                unsigned int hit3,
                                float dPhiChange) {
    storePixelMD(m, h, md, pixelModule, mdBase + 2 * tid, hit0, hit1);
    storePixelMD(m, h, md, pixelModule, mdBase + 2 * tid + 1, hit2, hit3);
    storePixelLS(m, h, s, pixelModule, mdBase, lsBase, tid, hit0, hit1, hit2, hit3, dPhiChange);
  }

}  // namespace lst

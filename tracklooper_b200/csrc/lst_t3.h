// Triplet (T3) selection: two line segments sharing a mini-doublet.  Cut
// arithmetic follows SDL/Triplet.h:154-870.
#pragma once

#include "lst_ls.h"

namespace lst {

  // Largest r-z residual of the middle hit against the line through the outer
  // two, by the three modules' layers in the sdlLayers numbering
  // (SDL/Triplet.h:241-299); 0 for the layers that never pass.
  LST_HD float t3RZCut(int layer1, int layer2, int layer3) {
    const int key = (layer1 << 10) | (layer2 << 5) | layer3;
    switch (key) {
      case (12 << 10) | (13 << 5) | 14:
      case (13 << 10) | (14 << 5) | 15:
      case (14 << 10) | (15 << 5) | 16:
        return 0.f;
      case (1 << 10) | (2 << 5) | 3:
        return 0.53f;
      case (2 << 10) | (3 << 5) | 4:
        return 1.21f;
      case (3 << 10) | (4 << 5) | 5:
        return 2.7f;
      case (4 << 10) | (5 << 5) | 6:
        return 3.06f;
      case (1 << 10) | (2 << 5) | 7:
      case (1 << 10) | (7 << 5) | 8:
      case (2 << 10) | (3 << 5) | 7:
      case (2 << 10) | (7 << 5) | 8:
      case (7 << 10) | (8 << 5) | 9:
      case (8 << 10) | (9 << 5) | 10:
      case (9 << 10) | (10 << 5) | 11:
        return 1.f;
    }
    return 5.f;
  }
  LST_HD bool t3PassRZ(float r1, float z1, float r2, float z2, float r3, float z3, float cut) {
    const float residual = z2 - ((z3 - z1) / (r3 - r1) * (r2 - r1) + z1);
    return fabs_(residual) < cut;
  }

  LST_HD float segmentDr(const MiniDoublets& md, unsigned int a, unsigned int b) {
    return fsqrt((md.rec[b].x - md.rec[a].x) * (md.rec[b].x - md.rec[a].x) +
                 (md.rec[b].y - md.rec[a].y) * (md.rec[b].y - md.rec[a].y));
  }

  // Pointing of the triplet and its first beta cut: barrel-barrel-barrel
  // (SDL/Triplet.h:301-402), barrel-barrel-endcap / barrel-endcap-endcap
  // (SDL/Triplet.h:404-531) and endcap-endcap-endcap (SDL/Triplet.h:533-658) in
  // one body: a warp holds candidates of all three, and the parts they share
  // (the extrapolation error, the atan2, the arcsine) run once for all of them.
  // f1, f2, f3: the modules' MDCutFlags.
  LST_HD bool t3Pointing(unsigned int f1,
                         unsigned int f2,
                         unsigned int f3,
                         float ptCut,
                         const MDRec& in,
                         const MDRec& mid,
                         const MDRec& out,
                         const Segments& s,
                         unsigned int innerSeg,
                         float& betaIn) {
    const bool eee = (f1 & f2 & f3 & kCutEndcap) != 0;
    const bool bbb = (f1 & f2 & f3 & kCutBarrel) != 0;
    // (the second module of a barrel-endcap triplet lies on either side)
    if (!(bbb or eee or ((f1 & kCutBarrel) and (f2 & (kCutBarrel | kCutEndcap)) and (f3 & kCutEndcap))))
      return false;
    const bool isPSIn = (f1 & kCutPS) != 0, isPSOut = (f3 & kCutPS) != 0;
    const float rtIn = in.rt, rtMid = mid.rt, rtOut = out.rt;
    const float zIn = in.z, zMid = mid.z, zOut = out.z;
    const float dzDrtScale = out.dzDrtScale;
    const float zGeom = (isPSIn ? kPixelPSZpitch : kStrip2SZpitch) + (isPSOut ? kPixelPSZpitch : kStrip2SZpitch);
    const float dz = zOut - zIn;
    float rtGeom = 0;
    if (bbb) {
      const float rtRatio_OutIn = rtOut / rtIn;
      const float zHi = zIn + (zIn + kDeltaZLum) * (rtRatio_OutIn - 1.f) * (zIn < 0.f ? 1.f : dzDrtScale) + zGeom;
      const float zLo = zIn + (zIn - kDeltaZLum) * (rtRatio_OutIn - 1.f) * (zIn > 0.f ? 1.f : dzDrtScale) - zGeom;
      if (!((zOut >= zLo) && (zOut <= zHi)))
        return false;
    } else {
      if (!(zIn * zOut > 0))
        return false;
      const float dLum = signTransfer(kDeltaZLum, zIn);
      float dzLo = dz, dzHi = dz, denLo = zIn + dLum, denHi = zIn - dLum;
      if (eee)
        rtGeom = (isPSIn and isPSOut)  ? 2.f * kPixelPSZpitch
                 : (isPSIn or isPSOut) ? kPixelPSZpitch + kStrip2SZpitch
                                       : 2.f * kStrip2SZpitch;
      else {
        rtGeom = isPSOut ? kPixelPSZpitch : kStrip2SZpitch;
        const float zGeom1 = signTransfer(zGeom, zIn);
        dzLo = dz - zGeom1;
        dzHi = dz + zGeom1;
        denLo = zIn + zGeom1 + dLum;
        denHi = zIn - zGeom1 - dLum;
        if (denHi * zIn < 0)
          denHi = signTransfer(0.1f, zIn);
      }
      const float rtLo = rtIn * (1.f + dzLo / denLo / dzDrtScale) - rtGeom;
      const float rtHi = rtIn * (1.f + dzHi / denHi) + rtGeom;
      if (!((rtOut >= rtLo) && (rtOut <= rtHi)))
        return false;
    }

    const float drtIn = rtMid - rtIn, dzIn = zMid - zIn;
    if (!bbb and (!eee or (isPSIn and isPSOut))) {
      const float kZ = dz / dzIn;
      if (!(kZ >= 0))
        return false;
    }
    if (bbb or (eee and isPSIn and isPSOut)) {
      const float r3In = fsqrt(zIn * zIn + rtIn * rtIn);
      const float dr3In = fsqrt(rtMid * rtMid + zMid * zMid) - r3In;
      const float coshEta = dr3In / drtIn;
      const float dzAbs = fabs_(dz);
      float theta = 0.015f * fsqrt(0.1f + 0.2f * (rtOut - rtIn) / 50.f);
      float lever, err;
      if (bbb) {
        theta = theta * fsqrt(r3In / rtIn);
        lever = rtOut - rtIn;
        err = zGeom * zGeom * 2.f;
      } else {
        lever = dzAbs * coshEta / (coshEta * coshEta - 1.f);
        err = kPixelPSZpitch * kPixelPSZpitch * 2.f / (dzIn * dzIn) * (dzAbs * dzAbs);
      }
      const float sdlMuls = theta * 3.f / ptCut * 4.f;
      err = fsqrt(err + sdlMuls * sdlMuls * lever * lever / 3.f * coshEta * coshEta);
      float lo, hi, x;
      if (bbb) {
        const float dzMean = dzIn / drtIn * lever;
        const float window = err / drtIn * lever + zGeom;
        lo = zIn + dzMean * (zIn > 0.f ? 1.f : dzDrtScale) - window;
        hi = zIn + dzMean * (zIn < 0.f ? 1.f : dzDrtScale) + window;
        x = zOut;
      } else {
        const float drtMean = drtIn * dzAbs / fabs_(dzIn);
        const float window = err + rtGeom;
        lo = rtIn + drtMean / dzDrtScale - window;
        hi = rtIn + drtMean + window;
        x = rtOut;
      }
      if (!((x >= lo) && (x <= hi)))
        return false;
    }

    const float alpha = s.dPhiChanges[innerSeg];
    const float tl_axis_x = out.x - in.x;
    const float tl_axis_y = out.y - in.y;
    betaIn = alpha - phiMpiPi(phiOf(tl_axis_x, tl_axis_y) - in.phi);
    float beta = betaIn;
    if (eee) {
      const float betaMin = betaIn + s.dPhiChangeMins[innerSeg] - alpha;
      const float betaMax = betaIn + s.dPhiChangeMaxs[innerSeg] - alpha;
      beta = fabs_(betaMin) > fabs_(betaMax) ? betaMax : betaMin;
    }
    const float drAxis = fsqrt(tl_axis_x * tl_axis_x + tl_axis_y * tl_axis_y);
    const float drIn = fsqrt((mid.x - in.x) * (mid.x - in.x) + (mid.y - in.y) * (mid.y - in.y));
    const float betaInCut = fasin(fmin_((-drIn + drAxis) * k2Rinv1GeVf / ptCut, kSinAlphaMax)) + (0.02f / drtIn);
    return fabs_(beta) < betaInCut;
  }

  // Circle through three points; radius -1 for collinear points
  // (SDL/Triplet.h:762-795).
  LST_HD float circleFrom3(float x1, float y1, float x2, float y2, float x3, float y3, float& g, float& f) {
    float radius = 0.f;
    float denomInv = 1.0f / ((y1 - y3) * (x2 - x3) - (x1 - x3) * (y2 - y3));
    float xy1sqr = x1 * x1 + y1 * y1;
    float xy2sqr = x2 * x2 + y2 * y2;
    float xy3sqr = x3 * x3 + y3 * y3;
    g = 0.5f * ((y3 - y2) * xy1sqr + (y1 - y3) * xy2sqr + (y2 - y1) * xy3sqr) * denomInv;
    f = 0.5f * ((x2 - x3) * xy1sqr + (x3 - x1) * xy2sqr + (x1 - x2) * xy3sqr) * denomInv;
    float c = ((x2 * y3 - x3 * y2) * xy1sqr + (x3 * y1 - x1 * y3) * xy2sqr + (x1 * y2 - x2 * y1) * xy3sqr) * denomInv;
    if (((y1 - y3) * (x2 - x3) - (x1 - x3) * (y2 - y3) == 0) || (g * g + f * f - c < 0))
      radius = -1.f;
    else
      radius = fsqrt(g * g + f * f - c);
    return radius;
  }

  struct T3Values {
    float betaIn, circleRadius, circleCenterX, circleCenterY;
  };

  // The tests after the r-z residual, and the circle.
  LST_HD bool t3Rest(unsigned int f1,
                     unsigned int f2,
                     unsigned int f3,
                     float ptCut,
                     const MDRec& in,
                     const MDRec& mid,
                     const MDRec& out,
                     const Segments& s,
                     unsigned int innerSeg,
                     T3Values& v) {
    if (!t3Pointing(f1, f2, f3, ptCut, in, mid, out, s, innerSeg, v.betaIn))
      return false;
    v.circleRadius = circleFrom3(in.x, in.y, mid.x, mid.y, out.x, out.y, v.circleCenterX, v.circleCenterY);
    return true;
  }

  // SDL/Triplet.h:797-870
  LST_HD bool t3Select(const Modules& m,
                       const MiniDoublets& md,
                       const Segments& s,
                       uint16_t lm1,
                       uint16_t lm2,
                       uint16_t lm3,
                       unsigned int innerSeg,
                       unsigned int outerSeg,
                       T3Values& v) {
    if (s.mdIndices[2 * innerSeg + 1] != s.mdIndices[2 * outerSeg])
      return false;
    unsigned int md1 = s.mdIndices[2 * innerSeg];
    unsigned int md2 = s.mdIndices[2 * outerSeg];
    unsigned int md3 = s.mdIndices[2 * outerSeg + 1];
    const MDRec &in = md.rec[md1], &mid = md.rec[md2], &out = md.rec[md3];
    const unsigned int f1 = cutFlags(m, lm1), f2 = cutFlags(m, lm2), f3 = cutFlags(m, lm3);
    if (!t3PassRZ(in.rt, in.z, mid.rt, mid.z, out.rt, out.z, t3RZCut(cutLayer(f1), cutLayer(f2), cutLayer(f3))))
      return false;
    return t3Rest(f1, f2, f3, m.ptCut, in, mid, out, s, innerSeg, v);
  }

  // SDL/Triplet.h:181-239
  LST_HD void storeT3(const Modules& m,
                      const MiniDoublets& md,
                      const Segments& s,
                      Triplets& t,
                      unsigned int innerSeg,
                      unsigned int outerSeg,
                      uint16_t lm1,
                      uint16_t lm2,
                      uint16_t lm3,
                      const T3Values& v,
                      unsigned int idx) {
    // (loads before stores, as in storeMD)
    const unsigned int md1 = s.mdIndices[2 * innerSeg];
    const unsigned int md2 = s.mdIndices[2 * innerSeg + 1];
    const unsigned int md3 = s.mdIndices[2 * outerSeg + 1];
    const uint8_t layer1 = m.layers[lm1] + (m.subdets[lm1] == 4) * 6;
    const uint8_t layer2 = m.layers[lm2] + (m.subdets[lm2] == 4) * 6;
    const uint8_t layer3 = m.layers[lm3] + (m.subdets[lm3] == 4) * 6;
    const unsigned int hits[6] = {md.rec[md1].anchorHit, md.rec[md1].outerHit, md.rec[md2].anchorHit,
                                  md.rec[md2].outerHit,  md.rec[md3].anchorHit, md.rec[md3].outerHit};
    t.segmentIndices[idx * 2] = innerSeg;
    t.segmentIndices[idx * 2 + 1] = outerSeg;
    t.lowerModuleIndices[idx * 3] = lm1;
    t.lowerModuleIndices[idx * 3 + 1] = lm2;
    t.lowerModuleIndices[idx * 3 + 2] = lm3;
    t.betaIn[idx] = v.betaIn;
    t.circleRadius[idx] = v.circleRadius;
    t.circleCenterX[idx] = v.circleCenterX;
    t.circleCenterY[idx] = v.circleCenterY;
    t.logicalLayers[idx * 3] = layer1;
    t.logicalLayers[idx * 3 + 1] = layer2;
    t.logicalLayers[idx * 3 + 2] = layer3;
    for (int i = 0; i < 6; ++i)
      t.hitIndices[idx * 6 + i] = hits[i];
    // The reference clears these flags for the whole store when it allocates it.
    t.partOfPT5[idx] = 0;
    t.partOfT5[idx] = 0;
    t.partOfPT3[idx] = 0;
  }

}  // namespace lst

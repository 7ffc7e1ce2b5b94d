// Mini-doublet (MD) selection: a pair of hits on the two sensors of one
// outer-tracker module.  Cut arithmetic follows SDL/MiniDoublet.h:193-892.
#pragma once

#include "lst_core.h"

namespace lst {

  // SDL/Constants.h:124-129 (double literals rounded to float, as there)
  LST_HD float miniMulsPtScaleBarrel(unsigned int i) {
    switch (i) {
      case 0: return static_cast<float>(0.0052);
      case 1: return static_cast<float>(0.0038);
      case 2: return static_cast<float>(0.0034);
      case 3: return static_cast<float>(0.0034);
      case 4: return static_cast<float>(0.0032);
      default: return static_cast<float>(0.0034);
    }
  }
  LST_HD float miniMulsPtScaleEndcap(unsigned int) { return static_cast<float>(0.006); }
  LST_HD float miniRminMeanBarrel(unsigned int i) {
    switch (i) {
      case 0: return static_cast<float>(25.007152356);
      case 1: return static_cast<float>(37.2186993757);
      case 2: return static_cast<float>(52.3104270826);
      case 3: return static_cast<float>(68.6658656666);
      case 4: return static_cast<float>(85.9770373007);
      default: return static_cast<float>(108.301772384);
    }
  }
  LST_HD float miniRminMeanEndcap(unsigned int i) {
    switch (i) {
      case 0: return static_cast<float>(130.992832231);
      case 1: return static_cast<float>(154.813883559);
      case 2: return static_cast<float>(185.352604327);
      case 3: return static_cast<float>(221.635123002);
      default: return static_cast<float>(265.022076742);
    }
  }

  // Tilted barrel modules with the smaller sensor spacing (SDL/MiniDoublet.h:268-286).
  LST_HD bool isTighterTilted(short subdet, short layer, short side, short rod) {
    return (subdet == Barrel) && (((side != Center) && (layer == 3)) ||
                                  ((side == NegZ) && (((layer == 2) && (rod > 5)) || ((layer == 1) && (rod > 9)))) ||
                                  ((side == PosZ) && (((layer == 2) && (rod < 8)) || ((layer == 1) && (rod < 4)))));
  }

  // Separation of the two sensors of a module (SDL/MiniDoublet.h:288-337).
  LST_HD float moduleGap(short layer, short ring, short subdet, short side, short rod) {
    unsigned int iL = layer - 1;
    unsigned int iR = ring - 1;
    if (subdet == Barrel && side == Center) {
      switch (iL) {
        case 0: return 0.26f;
        case 1: return 0.16f;
        case 2: return 0.16f;
        default: return 0.18f;
      }
    } else if (isTighterTilted(subdet, layer, side, rod)) {
      return 0.26f;
    } else if (subdet == Endcap) {
      unsigned int nWide = (iL <= 1) ? 10u : ((iL <= 3) ? 8u : 9u);
      return iR < nWide ? 0.4f : 0.18f;
    }
    return 0.4f;
  }
  LST_HD float moduleGap(const Modules& m, unsigned int i) {
    return moduleGap(m.layers[i], m.rings[i], m.subdets[i], m.sides[i], m.rods[i]);
  }

  // dPhi acceptance of a mini-doublet (SDL/MiniDoublet.h:340-402).
  // The slope term of mdDPhiThreshold, a function of the hit's rt alone
  // (computed once per hit by kHitPrep).
  LST_HD float mdMiniSlope(float rt, float ptCut) { return fasin(fmin_(rt * k2Rinv1GeVf / ptCut, kSinAlphaMax)); }

  // Moves the strip hit along the strip so that it lines up with the
  // interaction point and the pixel hit (SDL/MiniDoublet.h:404-568).
  // shiftStripHit (SDL/MiniDoublet.h:110-191) moves one hit of the pair (p)
  // along the strip direction onto the other sensor's plane and projects it
  // next to the other hit (o).  Which hit is p depends only on the lower
  // module lm: true = the lower hit.
  LST_HD bool shiftMovesLower(const Modules& m, uint16_t lm) {
    if (m.moduleType[lm] == PS)
      return m.subdets[lm] == Barrel ? m.moduleLayerType[lm] != Pixel : m.moduleLayerType[lm] == Pixel;
    return true;
  }

  // The part of shiftStripHit that depends on p alone: the moved point before
  // the projection (xa, ya) and the moved z (computed once per hit by kHitPrep).
  LST_HD void shiftStripPrep(const Modules& m, uint16_t lm, float xp, float yp, float zp, float rtp, float& xa, float& ya,
                             float& zn) {
    const float slope = m.dxdys[lm];
    const float drdz_ = m.drdzs[lm];
    const bool isEndcap = m.subdets[lm] == Endcap;
    float angleA = fabs_(fatan(rtp / zp));
    float angleB = isEndcap ? float(M_PI) / 2.f : fatan(drdz_);
    float moduleSeparation = moduleGap(m, lm);
    if (m.moduleType[lm] == PS and m.moduleLayerType[lm] != Pixel)
      moduleSeparation *= -1;
    float drprime = (moduleSeparation / fsin(angleA + angleB)) * fsin(angleA);
    float absArctanSlope = (slope != kInf) ? fabs_(fatan(slope)) : float(M_PI) / 2.f;
    float angleM;
    if (xp > 0 and yp > 0)
      angleM = absArctanSlope;
    else if (xp > 0 and yp < 0)
      angleM = float(M_PI) - absArctanSlope;
    else if (xp < 0 and yp < 0)
      angleM = float(M_PI) + absArctanSlope;
    else
      angleM = 2.f * float(M_PI) - absArctanSlope;
    float drprime_x = drprime * fsin(angleM);
    float drprime_y = drprime * fcos(angleM);
    xa = xp + drprime_x;
    ya = yp + drprime_y;
    float absdzprime = fabs_(moduleSeparation / fsin(angleA + angleB) * fcos(angleA));
    float abszn;
    if (m.moduleLayerType[lm] == Pixel)
      abszn = fabs_(zp) + absdzprime;
    else
      abszn = fabs_(zp) - absdzprime;
    zn = abszn * ((zp > 0) ? 1 : -1);
  }

  // What the mini-doublet cuts take from a lower module, formed once per module
  // when the event setup is loaded (kModuleCuts) instead of for every pair: the
  // terms of the dPhi threshold (SDL/MiniDoublet.h:340-402) and of the strip
  // shift's projection (:404-568).
  struct alignas(16) MDCut {
    float base, root;  // miniMuls^2 + miniPVoff^2, and its square root
    float tilt2;       // miniTilt^2
    float slope, slopeInv, slopeSum;  // the strip slope, 1 / slope, slope + 1 / slope
    unsigned int flags;
    unsigned int pad;
  };
  enum MDCutFlags : unsigned int {
    kCutBarrel = 1,         // barrel module
    kCutCenter = 2,         //   with sides == Center (not tilted)
    kCutPS = 4,
    kCutLowerIsPixel = 8,   // moduleLayerType == Pixel
    kCutMovesLower = 16,    // shiftMovesLower
    kCutEndcap = 32,
    kCutEndcapTwoS = 64,
    kCutInnerLayers = 128,  // layers 1 and 2
    kCutLayerShift = 8      // from this bit on: sdlLayers
  };

  LST_HD unsigned int cutFlags(const Modules& m, uint16_t mi) {
    const bool barrel = m.subdets[mi] == Barrel, endcap = m.subdets[mi] == Endcap;
    return (barrel ? kCutBarrel : 0u) | (barrel and m.sides[mi] == Center ? kCutCenter : 0u) |
           (m.moduleType[mi] == PS ? kCutPS : 0u) | (m.moduleLayerType[mi] == Pixel ? kCutLowerIsPixel : 0u) |
           (shiftMovesLower(m, mi) ? kCutMovesLower : 0u) | (endcap ? kCutEndcap : 0u) |
           (endcap and m.moduleType[mi] == TwoS ? kCutEndcapTwoS : 0u) | (m.layers[mi] <= 2 ? kCutInnerLayers : 0u) |
           (static_cast<unsigned int>(m.sdlLayers[mi]) << kCutLayerShift);
  }
  LST_HD int cutLayer(unsigned int flags) { return static_cast<int>(flags >> kCutLayerShift); }

  LST_HD MDCut mdCut(const Modules& m, uint16_t mi) {
    unsigned int iL = m.layers[mi] - 1;
    const bool barrel = m.subdets[mi] == Barrel;
    const float rLayNominal = barrel ? miniRminMeanBarrel(iL) : miniRminMeanEndcap(iL);
    const float miniPVoff = 0.1f / rLayNominal;
    const float miniMuls =
        barrel ? miniMulsPtScaleBarrel(iL) * 3.f / m.ptCut : miniMulsPtScaleEndcap(iL) * 3.f / m.ptCut;
    const bool isTilted = barrel and m.sides[mi] != Center;
    float drdz;
    if (isTilted) {
      if (m.moduleType[mi] == PS and m.moduleLayerType[mi] == Strip)
        drdz = m.drdzs[mi];
      else
        drdz = m.drdzs[m.partnerModuleIndices[mi]];
    } else {
      drdz = 0;
    }
    const float miniTilt =
        isTilted ? 0.5f * kPixelPSZpitch * drdz / fsqrt(1.f + drdz * drdz) / moduleGap(m, mi) : 0;
    MDCut c;
    c.base = miniMuls * miniMuls + miniPVoff * miniPVoff;
    c.root = fsqrt(miniMuls * miniMuls + miniPVoff * miniPVoff);
    c.tilt2 = miniTilt * miniTilt;
    c.slope = m.dxdys[mi];
    c.slopeInv = 1.f / c.slope;
    c.slopeSum = c.slope + (1.f / c.slope);
    c.flags = cutFlags(m, mi);
    c.pad = 0;
    return c;
  }

  // The dPhi threshold from the hit's slope term; dPhi and dz enter it for
  // endcap modules only.
  LST_HD float mdDPhiThreshold(const MDCut& c, float miniSlope, float dPhi, float dz) {
    if (c.flags & kCutCenter)
      return miniSlope + c.root;
    if (c.flags & kCutBarrel)
      return miniSlope + fsqrt(c.base + c.tilt2 * miniSlope * miniSlope);
    const float miniLum = fabs_(dPhi * kDeltaZLum / dz);
    return miniSlope + fsqrt(c.base + miniLum * miniLum);
  }

  // Per-hit values of the mini-doublet cuts computed once per hit: the slope
  // term of the dphi threshold and, for the hit that shiftStripHit moves, its
  // moved point (xa, ya) and z.  Arrays indexed by hit.
  struct MDHitPre {
    const float* miniSlope;
    const float* shiftXa;
    const float* shiftYa;
    const float* shiftZn;
  };

  // shiftStripHit's projection next to the other hit (xo, yo).
  LST_HD void shiftStripFinish(const MDCut& c, float xa, float ya, float xo, float yo, float& xn, float& yn) {
    if (c.slope == kInf) {
      xn = xa;
      yn = yo;
    } else if (c.slope == 0) {
      xn = xo;
      yn = ya;
    } else {
      xn = (c.slope * xa + c.slopeInv * xo - ya + yo) / c.slopeSum;
      yn = (xn - xa) * c.slope + ya;
    }
  }

  LST_HD void shiftStripHit(const MDCut& c,
                            const MDHitPre& pre,
                            unsigned int lowerIdx,
                            unsigned int upperIdx,
                            float xLower,
                            float yLower,
                            float xUpper,
                            float yUpper,
                            float& xn,
                            float& yn,
                            float& zn) {
    const bool fromLower = (c.flags & kCutMovesLower) != 0;
    const unsigned int p = fromLower ? lowerIdx : upperIdx;
    const float xo = fromLower ? xUpper : xLower, yo = fromLower ? yUpper : yLower;
    zn = pre.shiftZn[p];
    shiftStripFinish(c, pre.shiftXa[p], pre.shiftYa[p], xo, yo, xn, yn);
  }

  // The mini-doublet's record of what the later cuts read (MDRec).
  LST_HD void storeMDRec(MiniDoublets& md, unsigned int idx, float ptCut, const MDPos& p, float phi, float dphichange,
                         float dphi, float dz, float highEdgePhi, float lowEdgePhi, unsigned int anchorHit,
                         unsigned int outerHit) {
    const float slope = fasin(fmin_(p.rt * k2Rinv1GeVf / ptCut, kSinAlphaMax));
    const float tanSlope = ftan(slope);
    const float slope3 = fasin(fmin_(p.rt * k2Rinv1GeVf / 3.0f, kSinAlphaMax));
    md.rec[idx] = MDRec{p.x, p.y, p.z, p.rt, phi, slope, tanSlope / slope, dphichange, slope / tanSlope,
                        dphi * 15.0f / dz, highEdgePhi, lowEdgePhi, 0.1f / p.rt, slope3, anchorHit, outerHit};
  }
  // The same of a mini-doublet that storeMD has stored.
  LST_HD void storeMDDerived(MiniDoublets& md, unsigned int idx, float ptCut) {
    // (loads before stores, as in storeMDHits)
    const MDPos p = md.anchorPos[idx];
    const float phi = md.anchorPhi[idx], dphichange = md.dphichanges[idx], dphi = md.dphis[idx], dz = md.dzs[idx];
    const float highEdgePhi = md.anchorHighEdgePhi[idx], lowEdgePhi = md.anchorLowEdgePhi[idx];
    const unsigned int anchorHit = md.anchorHitIndices[idx], outerHit = md.outerHitIndices[idx];
    storeMDRec(md, idx, ptCut, p, phi, dphichange, dphi, dz, highEdgePhi, lowEdgePhi, anchorHit, outerHit);
  }

  struct MDValues {
    float dz, dphi, dphichange, shiftedX, shiftedY, shiftedZ, noShiftedDz, noShiftedDphi, noShiftedDphiChange;
  };

  // Barrel mini-doublet (SDL/MiniDoublet.h:645-777).
  LST_HD_BIG bool mdBarrel(const MDCut& c,
                       float xLower,
                       float yLower,
                       float zLower,
                       float rtLower,
                       float xUpper,
                       float yUpper,
                       float zUpper,
                       float rtUpper,
                       float phiLower,
                       float phiUpper,
                       const MDHitPre& pre,
                       unsigned int lowerIdx,
                       unsigned int upperIdx,
                       MDValues& v) {
    v.dz = zLower - zUpper;
    const float dzCut = (c.flags & kCutPS) ? 2.f : 10.f;
    const float sign = ((v.dz > 0) - (v.dz < 0)) * ((zLower > 0) - (zLower < 0));
    const float invertedcrossercut = (fabs_(v.dz) > 2) * sign;
    if (!((fabs_(v.dz) < dzCut) && (invertedcrossercut <= 0)))
      return false;

    const bool lowerIsPixel = (c.flags & kCutLowerIsPixel) != 0;
    float miniCut = mdDPhiThreshold(c, pre.miniSlope[lowerIsPixel ? lowerIdx : upperIdx], 0, 0);

    float shiftedRt = 0;
    const bool tilted = !(c.flags & kCutCenter);
    if (tilted) {
      float xn, yn, zn;
      shiftStripHit(c, pre, lowerIdx, upperIdx, xLower, yLower, xUpper, yUpper, xn, yn, zn);
      v.shiftedX = xn;
      v.shiftedY = yn;
      shiftedRt = fsqrt(xn * xn + yn * yn);
      if (lowerIsPixel) {
        v.shiftedZ = zUpper;
        v.dphi = phiMpiPi(phiOf(v.shiftedX, v.shiftedY) - phiLower);
      } else {
        v.shiftedZ = zLower;
        v.dphi = phiMpiPi(phiUpper - phiOf(v.shiftedX, v.shiftedY));
      }
      v.noShiftedDphi = phiMpiPi(phiUpper - phiLower);
    } else {
      v.shiftedX = 0;
      v.shiftedY = 0;
      v.shiftedZ = 0;
      v.dphi = phiMpiPi(phiUpper - phiLower);
      v.noShiftedDphi = v.dphi;
    }
    if (!(fabs_(v.dphi) < miniCut))
      return false;

    if (tilted) {
      if (!lowerIsPixel) {
        v.dphichange = (rtLower < shiftedRt) ? deltaPhiChangeFrom(phiLower, xLower, yLower, v.shiftedX, v.shiftedY)
                                             : deltaPhiChange(v.shiftedX, v.shiftedY, xLower, yLower);
      } else {
        v.dphichange = (shiftedRt < rtUpper) ? deltaPhiChange(v.shiftedX, v.shiftedY, xUpper, yUpper)
                                             : deltaPhiChangeFrom(phiUpper, xUpper, yUpper, v.shiftedX, v.shiftedY);
      }
      v.noShiftedDphiChange = rtLower < rtUpper ? deltaPhiChangeFrom(phiLower, xLower, yLower, xUpper, yUpper)
                                                : deltaPhiChangeFrom(phiUpper, xUpper, yUpper, xLower, yLower);
    } else {
      v.dphichange = deltaPhiChangeFrom(phiLower, xLower, yLower, xUpper, yUpper);
      v.noShiftedDphiChange = v.dphichange;
    }
    v.noShiftedDz = 0;
    return fabs_(v.dphichange) < miniCut;
  }

  // Endcap mini-doublet (SDL/MiniDoublet.h:779-892).  The stored "dz" of an
  // endcap mini-doublet is the transverse-radius difference.
  LST_HD_BIG bool mdEndcap(const MDCut& c,
                       float xLower,
                       float yLower,
                       float zLower,
                       float rtLower,
                       float xUpper,
                       float yUpper,
                       float zUpper,
                       float rtUpper,
                       float phiLower,
                       float phiUpper,
                       const MDHitPre& pre,
                       unsigned int lowerIdx,
                       unsigned int upperIdx,
                       MDValues& v) {
    float dz = zLower - zUpper;
    const float dzCut = 1.f;
    if (!(fabs_(dz) < dzCut))
      return false;
    const float drtCut = (c.flags & kCutPS) ? 2.f : 10.f;
    v.dz = rtLower - rtUpper;
    if (!(fabs_(v.dz) < drtCut))
      return false;

    float xn, yn, zn;
    shiftStripHit(c, pre, lowerIdx, upperIdx, xLower, yLower, xUpper, yUpper, xn, yn, zn);
    const bool isPS = (c.flags & kCutPS) != 0;
    const bool lowerIsPixel = (c.flags & kCutLowerIsPixel) != 0;
    v.shiftedX = xn;
    v.shiftedY = yn;
    if (isPS) {
      if (lowerIsPixel) {
        v.shiftedZ = zUpper;
        v.dphi = phiMpiPi(phiOf(v.shiftedX, v.shiftedY) - phiLower);
      } else {
        v.shiftedZ = zLower;
        v.dphi = phiMpiPi(phiUpper - phiOf(v.shiftedX, v.shiftedY));
      }
    } else {
      v.shiftedZ = zUpper;
      v.dphi = phiMpiPi(phiOf(xn, yn) - phiLower);
    }
    v.noShiftedDphi = phiMpiPi(phiUpper - phiLower);

    if (isPS)
      dz = lowerIsPixel ? zLower - zn : zUpper - zn;

    float miniCut = mdDPhiThreshold(c, pre.miniSlope[lowerIsPixel ? lowerIdx : upperIdx], v.dphi, dz);
    if (!(fabs_(v.dphi) < miniCut))
      return false;

    float dzFrac = fabs_(dz) / fabs_(zLower);
    v.dphichange = v.dphi / dzFrac * (1.f + dzFrac);
    v.noShiftedDphiChange = v.noShiftedDphi / dzFrac * (1.f + dzFrac);
    v.noShiftedDz = 0;
    return fabs_(v.dphichange) < miniCut;
  }

  // phiLower / phiUpper are the hits' stored phi (hits.phis, phi() of the same
  // coordinates), used wherever the reference takes deltaPhi of a hit itself.
  LST_HD bool mdSelect(const MDCut& c,
                       float xLower,
                       float yLower,
                       float zLower,
                       float rtLower,
                       float xUpper,
                       float yUpper,
                       float zUpper,
                       float rtUpper,
                       float phiLower,
                       float phiUpper,
                       const MDHitPre& pre,
                       unsigned int lowerIdx,
                       unsigned int upperIdx,
                       MDValues& v) {
    if (c.flags & kCutBarrel)
      return mdBarrel(c, xLower, yLower, zLower, rtLower, xUpper, yUpper, zUpper, rtUpper, phiLower, phiUpper, pre,
                      lowerIdx, upperIdx, v);
    return mdEndcap(c, xLower, yLower, zLower, rtLower, xUpper, yUpper, zUpper, rtUpper, phiLower, phiUpper, pre,
                    lowerIdx, upperIdx, v);
  }
  LST_HD bool mdSelect(const Modules& m,
                       uint16_t lm,
                       float xLower,
                       float yLower,
                       float zLower,
                       float rtLower,
                       float xUpper,
                       float yUpper,
                       float zUpper,
                       float rtUpper,
                       float phiLower,
                       float phiUpper,
                       const MDHitPre& pre,
                       unsigned int lowerIdx,
                       unsigned int upperIdx,
                       MDValues& v) {
    return mdSelect(mdCut(m, lm), xLower, yLower, zLower, rtLower, xUpper, yUpper, zUpper, rtUpper, phiLower, phiUpper,
                    pre, lowerIdx, upperIdx, v);
  }

  // A mini-doublet (SDL/MiniDoublet.h:193-266) is stored in two parts: its hits
  // and the values of its cuts by the kernel that finds it, where few lanes of a
  // warp have one, and the values of its hits by the next (kMDDerived), whose
  // lanes take stored mini-doublets in a row.
  //
  // On PS modules whose lower sensor is the strip sensor the anchor is the upper
  // (pixel) hit.
  LST_HD void storeMDPair(const Modules& m,
                          MiniDoublets& md,
                          unsigned int lowerHitIdx,
                          unsigned int upperHitIdx,
                          uint16_t lowerModuleIdx,
                          const MDValues& v,
                          unsigned int idx) {
    unsigned int anchor, outer;
    if (m.moduleType[lowerModuleIdx] == PS and m.moduleLayerType[lowerModuleIdx] == Strip) {
      anchor = upperHitIdx;
      outer = lowerHitIdx;
    } else {
      anchor = lowerHitIdx;
      outer = upperHitIdx;
    }
    md.moduleIndices[idx] = lowerModuleIdx;
    md.anchorHitIndices[idx] = anchor;
    md.outerHitIndices[idx] = outer;
    md.dphichanges[idx] = v.dphichange;
    md.dphis[idx] = v.dphi;
    md.dzs[idx] = v.dz;
    md.shiftedXs[idx] = v.shiftedX;
    md.shiftedYs[idx] = v.shiftedY;
    md.shiftedZs[idx] = v.shiftedZ;
    md.noShiftedDzs[idx] = v.noShiftedDz;
    md.noShiftedDphis[idx] = v.noShiftedDphi;
    md.noShiftedDphiChanges[idx] = v.noShiftedDphiChange;
  }

  struct MDAnchor {
    MDPos pos;
    float phi, highEdgePhi, lowEdgePhi;
  };
  LST_HD MDAnchor storeMDHits(const Modules& m,
                              const Hits& h,
                              MiniDoublets& md,
                              unsigned int anchor,
                              unsigned int outer,
                              uint16_t lowerModuleIdx,
                              unsigned int idx) {
    // All loads before the first store: a load after a store that might alias it
    // waits for its turn, some 25 round trips in a row per stored mini-doublet
    // (with the other objects' stores in the same way, the kernels of 64 PU200
    // events took 10.27 ms together, now 9.94; kCreateT3 1.29 and 1.12).
    const float ax = h.xs[anchor], ay = h.ys[anchor], az = h.zs[anchor], art = h.rts[anchor];
    const float aphi = h.phis[anchor], aeta = h.etas[anchor];
    const float hex = h.highEdgeXs[anchor], hey = h.highEdgeYs[anchor];
    const float lex = h.lowEdgeXs[anchor], ley = h.lowEdgeYs[anchor];
    const float ox = h.xs[outer], oy = h.ys[outer], oz = h.zs[outer], ort = h.rts[outer];
    const float ophi = h.phis[outer], oeta = h.etas[outer];
    const float ohex = h.highEdgeXs[outer], ohey = h.highEdgeYs[outer];
    const float olex = h.lowEdgeXs[outer], oley = h.lowEdgeYs[outer];
    // The strip ends of the other module types are all +0 (kHitPrep), and so are
    // their angles.
    float hphi = 0, lphi = 0;
    if (m.subdets[lowerModuleIdx] == Endcap and m.moduleType[lowerModuleIdx] == TwoS) {
      hphi = fatan2(hey, hex);
      lphi = fatan2(ley, lex);
    }
    md.anchorX[idx] = ax;
    md.anchorY[idx] = ay;
    md.anchorZ[idx] = az;
    md.anchorRt[idx] = art;
    md.anchorPos[idx] = MDPos{ax, ay, az, art};
    md.anchorPhi[idx] = aphi;
    md.anchorEta[idx] = aeta;
    md.anchorHighEdgeX[idx] = hex;
    md.anchorHighEdgeY[idx] = hey;
    md.anchorLowEdgeX[idx] = lex;
    md.anchorLowEdgeY[idx] = ley;
    md.anchorHighEdgePhi[idx] = hphi;
    md.anchorLowEdgePhi[idx] = lphi;

    md.outerX[idx] = ox;
    md.outerY[idx] = oy;
    md.outerZ[idx] = oz;
    md.outerRt[idx] = ort;
    md.outerPhi[idx] = ophi;
    md.outerEta[idx] = oeta;
    md.outerHighEdgeX[idx] = ohex;
    md.outerHighEdgeY[idx] = ohey;
    md.outerLowEdgeX[idx] = olex;
    md.outerLowEdgeY[idx] = oley;
    return MDAnchor{MDPos{ax, ay, az, art}, aphi, hphi, lphi};
  }

  LST_HD void storeMD(const Modules& m,
                      const Hits& h,
                      MiniDoublets& md,
                      unsigned int lowerHitIdx,
                      unsigned int upperHitIdx,
                      uint16_t lowerModuleIdx,
                      const MDValues& v,
                      unsigned int idx) {
    storeMDPair(m, md, lowerHitIdx, upperHitIdx, lowerModuleIdx, v, idx);
    storeMDHits(m, h, md, md.anchorHitIndices[idx], md.outerHitIndices[idx], lowerModuleIdx, idx);
  }

  // The second part and the record of a mini-doublet that storeMDPair stored.
  LST_HD void storeMDRest(const Modules& m, const Hits& h, MiniDoublets& md, uint16_t lowerModuleIdx,
                          unsigned int idx) {
    const unsigned int anchor = md.anchorHitIndices[idx], outer = md.outerHitIndices[idx];
    const float dphichange = md.dphichanges[idx], dphi = md.dphis[idx], dz = md.dzs[idx];
    const MDAnchor a = storeMDHits(m, h, md, anchor, outer, lowerModuleIdx, idx);
    storeMDRec(md, idx, m.ptCut, a.pos, a.phi, dphichange, dphi, dz, a.highEdgePhi, a.lowEdgePhi, anchor, outer);
  }

  // Per-module mini-doublet capacity from the (category, |eta|) occupancy table
  // (SDL/MiniDoublet.h:1019-1067).
  LST_HD int occupancyCategory(short layers, short subdets, short rings) {
    if (layers <= 3 && subdets == 5)
      return 0;
    if (layers >= 4 && subdets == 5)
      return 1;
    if (layers <= 2 && subdets == 4 && rings >= 11)
      return 2;
    if (layers >= 3 && subdets == 4 && rings >= 8)
      return 2;
    if (layers <= 2 && subdets == 4 && rings <= 10)
      return 3;
    if (layers >= 3 && subdets == 4 && rings <= 7)
      return 3;
    return -1;
  }
  LST_HD int occupancyEtaBin(float absEta) {
    if (absEta < 0.75)
      return 0;
    if (absEta > 0.75 && absEta < 1.5)
      return 1;
    if (absEta > 1.5 && absEta < 2.25)
      return 2;
    if (absEta > 2.25 && absEta < 3)
      return 3;
    return -1;
  }
  LST_HD int mdOccupancy(int category, int etaBin) {
    if (category == 0 && etaBin == 0) return 49;
    if (category == 0 && etaBin == 1) return 42;
    if (category == 0 && etaBin == 2) return 37;
    if (category == 0 && etaBin == 3) return 41;
    if (category == 1) return 100;
    if (category == 2 && etaBin == 1) return 16;
    if (category == 2 && etaBin == 2) return 19;
    if (category == 3 && etaBin == 1) return 14;
    if (category == 3 && etaBin == 2) return 20;
    if (category == 3 && etaBin == 3) return 25;
    return 0;
  }
  // SDL/Segment.h:954-994
  LST_HD int lsOccupancy(int category, int etaBin) {
    if (category == 0 && etaBin == 0) return 572;
    if (category == 0 && etaBin == 1) return 300;
    if (category == 0 && etaBin == 2) return 183;
    if (category == 0 && etaBin == 3) return 62;
    if (category == 1 && etaBin == 0) return 191;
    if (category == 1 && etaBin == 1) return 128;
    if (category == 2 && etaBin == 1) return 107;
    if (category == 2 && etaBin == 2) return 102;
    if (category == 3 && etaBin == 1) return 64;
    if (category == 3 && etaBin == 2) return 79;
    if (category == 3 && etaBin == 3) return 85;
    return 0;
  }
  // SDL/Triplet.h:1049-1089
  LST_HD int t3Occupancy(int category, int etaBin) {
    if (category == 0 && etaBin == 0) return 543;
    if (category == 0 && etaBin == 1) return 235;
    if (category == 0 && etaBin == 2) return 88;
    if (category == 0 && etaBin == 3) return 46;
    if (category == 1 && etaBin == 0) return 755;
    if (category == 1 && etaBin == 1) return 347;
    if (category == 2 && etaBin == 1) return 0;
    if (category == 2 && etaBin == 2) return 0;
    if (category == 3 && etaBin == 1) return 38;
    if (category == 3 && etaBin == 2) return 46;
    if (category == 3 && etaBin == 3) return 39;
    return 0;
  }
  // SDL/Quintuplet.h:3179-3198
  LST_HD int t5Occupancy(int category, int etaBin) {
    if (category == 0 && etaBin == 0) return 336;
    if (category == 0 && etaBin == 1) return 414;
    if (category == 0 && etaBin == 2) return 231;
    if (category == 0 && etaBin == 3) return 146;
    if (category == 3 && etaBin == 1) return 0;
    if (category == 3 && etaBin == 2) return 191;
    if (category == 3 && etaBin == 3) return 106;
    return 0;
  }

}  // namespace lst

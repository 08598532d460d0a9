/* Visplane rows, the per-column portal walk with its wall tiers and plane marks, two-sided middle textures.
 * Part of gd_render.cu (one translation unit); not meant to be included elsewhere. */
#ifndef GD_WALK_CUH
#define GD_WALK_CUH

/* ---- visplane rows (engine.py:10879-10954, 10588-10616, 13372-13405) ---- */
struct GdPlaneSpan {
  i64 basex, basey, pviewx, pviewy, phf, gv, shadeBase;
  unsigned tex;
  int wbits, hbits, texW;
};

/* Column-independent part of a span setup, one entry per (sector, floor or
 * ceiling), rebuilt for every lane: the three divisions of R_DrawSpan's setup
 * leave the per-crossing path.  GdPlane is the form the walk reads: it holds when every
 * operand fits 32 bits (`flags` says so), which leaves the pixel with 32 x 32 -> 64 multiplies. */
struct GdPlaneEntry {
  i64 phf, gv, shadeBase, xstep, ystep, bx0, by0, pviewx, pviewy;
  unsigned tex;
  int wbits, hbits, pad;
};
struct __align__(16) GdPlane {
  int phf, gv, shadeBase;
  unsigned flags;                 /* 32 - wbits | 32 - hbits << 8 | GD_PLANE_NARROW */
  int bx0, xstep, by0, ystep;
  unsigned pviewx, pviewy, tex;
  int pad;
};
#define GD_PLANE_NARROW 65536u

static_assert(sizeof(GdPlaneEntry) == GD_PLANE_ENTRY_BYTES && sizeof(GdPlane) == GD_PLANE_BYTES, "scratch layout");

__device__ __noinline__ void gd_plane_entry_setup(const GdScene &sc_, const GdView &v_, int sector, bool isFloor,
                                                  GdPlaneEntry &e, GdPlane &n) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const GdView &v = *gd_as_shared(&v_);
  float ph = isFloor ? (v.viewZ - gd_sec_floor(sc, sector)) : (gd_sec_ceil(sc, sector) - v.viewZ);
  int4 si = gd_sec_info(sc, sector);
  int tex = GD_CHECK_INDEX(isFloor ? si.y : si.z, sc.T);
  const int4 ti = *reinterpret_cast<const int4 *>(&sc.texInfo[tex * 4]);
  const int wbits = ti.z, hbits = ti.w;
  const unsigned texel0 = (unsigned)tex * (unsigned)(sc.texH * sc.texW);
  i64 xscale = 1LL << (32 - wbits), yscale = 1LL << (32 - hbits);
  i64 fs = v.vsin, fc = v.vcos;
  const i64 xstep = gd_div(xscale * fs, GD_FOCAL_X), ystep = gd_div(yscale * fc, GD_FOCAL_X);
  const i64 bx0 = (xscale * fc) >> 16, by0 = (yscale * -fs) >> 16;
  const i64 pviewx = gd_wmul(xscale, v.vx) >> 16, pviewy = gd_wmul(yscale, -v.vy) >> 16;
  const i64 phf = gd_rint(ph * 65536.0f);
  const i64 gv = gd_min(gd_div(GD_FLOOR_VIS << 16, gd_max(phf, 1)), (1LL << 31) - 1);
  i64 light = si.x + v.flashLight * 16;
  const i64 shadeBase = 64 * GD_FU - (light + 12) * (GD_FU / 4);
  e.wbits = wbits; e.hbits = hbits; e.tex = texel0; e.pad = 0;
  e.xstep = xstep; e.ystep = ystep; e.bx0 = bx0; e.by0 = by0;
  e.pviewx = pviewx; e.pviewy = pviewy; e.phf = phf; e.gv = gv; e.shadeBase = shadeBase;
  /* gv lies in [0, 2^31) by construction; columns run from -159 to 160; the screen centre is within
   * +-2^30 for any pitch short of +-89.5 degrees */
  const i64 big = 1LL << 30;
  const bool narrow = phf >= 0 && phf < 2 * big && shadeBase > -big && shadeBase < big && v.center > -big && v.center < big &&
                      gd_max(bx0, -bx0) + 160 * gd_max(xstep, -xstep) < 2 * big &&
                      gd_max(by0, -by0) + 160 * gd_max(ystep, -ystep) < 2 * big && wbits > 0 && hbits > 0;
  n.phf = (int)phf; n.gv = (int)gv; n.shadeBase = (int)shadeBase;
  n.flags = (unsigned)(32 - wbits) | ((unsigned)(32 - hbits) << 8) | (narrow ? GD_PLANE_NARROW : 0u);
  n.bx0 = (int)bx0; n.xstep = (int)xstep; n.by0 = (int)by0; n.ystep = (int)ystep;
  n.pviewx = (unsigned)pviewx; n.pviewy = (unsigned)pviewy; n.tex = texel0; n.pad = 0;
}

__device__ __forceinline__ void gd_plane_setup(const GdScene &sc, const GdPlaneEntry *table, int sector, bool isFloor,
                                               int x, GdPlaneSpan &p) {
  const GdPlaneEntry &e = table[gd_secidx(sc, sector) * 2 + (isFloor ? 1 : 0)];
  i64 col = (i64)x - 159;
  p.wbits = e.wbits; p.hbits = e.hbits; p.texW = sc.texW;
  p.tex = e.tex;
  p.basex = e.bx0 + col * e.xstep;
  p.basey = e.by0 + col * e.ystep;
  p.pviewx = e.pviewx;
  p.pviewy = e.pviewy;
  p.phf = e.phf;
  p.gv = e.gv;
  p.shadeBase = e.shadeBase;
}

/* One visplane pixel (R_DrawSpan, engine.py:10879-10954), any operands. */
__device__ __forceinline__ unsigned gd_plane_pixel_wide(const GdScene &sc, const GdPlaneSpan &p, i64 center, int y) {
  const unsigned yslope = ((const unsigned *)(gd_smem + GD_OFF_YSLOPE))[y];
  i64 distance = gd_wmul(p.phf, (i64)yslope) >> 16;
  i64 xfrac = ((gd_wmul(distance, p.basex) >> 16) + p.pviewx) & GD_U32MASK;
  i64 yfrac = ((gd_wmul(distance, p.basey) >> 16) + p.pviewy) & GD_U32MASK;
  int u = (int)(xfrac >> (32 - p.wbits)), tv = (int)(yfrac >> (32 - p.hbits));
  uint8_t texel = sc.texAtlas[p.tex + (unsigned)(tv * p.texW + u)];
  i64 rowDist = center - (i64)y * GD_FU;
  if (rowDist < 0) rowDist = -rowDist;
  i64 vis = gd_min(gd_wmul(p.gv, rowDist) >> 16, 24 * GD_FU);
  int shade = (int)gd_clamp((p.shadeBase - vis) >> 16, 0, 31);
  return gd_smem[GD_OFF_COLORMAP + shade * 256 + texel];
}

__device__ __noinline__ unsigned gd_plane_pixel(const GdScene &sc_, const GdPlaneSpan &p, i64 center, int y) {
  return gd_plane_pixel_wide(*gd_as_shared(&sc_), p, center, y);
}

/* The same in 32-bit arithmetic: the span is narrow and |distance| < 2^31 for its rows (see
 * gd_walk).  vis = min(gv * rowDist >> 16, 24 * 65536) is 24 * 65536 exactly when the 64-bit product is
 * at least 0x18 << 32. */
struct GdNarrowSpan { unsigned phf, pviewx, pviewy, tex; int basex, basey, gv, shadeBase, xshift, yshift; };
__device__ __forceinline__ unsigned gd_plane_pixel_narrow(const GdNarrowSpan &p, const uint8_t *atlas, int texW, int center, int y) {
  const unsigned yslope = ((const unsigned *)(gd_smem + GD_OFF_YSLOPE))[y];
  const int distance = (int)(((unsigned long long)p.phf * yslope) >> 16);
  const unsigned xfrac = (unsigned)(((i64)distance * p.basex) >> 16) + p.pviewx;
  const unsigned yfrac = (unsigned)(((i64)distance * p.basey) >> 16) + p.pviewy;
  const unsigned texel = atlas[p.tex + (yfrac >> p.yshift) * (unsigned)texW + (xfrac >> p.xshift)];
  const i64 vis64 = (i64)p.gv * (i64)abs(center - (y << 16));
  const int vis = (unsigned)(vis64 >> 32) >= 0x18u ? 24 * 65536 : (int)(unsigned)(vis64 >> 16);
  const int shade = min(max((p.shadeBase - vis) >> 16, 0), 31);
  return gd_smem[GD_OFF_COLORMAP + shade * 256 + texel];
}

/* A column's mask of 208 rows is one word column in shared memory: word k of column x is m[k * GD_SW]. */
/* bits of mask word k (rows 32k..32k+31) that lie in rows [a,b) */
__device__ __forceinline__ unsigned gd_range_word(int k, int a, int b) {
  int lo = max(a - (k << 5), 0), hi = min(b - (k << 5), 32);
  if (lo >= hi) return 0u;
  unsigned upto = hi == 32 ? 0xffffffffu : ((1u << hi) - 1u);
  return upto & ~((1u << lo) - 1u);
}

/* rows of line w at column x: fragment aware in the instantiation for scenes with split lines */
template <bool kSplit>
__device__ __forceinline__ int gd_rows(const GdScene &sc, const GdView &v, const GdShared &sh, int w, float worldZ, int x) {
  if (kSplit) return gd_line_rows(sc, v, sh.walls, sh.frags, w, worldZ, x);
  return gd_project_rows(v, sh.walls[w], worldZ, x);
}

/* ---- phase: per-column portal walk (engine.py:11561-13371) -------------- */
struct GdColState {
  int cur;
  int ceilClip, floorClip;
  float prev;
  bool pendOwnerBoundary, pendEpBoundary, pendEpBridgeBoundary, pendPortalBridge;
  float pendOwnerEpX, pendOwnerEpY, pendEpEpX, pendEpEpY;
  int pendEpWall, pendEpBridgeIndex, pendPortalBridgeIndex, pendPortalBridgeSector;
  float pendPortalBridgeExit;
};

__device__ __forceinline__ bool gd_state_equal(const GdColState &a, const GdColState &b) {
  return a.cur == b.cur && a.ceilClip == b.ceilClip && a.floorClip == b.floorClip && a.prev == b.prev &&
         a.pendOwnerBoundary == b.pendOwnerBoundary && a.pendEpBoundary == b.pendEpBoundary &&
         a.pendEpBridgeBoundary == b.pendEpBridgeBoundary && a.pendPortalBridge == b.pendPortalBridge &&
         a.pendOwnerEpX == b.pendOwnerEpX && a.pendOwnerEpY == b.pendOwnerEpY && a.pendEpEpX == b.pendEpEpX &&
         a.pendEpEpY == b.pendEpEpY && a.pendEpWall == b.pendEpWall && a.pendEpBridgeIndex == b.pendEpBridgeIndex &&
         a.pendPortalBridgeIndex == b.pendPortalBridgeIndex &&
         a.pendPortalBridgeSector == b.pendPortalBridgeSector && a.pendPortalBridgeExit == b.pendPortalBridgeExit;
}

/* What one iteration decided for a column; the part other columns of its
 * aligned group of four need is exchanged with shuffles. */
struct GdIter {
  int wall, side;
  bool rasterValid, valid, oneSided;
  int renderCurrent, renderOther, otherSector;
  float distance;
  i64 vis;
  int ctop, cbot, cupbot, clowtop;
  bool tier[3];
  bool markCeil, markFloor;
  float viewFloor, viewCeil, otherFloor, otherCeil;
  int tex[3];
  /* traversal */
  bool nokpp, pskpp, usesGeo, entersOther, entersShared, endpointOnly, epb, cppb, geometric;
  int nopOther, psOther, gpOther;
  float nopDist, psDist, gpDist, osd;
  bool startsOwner, continuesOwner, pendEpHasFwd;
  float selEpX, selEpY, epEpX, epEpY;
  int epFwdIdx, ppbIdx, psPathIndex;
  bool psFromFront;
};

/* kSplit: the scene has lines a node builder split; the other instantiation carries none of that code */
template <bool kSplit>
__device__ __forceinline__ void gd_column_decide(const GdScene &sc, const GdView &v, const GdShared &sh, const GdWall *walls, const GdWall *frags,
                                                 const GdRowProj *rowproj, int x, float rx, float ry, const GdColState &c, GdIter &it) {
  const unsigned *ownerMask = (const unsigned *)(gd_smem + GD_OFF_OWNER);
  const int curSector = c.cur;
  const int current = GD_CHECK_SECTOR(curSector < 0 ? 0 : curSector, sc.S);
  const float prev = c.prev;
  const unsigned short *secOff = sh.secOff, *secWalls = sh.secWalls;
  const int i0 = secOff[current], i1 = secOff[current + 1];
#define ONE_SIDED(w) ((gd_hot(w).bits & GD_HOT_ONESIDED) != 0)
#define HIT(w) gd_hit_slow(sc, w, x, rx, ry)
#define HITK(k) HIT(secWalls[k])
  float distance = GD_INF;
  int wallIndex = 0;
  if (curSector >= 0) {
    /* nearest wall, and the nearest one-sided one, which goes first when it is within 1e-3 */
    float sd = GD_INF;
    int sw = 0;
#pragma unroll 1
    for (int k = i0; k < i1; ++k) {
      const int w = secWalls[k];
      const GdHit h = HIT(w);
      if (!(h.d > prev)) continue;
      if (h.d < distance) { distance = h.d; wallIndex = w; }
      if (h.d < sd && ONE_SIDED(w)) { sd = h.d; sw = w; }
    }
    if (fabsf(sd - distance) <= 1e-3f) { distance = sd; wallIndex = sw; }
  }
  GdHit hSel = HIT(wallIndex);
  const float *selWall = &sc.walls[wallIndex * 4];
  bool selUsesStart = hSel.along <= 0.5f;
  float selEpX = selUsesStart ? selWall[0] : selWall[2], selEpY = selUsesStart ? selWall[1] : selWall[3];
  int selVtx = gd_vertex(sc, wallIndex, selUsesStart ? 0 : 1);
#define SHARES_SEL(w) (gd_vertex(sc, w, 0) == selVtx || gd_vertex(sc, w, 1) == selVtx)
  bool continuesOwner = c.pendOwnerBoundary && selEpX == c.pendOwnerEpX && selEpY == c.pendOwnerEpY;
  bool continuesEp = c.pendEpBoundary && selEpX == c.pendEpEpX && selEpY == c.pendEpEpY;
  int selSlot = hSel.along > 0.5f;
  int epFwdIdx = 0;
  bool pendEpHasFwd = false;
  if (continuesEp) {
    bool m = gd_portal_bridge(sc, selSlot, wallIndex, c.pendEpWall, epFwdIdx);
    pendEpHasFwd = m && (HIT(epFwdIdx).d > distance + 1e-3f);
  }
  bool completesPendEpBridge = c.pendEpBridgeBoundary && wallIndex == c.pendEpBridgeIndex;
  bool selIsProjected = hSel.proj;
  bool selExclRight = walls[wallIndex].sr == x;
  float psPathDist = distance;
  int psPathIndex = wallIndex;
  float psd = GD_INF;
  int psi = 0;
  if (!selIsProjected) {
#pragma unroll 1
    for (int k = i0; k < i1; ++k) {
      int w = secWalls[k];
      if (!ONE_SIDED(w) || !SHARES_SEL(w)) continue;
      GdHit h = HITK(k);
      if (h.proj && h.left && (h.d > prev + 1e-3f) && h.d < psd) { psd = h.d; psi = w; }
    }
    if (selExclRight) {
      const int32_t *off = selUsesStart ? sc.sbStartOff : sc.sbEndOff;
      const int32_t *idx = selUsesStart ? sc.sbStartIdx : sc.sbEndIdx;
      float sbd = GD_INF;
      int sbi = wallIndex;
#pragma unroll 1
      for (int k = off[wallIndex]; k < off[wallIndex + 1]; ++k) {
        int b = GD_CHECK_INDEX(idx[k], sc.W);
        bool inc = gd_hot_front(b) == current || gd_hot_back(b) == current;
        if (!inc || !ONE_SIDED(b)) continue;
        GdHit h = HIT(b);
        if (h.proj && h.left && (h.d > prev + 1e-3f) && h.d < sbd) { sbd = h.d; sbi = b; }
      }
      if (sbd < psd) { psd = sbd; psi = sbi; }
    }
  }
  bool hasProjectedSolidOwner = isfinite(psd);
  if (hasProjectedSolidOwner) { distance = psd; wallIndex = psi; }
  GdHit hW = (wallIndex == psPathIndex) ? hSel : HIT(wallIndex);
  int seo = wallIndex;
  float sed = hW.d;
  if (!hW.proj) gd_endpoint_owner(sc, walls, wallIndex, x, rx, ry, hW, seo, sed);
  bool eoPathIsGeo = hW.geo;
  bool replaceEo = (seo != wallIndex) && (sed > prev + 1e-3f);
  if (replaceEo) { distance = sed; wallIndex = seo; hW = HIT(wallIndex); }
  int nopIndex = wallIndex;
  float nopDist = distance;
  bool nopIsGeo = replaceEo ? eoPathIsGeo : hW.geo;
  bool nopFromFront = curSector == gd_hot_front(nopIndex);
  int nopOther = nopFromFront ? gd_hot_back(nopIndex) : gd_hot_front(nopIndex);
  bool selOwnerIsProjected = hW.proj;
  bool selOwnerExclRight = walls[wallIndex].sr == x;
  i64 selOwnerSpan = walls[wallIndex].sr - walls[wallIndex].sl;
  bool selOwnerShort = sc.wlen[wallIndex] <= 32.0f;
  float npd = GD_INF;
  int npi = 0;
  if (!selOwnerIsProjected) {
#pragma unroll 1
    for (int k = i0; k < i1; ++k) {
      int w = secWalls[k];
      if (ONE_SIDED(w)) continue;
      GdHit h = HITK(k);
      if (!h.proj || !(h.d > prev + 1e-3f)) continue;
      bool topological = false;
      if (h.left && selOwnerExclRight && selOwnerSpan <= 2) {
        int sbIdx;
        topological = gd_sector_bridge(sc, h.along > 0.5f, w, nopIndex, sbIdx);
      }
      bool a = gd_same_pair(sc, wallIndex, w) ||
               (h.left && selOwnerExclRight && (selOwnerSpan <= 2 || (SHARES_SEL(w) && selOwnerShort)));
      bool nearOwner = (a && (fabsf(h.d - distance) <= gd_tol(h.d))) || topological;
      if (nearOwner && h.d < npd) { npd = h.d; npi = w; }
    }
  }
  /* projected sector bridge (engine.py:12073-12164) */
  const int pew = c.pendEpWall;
  bool peFromCur = curSector == gd_hot_front(pew);
  int peOther = peFromCur ? gd_hot_back(pew) : gd_hot_front(pew);
  bool usePsb = false;
  if (c.pendEpBoundary && !selOwnerIsProjected && selOwnerExclRight && nopIsGeo) {
    bool peIncident = peFromCur || curSector == gd_hot_back(pew);
    const float *peWall = &sc.walls[pew * 4];
    int peSlot = (c.pendEpEpX == peWall[2] && c.pendEpEpY == peWall[3]) ? 1 : 0;
    int psbIndex;
    bool psbExists = gd_sector_bridge(sc, peSlot, pew, nopIndex, psbIndex);
    if (psbExists && peIncident && peOther >= 0 && nopOther >= 0 && (walls[pew].sr - walls[pew].sl <= 1)) {
      int b0 = gd_hot_front(psbIndex), b1 = gd_hot_back(psbIndex);
      bool matches = (b0 == peOther && b1 == nopOther) || (b1 == peOther && b0 == nopOther);
      GdHit hb = HIT(psbIndex);
      GdHit hp = HIT(pew);
      bool psb = matches && hb.proj && hb.left && (hb.d > prev - gd_tol(hp.d)) && (hb.d < nopDist);
      if (psb && hb.d < npd) { usePsb = true; npd = hb.d; npi = psbIndex; }
    }
  }
  bool replaceNp = isfinite(npd);
  if (replaceNp) { distance = npd; wallIndex = npi; hW = HIT(wallIndex); }
  bool finalIsProjected = hW.proj, finalIsGeo = hW.geo;
  bool completesOpposing =
      c.pendEpBoundary && finalIsProjected && !finalIsGeo && gd_opposing_pair(sc, pew, wallIndex);
  bool valid = isfinite(distance);
  bool boundaryHasOwner = (ownerMask[x >> 5] >> (x & 31)) & 1u;
  bool exclTraversalOnly =
      !selOwnerIsProjected && selOwnerExclRight && !replaceNp && selOwnerSpan <= 2 && !boundaryHasOwner;
  bool rasterValid = valid && !exclTraversalOnly && !continuesOwner &&
                     !((pendEpHasFwd || completesPendEpBridge) && !selIsProjected && selExclRight && !replaceNp);
  bool geometric = replaceNp ? nopIsGeo : (replaceEo ? eoPathIsGeo : hW.geo);
  bool nokpp = replaceNp && nopIsGeo && nopOther >= 0;
  int front = gd_hot_front(wallIndex), back = gd_hot_back(wallIndex);
  bool fromFront = curSector == front;
  int otherSector = fromFront ? back : front;
  int renderCurrent = usePsb ? peOther : (completesOpposing ? otherSector : current);
  bool renderFromFront = renderCurrent == front;
  int renderOther = renderFromFront ? back : front;
  int side = renderFromFront ? 0 : 1;
  const GdWall &wv = walls[wallIndex];
  const bool splitLine = kSplit && gd_line_is_split(sc, wallIndex);      /* a node builder cut this line: the slow way */
  i64 vis = splitLine ? gd_line_vis(sc, walls, frags, wallIndex, side, x)
                      : wv.visL[side] + ((i64)x - wv.visSl[side]) * wv.visStep[side];
  bool psFromFront = curSector == gd_hot_front(psPathIndex);
  int psOther = psFromFront ? gd_hot_back(psPathIndex) : gd_hot_front(psPathIndex);
  bool pskpp = hasProjectedSolidOwner && hSel.geo && psOther >= 0;
  int safeOther = renderOther < 0 ? 0 : renderOther;
  float viewFloor = gd_sec_floor(sc, renderCurrent), viewCeil = gd_sec_ceil(sc, renderCurrent);
  float otherFloor = gd_sec_floor(sc, safeOther), otherCeil = gd_sec_ceil(sc, safeOther);
  bool oneSided = otherSector < 0;
  const int32_t *stex = &sc.sideTex[(wallIndex * 2 + side) * 3];
  /* Row bounds: per (wall, sector height) tables built once per lane cover the
   * usual case of heights taken from the wall's own two sectors. */
  const GdRowProj *rp = rowproj + wallIndex * 4;
  int slotCur = (renderCurrent == front) ? 0 : ((renderCurrent == back && back >= 0) ? 2 : -1);
  int oneTop = 0, oneBottom = 0;
  /* the row bounds feed tiers, marks, clips and events, all of which need a
   * raster-valid crossing */
  if (!rasterValid) {
  } else if (splitLine) {
    oneTop = gd_line_rows(sc, v, walls, frags, wallIndex, viewCeil, x);
    oneBottom = gd_line_rows(sc, v, walls, frags, wallIndex, viewFloor, x);
  } else if (slotCur >= 0) {
    oneBottom = gd_rowproj_eval(v, wv, rp[slotCur], x);
    oneTop = gd_rowproj_eval(v, wv, rp[slotCur + 1], x);
  } else {
    oneTop = gd_project_rows(v, wv, viewCeil, x);
    oneBottom = gd_project_rows(v, wv, viewFloor, x);
  }
  int lowerTop = 0, upperBottom = 0;
  if (!oneSided && rasterValid) {  /* the tiers and clips below use them only for two-sided lines */
    int slotOther = (renderOther >= 0 && renderOther == back) ? 2 : ((renderOther >= 0 && renderOther == front) ? 0 : -1);
    if (splitLine) {
      lowerTop = gd_line_rows(sc, v, walls, frags, wallIndex, otherFloor, x);
      upperBottom = gd_line_rows(sc, v, walls, frags, wallIndex, otherCeil, x);
    } else if (slotOther >= 0) {
      lowerTop = gd_rowproj_eval(v, wv, rp[slotOther], x);
      upperBottom = gd_rowproj_eval(v, wv, rp[slotOther + 1], x);
    } else {
      lowerTop = gd_project_rows(v, wv, otherFloor, x);
      upperBottom = gd_project_rows(v, wv, otherCeil, x);
    }
  }
  int ctop = max(oneTop, c.ceilClip), cbot = min(oneBottom, c.floorClip);
  int cupbot = max(min(upperBottom, c.floorClip), ctop);
  int clowtop = min(max(lowerTop, c.ceilClip), cbot);
  int4 ri = gd_sec_info(sc, renderCurrent), oi = gd_sec_info(sc, safeOther);
  bool lightDiff = ri.x != oi.x;
  it.markCeil = oneSided || viewCeil != otherCeil || ri.z != oi.z || lightDiff;
  it.markFloor = oneSided || viewFloor != otherFloor || ri.y != oi.y || lightDiff;
  it.wall = wallIndex; it.side = side; it.rasterValid = rasterValid; it.valid = valid;
  it.oneSided = oneSided; it.renderCurrent = renderCurrent; it.renderOther = renderOther; it.otherSector = otherSector;
  it.distance = distance; it.vis = vis;
  it.ctop = ctop; it.cbot = cbot; it.cupbot = cupbot; it.clowtop = clowtop;
  it.viewFloor = viewFloor; it.viewCeil = viewCeil; it.otherFloor = otherFloor; it.otherCeil = otherCeil;
  it.tex[0] = stex[0]; it.tex[1] = stex[1]; it.tex[2] = stex[2];
  it.tier[0] = oneSided && rasterValid && stex[0] >= 0 && ctop < cbot;
  it.tier[1] = !oneSided && rasterValid && (viewFloor < otherFloor) && stex[1] >= 0 && clowtop < cbot;
  it.tier[2] = !oneSided && rasterValid && (viewCeil > otherCeil) && stex[2] >= 0 && ctop < cupbot;

  /* traversal decisions (engine.py:13070-13241) */
  bool endpointOnly = valid && !oneSided && !geometric;
  float cnd = GD_INF, ond = GD_INF, csd = GD_INF, osd = GD_INF, gpd = GD_INF;
  int cni = 0, oni = 0, gpi = 0;
  const float prior = prev;
  if (endpointOnly) {
#pragma unroll 1
    for (int k = i0; k < i1; ++k) {
      int w = secWalls[k];
      GdHit h = HITK(k);
      bool os = ONE_SIDED(w);
      bool fut = (h.geo || (os && isfinite(h.d))) && (h.d > distance + 1e-3f);
      if (fut && h.d < cnd) { cnd = h.d; cni = w; }
      bool sharesEp = gd_shares_endpoint(sc, w, wallIndex);
      bool sharedSolid = isfinite(h.d) && os && (sharesEp || h.left) && (h.d > prior + 1e-3f) &&
                         (h.d <= distance + 1e-3f);
      if (sharedSolid && h.d < csd) csd = h.d;
      bool sgp = h.geo && sharesEp && !os && (h.d > prior + 1e-3f) && (fabsf(h.d - distance) <= (1.0f / 16.0f));
      if (sgp && h.d < gpd) { gpd = h.d; gpi = w; }
    }
    /* endpointOnly implies otherSector >= 0 */
#pragma unroll 1
    for (int k = secOff[otherSector]; k < secOff[otherSector + 1]; ++k) {
      int w = secWalls[k];
      GdHit h = HIT(w);
      bool os = ONE_SIDED(w);
      bool fut = (h.geo || (os && isfinite(h.d))) && (h.d > distance + 1e-3f);
      if (fut && h.d < ond) { ond = h.d; oni = w; }
      bool sharesEp = gd_shares_endpoint(sc, w, wallIndex);
      bool sharedSolid = isfinite(h.d) && os && (sharesEp || h.left) && (h.d > prior + 1e-3f) &&
                         (h.d <= distance + 1e-3f);
      if (sharedSolid && h.d < osd) osd = h.d;
    }
  }
  bool tied = endpointOnly && isfinite(cnd) && cni == oni && gd_opposing_pair(sc, wallIndex, cni);
  bool entersOther = endpointOnly && otherSector >= 0 && ((ond < cnd) || tied);
  bool entersShared = endpointOnly && otherSector >= 0 && (osd < csd);
  bool gpFromFront = curSector == gd_hot_front(gpi);
  int gpOther = gpFromFront ? gd_hot_back(gpi) : gd_hot_front(gpi);
  bool usesGeo = endpointOnly && isfinite(gpd) && gpOther >= 0;
  int ppbIdx = 0;
  bool epb = false;
  if (usesGeo) {
    GdHit hg = HIT(gpi);
    bool ppbExists = gd_portal_bridge(sc, hg.along > 0.5f, gpi, wallIndex, ppbIdx);
    if (ppbExists) {
      GdHit hb = HIT(ppbIdx);
      epb = hb.proj && hb.left && (hb.d > prior + 1e-3f) && (fabsf(hb.d - gpd) <= gd_tol(hg.d));
    }
  }
  it.cppb = valid && c.pendPortalBridge && wallIndex == c.pendPortalBridgeIndex;
  it.nokpp = nokpp; it.pskpp = pskpp; it.usesGeo = usesGeo; it.entersOther = entersOther;
  it.entersShared = entersShared; it.endpointOnly = endpointOnly; it.epb = epb; it.geometric = geometric;
  it.nopOther = nopOther; it.psOther = psOther; it.gpOther = gpOther;
  it.nopDist = nopDist; it.psDist = psPathDist; it.gpDist = gpd; it.osd = osd;
  it.startsOwner = replaceNp; it.continuesOwner = continuesOwner; it.pendEpHasFwd = pendEpHasFwd;
  it.selEpX = selEpX; it.selEpY = selEpY;
  {
    const float *fw = &sc.walls[wallIndex * 4];
    bool us = hW.along <= 0.5f;
    it.epEpX = us ? fw[0] : fw[2];
    it.epEpY = us ? fw[1] : fw[3];
  }
  it.epFwdIdx = epFwdIdx; it.ppbIdx = ppbIdx; it.psPathIndex = psPathIndex; it.psFromFront = psFromFront;
#undef HIT
#undef HITK
#undef ONE_SIDED
#undef SHARES_SEL
}

/* What one iteration of a column hands to the drawing code, whichever path decided it. */
struct GdCross {
  int wall, side;
  unsigned flags;                 /* GD_C_* */
  unsigned tops, bots;            /* clamped rows: ctop | clowtop << 16, (255 - cbot) | (255 - cupbot) << 16 */
  int vis;                        /* wallscan light, saturated (see gd_vis_clamp) */
  int rc, ro;                     /* sector this side, sector beyond (0 when there is none) */
  float dist;
  int cur;                        /* next sector and distance */
  float prev;
  bool pend, pendEnd, settled;
  bool portalFront;               /* GD_C_PORTAL: the crossed portal behind the projected solid */
  int portalWall, portalOther;
  float portalDist;
};

/* The light term is min(vis, 24 * 65536) taken from a base of magnitude below 2^30 and clamped to 31 shades:
 * anything below -2^30 is shade 31 either way. */
__device__ __forceinline__ int gd_vis_clamp(i64 vis) { return (int)gd_clamp(vis, -(1LL << 30), 24 * GD_FU); }
__device__ __forceinline__ int gd_shade_base(int light) { return 64 * (int)GD_FU - (light + 12) * (int)(GD_FU / 4); }
__device__ __forceinline__ int gd_shade(int base, int vis) { return min(max((base - vis) >> 16, 0), 31); }

/* One iteration of a column by the full set of rules, with its traversal update (engine.py:13242-13371).  About
 * one column in eighty needs it: next to a wall's end the projected span and the ray test disagree, or a rule
 * carried something over from the crossing before. */
template <bool kSplit>
__device__ __noinline__ void gd_slow_step(const GdScene &sc_, const GdView &v_, const GdShared &sh_, const GdRowProj *rowproj, int x, float rx, float ry, bool stopsOutside, GdColState &c,
                                          GdCross &o) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const GdView &v = *gd_as_shared(&v_);
  const GdShared &sh = *gd_as_shared(&sh_);
  const GdColState before = c;
  GdIter it;
  gd_column_decide<kSplit>(sc, v, sh, sh.walls, sh.frags, rowproj, x, rx, ry, c, it);
  o.wall = it.wall; o.side = it.side; o.rc = gd_secidx(sc, it.renderCurrent); o.dist = it.distance;
  o.ro = it.renderOther < 0 ? 0 : it.renderOther;
  o.tops = (unsigned)it.ctop | ((unsigned)it.clowtop << 16);
  o.bots = (unsigned)(255 - it.cbot) | ((unsigned)(255 - it.cupbot) << 16);
  o.vis = gd_vis_clamp(it.vis);
  o.flags = (it.rasterValid ? GD_C_RASTER : 0u) | (it.oneSided ? GD_C_ONE_SIDED : 0u) |
            (it.markCeil ? GD_C_MARK_CEIL : 0u) | (it.markFloor ? GD_C_MARK_FLOOR : 0u) |
            (it.viewFloor < it.otherFloor ? GD_C_LOWER : 0u) | (it.viewCeil > it.otherCeil ? GD_C_UPPER : 0u) |
            (it.tier[0] ? GD_C_TIER0 : 0u) | (it.tier[1] ? GD_C_TIER1 : 0u) | (it.tier[2] ? GD_C_TIER2 : 0u) |
            (it.viewFloor > it.otherFloor ? GD_C_FLOOR_ABOVE : 0u) | (it.viewCeil < it.otherCeil ? GD_C_CEIL_BELOW : 0u) |
            (it.pskpp ? GD_C_PORTAL : 0u);
  o.portalWall = it.psPathIndex; o.portalOther = it.psOther; o.portalFront = it.psFromFront; o.portalDist = it.psDist;
  /* traversal update */
  float prior = c.prev;
  float np = prior;
  if (it.valid) {
    if (it.nokpp) np = it.nopDist;
    else if (it.pskpp) np = it.psDist;
    else if (it.entersShared && (it.osd < it.distance)) np = prior;
    else if (it.usesGeo) np = it.gpDist;
    else np = it.distance;
  }
  if (it.valid && it.epb) np = prior;
  if (it.valid && it.cppb) np = fmaxf(it.distance, c.pendPortalBridgeExit);
  c.prev = np;
  if (it.startsOwner) { c.pendOwnerEpX = it.selEpX; c.pendOwnerEpY = it.selEpY; }
  c.pendOwnerBoundary = it.startsOwner || (c.pendOwnerBoundary && it.continuesOwner);
  if (it.endpointOnly) { c.pendEpEpX = it.epEpX; c.pendEpEpY = it.epEpY; c.pendEpWall = it.wall; }
  c.pendEpBoundary = it.endpointOnly;
  if (it.pendEpHasFwd) c.pendEpBridgeIndex = it.epFwdIdx;
  c.pendEpBridgeBoundary = it.pendEpHasFwd;
  int next;
  if (it.nokpp) next = it.nopOther;
  else if (it.pskpp) next = it.psOther;
  else if (it.usesGeo) next = it.gpOther;
  else if (it.valid && !it.oneSided && (it.geometric || it.entersOther || it.entersShared)) next = it.otherSector;
  else if (it.endpointOnly) next = c.cur;
  else next = -1;
  if (it.epb) next = it.otherSector;
  if (it.cppb) next = c.pendPortalBridgeSector;
  if (it.epb) {
    c.pendPortalBridgeIndex = it.ppbIdx;
    c.pendPortalBridgeSector = it.gpOther;
    c.pendPortalBridgeExit = it.gpDist;
  }
  c.pendPortalBridge = it.epb;
  c.cur = next;
  o.cur = next; o.prev = np;
  o.pendEnd = c.pendEpBoundary && !(c.pendOwnerBoundary || c.pendEpBridgeBoundary || c.pendPortalBridge);
  o.pend = c.pendOwnerBoundary || c.pendEpBoundary || c.pendEpBridgeBoundary || c.pendPortalBridge;
  /* A column that has left the map repeats the same decision on the same state forever; once an iteration
   * changes nothing and draws nothing it can stop. */
  o.settled = (before.cur < 0 && !it.rasterValid && !it.pskpp && gd_state_equal(before, c)) || (next < 0 && stopsOutside);
}

__device__ __forceinline__ void gd_put_event(GdEvent *events, int &nEvents, int x, float dist, int wall, int sector, unsigned tiers,
                                             unsigned sil, unsigned floor) {
  if (nEvents < GD_MAX_EVENTS) {
    unsigned *e = (unsigned *)&events[nEvents * GD_SW + x];
    e[0] = (unsigned)__float_as_int(dist);
    e[1] = ((unsigned)wall & 0xFFFFu) | ((unsigned)sector << 16);
    e[2] = tiers; e[3] = sil; e[4] = floor;
  }
  nEvents++;
}
static_assert(sizeof(GdEvent) == 20, "written as five words");

/* Clips contributed by the portal crossed behind a projected solid (engine.py:12965-13069). */
template <bool kSplit>
__device__ __noinline__ int2 gd_portal_clips(const GdScene &sc_, const GdView &v_, const GdShared &sh_, int x, const GdCross &o, int clips,
                                             GdEvent *events, int nEvents) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const GdView &v = *gd_as_shared(&v_);
  const GdShared &sh = *gd_as_shared(&sh_);
  int ceilClip = clips & 255, floorClip = clips >> 8;
  const int pIdx = o.portalWall;
  const int pSafeOther = o.portalOther < 0 ? 0 : o.portalOther;
  const float viewFloor = gd_sec_floor(sc, o.rc), viewCeil = gd_sec_ceil(sc, o.rc);
  const float pOtherFloor = gd_sec_floor(sc, pSafeOther), pOtherCeil = gd_sec_ceil(sc, pSafeOther);
  const int pSide = o.portalFront ? 0 : 1;
  const int32_t *ptex = &sc.sideTex[(pIdx * 2 + pSide) * 3];
  int pTop = gd_rows<kSplit>(sc, v, sh, pIdx, viewCeil, x), pBottom = gd_rows<kSplit>(sc, v, sh, pIdx, viewFloor, x);
  int pLowerTop = gd_rows<kSplit>(sc, v, sh, pIdx, pOtherFloor, x);
  int pUpperBottom = gd_rows<kSplit>(sc, v, sh, pIdx, pOtherCeil, x);
  int pct = max(pTop, ceilClip), pcb = min(pBottom, floorClip);
  int pcub = max(min(pUpperBottom, floorClip), pct);
  int pclt = min(max(pLowerTop, ceilClip), pcb);
  int4 ri = gd_sec_info(sc, o.rc), oi = gd_sec_info(sc, pSafeOther);
  bool ld = ri.x != oi.x;
  bool pDrawsUpper = (viewCeil > pOtherCeil) && ptex[2] >= 0;
  bool pMarksCeil = (viewCeil != pOtherCeil) || ri.z != oi.z || ld;
  if (pDrawsUpper || pMarksCeil) ceilClip = pDrawsUpper ? pcub : pct;
  bool pDrawsLower = (viewFloor < pOtherFloor) && ptex[1] >= 0;
  bool pMarksFloor = (viewFloor != pOtherFloor) || ri.y != oi.y || ld;
  if (pDrawsLower || pMarksFloor) floorClip = pDrawsLower ? pclt : pcb;
  bool pMasked = ptex[0] >= 0;
  bool pBottomSil = (viewFloor > pOtherFloor) || (v.viewZ < pOtherFloor) || pMasked;
  bool pTopSil = (viewCeil < pOtherCeil) || (v.viewZ > pOtherCeil) || pMasked;
  if ((pBottomSil || pTopSil) && events)
    gd_put_event(events, nEvents, x, o.portalDist, pIdx, -1, 0u,
                 (pTopSil ? (unsigned)ceilClip : 0u) | ((pBottomSil ? (unsigned)floorClip : 255u) << 8), 0u);
  return make_int2(ceilClip | (floorClip << 8), nEvents);
}

/* ---- what a column's crossings claim (engine.py:10879-10954, 12637-12884) ---------------------------------- */
/* Crossings narrow a window of open rows from above and below, and nearly every plane or tier continues the rows claimed
 * so far: [0, top) and [bottom, GD_VH).  Such a claim can meet no other, and its rows are drawn as one run.  (Looking
 * every claim up in masks of 32 rows, a bit at a time, took 30 of 322 million warp instructions of 1024 lanes; a step of 4096
 * lanes took 3282 us, now 3104.)  A claim that
 * does not continue them (a crossing behind a projected solid, tiers that overlap) makes the column loose for good: its rows
 * are told apart by masks, tiers before planes and then the first claim, as the reference has it.
 * Until then the column's mask holds the bounds of its tiers, a bit where a row differs from the one before; then it
 * holds the rows of its tiers, and one in scratch those of its planes (on chip for every column it took 9 KB of what is L1
 * now). */
__device__ __forceinline__ bool gd_claim_fits(int top, int bottom, int ya, int yb, bool above) {
  return above ? ya == top && yb <= bottom : yb == bottom && ya >= top;       /* top and bottom are -1 in a loose column */
}
__device__ __forceinline__ void gd_note_tier(unsigned *filled, int ya, int yb) {
  filled[(ya >> 5) * GD_SW] ^= 1u << (ya & 31);
  filled[(yb >> 5) * GD_SW] ^= 1u << (yb & 31);
}
static_assert(GD_VH >> 5 < 7, "the bit past the last row");

struct GdTierRun { unsigned texel, frac, step; int shift; };

/* A claim of a loose column, or the one that makes it loose (`bounds`: top | bottom << 8, else -1).  plane: its place in the
 * span table, or -1 for a tier; rows: ya | yb << 8 | excluded rows << 16, << 24; tails: rows from the first byte
 * on, and between the other two, have the second shade. */
__device__ __noinline__ void gd_loose_claim(const GdScene &sc_, const GdView &v_, const GdShared &sh_, int x, int bounds, int plane,
                                            GdTierRun t, unsigned rows, unsigned tails, unsigned shades) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const GdView &v = *gd_as_shared(&v_);
  const GdShared &sh = *gd_as_shared(&sh_);
  unsigned *filled = (unsigned *)(gd_smem + GD_OFF_MASKS) + x, *owned = sh.planeRows + x;
  if (bounds >= 0) {
    unsigned carry = 0u;
#pragma unroll 1
    for (int k = 0; k < 7; ++k) {
      unsigned m = filled[k * GD_SW];
      m ^= m << 1; m ^= m << 2; m ^= m << 4; m ^= m << 8; m ^= m << 16;
      m ^= carry;
      carry = m >> 31 ? ~0u : 0u;
      filled[k * GD_SW] = m;
      owned[k * GD_SW] = gd_range_word(k, 0, bounds & 255) | gd_range_word(k, bounds >> 8, GD_VH);
    }
  }
  GdPlaneSpan p;
  if (plane >= 0) gd_plane_setup(sc, sh.planeTab, plane >> 1, (plane & 1) != 0, x, p);
#pragma unroll 1
  for (int k = 0; k < 7; ++k) {
    unsigned m = gd_range_word(k, rows & 255u, (rows >> 8) & 255u) & ~gd_range_word(k, (rows >> 16) & 255u, rows >> 24);
    if (plane >= 0) {
      m &= ~owned[k * GD_SW];
      owned[k * GD_SW] |= m;
      m &= ~filled[k * GD_SW];
    } else {
      m &= ~filled[k * GD_SW];
      filled[k * GD_SW] |= m;
    }
    const unsigned tail = gd_range_word(k, tails & 255u, GD_VH) | gd_range_word(k, (tails >> 8) & 255u, (tails >> 16) & 255u);
#pragma unroll 1
    while (m) {
      const int b = __ffs(m) - 1, y = (k << 5) + b;
      m &= m - 1;
      unsigned pixel;
      if (plane >= 0) {
        pixel = gd_plane_pixel(sc, p, v.center, y);
      } else {
        const unsigned shade = (tail >> b) & 1u ? shades >> 8 : shades & 255u;
        pixel = gd_smem[GD_OFF_COLORMAP + shade * 256u + sc.texAtlasCol[t.texel + ((t.frac + (unsigned)y * t.step) >> t.shift)]];
      }
      sh.frame[y * GD_SW + x] = (uint8_t)pixel;
    }
  }
}

/* Rows [ya, yb) of column x for a plane whose operands need 64 bits, as all do whose rows lie on both sides of the horizon.
 * The span stays in registers: as an argument in local memory, 88 bytes a thread are more than the L1 beside the shared
 * memory holds (a plane that fills the view took 513 thousand cycles, with the masks before 146, now 82). */
__device__ __noinline__ void gd_plane_rows_wide(const GdScene &sc_, const GdView &v_, const GdShared &sh_, int x, int ya, int yb, int plane) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const GdView &v = *gd_as_shared(&v_);
  const GdShared &sh = *gd_as_shared(&sh_);
  const i64 center = v.center;
  uint8_t *frame = sh.frame;
  GdPlaneSpan p;
  gd_plane_setup(sc, sh.planeTab, plane >> 1, (plane & 1) != 0, x, p);
#pragma unroll 1
  for (int y = ya; y < yb; ++y) frame[y * GD_SW + x] = (uint8_t)gd_plane_pixel_wide(sc, p, center, y);
}

/* The mask that the fallback reads: a bit for every claimed row. */
__device__ __noinline__ void gd_claimed_rows(const GdShared &sh_, int x, int top, int bottom) {
  const GdShared &sh = *gd_as_shared(&sh_);
  unsigned *claimed = (unsigned *)(gd_smem + GD_OFF_MASKS) + x;
#pragma unroll 1
  for (int k = 0; k < 7; ++k)
    claimed[k * GD_SW] = top < 0 ? claimed[k * GD_SW] | sh.planeRows[k * GD_SW + x] : gd_range_word(k, 0, top) | gd_range_word(k, bottom, GD_VH);
}

/* ---- two-sided middle textures (engine.py:13424-13745) -----------------------
 * Replayed after the planes: per column the nearest projected crossing of a
 * line that carries a middle texture on the viewer's side, clipped by the
 * drawseg snapshot the walk left for that column. */
__device__ __forceinline__ i64 gd_masked_iscale(i64 swall) {
  i64 s = (swall * GD_FU) >> 18;
  if (s >= 0 && s < 3) return 3;
  if (s > -3 && s < 0) return -3;
  return s;
}

template <bool kSplit>
__device__ __noinline__ void gd_masked_pass(const GdScene &sc_, const GdView &v_, const GdShared &sh_) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const GdView &v = *gd_as_shared(&v_);
  const GdShared &sh = *gd_as_shared(&sh_);
  const int x = threadIdx.x;
  float rx, ry;
  gd_ray(v, x, rx, ry);
  float best = GD_INF;
  int w = -1, side = 0, texId = -1;
  bool leftEdge = false;
#pragma unroll 1
  for (int i = 0; i < sc.M; ++i) {
    const int k = GD_CHECK_INDEX(sc.maskedWalls[i], sc.W);
#ifndef GD_CHECKED
    const unsigned span = gd_hot(k).span;              /* the wall has to own the column */
    if (x < (int)(short)(span & 0xFFFFu) || x >= (int)(span >> 16)) continue;
#endif
    const int sd = (gd_hot(k).bits & GD_HOT_FRONT) ? 0 : 1;
    const int t = sc.sideTex[(k * 2 + sd) * 3];
    if (t < 0) continue;
#ifdef GD_CHECKED
    if (t >= sc.T) { atomicOr(gdCheckedStatus, GD_STATUS_BAD_INDEX); continue; }
#endif
    GdHit h = gd_hit_slow(sc, k, x, rx, ry);
    if (h.proj && h.d < best) { best = h.d; w = k; side = sd; texId = t; leftEdge = h.left; }
  }
  /* what this column drew, for the decal layer's depth test: the crossing's distance in
   * maskedDist (infinite: nothing), first row | end row << 8 in maskedInfo */
  if (!isfinite(best)) { sh.maskedDist[x] = GD_INF; return; }
  const GdWall &wv = sh.walls[w];
  const int front = gd_wsec(sc, w * 2), back = gd_wsec(sc, w * 2 + 1) < 0 ? 0 : gd_wsec(sc, w * 2 + 1);
  const int lightSector = side == 0 ? front : back;
  const float worldTop = fminf(gd_sec_ceil(sc, front), gd_sec_ceil(sc, back));
  const int4 ti = *reinterpret_cast<const int4 *>(&sc.texInfo[texId * 4]);
  const int tw = ti.x, th = ti.y, hbits = ti.w;
  const i64 owallTop = gd_rows<kSplit>(sc, v, sh, w, worldTop, x);
  const i64 owallBottom = gd_rows<kSplit>(sc, v, sh, w, worldTop - (float)th, x);
  const unsigned info = sh.maskedInfo[x];
  const bool hasSaved = (int)(info >> 16) == w;
  const i64 ceilClip = gd_max(owallTop, hasSaved ? (i64)((info >> 8) & 0xFF) : 0);
  const i64 floorClip = gd_min(owallBottom, hasSaved ? (i64)(info & 0xFF) : GD_VH);
  const float *soff = &sc.sideOff[(w * 2 + side) * 2];
  i64 hoff, vstepBase;
  gd_prep_wall(sc, wv, w, x, hoff, vstepBase);
  const i64 repeat = gd_rint(sc.wlen[w] * 65536.0f);
  if (side != 0) hoff = repeat - hoff;
  if (wv.sl > 0 && hoff < 0) hoff = 0;
  if (hoff >= repeat) hoff = repeat - 1;
  const int u = gd_pymod_width((hoff + gd_rint(soff[0] * 65536.0f)) >> 16, tw);
  const i64 vstep = vstepBase * (1LL << (14 - hbits));
  const i64 texMid = gd_rint((worldTop - v.viewZ) * 65536.0f + soff[1] * 65536.0f);
  /* R_DrawMaskedColumn: post rows from the drawseg's interpolated scale */
  const i64 sLeft = gd_clamp(wv.sl, 0, GD_SW - 1), sLast = gd_clamp(wv.sr - 1, 0, GD_SW - 1);
  i64 unused, startSwall, endSwall;
  gd_prep_wall(sc, wv, w, (int)sLeft, unused, startSwall);
  gd_prep_wall(sc, wv, w, (int)sLast, unused, endSwall);
  const i64 startScale = gd_div(1LL << 32, gd_masked_iscale(startSwall));
  const i64 endScale = gd_div(1LL << 32, gd_masked_iscale(endSwall));
  const i64 scaleStep = gd_div(endScale - startScale, gd_max(wv.sr - wv.sl, 1));
  const i64 spriteScale = startScale + gd_wmul(scaleStep, (i64)x - wv.sl);
  const i64 topScreen = v.center - (gd_wmul(texMid, spriteScale) >> 16);
  const i64 postTop = topScreen >> 16;
  const i64 postBottom = ((topScreen + gd_wmul(spriteScale, th) - GD_FU) >> 16) + 1;
  const i64 clippedTop = gd_max(postTop, ceilClip);
  i64 clippedBottom = gd_min(postBottom, floorClip);
  const i64 dcIscale = (vstepBase * GD_FU) >> 18;
  const i64 fracStart = texMid + gd_wmul(clippedTop, dcIscale) - (gd_wmul(v.center - GD_FU, dcIscale) >> 16);
  const i64 fracEnd = fracStart + gd_wmul(clippedBottom - clippedTop - 1, dcIscale);
  if (clippedTop < clippedBottom && clippedBottom < floorClip && fracEnd < (i64)th * GD_FU - dcIscale)
    clippedBottom += 1;
  if (!(hasSaved || leftEdge)) { sh.maskedDist[x] = GD_INF; return; }
  const float *wl = &sc.walls[w * 4];
  const bool horizontal = fabsf(wl[3] - wl[1]) < 1e-6f, vertical = fabsf(wl[2] - wl[0]) < 1e-6f;
  const i64 light = gd_sec_info(sc, lightSector).x + v.flashLight * 16 + (vertical ? 16 : (horizontal ? -16 : 0));
  const i64 vis = kSplit ? gd_line_vis(sc, sh.walls, sh.frags, w, side, x)
                         : wv.visL[side] + ((i64)x - wv.visSl[side]) * wv.visStep[side];
  const uint8_t *cm = sh.colormap + gd_wall_shade(light, vis) * 256;
  const uint8_t *col = sc.texAtlasCol + ((size_t)texId * sc.texW + u) * sc.texH;
  const unsigned base = (unsigned)(gd_shl(texMid, 16 - hbits) + (gd_wmul(vstep, GD_FU - v.center) >> 16));
  const unsigned step = (unsigned)vstep;
  const int rowA = (int)gd_max(clippedTop, 0), rowB = (int)gd_min(clippedBottom, GD_VH);
#pragma unroll 1
  for (int y = rowA; y < rowB; ++y)
    sh.frame[y * GD_SW + x] = cm[col[(base + (unsigned)y * step) >> (32 - hbits)]];
  sh.maskedDist[x] = rowA < rowB ? best : GD_INF;
  sh.maskedInfo[x] = (unsigned)max(rowA, 0) | ((unsigned)max(rowB, 0) << 8);
}

#define GD_FALLBACK_MAX (8 * GD_SW)
static_assert(GD_FALLBACK_MAX * 4 <= GD_AUX_BYTES, "the fallback queue");

/* A column that has left the map (current sector -1) still takes part in the reference's
 * vectorised iterations: its decision is made against sector 0 with wall 0 selected at an
 * infinite distance (engine.py:11561-11588 clamp the sector index).  That decision can only
 * become a valid crossing through a projected left-edge owner: a one-sided wall of sector 0
 * that shares an endpoint with wall 0 (engine.py:11905-11930), or a neighbour of wall 0 at one
 * of its endpoints (11589-11730), whose ray-owned span starts at this very column, or
 * through the rules that need
 * wall 0's projected span to end at this column (engine.py:11930-11962, 12073-12164).  Every
 * other column draws nothing, records nothing and changes nothing the frame depends on once
 * it is outside, so its walk can stop there.  This marks the columns that may have to go on; all these rules
 * ask for some wall whose projected span starts at the column, which the walk tests as well. */
__device__ void gd_mark_afterlife_columns(const GdScene &sc, const GdShared &sh) {
  unsigned *busy = sh.ownerMask + 16;
  const int n0 = sc.secOff[1] - sc.secOff[0];
  const int nb0 = sc.nbDirect ? 0 : sc.nbOff[0], nb1 = sc.nbDirect ? 2 : sc.nbOff[1];
  const int total = n0 + (nb1 - nb0) + 1;
#pragma unroll 1
  for (int i = threadIdx.x; i < total; i += GD_THREADS) {
    int xl;
    if (i == total - 1) {
      const i64 sr = sh.walls[0].sr;
      xl = (sr >= 0 && sr < GD_SW) ? (int)sr : -1;
    } else {
      int w = i < n0 ? sc.secWalls[sc.secOff[0] + i]
                     : (sc.nbDirect ? sc.nbDirectTab[i - n0] : sc.nbIdx[nb0 + (i - n0)]);
      if (w < 0) continue;                            /* no neighbour at that endpoint */
      w = GD_CHECK_INDEX(w, sc.W);
      if (i < n0 && (!(gd_hot(w).bits & GD_HOT_ONESIDED) || !gd_shares_endpoint(sc, w, 0))) continue;
      xl = (int)(short)(gd_hot(w).span & 0xFFFFu);
    }
    if (xl >= 0 && xl < GD_SW) atomicOr(&busy[xl >> 5], 1u << (xl & 31));
  }
}

/* ---- phase: per-column portal walk (engine.py:11561-13371) -------------- */
/* Thread x walks column x front to back; true: it is one of the slice's, and its mask tells which of its
 * rows are claimed; else all are.  Nearly every crossing is plain: nothing is carried over from the one
 * before, and the nearest wall of the current sector is both crossed by the column's ray and owned by its
 * projected span.  None of the ownership rules can then change the outcome: the owner rules ask for a selected
 * wall that is not projected here (engine.py:11589-11730, 11905-12164), the endpoint rules for one that is not
 * crossed (13070-13241), the bridges for something pending.  Such a crossing is decided below in one pass over
 * the sector's walls; every other one takes gd_slow_step.  What bounds the walk is instruction fetch and issue:
 * the loop is kept small enough for the instruction cache, and its operands are shared-memory tables at offsets
 * that are launch constants. */
/* Does the ray cross `wall` nearer to the endpoint (ex, ey) than to its other one (engine.py:11650-11668)? */
__device__ __noinline__ bool gd_meets_end(int wall, float rx, float ry, const float *walls, float ex, float ey) {
  const GdHot &h = gd_hot(wall);
  const bool usesStart = (h.offx * ry - h.offy * rx) / (rx * h.segy - ry * h.segx) <= 0.5f;
  const float2 e = *reinterpret_cast<const float2 *>(&walls[wall * 4 + (usesStart ? 0 : 2)]);
  return e.x == ex && e.y == ey;
}

/* The ray of column x crosses wall `sel`, the nearest of the sector, but its projected span does not own the column, and
 * nothing is pending.  True when no rule can hand the crossing to another wall (a superset of their conditions, without
 * the distances): no one-sided wall of the sector at the same vertex, and none that may own the columns past the wall's
 * end, starts its span here (engine.py:11905-11962), no line between the same two sectors touches it (11589-11730), no
 * wall that owns the column is between the same sectors or takes over past a short line's right end (12005-12072), and
 * the line is not itself too narrow to draw. */
__device__ __noinline__ bool gd_quiet_crossing(const GdScene &sc_, const unsigned short *secWalls, int k0, int k1, int sel, int x,
                                               float rx, float ry, bool spanStarts) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const GdHot s = gd_hot(sel);
  const bool endsHere = GD_HOT_SR(s.bits) == x;
  /* the clamped span is never wider than the real one */
  if (endsHere && GD_HOT_SR(s.bits) - GD_HOT_SL(s.bits) <= 2) return false;
  int vertex = -1;
  if (spanStarts) {
    if (s.bits & GD_HOT_NEIGHBOUR) return false;
    if (endsHere && sc.wlen[sel] <= 32.0f) return false;
    const bool usesStart = (s.offx * ry - s.offy * rx) / (rx * s.segy - ry * s.segx) <= 0.5f;
    vertex = gd_vertex(sc, sel, usesStart ? 0 : 1);
    if (endsHere && (s.bits & (usesStart ? GD_HOT_BRIDGE0 : GD_HOT_BRIDGE1))) {
      const int32_t *off = usesStart ? sc.sbStartOff : sc.sbEndOff, *idx = usesStart ? sc.sbStartIdx : sc.sbEndIdx;
#pragma unroll 1
      for (int k = off[sel]; k < off[sel + 1]; ++k) {
        const GdHot &h = gd_hot(GD_CHECK_INDEX(idx[k], sc.W));
        if ((h.bits & GD_HOT_ONESIDED) && x == (int)(short)(h.span & 0xFFFFu) && x < (int)(h.span >> 16) && gd_ray_meets_line(h, rx, ry)) return false;
      }
    }
  }
  const int swapped = (int)(((unsigned)s.secs << 16) | ((unsigned)s.secs >> 16));
#pragma unroll 1
  for (int k = k0; k < k1; ++k) {
    const int w = secWalls[k];
    const GdHot &h = gd_hot(w);
    const int isl = (int)(short)(h.span & 0xFFFFu);
    if (w == sel || x < isl || x >= (int)(h.span >> 16) || !gd_ray_meets_line(h, rx, ry)) continue;
    if (h.bits & GD_HOT_ONESIDED) {
      if (x == isl && (gd_vertex(sc, w, 0) == vertex || gd_vertex(sc, w, 1) == vertex)) return false;
    } else if (h.secs == s.secs || h.secs == swapped) {
      return false;
    }
  }
  return true;
}

__device__ __noinline__ int gd_light_wide(const GdWall &wv, int side, int x) {
  return gd_vis_clamp(wv.visL[side] + gd_wmul((i64)x - wv.visSl[side], wv.visStep[side]));
}

/* Row bounds of a column outside the wall's projected span: the whole-wall projection (engine.py:12393-12410).
 * Returns floor | ceiling << 8 of this side and of the side beyond, and the light. */
__device__ __noinline__ uint3 gd_rows_outside(const GdView &v_, const GdWall &wv, const GdRowProj *rp, int side, bool beyond, int x) {
  const GdView &v = *gd_as_shared(&v_);
  const i64 column = (i64)x - wv.sl;
  unsigned r[2] = {0u, 0u};
#pragma unroll 1
  for (int k = 0; k < (beyond ? 4 : 2); ++k) {
    const GdRowProj &q = rp[((k >> 1) ^ side) * 2 + (k & 1)];
    r[k >> 1] |= (unsigned)gd_clamp((v.center + q.opl + gd_wmul(column, q.ostep)) >> 16, 0, GD_VH) << (8 * (k & 1));
  }
  return make_uint3(r[0], r[1], (unsigned)gd_light_wide(wv, side, x));
}

template <bool kSplit, bool kChip>
__device__ __forceinline__ bool gd_walk(const GdParams &p, const GdScene &sc, const GdView &v, const GdShared &sh, uint8_t *frame,
                                        uint8_t *tables, GdEvent *events, int *eventCount, const GdRowProj *rowproj, int startSector, bool mine) {
  const int x = threadIdx.x;
  const int quadBase = x & 28;
  const unsigned quad = 15u << quadBase;
  float rx, ry;
  gd_ray(v, x, rx, ry);
  const GdRow *rows = (const GdRow *)(kChip ? gd_smem + p.offRows : tables + p.offRows);
  const GdRow *fragRows = kChip ? rows + p.sc.W * 4 : (const GdRow *)(p.frags + blockIdx.x * p.fragStride + gd_frag_rows(p.sc.F));
  const float4 *prep = (const float4 *)(kChip ? gd_smem + p.offPrep : tables + p.offPrep);
  const GdPlane *planes = (const GdPlane *)(kChip ? gd_smem + p.offPlanes : tables + p.offPlanes);
  const GdSide *sides = kChip ? (const GdSide *)(gd_smem + p.offSides) : p.sides;
  const float4 *sectors = (const float4 *)(gd_smem + p.offSectors);
  const unsigned short *secOff = (const unsigned short *)(gd_smem + p.offSecOff), *secWalls = (const unsigned short *)(gd_smem + p.offSecWalls);
  const unsigned *yslope = (const unsigned *)(gd_smem + GD_OFF_YSLOPE);
  unsigned *filled = (unsigned *)(gd_smem + GD_OFF_MASKS) + x;
#pragma unroll
  for (int k = 0; k < 7; ++k) filled[k * GD_SW] = 0;
  int top = 0, bottom = GD_VH;      /* the rows not in between are claimed; -1: the masks tell */
  float *maskedDist = (float *)(gd_smem + GD_OFF_MASKED_DIST) + x;
  unsigned *maskedInfo = (unsigned *)(gd_smem + GD_OFF_MASKED_INFO) + x;
  if (p.sc.M > 0) { *maskedDist = GD_INF; *maskedInfo = 0xFFFF0000u | GD_VH; }
  GdColState c;                     /* read and written by the slow path only */
  c.pendOwnerBoundary = c.pendEpBoundary = c.pendEpBridgeBoundary = c.pendPortalBridge = false;
  c.pendOwnerEpX = c.pendOwnerEpY = c.pendEpEpX = c.pendEpEpY = 0.0f;
  c.pendEpWall = c.pendEpBridgeIndex = c.pendPortalBridgeIndex = 0;
  c.pendPortalBridgeSector = -1;
  c.pendPortalBridgeExit = 0.0f;
  GdCross o;
  int cur = startSector, ceilClip = 0, floorClip = GD_VH;
  float prev = 0.0f;
  bool pend = false, settled = !mine;
  bool pendEnd = false;             /* all that is pending is that the last crossing met a wall's end only */
  const unsigned *columns = (const unsigned *)(gd_smem + GD_OFF_OWNER) + (x >> 5);
  const bool spanStarts = (columns[32] >> (x & 31)) & 1u;         /* some wall's projected span starts here */
  const bool stopsOutside = !(spanStarts && ((columns[16] >> (x & 31)) & 1u));
  /* clip events are read where sprites or chips may cover the column */
  const bool wantEvents = p.decals != nullptr || ((const unsigned long long *)(gd_smem + GD_OFF_CAND))[x] != 0;
  int nEvents = 0;

#pragma unroll 1
  for (int iter = 0; iter < p.sc.S; ++iter) {
    if (__all_sync(0xffffffffu, settled)) break;
    const bool active = !settled;
    int wall = -1 - x, side = 0, vis = 0, rc = 0, ro = 0, next = -1;
    unsigned flags = 0, tops = 0, bots = 0;
    float dist = 0.0f, nextPrev = 0.0f;
    if (active) {
      bool slow = (pend && !pendEnd) || cur < 0;
      if (!slow) {
        /* nearest wall beyond prev; a one-sided one within 1e-3 of it goes first (engine.py:11589-11640) */
        float best = GD_INF, solid = GD_INF;
        unsigned bestTag = 0, solidTag = 0;           /* wall | 1 << 31: crossed by the ray | 1 << 30: owned by the projected span */
        const int k1 = secOff[cur + 1];
#pragma unroll 1
        for (int k = secOff[cur]; k < k1; ++k) {
          const int w = secWalls[k];
          const float4 g = *reinterpret_cast<const float4 *>(&gd_hot(w));
          const int4 h = *(reinterpret_cast<const int4 *>(&gd_hot(w)) + 1);
          const float dn = __int_as_float(h.x);
          const float den = rx * g.y - ry * g.x;
          if (fabsf(den) < 1e-6f || dn == 0.0f || (dn < 0) != (den < 0)) continue;
          const float an = g.z * ry - g.w * rx;
          const bool geo = an == 0.0f || ((an < 0) == (den < 0) && fabsf(an) <= fabsf(den));
          const bool proj = x >= (int)(short)(h.y & 0xFFFF) && x < (int)((unsigned)h.y >> 16);
          const bool oneSided = ((unsigned)h.w & GD_HOT_ONESIDED) != 0;
          if (!(oneSided ? (proj && ((unsigned)h.w & GD_HOT_FRONT)) : (geo || proj))) continue;
          const float d = dn / den;
          if (!(d > prev)) continue;
          const unsigned tag = (unsigned)w | (geo ? 0x80000000u : 0u) | (proj ? 0x40000000u : 0u);
          if (d < best) { best = d; bestTag = tag; }
          if (oneSided && d < solid) { solid = d; solidTag = tag; }
        }
        if (fabsf(solid - best) <= 1e-3f) { best = solid; bestTag = solidTag; }
        wall = (int)(bestTag & 0x3FFFFFFFu);
        const unsigned kind = bestTag >> 30;          /* 3: crossed and owned, 2: crossed, 1: owned, 0: nothing beyond prev */
        if (kind == 3u) slow = pendEnd && gd_meets_end(wall, rx, ry, p.sc.walls, c.pendEpEpX, c.pendEpEpY);
        else if (pendEnd) slow = true;
        else if (kind == 2u) slow = !gd_quiet_crossing(sc, secWalls, secOff[cur], k1, wall, x, rx, ry, spanStarts);
        else if (kind == 1u) slow = !(gd_hot(wall).bits & GD_HOT_ONESIDED);     /* a one-sided end of the column either way */
        else slow = !stopsOutside;
        if (!slow && kind == 0u) {
          /* no wall of the sector is left and nothing is pending: the rules start from wall 0 at an infinite distance
           * like those of a column outside the map, and of the sector's walls none can take over, because a
           * projected one would have been found.  What can is a neighbour of wall 0 whose span starts here
           * (engine.py:11650-11730), which gd_mark_afterlife_columns marks; every other column leaves the map.
           * (Any span's start used to send the column to gd_slow_step: 5.7 of 9 such steps per lane of the
           * 64-sector map, each a warp's wait of 28 thousand cycles.) */
          wall = -1 - x;
        } else
        if (!slow) {
          const int secs = gd_hot(wall).secs;
          const unsigned bits = gd_hot(wall).bits;
          const int front = (int)(short)(secs & 0xFFFF), back = secs >> 16;
          side = cur == front ? 0 : 1;
          const int other = side ? front : back;
          const GdRow *unit = rows + wall * 4;
          if (kSplit && (bits & GD_HOT_SPLIT)) {
            /* the first fragment whose half-open span holds the column (engine.py:12310-12376) */
            const unsigned *spans = (const unsigned *)(gd_smem + p.offFrags);
            const int f1 = p.sc.fragOff[wall + 1];
            int f = p.sc.fragOff[wall];
#pragma unroll 1
            for (; f < f1; ++f)
              if (x >= (int)(spans[f] & 0xFFFFu) && x < (int)(spans[f] >> 16)) break;
            unit = f < f1 ? fragRows + f * 4 : nullptr;      /* none: the whole line's projection */
          } else {
            if (x < GD_HOT_SL(bits) || x >= GD_HOT_SR(bits)) unit = nullptr;
          }
          slow = side && cur != back;
          if (!slow) {
            unsigned wide = 0u;
            int bottom, top, beyondBottom = 0, beyondTop = 0;
            if (unit) {
              const GdRow rf = unit[side * 2], rt = unit[side * 2 + 1];
              wide = rf.lim | rt.lim;
              bottom = gd_row_eval(rf, x); top = gd_row_eval(rt, x);
              vis = min((int)((unsigned)rf.vis + (unsigned)x * (unsigned)rt.vis), 24 * (int)GD_FU);
              if (rf.lim & GD_ROW_LIGHT_WIDE)
                vis = gd_light_wide(kSplit && (bits & GD_HOT_SPLIT) ? sh.frags[(unit - fragRows) >> 2] : sh.walls[wall], side, x);
              if (other >= 0) {
                const GdRow ol = unit[(side ^ 1) * 2], ou = unit[(side ^ 1) * 2 + 1];
                wide |= ol.lim | ou.lim;
                beyondBottom = gd_row_eval(ol, x); beyondTop = gd_row_eval(ou, x);
              }
            } else {
              const uint3 r = gd_rows_outside(v, sh.walls[wall], rowproj + wall * 4, side, other >= 0, x);
              bottom = r.x & 255u; top = (r.x >> 8) & 255u;
              beyondBottom = r.y & 255u; beyondTop = (r.y >> 8) & 255u;
              vis = (int)r.z;
            }
            const GdSide &sd = sides[wall * 2 + side];
            flags = sd.flags;
            const int ctop = max(top, ceilClip), cbot = min(bottom, floorClip);
            int cupbot = ctop, clowtop = cbot;
            if (other >= 0) {
              clowtop = min(max(beyondBottom, ceilClip), cbot);
              cupbot = max(min(beyondTop, floorClip), ctop);
            }
            slow = (wide & GD_ROW_WIDE) != 0;
            tops = (unsigned)ctop | ((unsigned)clowtop << 16);
            bots = (unsigned)(255 - cbot) | ((unsigned)(255 - cupbot) << 16);
            /* the static flags name the tiers that have a texture; they need rows as well */
            if (ctop >= cbot) flags &= ~GD_C_TIER0;
            if (clowtop >= cbot) flags &= ~GD_C_TIER1;
            if (ctop >= cupbot) flags &= ~GD_C_TIER2;
            rc = cur; ro = other < 0 ? 0 : other;
            dist = best;
            next = other; nextPrev = best;
          }
        }
      }
      if (slow) {
        c.cur = cur; c.prev = prev; c.ceilClip = ceilClip; c.floorClip = floorClip;
        gd_slow_step<kSplit>(sc, v, sh, rowproj, x, rx, ry, stopsOutside, c, o);
        wall = o.wall; side = o.side; flags = o.flags; tops = o.tops; bots = o.bots; vis = o.vis; rc = o.rc; ro = o.ro;
        dist = o.dist; next = o.cur; nextPrev = o.prev; pend = o.pend; pendEnd = o.pendEnd; settled = o.settled;
      } else {
        settled = next < 0 && stopsOutside;
        if (pend) { pend = pendEnd = false; c.pendEpBoundary = false; }
      }
    }
    /* aligned four-column wallscan groups (engine.py:12694-12761): tops and bottoms travel as byte maxima */
    const int key = wall * 2 + side;
    const bool same = (__ballot_sync(0xffffffffu, key == __shfl_sync(0xffffffffu, key, quadBase)) & quad) == quad;
    const bool all0 = (__ballot_sync(0xffffffffu, (flags & GD_C_TIER0) != 0) & quad) == quad;
    const bool all1 = (__ballot_sync(0xffffffffu, (flags & GD_C_TIER1) != 0) & quad) == quad;
    const bool all2 = (__ballot_sync(0xffffffffu, (flags & GD_C_TIER2) != 0) & quad) == quad;
    unsigned topMax = __vmaxu2(tops, __shfl_xor_sync(0xffffffffu, tops, 1)), botMax = __vmaxu2(bots, __shfl_xor_sync(0xffffffffu, bots, 1));
    topMax = __vmaxu2(topMax, __shfl_xor_sync(0xffffffffu, topMax, 2));
    botMax = __vmaxu2(botMax, __shfl_xor_sync(0xffffffffu, botMax, 2));
    const int firstVis = __shfl_sync(0xffffffffu, vis, quadBase);
    if (!active) continue;

    if (flags & GD_C_RASTER) {
      const int ctop = (int)(tops & 0xFFFFu), clowtop = (int)(tops >> 16), cbot = 255 - (int)(bots & 0xFFFFu), cupbot = 255 - (int)(bots >> 16);
      const int oldCeil = ceilClip, oldFloor = floorClip;
      const float4 here = sectors[rc], there = sectors[ro];    /* floor, ceiling, light */
      const int centerRow = (int)(v.center >> 16);
      /* visplane rows uncovered by this seg (engine.py:12637-12655) */
#pragma unroll 1
      for (int q = 0; q < 2; ++q) {
        const bool isFloor = q == 0;
        const int ya = isFloor ? max(cbot, ceilClip) : ceilClip, yb = isFloor ? floorClip : min(ctop, floorClip);
        if (!(flags & (isFloor ? GD_C_MARK_FLOOR : GD_C_MARK_CEIL)) || ya >= yb) continue;
        const int plane = rc * 2 + (isFloor ? 1 : 0);
        if (!gd_claim_fits(top, bottom, ya, yb, !isFloor)) {
          gd_loose_claim(sc, v, sh, x, top < 0 ? -1 : top | (bottom << 8), plane, GdTierRun{0u, 0u, 0u, 0},
                         (unsigned)ya | ((unsigned)yb << 8), 255u, 0u);
          top = bottom = -1;
          continue;
        }
        if (isFloor) bottom = ya; else top = yb;
        const int4 *e = reinterpret_cast<const int4 *>(&planes[plane]);
        const int4 e0 = e[0];
        /* rows lie farther from the viewer towards the horizon: the row that bounds the span's distance */
        const unsigned far = ya > centerRow ? yslope[ya] : (yb <= centerRow ? yslope[yb - 1] : 0xffffffffu);
        if (!((unsigned)e0.w & GD_PLANE_NARROW) || ((unsigned long long)(unsigned)e0.x * far) >> 47) {
          gd_plane_rows_wide(sc, v, sh, x, ya, yb, plane);
          continue;
        }
        const int4 e1 = e[1], e2 = e[2];
        GdNarrowSpan s;
        s.phf = (unsigned)e0.x; s.gv = e0.y; s.shadeBase = e0.z;
        s.xshift = e0.w & 63; s.yshift = (e0.w >> 8) & 63;
        s.basex = e1.x + (x - 159) * e1.y; s.basey = e1.z + (x - 159) * e1.w;
        s.pviewx = (unsigned)e2.x; s.pviewy = (unsigned)e2.y; s.tex = (unsigned)e2.z;
        const int center = (int)v.center;
        /* two rows per trip; an odd last row is simply drawn twice */
#pragma unroll 1
        for (int y = ya; y < yb; y += 2) {
          const int y1 = min(y + 1, yb - 1);
          const unsigned p0 = gd_plane_pixel_narrow(s, p.sc.texAtlas, p.sc.texW, center, y);
          const unsigned p1 = gd_plane_pixel_narrow(s, p.sc.texAtlas, p.sc.texW, center, y1);
          frame[(unsigned)(y * GD_SW + x)] = (uint8_t)p0;
          frame[(unsigned)(y1 * GD_SW + x)] = (uint8_t)p1;
        }
      }
      /* wall tiers: middle or lower first, then upper; the lower one has priority where they overlap
       * (engine.py:12762-12884) */
      const GdSide &sd = sides[wall * 2 + side];
      const bool oneSided = (flags & GD_C_ONE_SIDED) != 0;
      const bool lowRange = !oneSided && (flags & GD_C_LOWER) && clowtop < cbot, upRange = !oneSided && (flags & GD_C_UPPER) && ctop < cupbot;
      if (flags & (GD_C_TIER0 | GD_C_TIER1 | GD_C_TIER2)) {
        /* the sector beyond has its ceiling below its floor: the rows that both ranges hold are the lower one's, drawn or
         * not, and take the second shade of either, so neither tier is one run */
        const bool meet = lowRange && upRange && clowtop < cupbot;
        const i64 repeat = sd.repeat;
        i64 hoff, vstepBase;
        gd_prep_eval(prep[wall], repeat, x, hoff, vstepBase);
        if (side != 0) hoff = repeat - hoff;
        if (GD_HOT_SL(gd_hot(wall).bits) > 0 && hoff < 0) hoff = 0;
        if (hoff >= repeat) hoff = repeat - 1;
        const i64 column = (hoff + sd.tox) >> 16;
        const int base = gd_shade_base(__float_as_int(here.z) + v.flashLight * 16 + sd.contrast);
        const unsigned shadeN = (unsigned)gd_shade(base, vis), shadeT = (unsigned)gd_shade(base, firstVis);
#pragma unroll 1
        for (int q = 0; q < 2; ++q) {
          const bool upper = q == 1;
          if (!(flags & (upper ? GD_C_TIER2 : (oneSided ? GD_C_TIER0 : GD_C_TIER1)))) continue;
          const int texId = sd.tex[upper ? 2 : (oneSided ? 0 : 1)];
#ifdef GD_CHECKED
          if (texId >= sc.T) {                         /* the tier stays undrawn, and its rows are nobody's */
            atomicOr(gdCheckedStatus, GD_STATUS_BAD_INDEX);
            gd_loose_claim(sc, v, sh, x, top < 0 ? -1 : top | (bottom << 8), -1, GdTierRun{0u, 0u, 0u, 0}, 0u, 255u, 0u);
            top = bottom = -1;
            continue;
          }
#endif
          const int ya = upper || oneSided ? ctop : clowtop, yb = upper ? cupbot : cbot;
          const float originZ = upper ? there.y : (oneSided ? here.y : there.x);
          /* rows lit with the group's first-column light: below the group's highest bottom */
          const int gb0 = 255 - (int)(botMax & 0xFFFFu), gb2 = 255 - (int)(botMax >> 16);
          const bool group2 = same && all2 && (int)(topMax & 0xFFFFu) < gb2;
          const bool group = upper ? group2 : (same && (oneSided ? (all0 && (int)(topMax & 0xFFFFu) < gb0) : (all1 && (int)(topMax >> 16) < gb0)));
          const int tailA = group && shadeN != shadeT ? (upper ? gb2 : gb0) : GD_VH;
          const int4 ti = *reinterpret_cast<const int4 *>(&p.sc.texInfo[texId * 4]);
          const int hbits = ti.w;
          const unsigned u = (unsigned)gd_pymod_width(column, ti.x);
          const i64 vstep = vstepBase * (1LL << (14 - hbits));
          const i64 texMid = gd_rint((originZ - v.viewZ) * 65536.0f + sd.yoff * 65536.0f);
          /* frac(y) = (texMid << (16-bits)) + ((vstep * (y*FU - center + FU)) >> 16); the
           * y term is a multiple of 2^16 inside the shift, so it steps by vstep exactly. */
          GdTierRun t;
          t.frac = (unsigned)(gd_shl(texMid, 16 - hbits) + (gd_wmul(vstep, GD_FU - v.center) >> 16));
          t.step = (unsigned)vstep;
          t.texel = ((unsigned)texId * (unsigned)p.sc.texW + u) * (unsigned)p.sc.texH;
          t.shift = 32 - hbits;
          if (meet || !gd_claim_fits(top, bottom, ya, yb, upper || oneSided)) {
            const bool otherTail = !upper && !oneSided && upRange && group2 && shadeN != shadeT;
            const unsigned oTailA = otherTail ? (unsigned)max(ctop, gb2) : 0u, oTailB = otherTail ? (unsigned)cupbot : 0u;
            gd_loose_claim(sc, v, sh, x, top < 0 ? -1 : top | (bottom << 8), -1, t,
                           (unsigned)ya | ((unsigned)yb << 8) | (upper && lowRange ? ((unsigned)clowtop << 16) | ((unsigned)cbot << 24) : 0u),
                           (unsigned)tailA | (oTailA << 8) | (oTailB << 16), shadeN | (shadeT << 8));
            top = bottom = -1;
            continue;
          }
          if (upper || oneSided) top = yb; else bottom = ya;
          gd_note_tier(filled, ya, yb);
          const unsigned cmN = shadeN * 256u, cmT = shadeT * 256u;
          unsigned f = t.frac + (unsigned)ya * t.step;
#pragma unroll 1
          for (int y = ya; y < yb; y += 2) {
            const int odd = y + 1 < yb ? 1 : 0;
            const unsigned f1 = odd ? f + t.step : f;
            const unsigned t0 = p.sc.texAtlasCol[t.texel + (f >> t.shift)], t1 = p.sc.texAtlasCol[t.texel + (f1 >> t.shift)];
            f += 2u * t.step;
            frame[(unsigned)(y * GD_SW + x)] = gd_smem[GD_OFF_COLORMAP + (y >= tailA ? cmT : cmN) + t0];
            frame[(unsigned)((y + odd) * GD_SW + x)] = gd_smem[GD_OFF_COLORMAP + (y + odd >= tailA ? cmT : cmN) + t1];
          }
        }
      }
      /* clip updates (engine.py:12885-12913) */
      const bool masked = sd.tex[0] >= 0;
      if (!oneSided) {
        const bool drawsUpper = (flags & GD_C_UPPER) && sd.tex[2] >= 0, drawsLower = (flags & GD_C_LOWER) && sd.tex[1] >= 0;
        if (drawsUpper || (flags & GD_C_MARK_CEIL)) ceilClip = drawsUpper ? cupbot : ctop;
        if (drawsLower || (flags & GD_C_MARK_FLOOR)) floorClip = drawsLower ? clowtop : cbot;
        /* masked drawseg snapshot (engine.py:12914-12939) */
        if (masked && p.sc.M > 0 && dist < *maskedDist) {
          *maskedDist = dist;
          *maskedInfo = ((unsigned)wall << 16) | ((unsigned)ceilClip << 8) | (unsigned)floorClip;
        }
      }
      if (wantEvents) {
        /* sprite silhouettes (engine.py:12940-12964); a crossing that draws, marks and clips nothing leaves no trace */
        const bool bottomSil = !oneSided && ((flags & GD_C_FLOOR_ABOVE) || v.viewZ < there.x || masked);
        const bool topSil = !oneSided && ((flags & GD_C_CEIL_BELOW) || v.viewZ > there.y || masked);
        const int fa = max(cbot, oldCeil), cb = min(ctop, oldFloor);
        const bool floorOn = (flags & GD_C_MARK_FLOOR) && fa < oldFloor, ceilOn = (flags & GD_C_MARK_CEIL) && oldCeil < cb;
        const bool mid = oneSided && ctop < cbot;
        const unsigned sil = (topSil ? (unsigned)ceilClip : 0u) | ((bottomSil ? (unsigned)floorClip : 255u) << 8);
        const unsigned tiers = (mid ? (unsigned)ctop | ((unsigned)cbot << 8) : (upRange ? (unsigned)ctop | ((unsigned)cupbot << 8) : 0u)) |
                               (lowRange ? ((unsigned)clowtop << 16) | ((unsigned)cbot << 24) : 0u);
        if (mid || upRange || lowRange || sil != (255u << 8) || floorOn || ceilOn) {
          const unsigned drawn = ((mid && masked) || (upRange && sd.tex[2] >= 0) ? 1u : 0u) | (lowRange && sd.tex[1] >= 0 ? 2u : 0u);
          gd_put_event(events, nEvents, x, dist, wall, rc, tiers,
                       sil | (ceilOn ? ((unsigned)oldCeil << 16) | ((unsigned)cb << 24) : 0u),
                       (floorOn ? (unsigned)fa | ((unsigned)oldFloor << 8) : 0u) | (drawn << 16));
        }
      }
    }
    if (flags & GD_C_PORTAL) {
      const int2 clips = gd_portal_clips<kSplit>(sc, v, sh, x, o, ceilClip | (floorClip << 8), wantEvents ? events : nullptr, nEvents);
      ceilClip = clips.x & 255; floorClip = clips.x >> 8; nEvents = clips.y;
    }
    cur = next; prev = nextPrev;
  }
  eventCount[x] = nEvents < GD_MAX_EVENTS ? nEvents : GD_MAX_EVENTS;
  if (nEvents > GD_MAX_EVENTS) atomicOr(p.status, GD_STATUS_EVENT_OVERFLOW);
  const bool open = mine && (top < bottom || top < 0);
  if (open) gd_claimed_rows(sh, x, top, bottom);
  return open;
}

#endif

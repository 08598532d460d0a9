/* View setup, wall projection, per-(column, wall) ray tests, static topology predicates, ray-owned spans, blocking rays.
 * Part of gd_render.cu (one translation unit); not meant to be included elsewhere. */
#ifndef GD_GEOMETRY_CUH
#define GD_GEOMETRY_CUH

/* ---- view (engine.py:10648-10670, 10596-10601, 14949-14967) ------------- */
__device__ void gd_view_setup(const GdScene &sc, const int32_t *lane, GdView &v) {
  v.x = __int_as_float(lane[GD_L_X]);
  v.y = __int_as_float(lane[GD_L_Y]);
  v.angle = __int_as_float(lane[GD_L_ANGLE]);
  v.viewZ = __int_as_float(lane[GD_L_VIEW_Z]);
  v.vx = lane[GD_L_X_FIXED];
  v.vy = lane[GD_L_Y_FIXED];
  i64 bam = (i64)(uint32_t)lane[GD_L_ANGLE_BAM];
  v.pitchBam = lane[GD_L_PITCH_BAM];
  int fine = (int)((bam >> 19) & 8191);
  v.vsin = sc.fineSine[fine];
  v.vcos = sc.fineSine[(fine + 2048) & 8191];
  v.fsin = (float)v.vsin / 65536.0f;
  v.fcos = (float)v.vcos / 65536.0f;
  i64 ti = gd_clamp((GD_ANG90 - v.pitchBam) >> 19, 0, 4095);
  v.center = 104 * GD_FU + ((GD_FOCAL_Y * (i64)sc.fineTan[ti]) >> 16);
  v.upperClip = gd_div((-v.center) * GD_FU, GD_FOCAL_Y);
  v.lowerClip = gd_div((GD_VH * GD_FU - v.center) * GD_FU, GD_FOCAL_Y);
  int weapon = (int)gd_clamp(lane[GD_L_WEAPON], 0, 7);
  int cooldown = (int)gd_clamp(lane[GD_L_WPN_COOLDOWN], 0, sc.wpnTics - 1);
  int parity = (int)gd_pymod(lane[GD_L_WPN_FIRE_COUNT], 2);
  if (weapon == 1 && cooldown == 0) parity = (int)gd_pymod(gd_max(lane[GD_L_WPN_READY_TICS] - 1, 0) / 4, 2);
  v.flashLight = sc.wpnFlashLights[(weapon * 2 + parity) * sc.wpnTics + cooldown];
}

__device__ __forceinline__ void gd_ray(const GdView &v, int x, float &rx, float &ry) {
  float c = ((float)x - 160.0f) / 160.0f;
  rx = v.fcos + v.fsin * c;
  ry = v.fsin - v.fcos * c;
}

/* View coordinates of a segment's 16.16 endpoints, and the screen column that each projects to (engine.py:10747-10790).
 * Two divisions serve everything below: FWallCoords and the light of either side start from these columns. */
__device__ __forceinline__ void gd_project_ends(const GdView &v, const i64 fx[2], const i64 fy[2], GdEnds &e) {
#pragma unroll 1
  for (int k = 0; k < 2; ++k) {
    const i64 rx = (k ? fx[1] : fx[0]) - v.vx, ry = (k ? fy[1] : fy[0]) - v.vy;
    const i64 tx = (rx * v.vsin - ry * v.vcos) >> 20, ty = (rx * v.vcos + ry * v.vsin) >> 20;
    const i64 cf = 160 * GD_FU;
    const i64 column = ((cf + gd_div(tx * cf, ty == 0 ? 1 : ty)) >> 16) + (tx >= 0);
    if (k) { e.tx1 = tx; e.ty1 = ty; e.column1 = column; } else { e.tx0 = tx; e.ty0 = ty; e.column0 = column; }
  }
  const i64 wvx = fx[1] - fx[0], wvy = fy[1] - fy[0];
  const i64 fsx = v.vx - fx[0], fsy = v.vy - fy[0];
  e.front = (wvx * fsy - wvy * fsx) < 0;
}

/* The segment taken in its stored order (side 0) or the other way round (side 1): wallscan light of that side
 * (engine.py:11217-11291), and FWallCoords (10791-10869) of the side that faces the viewer. */
__device__ __noinline__ void gd_project_side(const GdEnds &e, int side, GdWall &out) {
  const i64 tx1 = side ? e.tx1 : e.tx0, ty1 = side ? e.ty1 : e.ty0, tx2 = side ? e.tx0 : e.tx1, ty2 = side ? e.ty0 : e.ty1;
  const i64 lp = side ? e.column1 : e.column0, rp = side ? e.column0 : e.column1;
  const i64 lden = tx1 - tx2 - ty2 + ty1, rden = ty2 - ty1 - tx2 + tx1;
  const bool lin = tx1 >= -ty1, rin = tx2 <= ty2;
  const i64 wsl = lin ? lp : 0, wsr = rin ? rp : GD_SW;
  i64 depthL = ty1, depthR = ty2;
  if (!lin) depthL = ty1 + gd_div((ty2 - ty1) * (tx1 + ty1), lden == 0 ? 1 : lden);
  if (!rin) depthR = ty1 + gd_div((ty2 - ty1) * (tx1 - ty1), rden == 0 ? 1 : rden);
  const i64 ll = gd_div(GD_WALL_VIS << 12, gd_max(depthL, 1));
  const i64 lr = gd_div(GD_WALL_VIS << 12, gd_max(depthR, 1));
  out.visStep[side] = gd_div(lr - ll, gd_max(wsr - wsl, 1));
  out.visL[side] = ll;
  out.visSl[side] = wsl;
  if (e.front != (side == 0)) return;
  const i64 screenL = lin && tx1 >= 0 ? gd_min(wsl, GD_SW) : wsl;
  i64 screenR = rin && tx2 >= 0 ? gd_min(wsr, GD_SW) : wsr;
  const bool invL = (lin ? ((tx1 > ty1) || (ty1 == 0)) : ((tx2 < -ty2) || (lden == 0))) || (depthL < 32);
  const bool invR = (rin ? ((tx2 < -ty2) || (ty2 == 0)) : ((tx1 > ty1) || (rden == 0))) || (depthR < 32);
  if (invL || invR || (screenR <= screenL)) screenR = screenL;
  out.sl = screenL; out.sr = screenR; out.dl = depthL; out.dr = depthR;
}

/* Crossing record of side i & 1 of wall i >> 1.  Texture indices are passed on as they are (the checked build tests
 * them where they are drawn); sectors out of range count as absent.  Inline: as a function of its own it moves the
 * walk's functions to addresses that cost 4096 lanes of the 64-sector map 3.46 instead of 3.40 ms. */
__device__ __forceinline__ void gd_side_setup(const GdScene &sc, int i, GdSide &out) {
  const int w = i >> 1;
  int here = sc.wsec[i], there = sc.wsec[i ^ 1];
  if (here < 0 || here >= sc.S) here = 0;
  if (there < -1 || there >= sc.S) there = -1;
  const bool oneSided = there < 0;
  const int other = oneSided ? 0 : there;
  const float vf = sc.secF[here * 2], vc = sc.secF[here * 2 + 1], of = sc.secF[other * 2], oc = sc.secF[other * 2 + 1];
  const int4 ri = *reinterpret_cast<const int4 *>(&sc.secI[here * 4]), oi = *reinterpret_cast<const int4 *>(&sc.secI[other * 4]);
  const float4 wl = *reinterpret_cast<const float4 *>(&sc.walls[w * 4]);
  const bool horizontal = fabsf(wl.w - wl.y) < 1e-6f, vertical = fabsf(wl.z - wl.x) < 1e-6f;
  GdSide o;
  for (int k = 0; k < 3; ++k) o.tex[k] = sc.sideTex[i * 3 + k];
  o.contrast = vertical ? 16 : (horizontal ? -16 : 0);
  o.tox = gd_rint(sc.sideOff[i * 2] * 65536.0f);
  o.yoff = sc.sideOff[i * 2 + 1];
  o.repeat = gd_rint(sc.wlen[w] * 65536.0f);
  o.pad = 0;
  unsigned f = GD_C_RASTER;
  const bool lightDiff = ri.x != oi.x;
  if (oneSided || vc != oc || ri.z != oi.z || lightDiff) f |= GD_C_MARK_CEIL;
  if (oneSided || vf != of || ri.y != oi.y || lightDiff) f |= GD_C_MARK_FLOOR;
  if (oneSided) {
    f |= GD_C_ONE_SIDED | (o.tex[0] >= 0 ? GD_C_TIER0 : 0u);
  } else {
    if (vf < of) f |= GD_C_LOWER | (o.tex[1] >= 0 ? GD_C_TIER1 : 0u);
    if (vc > oc) f |= GD_C_UPPER | (o.tex[2] >= 0 ? GD_C_TIER2 : 0u);
    if (vf > of) f |= GD_C_FLOOR_ABOVE;
    if (vc < oc) f |= GD_C_CEIL_BELOW;
  }
  o.flags = f;
  out = o;
}

/* Does the column ray (rx, ry) cross the wall (engine.py:11317-11331)?  The
 * comparisons of the rounded quotients dn / den and an / den with 0 and 1 depend
 * only on signs and magnitudes: both numerators are differences of products of
 * map-scale numbers, so a nonzero one is far too large for its quotient to
 * underflow, and a quotient of two floats rounds to at most 1 only when the
 * numerator is not larger. */
__device__ __forceinline__ bool gd_ray_geo(const GdHot &h, float rx, float ry) {
  const float den = rx * h.segy - ry * h.segx;
  const float safe = fabsf(den) < 1e-6f ? 1.0f : den;
  const float an = h.offx * ry - h.offy * rx;
  const bool positive = (h.dn != 0.0f) && ((h.dn < 0) == (safe < 0));
  const bool alongOk = (an == 0.0f) || (((an < 0) == (safe < 0)) && fabsf(an) <= fabsf(safe));
  return !(fabsf(den) < 1e-6f) && positive && alongOk;
}

/* First and last column whose ray crosses a wall, as a span word, found at the projections of its ends.
 * A ray's cross product with an endpoint is linear in the column, with a slope of its depth / 160.  With both ends
 * at least 8 units deep and no coordinate above 16384 the rounding of the test moves a crossing's edge by less than
 * half a column, and that of the projections below by less than a tenth: every column more than one inside the
 * projected ends gives the same answer, and every one more than one outside is not crossed.  So the four columns
 * around either end decide.  A wall that does not qualify gets GD_SPAN_SWEEP: all columns are tried. */
#define GD_SPAN_SWEEP 0xFFFEFFFEu
__device__ __forceinline__ unsigned gd_crossed_columns(const GdView &v, const GdHot &h) {
  const float bx = h.offx + h.segx, by = h.offy + h.segy;
  const float size = fmaxf(fmaxf(fabsf(h.offx), fabsf(h.offy)), fmaxf(fabsf(bx), fabsf(by)));
  const float da = h.offx * v.fcos + h.offy * v.fsin, db = bx * v.fcos + by * v.fsin;
  if (!(size <= 16384.0f && fminf(da, db) >= 8.0f)) return GD_SPAN_SWEEP;
  const float ca = 160.0f + 160.0f * ((h.offx * v.fsin - h.offy * v.fcos) / da);
  const float cb = 160.0f + 160.0f * ((bx * v.fsin - by * v.fcos) / db);
  const float low = floorf(fminf(ca, cb)) - 1.0f, high = ceilf(fmaxf(ca, cb)) + 1.0f;
  if (high < 0.0f || low > (float)(GD_SW - 1)) return 0xFFFFu;
  const int lo = (int)fmaxf(low, 0.0f), hi = (int)fminf(high, (float)(GD_SW - 1));
  int first = -1, last = -1;
#pragma unroll 1
  for (int k = 0; k < 8; ++k) {
    const int x = min(max(k < 4 ? lo + k : hi - 7 + k, lo), hi);
    float rx, ry;
    gd_ray(v, x, rx, ry);
    if (!gd_ray_geo(h, rx, ry)) continue;
    if (first < 0) first = x;
    last = max(last, x);
  }
  return ((unsigned)first & 0xFFFFu) | ((unsigned)(last + 1) << 16);
}

/* One half of the projection of wall w for this lane (engine.py:10747-10869, 11207-11302, 11359-11427), by a
 * thread of its own: side 0, the lane-dependent operands of the column-ray test and the ends' columns, or side 1 and the
 * columns whose rays cross the wall.  What bounds it is the latency of one thread's divisions: one after the other, for
 * both sides, the ends and the light terms more than once, they were twenty, and span tables and things went before them
 * (one lane alone 112 us a step, now 109; 4096 lanes 3036 and 2998). */
__device__ __noinline__ void gd_project_wall(const GdScene &sc, const GdView &v, int w, int side, GdWall &out, GdHot &hot, int2 &columns) {
  const float4 wl = *reinterpret_cast<const float4 *>(&sc.walls[w * 4]);
  const i64 fx[2] = {gd_rint(wl.x * 65536.0f), gd_rint(wl.z * 65536.0f)};
  const i64 fy[2] = {gd_rint(wl.y * 65536.0f), gd_rint(wl.w * 65536.0f)};
  GdEnds e;
  gd_project_ends(v, fx, fy, e);
  gd_project_side(e, side, out);
  GdHot mine;
  mine.segx = wl.z - wl.x; mine.segy = wl.w - wl.y;
  mine.offx = wl.x - v.x; mine.offy = wl.y - v.y;
  mine.dn = mine.offx * mine.segy - mine.offy * mine.segx;
  if (e.front == (side == 0)) {
    const float vfsx = v.x - wl.x, vfsy = v.y - wl.y;
    const bool front = (mine.segx * vfsy - mine.segy * vfsx) < 0;
    const unsigned sl = (unsigned)(gd_clamp(out.sl, -1, GD_SW + 1) + 1), sr = (unsigned)(gd_clamp(out.sr, -1, GD_SW + 1) + 1);
    hot.bits = sl | (sr << 10) | (front ? GD_HOT_FRONT : 0u) | (hot.bits & GD_HOT_STATIC);
  }
  if (side == 0) {
    hot.segx = mine.segx; hot.segy = mine.segy; hot.offx = mine.offx; hot.offy = mine.offy; hot.dn = mine.dn;
    out.tx[0] = (int)e.tx0; out.tx[1] = (int)e.tx1;
    out.ty[0] = (int)e.ty0; out.ty[1] = (int)e.ty1;
    columns = make_int2((int)gd_clamp(e.column0, -1, GD_SW + 1), (int)gd_clamp(e.column1, -1, GD_SW + 1));
  } else {
    hot.span = gd_crossed_columns(v, mine);
  }
}

/* One piece of a line a node builder split (engine.py:11478-11500): projected like a line, from its
 * own fixed-point endpoints.  Only its FWallCoords and its wallscan light are ever read. */
__device__ __forceinline__ void gd_project_fragment(const GdScene &sc, const GdView &v, int f, GdWall &out) {
  const int4 q = *reinterpret_cast<const int4 *>(&sc.fragFixed[f * 4]);
  const i64 fx[2] = {q.x, q.z}, fy[2] = {q.y, q.w};
  GdEnds e;
  gd_project_ends(v, fx, fy, e);
#pragma unroll 1
  for (int side = 0; side < 2; ++side) gd_project_side(e, side, out);
}

/* Does the ray meet the wall's line in front of the viewer (the `positive` of engine.py:11317-11331)? */
__device__ __forceinline__ bool gd_ray_meets_line(const GdHot &h, float rx, float ry) {
  const float den = rx * h.segy - ry * h.segx;
  return !(fabsf(den) < 1e-6f) && h.dn != 0.0f && ((h.dn < 0) == (den < 0));
}

/* ---- per (column, wall) hit -------------------------------------------- */
struct GdHit {
  float d;       /* ray distance, +inf when the wall does not count here */
  float along;   /* clamped to [0,1] */
  bool geo, proj, left;
};

/* engine.py:11317-11331, 11440-11459 */
__device__ __forceinline__ GdHit gd_hit(const GdScene &sc, int w, int x, float rx, float ry) {
  GdHit h;
  w = GD_CHECK_INDEX(w, sc.W);
  const GdHot hot = gd_hot(w);
  const float den = rx * hot.segy - ry * hot.segx;
  const bool small = fabsf(den) < 1e-6f;
  const float safe = small ? 1.0f : den;
  const float distance = hot.dn / safe;
  const float along = (hot.offx * ry - hot.offy * rx) / safe;
  const bool positive = !small && distance > 0;
  const int isl = (short)(hot.span & 0xFFFFu), isr = (int)(hot.span >> 16);
  const bool geo = positive && along >= 0 && along <= 1;
  const bool pv = positive && x >= isl && x < isr;
  const bool valid = (hot.bits & GD_HOT_ONESIDED) ? (pv && (hot.bits & GD_HOT_FRONT)) : (geo || pv);
  h.d = valid ? distance : GD_INF;
  float ac = along;
  if (!(ac >= 0.0f)) ac = (ac != ac) ? ac : 0.0f;
  if (ac > 1.0f) ac = 1.0f;
  h.along = ac;
  h.geo = geo;
  h.proj = pv;
  h.left = (x == isl);
  return h;
}

/* the same out of line, as three words */
__device__ __noinline__ uint3 gd_hit_words(const GdScene &sc_, int w, int x, float rx, float ry) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const GdHit h = gd_hit(sc, w, x, rx, ry);
  return make_uint3(__float_as_uint(h.d), __float_as_uint(h.along), (h.geo ? 1u : 0u) | (h.proj ? 2u : 0u) | (h.left ? 4u : 0u));
}
__device__ __forceinline__ GdHit gd_hit_slow(const GdScene &sc, int w, int x, float rx, float ry) {
  const uint3 q = gd_hit_words(sc, w, x, rx, ry);
  GdHit h;
  h.d = __uint_as_float(q.x); h.along = __uint_as_float(q.y);
  h.geo = q.z & 1u; h.proj = (q.z & 2u) != 0; h.left = (q.z & 4u) != 0;
  return h;
}

__device__ __forceinline__ float gd_tol(float d) { return fmaxf(fabsf(d) / 128.0f, 4.0f); }

/* Endpoint owner of wall w at column x (engine.py:11589-11730). */
__device__ __noinline__ void gd_endpoint_owner(const GdScene &sc_, const GdWall *walls, int w, int x, float rx, float ry,
                                               const GdHit &hw, int &ownerIdx, float &ownerDist) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const GdWall &wv = walls[w];
  float d = hw.d;
  float tol = gd_tol(d);
  bool subpixel = (wv.sr - wv.sl <= 1) && !(gd_hot(w).bits & GD_HOT_ONESIDED);
  bool usesStart = hw.along <= 0.5f;
  int oi = w;
  float od = d;
  bool ownerValid = false;
  if (sc.nbDirect) {
    const int32_t *nd = &sc.nbDirectTab[w * 4];
    int sIdx = nd[0] >= 0 ? GD_CHECK_INDEX(nd[0], sc.W) : w, eIdx = nd[1] >= 0 ? GD_CHECK_INDEX(nd[1], sc.W) : w;
    bool hasS = nd[0] >= 0, hasE = nd[1] >= 0;
    int rIdx = usesStart ? sIdx : eIdx, rSlot = usesStart ? nd[2] : nd[3];
    bool rHas = usesStart ? hasS : hasE;
    int oIdx = usesStart ? eIdx : sIdx, oSlot = usesStart ? nd[3] : nd[2];
    bool oHas = usesStart ? hasE : hasS;
    GdHit hr = (rIdx == w) ? hw : gd_hit_slow(sc, rIdx, x, rx, ry);
    GdHit ho = (oIdx == w) ? hw : gd_hit_slow(sc, oIdx, x, rx, ry);
    bool rOwns = rHas && hr.proj && hr.left;
    bool oOwns = subpixel && oHas && ho.proj && ho.left && (fabsf(ho.d - d) <= tol);
    bool useO = oOwns && (!rOwns || ho.d < hr.d || (ho.d == hr.d && oSlot < rSlot));
    oi = useO ? oIdx : rIdx;
    od = useO ? ho.d : hr.d;
    ownerValid = rOwns || oOwns;
  } else {
    float best = GD_INF;
    int bestSlot = 0;
    int n0 = sc.nbOff[w], n1 = sc.nbOff[w + 1];
#pragma unroll 1
    for (int k = n0; k < n1; ++k) {
      int nb = GD_CHECK_INDEX(sc.nbIdx[k], sc.W), fl = sc.nbFlags[k];
      GdHit hn = gd_hit_slow(sc, nb, x, rx, ry);
      bool rayNb = usesStart ? (fl & 1) : ((fl >> 1) & 1);
      bool sel = rayNb || (subpixel && (fabsf(hn.d - d) <= tol));
      float cand = (hn.proj && hn.left && sel) ? hn.d : GD_INF;
      if (cand < best) { best = cand; bestSlot = k - n0; }
    }
    od = best;
    oi = (n1 > n0) ? GD_CHECK_INDEX(sc.nbIdx[n0 + bestSlot], sc.W) : w;
    ownerValid = isfinite(best);
  }
  bool has = !hw.proj && ownerValid;
  ownerIdx = has ? oi : w;
  ownerDist = has ? od : d;
}

/* PrepWall (engine.py:10672-10739): the operands that depend on the wall alone, and the evaluation at
 * one column.  `repeat`: the wall's length in 16.16. */
__device__ __forceinline__ float4 gd_prep_setup(const GdWall &wv) {
  const i64 tx1 = wv.tx[0], tx2 = wv.tx[1], ty1 = wv.ty[0], ty2 = wv.ty[1];
  return make_float4((float)tx1 * 160.0f, (float)ty1, (float)(tx1 - tx2) * 160.0f, (float)(ty2 - ty1));
}
__device__ __forceinline__ void gd_prep_eval(const float4 q, i64 repeat, int x, i64 &hoff, i64 &vstep) {
  const double col = (double)x - 160.0;
  const double top = (double)q.x + (double)(-q.y) * col;
  const double bottom = (double)q.z + (double)q.w * col;
  const double safeBottom = bottom == 0 ? 1.0 : bottom;
  const double fraction = top / safeBottom;
  hoff = (i64)floor(fraction * (double)repeat + 0.5);
  const double wms = (320 * 200.0 / 320.0 / 240) * 64.0 / (320 / 2.0);
  const double depthScale = (double)(q.w * (float)wms);
  const double depthOrigin = (double)(q.y * (float)wms);
  vstep = (i64)floor(fraction * depthScale + depthOrigin + 0.5);
}
__device__ __noinline__ void gd_prep_wall(const GdScene &sc_, const GdWall &wv, int w, int x, i64 &hoff, i64 &vstep) {
  const GdScene &sc = *gd_as_shared(&sc_);
  gd_prep_eval(gd_prep_setup(wv), gd_rint(sc.wlen[w] * 65536.0f), x, hoff, vstep);
}

/* OWallMost row projection (engine.py:12294-12605), one fragment per wall. */
__device__ __noinline__ int gd_project_rows(const GdView &v_, const GdWall &wv, float worldZ, int x) {
  const GdView &v = *gd_as_shared(&v_);
  i64 wsl = wv.sl, wsr = wv.sr;
  i64 wdl = gd_max(wv.dl, 1), wdr = gd_max(wv.dr, 1);
  bool owns = (wsr > wsl) && x >= wsl && x < wsr;
  i64 relZ = gd_rint((worldZ - v.viewZ) * 65536.0f);
  i64 pz = -(relZ >> 4);
  i64 center = v.center;
  i64 num = pz * GD_FOCAL_Y;
  if (!owns) {
    i64 ospan = gd_max(wsr - wsl, 1);
    i64 opl = gd_div(num, wdl), opr = gd_div(num, wdr);
    i64 ostep = gd_div(opr - opl, ospan);
    return (int)gd_clamp((center + opl + (x - wsl) * ostep) >> 16, 0, GD_VH);
  }
  i64 sl = wsl, sr = wsr, dl = wdl, dr = wdr;
  i64 upperClip = v.upperClip, lowerClip = v.lowerClip;
  i64 ul = (upperClip * dl) >> 16, ur = (upperClip * dr) >> 16;
  i64 ll = (lowerClip * dl) >> 16, lr = (lowerClip * dr) >> 16;
  bool aboveL = pz < ul, aboveR = pz < ur, belowL = pz > ll, belowR = pz > lr;
  bool entAbove = aboveL && aboveR, entBelow = belowL && belowR;
  i64 cl = sl, cr = sr, cdl = dl, cdr = dr;
  bool outTop = false, outBottom = false;
  bool crossesTop = aboveL != aboveR;
  if (crossesTop) {
    i64 sud = (ur != ul) ? (ur - ul) : 1;
    i64 tf = gd_div(gd_shl(pz - ul, 30), sud);
    i64 td = dl + (((dr - dl) * tf) >> 30);
    i64 tc = sl + gd_div(((dr * tf) >> 30) * (sr - sl), gd_max(td, 1));
    if (aboveR && (sl <= tc)) { cr = tc; cdr = td; }
    outTop |= aboveR && (sr > tc) && (x >= tc) && (x < sr);
    if (aboveL && (tc <= sr)) { cl = tc; cdl = td; }
    outTop |= aboveL && (tc > sl) && (x >= sl) && (x < tc);
  }
  bool crossesBottom = belowL != belowR;
  if (crossesBottom) {
    i64 sld = (lr != ll) ? (lr - ll) : 1;
    i64 bf = gd_div(gd_shl(pz - ll, 30), sld);
    i64 bd = dl + (((dr - dl) * bf) >> 30);
    i64 bc = sl + gd_div(((dr * bf) >> 30) * (sr - sl), gd_max(bd, 1));
    if (belowR && (sl <= bc)) { cr = bc; cdr = bd; }
    outBottom |= belowR && (sr > bc) && (x >= bc) && (x < sr);
    if (belowL && (bc <= sr)) { cl = bc; cdl = bd; }
    outBottom |= belowL && (bc > sl) && (x >= sl) && (x < bc);
  }
  bool collapsed = (cr == cl) && (x == cl) && !(entAbove || entBelow);
  if (entAbove || (outTop && !collapsed)) return 0;
  if (entBelow || (outBottom && !collapsed)) return GD_VH;
  i64 pl = gd_div(num, gd_max(cdl, 1)), pr = gd_div(num, gd_max(cdr, 1));
  i64 span = gd_max(cr - cl, 1);
  i64 pstep = gd_div(pr - pl, span);
  return (int)gd_clamp((center + pl + (x - cl) * pstep) >> 16, 0, GD_VH);
}

/* The unclipped whole-line projection: what a column of a split line falls back to when none of
 * the line's fragments owns it (engine.py:12393-12410, 12596-12604). */
__device__ __noinline__ int gd_project_rows_whole(const GdView &v, const GdWall &wv, float worldZ, int x) {
  const i64 wdl = gd_max(wv.dl, 1), wdr = gd_max(wv.dr, 1);
  const i64 relZ = gd_rint((worldZ - v.viewZ) * 65536.0f);
  const i64 num = -(relZ >> 4) * GD_FOCAL_Y;
  const i64 opl = gd_div(num, wdl), opr = gd_div(num, wdr);
  const i64 ostep = gd_div(opr - opl, gd_max(wv.sr - wv.sl, 1));
  return (int)gd_clamp((v.center + opl + (x - wv.sl) * ostep) >> 16, 0, GD_VH);
}

/* Is line w split, and if so which of its fragments owns column x: the first whose half-open
 * span holds it (engine.py:12310-12376, 11511-11545), or null. */
__device__ __forceinline__ bool gd_line_is_split(const GdScene &sc, int w) {
  return sc.F > 0 && sc.fragOff[w + 1] > sc.fragOff[w];
}
__device__ __noinline__ const GdWall *gd_fragment_at(const GdScene &sc, const GdWall *frags, int w, int x) {
#pragma unroll 1
  for (int f = sc.fragOff[w]; f < sc.fragOff[w + 1]; ++f) {
    const GdWall &q = frags[f];
    if (q.sr > q.sl && x >= q.sl && x < q.sr) return &q;
  }
  return nullptr;
}
/* Row projection and wallscan light of line w at column x, fragments considered. */
__device__ __noinline__ int gd_line_rows(const GdScene &sc, const GdView &v, const GdWall *walls, const GdWall *frags, int w,
                                         float worldZ, int x) {
  if (!gd_line_is_split(sc, w)) return gd_project_rows(v, walls[w], worldZ, x);
  const GdWall *q = gd_fragment_at(sc, frags, w, x);
  return q ? gd_project_rows(v, *q, worldZ, x) : gd_project_rows_whole(v, walls[w], worldZ, x);
}
__device__ __forceinline__ i64 gd_line_vis(const GdScene &sc, const GdWall *walls, const GdWall *frags, int w, int side, int x) {
  const GdWall *q = &walls[w];
  if (gd_line_is_split(sc, w)) {
    const GdWall *f = gd_fragment_at(sc, frags, w, x);
    if (f) q = f;
  }
  return q->visL[side] + ((i64)x - q->visSl[side]) * q->visStep[side];
}

/* Column-independent part of gd_project_rows for one (wall, height): the full record, and the form
 * the walk reads (its `vis` word is the caller's). */
__device__ __noinline__ void gd_rowproj_setup(const GdView &v_, const GdWall &wv, float worldZ, GdRowProj &o, GdRow &row) {
  const GdView &v = *gd_as_shared(&v_);
  i64 wsl = wv.sl, wsr = wv.sr;
  i64 wdl = gd_max(wv.dl, 1), wdr = gd_max(wv.dr, 1);
  i64 relZ = gd_rint((worldZ - v.viewZ) * 65536.0f);
  i64 pz = -(relZ >> 4);
  i64 num = pz * GD_FOCAL_Y;
  {
    i64 ospan = gd_max(wsr - wsl, 1);
    i64 opl = gd_div(num, wdl), opr = gd_div(num, wdr);
    o.opl = opl;
    o.ostep = gd_div(opr - opl, ospan);
  }
  i64 sl = wsl, sr = wsr, dl = wdl, dr = wdr;
  i64 upperClip = v.upperClip, lowerClip = v.lowerClip;
  i64 ul = (upperClip * dl) >> 16, ur = (upperClip * dr) >> 16;
  i64 ll = (lowerClip * dl) >> 16, lr = (lowerClip * dr) >> 16;
  bool aboveL = pz < ul, aboveR = pz < ur, belowL = pz > ll, belowR = pz > lr;
  bool entAbove = aboveL && aboveR, entBelow = belowL && belowR;
  i64 cl = sl, cr = sr, cdl = dl, cdr = dr;
  i64 topA = 0, topB = 0, botA = 0, botB = 0;
  if (aboveL != aboveR) {
    i64 sud = (ur != ul) ? (ur - ul) : 1;
    i64 tf = gd_div(gd_shl(pz - ul, 30), sud);
    i64 td = dl + (((dr - dl) * tf) >> 30);
    i64 tc = sl + gd_div(((dr * tf) >> 30) * (sr - sl), gd_max(td, 1));
    if (aboveR && (sl <= tc)) { cr = tc; cdr = td; }
    if (aboveR && (sr > tc)) { topA = tc; topB = sr; }
    if (aboveL && (tc <= sr)) { cl = tc; cdl = td; }
    if (aboveL && (tc > sl)) { topA = sl; topB = tc; }
  }
  if (belowL != belowR) {
    i64 sld = (lr != ll) ? (lr - ll) : 1;
    i64 bf = gd_div(gd_shl(pz - ll, 30), sld);
    i64 bd = dl + (((dr - dl) * bf) >> 30);
    i64 bc = sl + gd_div(((dr * bf) >> 30) * (sr - sl), gd_max(bd, 1));
    if (belowR && (sl <= bc)) { cr = bc; cdr = bd; }
    if (belowR && (sr > bc)) { botA = bc; botB = sr; }
    if (belowL && (bc <= sr)) { cl = bc; cdl = bd; }
    if (belowL && (bc > sl)) { botA = sl; botB = bc; }
  }
  bool collapsed = (cr == cl) && !(entAbove || entBelow);
  o.collapsedX = (short)((collapsed && cl >= 0 && cl < GD_SW) ? cl : -1);
  o.entAbove = entAbove; o.entBelow = entBelow;
  o.topA = (short)gd_clamp(topA, -1, GD_SW + 1); o.topB = (short)gd_clamp(topB, -1, GD_SW + 1);
  o.botA = (short)gd_clamp(botA, -1, GD_SW + 1); o.botB = (short)gd_clamp(botB, -1, GD_SW + 1);
  i64 pl = gd_div(num, gd_max(cdl, 1)), pr = gd_div(num, gd_max(cdr, 1));
  o.pl = pl;
  const i64 pstep = gd_div(pr - pl, gd_max(cr - cl, 1));
  o.pstep = pstep;
  o.cl = cl;
  o.pad = 0;
  /* The walk's form computes center + pl + (x - cl) * pstep modulo 2^32, which is exact where the result fits: the
   * row is linear, so it is enough to look at the first and last owned column that is not forced. */
  unsigned lim = GD_ROW_PLAIN;
  bool wide = false;
  i64 a = v.center + pl - gd_wmul(cl, pstep), step = pstep;
  if (entAbove || entBelow) {
    lim = 1023u | (1023u << 10) | (entAbove ? GD_ROW_LEFT_TOP : 0u);
    a = 0; step = 0;
  } else {
    int la = 0, lb = 1023;
    const bool top = topA < topB, bottom = botA < botB;
    if (bottom && belowL) la = o.botB;
    if (bottom && belowR) lb = o.botA;
    if (top && aboveL) { la = o.topB; lim |= GD_ROW_LEFT_TOP; }
    if (top && aboveR) { lb = o.topA; lim |= GD_ROW_RIGHT_TOP; }
    la = max(la, 0); lb = max(lb, 0);
    if (la > lb) { if (lim & GD_ROW_LEFT_TOP) lb = la; else la = lb; }    /* where both reach a column, the top wins */
    /* the one column exempt from both: next to the forced columns as a rule, where it moves their bound */
    const int cx = o.collapsedX;
    if (cx >= 0 && (cx < la || cx >= lb)) {
      if (cx == la - 1) la = cx;
      else if (cx == lb) lb = cx + 1;
      else wide = true;
    }
    lim = (lim & ~GD_ROW_PLAIN) | (unsigned)la | ((unsigned)lb << 10);
    const i64 x0 = gd_max(gd_max(wsl, 0), la), x1 = gd_min(gd_min(wsr, GD_SW), lb) - 1;
    if (x0 <= x1) {
      const i64 r0 = v.center + pl + gd_wmul(x0 - cl, pstep), r1 = v.center + pl + gd_wmul(x1 - cl, pstep);
      wide = wide || r0 != (i64)(int)r0 || r1 != (i64)(int)r1;
    }
    wide = wide || (aboveL && belowL) || (aboveR && belowR);
  }
  if (wide) lim |= GD_ROW_WIDE;
  row.a = (int)a; row.step = (int)step; row.lim = lim;
}

__device__ __forceinline__ int gd_row_eval(const GdRow &r, int x) {
  int y = min(max((int)((unsigned)r.a + (unsigned)x * (unsigned)r.step) >> 16, 0), GD_VH);
  if ((r.lim & 0xFFFFFu) != GD_ROW_PLAIN) {
    if (x < (int)(r.lim & 1023u)) y = (r.lim & GD_ROW_LEFT_TOP) ? 0 : GD_VH;
    if (x >= (int)((r.lim >> 10) & 1023u)) y = (r.lim & GD_ROW_RIGHT_TOP) ? 0 : GD_VH;
  }
  return y;
}

__device__ __forceinline__ int gd_rowproj_eval(const GdView &v, const GdWall &wv, const GdRowProj &o, int x) {
  bool owns = (wv.sr > wv.sl) && x >= wv.sl && x < wv.sr;
  if (!owns) return (int)gd_clamp((v.center + o.opl + (x - wv.sl) * o.ostep) >> 16, 0, GD_VH);
  bool collapsed = x == o.collapsedX;
  bool outTop = x >= o.topA && x < o.topB, outBottom = x >= o.botA && x < o.botB;
  if (o.entAbove || (outTop && !collapsed)) return 0;
  if (o.entBelow || (outBottom && !collapsed)) return GD_VH;
  return (int)gd_clamp((v.center + o.pl + (x - o.cl) * o.pstep) >> 16, 0, GD_VH);
}

__device__ __forceinline__ int gd_wall_shade(i64 light, i64 vis) {
  i64 base = 64 * GD_FU - (light + 12) * (GD_FU / 4);
  return (int)gd_clamp((base - gd_min(vis, 24 * GD_FU)) >> 16, 0, 31);
}

/* ---- static topology predicates (engine.py:399-484, 1596-1612) ---------- */
__device__ __forceinline__ int gd_secidx(const GdScene &sc, int s) { return GD_CHECK_SECTOR(s < 0 ? s + sc.S : s, sc.S); }
__device__ __forceinline__ float gd_sec_floor(const GdScene &sc, int s) { return sc.secF[gd_secidx(sc, s) * 2]; }
__device__ __forceinline__ float gd_sec_ceil(const GdScene &sc, int s) { return sc.secF[gd_secidx(sc, s) * 2 + 1]; }
__device__ __forceinline__ int4 gd_sec_info(const GdScene &sc, int s) {
  return *reinterpret_cast<const int4 *>(&sc.secI[gd_secidx(sc, s) * 4]);
}

__device__ __forceinline__ bool gd_same_pair(const GdScene &sc, int a, int b) {
  int a0 = gd_hot_front(a), a1 = gd_hot_back(a), b0 = gd_hot_front(b), b1 = gd_hot_back(b);
  return (a0 == b0 && a1 == b1) || (a0 == b1 && a1 == b0);
}
__device__ __forceinline__ bool gd_shares_endpoint(const GdScene &sc, int a, int b) {
  int a0 = gd_vertex(sc, a, 0), a1 = gd_vertex(sc, a, 1), b0 = gd_vertex(sc, b, 0), b1 = gd_vertex(sc, b, 1);
  return a0 == b0 || a0 == b1 || a1 == b0 || a1 == b1;
}
__device__ __noinline__ bool gd_opposing_pair(const GdScene &sc_, int a, int b) {
  const GdScene &sc = *gd_as_shared(&sc_);
  if (!gd_same_pair(sc, a, b)) return false;
  if (gd_hot_back(a) < 0 || gd_hot_back(b) < 0) return false;
  if (gd_shares_endpoint(sc, a, b)) return false;
  const float *A = &sc.walls[a * 4], *B = &sc.walls[b * 4];
  float adx = A[2] - A[0], ady = A[3] - A[1], bdx = B[2] - B[0], bdy = B[3] - B[1];
  float dot = adx * bdx + ady * bdy;
  float cross = adx * bdy - ady * bdx;
  return dot < 0 && fabsf(cross) < 1e-6f;
}
__device__ __forceinline__ bool gd_two_distinct(const GdScene &sc, int w) {
  return gd_hot_back(w) >= 0 && gd_hot_front(w) != gd_hot_back(w);
}
__device__ bool gd_bridge_pair_of(const GdScene &sc, int a, int b, int &p0, int &p1) {
  int a0 = gd_hot_front(a), a1 = gd_hot_back(a), b0 = gd_hot_front(b), b1 = gd_hot_back(b);
  int shared = 0, sv = -2;
  if (a0 == b0 || a0 == b1) { shared++; sv = a0; }
  if (a1 == b0 || a1 == b1) { shared++; sv = a1; }
  if (shared != 1) return false;
  p0 = (a0 == sv) ? a1 : a0;
  p1 = (b0 == sv) ? b1 : b0;
  return true;
}
__device__ __forceinline__ bool gd_set_equals(const GdScene &sc, int w, int p0, int p1) {
  int s0 = gd_hot_front(w), s1 = gd_hot_back(w);
  if (p0 == p1) return s0 == p0 && s1 == p0;
  return (s0 == p0 && s1 == p1) || (s0 == p1 && s1 == p0);
}
__device__ bool gd_unique_at_vertex(const GdScene &sc, int v, int skipA, int skipB, int p0, int p1, int &index) {
  int count = 0, found = 0;
#pragma unroll 1
  for (int k = sc.vtxOff[v]; k < sc.vtxOff[v + 1]; ++k) {
    int c = GD_CHECK_INDEX(sc.vtxWalls[k], sc.W);
    if (c == skipA || c == skipB) continue;
    if (gd_set_equals(sc, c, p0, p1)) { count++; found = c; }
  }
  index = (count == 1) ? found : 0;
  return count == 1;
}
__device__ __noinline__ bool gd_portal_bridge(const GdScene &sc_, int slot, int path, int owner, int &index) {
  const GdScene &sc = *gd_as_shared(&sc_);
  index = 0;
  if (!gd_two_distinct(sc, path) || owner == path) return false;
  int v = gd_vertex(sc, path, slot);
  if (gd_vertex(sc, owner, 0) != v && gd_vertex(sc, owner, 1) != v) return false;
  if (!gd_two_distinct(sc, owner)) return false;
  int p0, p1;
  if (!gd_bridge_pair_of(sc, path, owner, p0, p1)) return false;
  return gd_unique_at_vertex(sc, v, path, owner, p0, p1, index);
}
__device__ __noinline__ bool gd_sector_bridge(const GdScene &sc_, int slot, int pending, int path, int &index) {
  const GdScene &sc = *gd_as_shared(&sc_);
  index = 0;
  if (!gd_two_distinct(sc, pending) || path == pending || !gd_two_distinct(sc, path)) return false;
  int p0, p1;
  if (!gd_bridge_pair_of(sc, pending, path, p0, p1)) return false;
  return gd_unique_at_vertex(sc, gd_vertex(sc, pending, slot), pending, path, p0, p1, index);
}

/* ---- phase: ray-owned spans (engine.py:11333-11438) --------------------- */
/* A wall whose two endpoints lie behind the viewer, or both beyond the same
 * edge of the 90-degree frustum, is crossed by no column ray at a positive
 * distance.  The two-unit margin is four orders of magnitude above the float
 * error of these dot products at map scale, so the test only ever drops walls
 * for which the exact sweep below finds no column. */
__device__ __forceinline__ bool gd_wall_in_frustum(const float4 wl, const GdView &v) {
  float ax = wl.x - v.x, ay = wl.y - v.y, bx = wl.z - v.x, by = wl.w - v.y;
  float fa = ax * v.fcos + ay * v.fsin, fb = bx * v.fcos + by * v.fsin;      /* forward */
  float sa = ax * v.fsin - ay * v.fcos, sb = bx * v.fsin - by * v.fcos;      /* to the right */
  const float m = -2.0f;
  if (fa < m && fb < m) return false;
  if (fa + sa < m && fb + sb < m) return false;
  if (fa - sa < m && fb - sb < m) return false;
  return true;
}

/* Lists the walls that a column ray may cross, and with them wall 0 and the first blocking wall, which the
 * rules fall back to.  Every other wall gets the record no ray meets.  The list stays in aux until the walk begins. */
__device__ __forceinline__ void gd_wall_list(const GdScene &sc, const GdView &v) {
  short *list = (short *)(gd_smem + GD_OFF_AUX);
  int *listed = (int *)(gd_smem + GD_OFF_MISC) + 2;
  const int block0 = GD_CHECK_INDEX(sc.blocking[0], sc.W);
#pragma unroll 1
  for (int w = threadIdx.x; w < sc.W; w += GD_THREADS) {
    const float4 wl = *reinterpret_cast<const float4 *>(&sc.walls[w * 4]);
    if (gd_wall_in_frustum(wl, v) || w == 0 || w == block0) {
      list[atomicAdd(listed, 1)] = (short)w;
    } else {
      gd_hot(w).dn = 0.0f;
      gd_hot(w).span = 0xFFFFu;
    }
  }
}

/* The ray-owned spans of the listed walls, which are projected; `prep` still holds the columns of their ends. */
__device__ __forceinline__ void gd_wall_spans(const GdView &v_, const GdShared &sh_, const float4 *prep) {
  const GdView &v = *gd_as_shared(&v_);
  const GdShared &sh = *gd_as_shared(&sh_);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const GdWall *walls = sh.walls;
  const short *list = (const short *)(gd_smem + GD_OFF_AUX);
  const int n = ((const int *)(gd_smem + GD_OFF_MISC))[2];
#pragma unroll 1
  for (int i = warp; i < n; i += GD_WARPS) {
    const int w = list[i];
    if (gd_hot(w).span != GD_SPAN_SWEEP) continue;
    const GdHot h = gd_hot(w);
    int first = -1, last = -1;
#pragma unroll 1
    for (int chunk = 0; chunk < GD_SW / 32; ++chunk) {
      float rx, ry;
      gd_ray(v, chunk * 32 + lane, rx, ry);
      const unsigned m = __ballot_sync(0xffffffffu, gd_ray_geo(h, rx, ry));
      if (m) {
        if (first < 0) first = chunk * 32 + __ffs(m) - 1;
        last = chunk * 32 + 31 - __clz(m);
      }
    }
    if (lane == 0) gd_hot(w).span = ((unsigned)first & 0xFFFFu) | ((unsigned)(last + 1) << 16);
  }
  __syncthreads();
#pragma unroll 1
  for (int i = threadIdx.x; i < n; i += GD_THREADS) {
    const int w = list[i];
    const GdWall &wv = walls[w];
    const int2 ends = *reinterpret_cast<const int2 *>(&prep[w]);
    const int column[2] = {ends.x, ends.y};
    GdHot &hot = gd_hot(w);
    const int first = (short)(hot.span & 0xFFFFu), end = (int)(hot.span >> 16);
    bool hasColumns = first >= 0;
    int isl = hasColumns ? first : 0;
    int isr = hasColumns ? end : GD_SW;
    bool evis[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int ty = wv.ty[e], tx = wv.tx[e];
      evis[e] = ty > 0 && tx >= -ty && tx <= ty && column[e] >= 0 && column[e] <= GD_SW;
    }
    bool fff = (hot.bits & GD_HOT_FRONT) != 0;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      bool visible = evis[e] && hasColumns;
      bool ownsLeft = fff ? (e == 0) : (e == 1);
      if (visible && ownsLeft) isl = column[e];
      if (visible && !ownsLeft) isr = column[e];
    }
    if (evis[0] && evis[1]) {
      isl = column[fff ? 0 : 1];
      isr = column[fff ? 1 : 0];
      hasColumns = isr > isl;
    }
    hasColumns = hasColumns && (wv.sr > wv.sl);
    hot.span = ((unsigned)isl & 0xFFFFu) | (hasColumns ? (unsigned)isr << 16 : 0u);
  }
}

/* ---- phase: blocking ray cast of column x (engine.py:10534-10557) ------- */
/* Nearest one-sided wall the column ray crosses; among equal distances the
 * lowest wall index, as the reference's first-minimum over its ascending
 * blocking list.  Only walls that passed the frustum test can be crossed, and
 * the division is spent only on walls the sign test says are crossed. */
__device__ void gd_blocking_raycast(const GdScene &sc_, const short *list, int listed, float rx, float ry, float &wallDistance,
                                    int &blockingWall) {
  const GdScene &sc = *gd_as_shared(&sc_);
  float best = GD_INF;
  int bestWall = GD_CHECK_INDEX(sc.blocking[0], sc.W);
#pragma unroll 1
  for (int i = 0; i < listed; ++i) {
    const int w = list[i];
    if (!(gd_hot(w).bits & GD_HOT_ONESIDED)) continue;
    const GdHot h = gd_hot(w);
    if (!gd_ray_geo(h, rx, ry)) continue;
    const float d = h.dn / (rx * h.segy - ry * h.segx);
    if (d < best || (d == best && w < bestWall && isfinite(d))) { best = d; bestWall = w; }
  }
  blockingWall = bestWall;
  wallDistance = fminf(fmaxf(best, 1.0f), 4096.0f);
}

#endif

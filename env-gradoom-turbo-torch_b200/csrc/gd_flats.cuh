/* Point-in-sector tests and the per-pixel flat fallback layer.
 * Part of gd_render.cu (one translation unit); not meant to be included elsewhere. */
#ifndef GD_FLATS_CUH
#define GD_FLATS_CUH

/* ---- point in sector (engine.py:9598-9617) ------------------------------ */
/* Crossing parity of a +x ray over the sector's edges.  The bounding box only
 * skips sectors whose parity is provably even. */
__device__ __forceinline__ bool gd_outside_box(const GdScene &sc, int s, float px, float py) {
  const float4 bb = *reinterpret_cast<const float4 *>(&sc.secBBox[s * 4]);
  return py >= bb.w || py < bb.z                             /* no edge straddles the ray's row */
         || px > bb.y + 1.0f                                 /* every crossing lies left of the point */
         || (px < bb.x - 1.0f && sc.secI[s * 4 + 3]);        /* closed loops cross an even number of times */
}
__device__ __forceinline__ bool gd_crosses_edge(const GdScene &sc, int k, float px, float py) {
  const float4 e = *reinterpret_cast<const float4 *>(&sc.walls[GD_CHECK_INDEX(sc.edgeWalls[k], sc.W) * 4]);
  const bool crosses = (e.y > py) != (e.w > py);
  const float dy = e.w - e.y;
  const float safe = fabsf(dy) < 1e-6f ? 1.0f : dy;
  const float cx = e.x + (py - e.y) * (e.z - e.x) / safe;
  return crosses && (px < cx);
}
__device__ __forceinline__ bool gd_point_in_sector(const GdScene &sc, int s, float px, float py) {
  s = GD_CHECK_SECTOR(s, sc.S);
  if (gd_outside_box(sc, s, px, py)) return false;
  int crossings = 0;
#pragma unroll 1
  for (int k = sc.edgeOff[s]; k < sc.edgeOff[s + 1]; ++k) crossings += gd_crosses_edge(sc, k, px, py) ? 1 : 0;
  return crossings & 1;
}

/* The cell of a point; any cell will do for a point that is not a number, no sector contains it. */
__device__ __forceinline__ int gd_cell_axis(float c, float c0, float per) { return min(max((int)((c - c0) * per), 0), GD_CELLS - 1); }
__device__ __forceinline__ int gd_cell(const GdCells &g, float px, float py) {
  return gd_cell_axis(py, g.y0, g.perY) * GD_CELLS + gd_cell_axis(px, g.x0, g.perX);
}

/* Along a ray (rc, rs) the points only move on: once one is past every sector in the ray's direction (the roundings
 * are monotone, so is the distance from group to group), no later one lies in a sector. */
__device__ __forceinline__ bool gd_past_map(const GdCells &g, float px, float py, float rc, float rs) {
  return (rc > 0 && px > g.xHi) || (rc < 0 && px < g.xLo) || (rs > 0 && py >= g.yHi) || (rs < 0 && py < g.yLo);
}

/* The lowest-numbered sector of height group g (f: floors, else ceilings) below `end` that contains the point,
 * or -1.  A point's cell names the one to four sectors that can; testing all of a group's took most of the
 * time of views with many such pixels (a lane of the 256-sector map: 11 million cycles at worst, now 4). */
__device__ __noinline__ int gd_group_sector(const GdScene &sc_, int f, int g, float px, float py, int end) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const GdCells &cells = *sc.cells;
  uint4 list = *reinterpret_cast<const uint4 *>(cells.cell[gd_cell(cells, px, py)]);
  const int count = (int)(list.x & 0xFFFFu);
  const bool listed = count <= GD_CELL_SECTORS;
  const float height = sc.groupH[f][g];
  int k = listed ? 0 : sc.groupOff[f][g];
  const int k1 = listed ? count : sc.groupOff[f][g + 1];
#pragma unroll 1
  for (; k < k1; ++k) {
    list.x = __funnelshift_r(list.x, list.y, 16); list.y = __funnelshift_r(list.y, list.z, 16);
    list.z = __funnelshift_r(list.z, list.w, 16); list.w >>= 16;
    const int s = GD_CHECK_SECTOR(listed ? (int)(list.x & 0xFFFFu) : sc.groupSec[f][k], sc.S);
    if (s >= end) break;
    if (listed && sc.secF[s * 2 + (f ? 0 : 1)] != height) continue;
    if (gd_point_in_sector(sc, s, px, py)) return s;
  }
  return -1;
}

/* Lowest-numbered sector that contains a point (engine.py:9598-9617), 0x7fffffff for none; by eight threads.  What bounds
 * it is a chain of loads, so the few sectors of the point's cell are looked at one after the other, an edge a thread (it
 * was a sector a thread, edge after edge, and a warp for each point: one lane alone 114 us a step, now 112).  Where the cell has no list, each thread takes
 * every eighth sector. */
#define GD_POINT_THREADS 8
__device__ __forceinline__ int gd_sector_of_point(const GdScene &sc, float px, float py) {
  const unsigned short *cell = sc.cells->cell[gd_cell(*sc.cells, px, py)];
  const int lane = threadIdx.x & (GD_POINT_THREADS - 1), count = cell[0];
  const unsigned group = ((1u << GD_POINT_THREADS) - 1u) << (threadIdx.x & 31 & ~(GD_POINT_THREADS - 1));
  unsigned found = 0x7fffffff;
  if (count <= GD_CELL_SECTORS) {
#pragma unroll 1
    for (int i = 0; i < count && found == 0x7fffffff; ++i) {
      const int s = GD_CHECK_SECTOR(cell[1 + i], sc.S);
      if (gd_outside_box(sc, s, px, py)) continue;
      bool odd = false;
#pragma unroll 1
      for (int k = sc.edgeOff[s] + lane; k < sc.edgeOff[s + 1]; k += GD_POINT_THREADS) odd = odd != gd_crosses_edge(sc, k, px, py);
      if (__popc(__ballot_sync(group, odd)) & 1) found = (unsigned)s;
    }
    return (int)found;
  }
#pragma unroll 1
  for (int s = lane; s < sc.S; s += GD_POINT_THREADS)
    if (gd_point_in_sector(sc, s, px, py)) { found = (unsigned)s; break; }
  return (int)__reduce_min_sync(group, found);
}

/* Flat-fallback resolution of a pixel (engine.py:10961-11026): true when the
 * column ray meets no sector's plane inside that sector's polygon. */
__device__ __noinline__ bool gd_pixel_unresolved(const GdScene &sc_, const GdView &v_, int x, int y, int hint) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const GdView &v = *gd_as_shared(&v_);
  const float rayAngle = v.angle + sc.rayOffsets[x], rc = cosf(rayAngle), rs = sinf(rayAngle);
  i64 ti = gd_clamp((GD_ANG90 - v.pitchBam) >> 19, 0, 4095);
  i64 offFixed = ((i64)sc.fineTan[ti] * 12582912LL) >> 16;
  float center = 103.5f + (float)offFixed / 65536.0f;
  float cc = sc.rayCosCorr[x];
  float delta = (float)y - center;
  bool floorPixel = delta > 0;
  float den = fmaxf(fabsf(delta), 0.5f);
  /* An existence test, so the order is free: `hint` (the sector whose plane
   * was marked on this pixel) is nearly always the one that answers it; the
   * others are visited by plane height, one plane point per distinct height. */
  {
    float ph = floorPixel ? (v.viewZ - sc.secF[hint * 2]) : (sc.secF[hint * 2 + 1] - v.viewZ);
    float cd = ph * 192.0f / den / cc;
    if (ph > 0 && isfinite(cd) && cd > 0 && gd_point_in_sector(sc, hint, v.x + rc * cd, v.y + rs * cd)) return false;
  }
  const int f = floorPixel ? 1 : 0;
  const float *gh = sc.groupH[f];
#pragma unroll 1
  for (int g = 0; g < sc.groups[f]; ++g) {
    float ph = floorPixel ? (v.viewZ - gh[g]) : (gh[g] - v.viewZ);
    float perp = ph * 192.0f / den;
    float cd = perp / cc;
    if (!(ph > 0) || !isfinite(cd) || !(cd > 0)) continue;
    float px = v.x + rc * cd, py = v.y + rs * cd;
    if (gd_past_map(*sc.cells, px, py, rc, rs)) break;
    if (gd_group_sector(sc, f, g, px, py, 0x7fffffff) >= 0) return false;
  }
  return true;
}

/* Row of the horizon, for gd_plane_depth. */
__device__ __forceinline__ float gd_flat_center(const GdScene &sc, const GdView &v) {
  i64 ti = gd_clamp((GD_ANG90 - v.pitchBam) >> 19, 0, 4095);
  i64 offFixed = ((i64)sc.fineTan[ti] * 12582912LL) >> 16;
  return (103.0f + (float)offFixed / 65536.0f) + 0.5f;
}
__device__ __forceinline__ float gd_plane_depth(const GdScene &sc, const GdView &v, float flatCenter, int sector, bool isFloor, int y) {
  float ph = isFloor ? (v.viewZ - gd_sec_floor(sc, sector)) : (gd_sec_ceil(sc, sector) - v.viewZ);
  float den = fmaxf(fabsf((float)y - flatCenter), 0.5f);
  return ph * 192.0f / den;
}

__device__ __forceinline__ float gd_wrap_angle(float a) {
  const float pi = 3.14159265358979323846f, twoPi = 6.28318530717958647692f;
  float t = a + pi;
  float r = fmodf(t, twoPi);
  if (r != 0 && (r < 0)) r += twoPi;
  return r - pi;
}

/* ---- per-pixel flat fallback (engine.py:10956-11171) ------------------------
 * Only pixels that no seg and no visplane claimed show this layer, so it is
 * evaluated lazily for exactly those pixels.  The reference resolves every
 * pixel, repairs unresolved ones from the next resolved row below and then
 * from the nearest anchors left and right; here a pixel that resolves by
 * itself costs one probe, and only when some do not is the repair state built, for
 * the columns near them as a rule. */
struct GdFlatProbe { bool unresolved, isFloor; int sector; };

/* the part of a probe that depends on the column only */
struct GdFlatRay { float rc, rs, cc, center; };

/* Per-lane bounds that let a probe prove "no sector" without visiting any:
 * the smallest positive plane height of either orientation (the nearest plane
 * point of every sector lies at least that far along the ray) and the box
 * outside which gd_point_in_sector rejects every sector. */
struct GdFlatBounds { float phFloor, phCeil, xHi, xLo, yHi, yLo; int allClosed; };

__device__ __forceinline__ GdFlatBounds gd_flat_bounds_load(const int *misc) {
  GdFlatBounds b;
  b.phFloor = __int_as_float(misc[4]); b.phCeil = __int_as_float(misc[5]);
  b.xHi = __int_as_float(misc[6]); b.xLo = __int_as_float(misc[7]);
  b.yHi = __int_as_float(misc[8]); b.yLo = __int_as_float(misc[9]);
  b.allClosed = misc[10];
  return b;
}

/* warp 0 fills misc[4..10] */
__device__ void gd_flat_bounds_setup(const GdScene &sc, const GdView &v, int *misc) {
  const int lane = threadIdx.x & 31;
  float phF = GD_INF, phC = GD_INF, xHi = -GD_INF, xLo = GD_INF, yHi = -GD_INF, yLo = GD_INF;
  int closed = 1;
#pragma unroll 1
  for (int s = lane; s < sc.S; s += 32) {
    float f = v.viewZ - sc.secF[s * 2], c = sc.secF[s * 2 + 1] - v.viewZ;
    if (f > 0) phF = fminf(phF, f);
    if (c > 0) phC = fminf(phC, c);
    const float4 bb = *reinterpret_cast<const float4 *>(&sc.secBBox[s * 4]);
    xHi = fmaxf(xHi, bb.y + 1.0f);
    xLo = fminf(xLo, bb.x - 1.0f);
    yHi = fmaxf(yHi, bb.w);
    yLo = fminf(yLo, bb.z);
    closed &= sc.secI[s * 4 + 3] != 0;
  }
#pragma unroll 1
  for (int o = 16; o > 0; o >>= 1) {
    phF = fminf(phF, __shfl_xor_sync(0xffffffffu, phF, o));
    phC = fminf(phC, __shfl_xor_sync(0xffffffffu, phC, o));
    xHi = fmaxf(xHi, __shfl_xor_sync(0xffffffffu, xHi, o));
    xLo = fminf(xLo, __shfl_xor_sync(0xffffffffu, xLo, o));
    yHi = fmaxf(yHi, __shfl_xor_sync(0xffffffffu, yHi, o));
    yLo = fminf(yLo, __shfl_xor_sync(0xffffffffu, yLo, o));
    closed &= __shfl_xor_sync(0xffffffffu, closed, o);
  }
  if (lane == 0) {
    misc[4] = __float_as_int(phF); misc[5] = __float_as_int(phC);
    misc[6] = __float_as_int(xHi); misc[7] = __float_as_int(xLo);
    misc[8] = __float_as_int(yHi); misc[9] = __float_as_int(yLo);
    misc[10] = closed;
  }
}

__device__ __noinline__ GdFlatRay gd_flat_ray(const GdScene &sc_, const GdView &v_, int x) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const GdView &v = *gd_as_shared(&v_);
  i64 ti = gd_clamp((GD_ANG90 - v.pitchBam) >> 19, 0, 4095);
  i64 offFixed = ((i64)sc.fineTan[ti] * 12582912LL) >> 16;
  GdFlatRay r;
  r.center = 103.5f + (float)offFixed / 65536.0f;
  float rayAngle = v.angle + sc.rayOffsets[x];
  r.rc = cosf(rayAngle);
  r.rs = sinf(rayAngle);
  r.cc = sc.rayCosCorr[x];
  return r;
}

/* The bounds are set up.  Neither they nor the ray are passed through local memory, which the L1 has little room for. */
__device__ __noinline__ GdFlatProbe gd_flat_probe(const GdScene &sc_, const GdView &v_, GdFlatRay r, int y, int currentSector) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const GdView &v = *gd_as_shared(&v_);
  const GdFlatBounds b = gd_flat_bounds_load((const int *)(gd_smem + GD_OFF_MISC));
  float delta = (float)y - r.center;
  GdFlatProbe out;
  out.isFloor = delta > 0;
  float den = fmaxf(fabsf(delta), 0.5f);
  out.sector = currentSector;
  out.unresolved = true;
  {
    /* Every sector's plane point lies at cd >= cd0 along the ray, and each
     * coordinate moves monotonically with cd (the roundings are monotone too):
     * once the nearest candidate is past the box on the side the ray is
     * heading to, every sector rejects every candidate. */
    float ph0 = out.isFloor ? b.phFloor : b.phCeil;
    float cd0 = ph0 * 192.0f / den / r.cc;
    if (!isfinite(cd0)) return out;
    if (cd0 > 0) {
      float px0 = v.x + r.rc * cd0, py0 = v.y + r.rs * cd0;
      if (r.rc > 0 && px0 > b.xHi) return out;
      if (r.rc < 0 && b.allClosed && px0 < b.xLo) return out;
      if (r.rs > 0 && py0 >= b.yHi) return out;
      if (r.rs < 0 && py0 < b.yLo) return out;
    }
  }
  /* Sectors are visited by plane height, nearest plane first, so the distance
   * along the ray never decreases from group to group: the first group with a
   * sector that contains its plane point holds the answer, except that a later
   * group whose distance rounds to the same value may still own it with a lower
   * sector index (the reference keeps the first index among equal distances). */
  float best = GD_INF;
  const int f = out.isFloor ? 1 : 0;
  const float *gh = sc.groupH[f];
#pragma unroll 1
  for (int g = 0; g < sc.groups[f]; ++g) {
    float ph = out.isFloor ? (v.viewZ - gh[g]) : (gh[g] - v.viewZ);
    float perp = ph * 192.0f / den;
    float cd = perp / r.cc;
    if (!(ph > 0) || !isfinite(cd) || !(cd > 0)) continue;
    if (cd > best) break;
    float px = v.x + r.rc * cd, py = v.y + r.rs * cd;
    if (gd_past_map(*sc.cells, px, py, r.rc, r.rs)) break;
    const int s = gd_group_sector(sc, f, g, px, py, cd == best ? out.sector + 1 : 0x7fffffff);
    if (s >= 0) { best = cd; out.sector = s; }
  }
  out.unresolved = !isfinite(best);
  return out;
}

/* Repairs, for the `c` listed columns, rows minY .. maxY: `vsec` gets the vertically repaired sector of every such pixel,
 * and `anchors` a bit per pixel telling whether it anchors horizontal spans.  First every pixel is probed; then the columns
 * that are unresolved at maxY have the nearest resolved row below it looked for, of its orientation; then a thread a
 * column carries the nearest resolved row upwards.  The threads are dealt to the columns evenly, so that each keeps its
 * column's ray (600 viewers outside the 64-sector map 9879 us with a ray a pixel, now 9269), and the fewer columns are left
 * without a resolved row the more threads look for it, at GD_FLAT_ROWS rows or so between two barriers.  All columns'
 * anchors are stored a warp's word at a time (140 rows: an atomic an anchor 277 of a lane's 2400 thousand cycles). */
#define GD_FLAT_UNRESOLVED 0xFFFFu
#define GD_FLAT_ROWS 8
__device__ __noinline__ void gd_flat_sweep(const GdScene &sc_, const GdView &v_, const GdShared &sh_, int currentSector,
                                           unsigned short *vsec, int c, int minY, int maxY) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const GdView &v = *gd_as_shared(&v_);
  const GdShared &sh = *gd_as_shared(&sh_);
  const int tid = threadIdx.x;
  unsigned *first = (unsigned *)(gd_smem + GD_OFF_AUX2);             /* row << 16 | sector */
  const short *list = (const short *)(gd_smem + GD_OFF_FLAT_LIST);
  short *pending = (short *)(gd_smem + GD_OFF_FLAT_LIST) + GD_SW, *others = pending + GD_SW;
  int *count = (int *)(gd_smem + GD_OFF_MISC) + 13;
  const int flipRow = gd_clamp((int)floorf(gd_flat_ray(sc, v, 0).center) + 1, 0, GD_VH);   /* first floor row */
  const int limit = maxY < flipRow ? flipRow : GD_VH;
  if (tid == 0) *count = 0;
#pragma unroll 1
  for (int i = tid; i < (maxY - minY + 1) * GD_WARPS; i += GD_THREADS) sh.anchors[minY * GD_WARPS + i] = 0u;
  const int each = GD_THREADS / c;                                   /* threads of a column */
  if (tid < each * c) {
    const int x = list[tid % c];
    const GdFlatRay r = gd_flat_ray(sc, v, x);
#pragma unroll 1
    for (int y = minY + tid / c; y <= maxY; y += each) {
      const GdFlatProbe q = gd_flat_probe(sc, v, r, y, currentSector);
      vsec[y * GD_SW + x] = (unsigned short)(q.unresolved ? GD_FLAT_UNRESOLVED : (unsigned)q.sector);
    }
  }
  __threadfence_block();
  __syncthreads();
  if (tid < c) {
    first[tid] = 0xffffffffu;
    if (vsec[maxY * GD_SW + list[tid]] == GD_FLAT_UNRESOLVED) pending[atomicAdd(count, 1)] = (short)tid;
  }
  __syncthreads();
  int n = *count;
  __syncthreads();
#pragma unroll 1
  for (int y = maxY + 1; n > 0 && y < limit;) {
    const int k = GD_THREADS / n, i = tid / k, end = min(y + max(k, GD_FLAT_ROWS / k * k), limit);
    if (tid == 0) *count = 0;
    __syncthreads();
    if (i < n) {
      const GdFlatRay r = gd_flat_ray(sc, v, list[pending[i]]);
#pragma unroll 1
      for (int row = y + tid % k; row < end; row += k) {
        const GdFlatProbe q = gd_flat_probe(sc, v, r, row, currentSector);
        if (q.unresolved) continue;
        atomicMin(&first[pending[i]], ((unsigned)row << 16) | (unsigned)q.sector);
        break;
      }
    }
    __syncthreads();
    if (tid < n && first[pending[tid]] == 0xffffffffu) others[atomicAdd(count, 1)] = pending[tid];
    __syncthreads();
    n = *count;
    y = end;
    short *swap = pending; pending = others; others = swap;
    __syncthreads();
  }
  if (tid < c) {
    const int x = list[tid];
    bool haveBelow = first[tid] != 0xffffffffu, belowFloor = (int)(first[tid] >> 16) >= flipRow;
    int belowSector = (int)(first[tid] & 0xFFFFu);
    unsigned next = vsec[maxY * GD_SW + x];
#pragma unroll 1
    for (int y = maxY; y >= minY; --y) {
      const unsigned own = next;
      if (y > minY) next = vsec[(y - 1) * GD_SW + x];
      const bool isFloor = y >= flipRow;
      bool anchor = true;
      int repaired = (int)own;
      if (own != GD_FLAT_UNRESOLVED) {
        haveBelow = true; belowFloor = isFloor; belowSector = repaired;
      } else {
        const bool spans = haveBelow && belowFloor == isFloor;
        repaired = spans ? belowSector : currentSector;
        anchor = spans && belowSector != currentSector;
      }
      vsec[y * GD_SW + x] = (unsigned short)repaired;
      unsigned *word = &sh.anchors[y * GD_WARPS + (x >> 5)];
      if (c == GD_SW) {                                              /* thread x has column x */
        const unsigned bits = __ballot_sync(0xffffffffu, anchor);
        if ((x & 31) == 0) *word = bits;
      } else if (anchor) {
        atomicOr(word, 1u << (x & 31));
      }
    }
  }
  __threadfence_block();
  __syncthreads();
}

/* Draws the queued pixels that are left: each with its own repaired sector, or with the one its nearest anchors left and
 * right agree on.  Only columns up to `window` from a pixel's own have been repaired: one whose anchors may lie
 * farther away stays in the queue, and misc[12] tells. */
__device__ __noinline__ void gd_flat_repaired(const GdScene &sc_, const GdView &v_, const GdShared &sh_, const unsigned short *vsec, int *queue,
                                              int count, int window) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const GdView &v = *gd_as_shared(&v_);
  const GdShared &sh = *gd_as_shared(&sh_);
#pragma unroll 1
  for (int i = threadIdx.x; i < count; i += GD_THREADS) {
    if (queue[i] < 0) continue;
    const int px = queue[i] & 0xFFFF, py = queue[i] >> 16;
    int sector = vsec[py * GD_SW + px];
    /* nearest anchor at or left of px, at or right of px */
    int left = -1, right = -1;
#pragma unroll 1
    for (int w = 0; w < GD_WARPS; ++w) {
      unsigned bits = sh.anchors[py * GD_WARPS + w];
      int base = w * 32;
      if (base <= px) {
        unsigned lo = px - base >= 31 ? bits : (bits & ((2u << (px - base)) - 1u));
        if (lo) left = base + 31 - __clz(lo);
      }
      if (base + 31 >= px && right < 0) {
        unsigned hi = px - base <= 0 ? bits : (bits & ~((1u << (px - base)) - 1u));
        if (hi) right = base + __ffs(hi) - 1;
      }
    }
    const bool sure = px - left <= window && (right >= 0 ? right : GD_SW) - px <= window;   /* no anchor up to the edge counts too */
    if (!sure) { sh.misc[12] = 1; continue; }
    if (left >= 0 && right >= 0) {
      int sl = vsec[py * GD_SW + left], sr = vsec[py * GD_SW + right];
      if (sl == sr) sector = sl;
    }
    const bool isFloor = ((float)py - gd_flat_ray(sc, v, px).center) > 0;
    GdPlaneSpan p;
    gd_plane_setup(sc, sh.planeTab, sector, isFloor, px, p);
    sh.frame[py * GD_SW + px] = (uint8_t)gd_plane_pixel(sc, p, v.center, py);
    atomicOr(&sh.masks[(py >> 5) * GD_SW + px], 1u << (py & 31));
    queue[i] = -1;
  }
}

/* Pass over the queued pixels.
 *   A  one thread per queued pixel probes it; a resolved pixel is drawn at
 *      once and leaves the queue.
 *   B  Only when unresolved pixels remain: the columns near theirs are repaired in their rows, which as a rule says what
 *      they are.  Unresolved pixels are few and lie in a column or two where two lines meet, near the horizon, and repairing
 *      all 320 columns, down to the first resolved row in each, took up to 1.2 million of a lane's cycles (148 lanes of the
 *      64-sector map: 325 us a step, now 253; 1024 lanes with RGB24 1313 and 891).  With 3 or 20 columns either side
 *      the times are the same.
 *   C  Pixels whose anchors lie farther away, or too many columns: all columns are repaired, once per lane, in the rows
 *      of every pixel that is still unclaimed. */
#define GD_FLAT_WINDOW 8
__device__ void gd_fallback_pass(const GdScene &sc_, const GdView &v_, const GdShared &sh_, int currentSector,
                                 unsigned short *vsec, bool &sweepDone) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const GdView &v = *gd_as_shared(&v_);
  const GdShared &sh = *gd_as_shared(&sh_);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int queued = sh.misc[1], count = min(queued, GD_FALLBACK_MAX);
  int *queue = (int *)sh.hitD;
  unsigned *owned = sh.masks;                        /* drawn pixels are marked as claimed */
  unsigned *columns = sh.ownerMask;                  /* with unresolved pixels; 16 words on: to be repaired */
  short *list = (short *)(gd_smem + GD_OFF_FLAT_LIST);
  if (tid == 0) { sh.misc[2] = GD_VH; sh.misc[3] = -1; sh.misc[11] = 0; sh.misc[12] = 0; }
  if (tid < GD_WARPS) columns[tid] = 0u;
  if (warp == 0) gd_flat_bounds_setup(sc, v, sh.misc);
  __syncthreads();
#pragma unroll 1
  for (int i = tid; i < count; i += GD_THREADS) {
    const int px = queue[i] & 0xFFFF, py = queue[i] >> 16;
    const GdFlatRay r = gd_flat_ray(sc, v, px);
    GdFlatProbe own = gd_flat_probe(sc, v, r, py, currentSector);
    if (!own.unresolved) {
      GdPlaneSpan p;
      gd_plane_setup(sc, sh.planeTab, own.sector, own.isFloor, px, p);
      sh.frame[py * GD_SW + px] = (uint8_t)gd_plane_pixel(sc, p, v.center, py);
      atomicOr(&owned[(py >> 5) * GD_SW + px], 1u << (py & 31));
      queue[i] = -1;
    } else {
      sh.misc[11] = 1;
      atomicMin(&sh.misc[2], py); atomicMax(&sh.misc[3], py);
      atomicOr(&columns[px >> 5], 1u << (px & 31));
    }
  }
  __syncthreads();
  if (sh.misc[11] == 0) return;                       /* block-uniform: nothing unresolved */
  if (!sweepDone) {
    if (queued <= GD_FALLBACK_MAX) {
      if (tid < GD_WARPS) {
        const unsigned a = columns[tid], l = tid > 0 ? columns[tid - 1] : 0u, r = tid < GD_WARPS - 1 ? columns[tid + 1] : 0u;
        unsigned near = a;
#pragma unroll 1
        for (int s = 1; s <= GD_FLAT_WINDOW; ++s) near |= (a << s) | (l >> (32 - s)) | (a >> s) | (r << (32 - s));
        columns[16 + tid] = near;
      }
      __syncthreads();
      int c = 0, rank = 0;
#pragma unroll 1
      for (int w = 0; w < GD_WARPS; ++w) {
        const unsigned near = columns[16 + w];
        if (w < warp) rank += __popc(near);
        else if (w == warp) rank += __popc(near & ((1u << (tid & 31)) - 1u));
        c += __popc(near);
      }
      if (c <= GD_SW / 2) {                           /* block-uniform */
        if ((columns[16 + warp] >> (tid & 31)) & 1u) list[rank] = (short)tid;
        const int minY = sh.misc[2], maxY = sh.misc[3];
        __syncthreads();
        gd_flat_sweep(sc, v, sh, currentSector, vsec, c, minY, maxY);
        gd_flat_repaired(sc, v, sh, vsec, queue, count, GD_FLAT_WINDOW);
        __syncthreads();
        if (sh.misc[12] == 0) return;                 /* block-uniform */
      }
    }
    __syncthreads();
    if (tid == 0) { sh.misc[2] = GD_VH; sh.misc[3] = -1; }
    list[tid] = (short)tid;
    __syncthreads();
    {
      const unsigned *own = owned + tid;
      int lo = GD_VH, hi = -1;
#pragma unroll 1
      for (int k = 0; k < 7; ++k) {
        unsigned m = gd_range_word(k, 0, GD_VH) & ~own[k * GD_SW];
        if (m) { lo = min(lo, (k << 5) + __ffs(m) - 1); hi = max(hi, (k << 5) + 31 - __clz(m)); }
      }
      if (hi >= 0) { atomicMin(&sh.misc[2], lo); atomicMax(&sh.misc[3], hi); }
    }
    __syncthreads();
    const int minY = sh.misc[2], maxY = sh.misc[3];
    gd_flat_sweep(sc, v, sh, currentSector, vsec, GD_SW, minY, maxY);
    sweepDone = true;
  }
  gd_flat_repaired(sc, v, sh, vsec, queue, count, GD_SW);
  __syncthreads();
}

#endif

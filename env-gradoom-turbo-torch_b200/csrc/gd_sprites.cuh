/* Sprites, the weapon overlay and the status bar.
 * Part of gd_render.cu (one translation unit); not meant to be included elsewhere. */
#ifndef GD_SPRITES_CUH
#define GD_SPRITES_CUH

/* ---- phase: sprites (engine.py:14138-14228, 14684-14947) ----------------- */
__device__ __noinline__ void gd_actor_setup(const GdScene &sc_, const GdView &v_, const gd_thing &t, int sector,
                                            GdActor &ac) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const GdView &v = *gd_as_shared(&v_);
  ac.alive = (t.flags & GD_THING_ALIVE) != 0;
  ac.style = t.style;
  ac.x = t.x; ac.y = t.y;
  int sprite = t.sprite < sc.P ? t.sprite : 0;
  ac.sprite = sprite;
  const int4 si = *reinterpret_cast<const int4 *>(&sc.sprInfo[sprite * 4]);
  ac.w = si.x; ac.h = si.y;
#ifdef GD_CHECKED
  {
    /* a record that names no patch of the scene, or lies nowhere, is not drawn */
    const bool badIndex = t.sprite >= sc.P || si.x > sc.sprW || si.y > sc.sprH || si.x < 0 || si.y < 0;
    const bool badState = !isfinite(t.x) || !isfinite(t.y) || !isfinite(t.z) || sector < 0 || sector >= sc.S;
    if (badIndex) atomicOr(gdCheckedStatus, GD_STATUS_BAD_INDEX);
    if (badState) atomicOr(gdCheckedStatus, GD_STATUS_BAD_STATE);
    if (badIndex || badState) { ac.alive = 0; ac.w = ac.h = 0; if (badState) sector = 0; }
  }
#endif
  float dx = t.x - v.x, dy = t.y - v.y;
  float dist = sqrtf(dx * dx + dy * dy);
  if (dist < 1.0f) dist = 1.0f;
  float rel = gd_wrap_angle(atan2f(dy, dx) - v.angle);
  ac.depth = dist * cosf(rel);
  i64 ax = gd_rint(t.x * 65536.0f), ay = gd_rint(t.y * 65536.0f);
  i64 rx = ax - v.vx, ry = ay - v.vy;
  i64 depthFixed = (rx * v.vcos + ry * v.vsin) >> 20;
  i64 sideFixed = (rx * v.vsin - ry * v.vcos) >> 16;
  ac.depthFixed = depthFixed;
  i64 xscale = gd_div(GD_FOCAL_X << 12, gd_max(depthFixed, GD_SPRITE_MIN_DEPTH));
  i64 leftFixed = sideFixed - (i64)si.z * GD_FU;
  i64 left = 160 + (gd_wmul(leftFixed, xscale) >> 32);
  i64 rightFixed = leftFixed + (i64)si.x * GD_FU;
  i64 right = 160 + (gd_wmul(rightFixed, xscale) >> 32);
  ac.xstep = gd_div((i64)si.x << 16, gd_max(right - left, 1));
  ac.left = (int)gd_clamp(left, -(1 << 30), 1 << 30);
  ac.right = (int)gd_clamp(right, -(1 << 30), 1 << 30);
  ac.yscale = gd_div(GD_FOCAL_Y << 12, gd_max(depthFixed, GD_SPRITE_MIN_DEPTH));
  const i64 texMid = (i64)si.w * GD_FU - gd_rint((v.viewZ - t.z) * 65536.0f);
  ac.topFixed = v.center - (gd_wmul(texMid, ac.yscale) >> 16);
  ac.iscale = gd_div(GD_U32MASK, gd_max(ac.yscale, 1));
  ac.fracBase = texMid - (gd_wmul(v.center - GD_FU, ac.iscale) >> 16);
  ac.row0 = 0; ac.row1 = GD_VH;
  if (ac.iscale > 0) {
    /* frac(y) >> 16 in [0,h)  <=>  0 <= fracBase + y*iscale < h*FU */
    const i64 lo = -ac.fracBase, hi = (i64)ac.h * GD_FU - ac.fracBase;
    ac.row0 = (short)gd_clamp(lo <= 0 ? 0 : gd_div(lo + ac.iscale - 1, ac.iscale), 0, GD_VH);
    ac.row1 = (short)gd_clamp(hi <= 0 ? 0 : gd_div(hi + ac.iscale - 1, ac.iscale), 0, GD_VH);
  }
  i64 light = sc.secI[sector * 4] + v.flashLight * 16;
  if (t.flags & GD_THING_BRIGHT) light = 255;
  float base = 61.0f - (float)light / 4.0f;
  float visf = fminf(1280.0f / fmaxf(ac.depth, 1.0f), 24.0f);
  ac.shade = (short)gd_clamp((i64)floorf(base - visf), 0, 31);
}

__device__ __forceinline__ bool gd_behind(const GdScene &sc, const GdWall &wv, int w, const GdActor &ac) {
  i64 nearD = gd_min(wv.dl, wv.dr), farD = gd_max(wv.dl, wv.dr);
  const float4 g = *reinterpret_cast<const float4 *>(&sc.walls[w * 4]);
  float dx = g.z - g.x, dy = g.w - g.y;
  float side = dx * (ac.y - g.y) - dy * (ac.x - g.x);
  return (nearD > ac.depthFixed) || ((farD > ac.depthFixed) && (side <= 0));
}

/* The things that may show in column x = threadIdx.x (engine.py:14684-14720): in front of the viewer, across the
 * column, and not behind the nearest one-sided wall of the column's ray.  The ray is cast where a thing lies across
 * the column at all: most warps have none (one lane alone: 120 us a step, 117 without the other rays). */
__device__ __noinline__ unsigned long long gd_sprite_candidates(const GdScene &sc_, const GdView &v_, const GdShared &sh_, int nThings,
                                                                const short *list, int listed) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const GdView &v = *gd_as_shared(&v_);
  const GdShared &sh = *gd_as_shared(&sh_);
  const int x0 = threadIdx.x;
  unsigned long long across = 0;
#pragma unroll 1
  for (int a = 0; a < nThings; ++a) {
    const GdActor &ac = *gd_as_shared(&sh.actors[a]);
    if (ac.alive && x0 >= ac.left && x0 < ac.right && ac.depth > 0) across |= 1ull << a;
  }
  if (!across) return 0;
  float rx, ry, wd;
  int bw;
  gd_ray(v, x0, rx, ry);
  gd_blocking_raycast(sc, list, listed, rx, ry, wd, bw);
  const GdWall &bwv = sh.walls[bw];
  unsigned long long cand = 0;
#pragma unroll 1
  while (across) {
    const int a = __ffsll((long long)across) - 1;
    across &= across - 1;
    const GdActor &ac = *gd_as_shared(&sh.actors[a]);
    if (ac.depth < wd || !(x0 >= bwv.sl && x0 < bwv.sr) || gd_behind(sc, bwv, bw, ac)) cand |= 1ull << a;
  }
  return cand;
}

/* Sprites cluster in a few screen columns, so the drawing is spread by rows:
 * the columns with candidates are listed; then the warps take
 * the listed columns from a counter and draw each candidate's rows 32 at a
 * time, far to near.  A column's clip events are fetched once, by all threads of the warp at once, into its
 * share of shared memory, and what a thing's depth says about each of them (gd_behind) is decided once per thing,
 * one event a thread, so that a row's loop over the events reads nothing from global memory. */
#define GD_SPRITE_EVENTS (GD_MAX_EVENTS * 20)      /* bytes per warp: 16 of clip rows and 4 of wall and sector an event */
static_assert(GD_SPRITE_EVENTS * GD_WARPS <= GD_AUX_BYTES && GD_SPRITE_EVENTS % 16 == 0, "staged events");
__device__ void gd_sprites(const GdScene &sc_, const GdView &v_, const GdShared &sh_, const GdEvent *events,
                           const int *eventCount, int nThings) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const GdView &v = *gd_as_shared(&v_);
  const GdShared &sh = *gd_as_shared(&sh_);
  const int x0 = threadIdx.x, lane = threadIdx.x & 31;
  if (nThings <= 0) return;                          /* block-uniform */
  const unsigned long long *candOf = (const unsigned long long *)(gd_smem + GD_OFF_CAND);
  short *list = (short *)sh.hitA;
  int *counters = &sh.misc[2];                       /* [0] listed columns, [1] next to draw */
  if (x0 == 0) { counters[0] = 0; counters[1] = 0; }
  __syncthreads();
  if (candOf[x0]) list[atomicAdd(&counters[0], 1)] = (short)x0;
  __syncthreads();
  const int listed = counters[0];
  const float flatCenter = gd_flat_center(sc, v);
  uint4 *staged = (uint4 *)(gd_smem + GD_OFF_AUX + (x0 >> 5) * GD_SPRITE_EVENTS);   /* distance, tiers, silhouettes, plane marks */
  unsigned *owners = (unsigned *)(staged + GD_MAX_EVENTS);
  for (;;) {
    int slot = 0;
    if (lane == 0) slot = atomicAdd(&counters[1], 1);
    slot = __shfl_sync(0xffffffffu, slot, 0);
    if (slot >= listed) break;
    const int x = list[slot];
    unsigned long long cand = candOf[x];
    const int nEv = eventCount[x];
    __syncwarp();                                      /* the column before has read its events */
#pragma unroll 1
    for (int e = lane; e < nEv; e += 32) {
      const unsigned *ev = (const unsigned *)&events[e * GD_SW + x];
      staged[e] = make_uint4(ev[0], ev[2], ev[3], ev[4]);
      owners[e] = ev[1];
    }
    __syncwarp();
    /* the walk goes front to back: as a rule the first event that covers a row is the nearest one (4096 lanes of the
     * 64-sector map: 3315 us a step with every event looked at, 3251 without) */
    bool sorted = true;
#pragma unroll 1
    for (int e = lane + 1; e < nEv; e += 32) sorted = sorted && __uint_as_float(staged[e].x) >= __uint_as_float(staged[e - 1].x);
    sorted = __all_sync(0xffffffffu, sorted);
    /* far to near: repeatedly take the remaining candidate with the largest
     * (depth, index) key */
#pragma unroll 1
    while (cand) {
      int pick = -1;
      float pd = 0.0f;
      unsigned long long m = cand;
#pragma unroll 1
      while (m) {
        int a = __ffsll((long long)m) - 1;
        m &= m - 1;
        float d = sh.actors[a].depth;
        if (pick < 0 || d >= pd) { pick = a; pd = d; }
      }
      cand &= ~(1ull << pick);
      const GdActor &ac = sh.actors[pick];
      i64 u = (((i64)x - ac.left) * ac.xstep) >> 16;
      if (u < 0 || u >= ac.w) continue;
      const uint8_t *cm = sh.colormap + ac.shade * 256;
      const i64 fracBase = ac.fracBase;
      const int y0 = ac.row0, y1 = ac.row1;            /* two divisions that every column made for itself before
                                                        * (256 sectors, 32 things: 14653 us a step, now 14271) */
      unsigned long long behind = 0;                 /* events whose wall lies behind the thing */
#pragma unroll 1
      for (int e0 = 0; e0 < nEv; e0 += 32) {
        const int wall = e0 + lane < nEv ? (int)(short)(owners[e0 + lane] & 0xFFFFu) : -1;
        behind |= (unsigned long long)__ballot_sync(0xffffffffu, wall >= 0 && gd_behind(sc, sh.walls[wall], wall, ac)) << e0;
      }
      __syncwarp();                                  /* the farther sprite's pixels are in place */
#pragma unroll 1
      for (int y = y0 + lane; y < y1; y += 32) {
        i64 frac = fracBase + (i64)y * ac.iscale;
        i64 tv = frac >> 16;
        if (tv < 0 || tv >= ac.h) continue;
        size_t si = ((size_t)ac.sprite * sc.sprH + (size_t)tv) * sc.sprW + (size_t)u;
        const uint8_t post = sc.sprPost[si], source = sc.sprAtlas[si];
        if (post == 255) continue;
        i64 postTop = (ac.topFixed + ac.yscale * (i64)post) >> 16;
        if (y < postTop) continue;
        /* nearest clip event covering this pixel */
        float bestD = GD_INF;
        int bestE = -1, ownerSector = -1;
        bool filled = false, ownerFloor = false;
        const unsigned row = (unsigned)y;
#pragma unroll 1
        for (int e = 0; e < nEv; ++e) {
          const uint4 q = staged[e];
          const bool inLower = row >= ((q.y >> 16) & 255u) && row < (q.y >> 24), inUpper = row >= (q.y & 255u) && row < ((q.y >> 8) & 255u);
          const bool drawn = inLower ? (q.w & (2u << 16)) != 0 : (inUpper && (q.w & (1u << 16)) != 0);
          bool covers = row < (q.z & 255u) || row >= ((q.z >> 8) & 255u);
          if (drawn && !filled) { filled = true; covers = true; }
          const float d = __uint_as_float(q.x);
          if (covers && d < bestD) {
            bestD = d; bestE = e;
            if (sorted) break;
          }
          if (ownerSector < 0) {
            const bool onFloor = row >= (q.w & 255u) && row < ((q.w >> 8) & 255u);
            if (onFloor || (row >= ((q.z >> 16) & 255u) && row < (q.z >> 24))) {
              const int sector = (int)(short)(owners[e] >> 16);
              if (sector >= 0) { ownerSector = sector; ownerFloor = onFloor; }
            }
          }
        }
        bool visible;
        if (bestE >= 0) {
          visible = (behind >> bestE) & 1ull;
        } else {
          /* The plane's depth limits the thing only where the pixel resolves to no sector: that search, plane by
           * plane along the ray, is left for things beyond the plane (made for every pixel, and with a test of every
           * sector, it took up to 3.2 million cycles for a thing that fills the view). */
          visible = ac.depth < GD_INF &&
                    (filled || ownerSector < 0 || ac.depth < gd_plane_depth(sc, v, flatCenter, ownerSector, ownerFloor, y) ||
                     !gd_pixel_unresolved(sc, v, x, y, ownerSector));
        }
        if (!visible) continue;
        uint8_t out = cm[source];
        if (ac.style == -2) out = sc.transLut[sh.frame[y * GD_SW + x] * 256 + out];
        else if (ac.style >= 0) out = sc.addLut[((ac.style > 1 ? 1 : ac.style) * 256 + sh.frame[y * GD_SW + x]) * 256 + out];
        sh.frame[y * GD_SW + x] = out;
      }
    }
    __syncwarp();
  }
}

/* ---- phase: weapon (engine.py:14994-15121) ------------------------------ */
#define GD_WEAPON_ROWS 4
__device__ __noinline__ void gd_weapon_patch(const GdScene &sc_, const GdShared &sh_, uint8_t *frame, int id, i64 hoff, i64 voff) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const GdShared &sh = *gd_as_shared(&sh_);
#ifdef GD_CHECKED
  if (id >= sc.Q || id < -1) { if (threadIdx.x == 0) atomicOr(gdCheckedStatus, GD_STATUS_BAD_INDEX); }
#endif
  if (id < 0 || id >= sc.Q) return;
  const int4 wi = *reinterpret_cast<const int4 *>(&sc.wpnInfo[id * 4]);
  int w = wi.x, h = wi.y;
  if (w <= 0 || h <= 0) return;
  i64 screenLeft = (hoff - (i64)wi.z * GD_FU) >> 16;
  i64 texMid = 100 * GD_FU - (32 * GD_FU + 0x6000) - voff + (i64)wi.w * GD_FU;
  const i64 yscale = GD_SCREEN_H * GD_FU / 200;
  const i64 iscale = GD_U32MASK / yscale;
  /* rows whose source row lies inside the patch: 0 <= base + y*iscale < h*FU */
  const i64 base = texMid - (i64)(GD_VH / 2 - 1) * iscale;
  const i64 lo = -base, hi = (i64)h * GD_FU - base;
  const int y0 = (int)gd_clamp(lo <= 0 ? 0 : gd_div(lo + iscale - 1, iscale), 0, GD_VH);
  const int y1 = (int)gd_clamp(hi <= 0 ? 0 : gd_div(hi + iscale - 1, iscale), 0, GD_VH);
  /* a warp takes a row of 32 pixels, GD_WEAPON_ROWS such rows at once: what bounds it is the latency of the texels
   * (a pixel at a time, with a division for each, 13 of a lane's 426 thousand cycles; now 11, and of a lane alone 17 and 10) */
  const uint8_t *opaques = sc.wpnOpaque + (size_t)id * sc.wpnH * sc.wpnW, *texels = sc.wpnAtlas + (size_t)id * sc.wpnH * sc.wpnW;
#pragma unroll 1
  for (int sx = threadIdx.x & 31; sx < w; sx += 32) {
    const i64 xx = screenLeft + sx;
    if (xx < sh.misc[14] || xx >= sh.misc[15]) continue;
    const int cx = min(sx, sc.wpnW - 1);
#pragma unroll 1
    for (int y = y0 + (threadIdx.x >> 5); y < y1; y += GD_WARPS * GD_WEAPON_ROWS) {
      uint8_t opaque[GD_WEAPON_ROWS], texel[GD_WEAPON_ROWS];
#pragma unroll
      for (int r = 0; r < GD_WEAPON_ROWS; ++r) {
        const int row = y + r * GD_WARPS;
        const i64 sy = (base + (i64)row * iscale) >> 16;
        opaque[r] = texel[r] = 0;
        if (row < y1 && sy >= 0 && sy < h) {
          const int si = (int)gd_min(sy, sc.wpnH - 1) * sc.wpnW + cx;
          opaque[r] = opaques[si]; texel[r] = texels[si];
        }
      }
#pragma unroll
      for (int r = 0; r < GD_WEAPON_ROWS; ++r)
        if (opaque[r]) frame[(y + r * GD_WARPS) * GD_SW + (int)xx] = texel[r];
    }
  }
}

__device__ void gd_weapon(const GdScene &sc_, const GdShared &sh, const int32_t *lane, uint8_t *frame) {
  const GdScene &sc = *gd_as_shared(&sc_);
  if (!sc.wpnAvailable) return;
  if (lane[GD_L_FLAGS] & 1) return;
  int weapon = (int)gd_clamp(lane[GD_L_WEAPON], 0, 7);
  int cooldown = (int)gd_clamp(lane[GD_L_WPN_COOLDOWN], 0, sc.wpnTics - 1);
  int parity = (int)gd_pymod(lane[GD_L_WPN_FIRE_COUNT], 2);
  if (weapon == 1 && cooldown == 0) parity = (int)gd_pymod(gd_max(lane[GD_L_WPN_READY_TICS] - 1, 0) / 4, 2);
  int ti = (weapon * 2 + parity) * sc.wpnTics + cooldown;
  int frameId = sc.wpnFrameIds[ti], flashId = sc.wpnFlashIds[ti];
  i64 lowerTics = gd_clamp(16 - (i64)lane[GD_L_WPN_LOWER], 0, 16);
  i64 verticalTics = lane[GD_L_WPN_PENDING] >= 0 ? lowerTics : (i64)lane[GD_L_WPN_RAISE];
  i64 spawnRaise = gd_clamp(14 - ((i64)lane[GD_L_EPISODE_TIME] - 1), 0, 14);
  verticalTics = gd_max(verticalTics, spawnRaise);
  bool ready = lane[GD_L_WPN_COOLDOWN] <= 0 && lane[GD_L_WPN_RAISE] <= 0 && lane[GD_L_WPN_PENDING] < 0;
  i64 bobAngle = ((i64)lane[GD_L_EPISODE_TIME] * 128) & 8191;
  i64 bob = lane[GD_L_BOB_FIXED];
  i64 bobx = (bob * sc.fineSine[(bobAngle + 2048) & 8191]) >> 16;
  i64 boby = (bob * sc.fineSine[bobAngle & 4095]) >> 16;
  if (!ready) { bobx = 0; boby = 0; }
  i64 voff = verticalTics * 6 * GD_FU + boby;
  gd_weapon_patch(sc, sh, frame, frameId, bobx, voff);
  __syncthreads();
  if (flashId >= 0) gd_weapon_patch(sc, sh, frame, flashId, bobx, voff);
}

/* ---- phase: status bar (engine.py:15158-15267) --------------------------- */
/* The status bar is a list of opaque-masked blits drawn in a fixed order, later ones on top.  Every glyph that may
 * be drawn has its place in the list: one thread fills in one place (patch, position, clipped against the canvas),
 * and then every column thread resolves its 32 pixels from the entries that cross its column, topmost first.
 * What bounds it is latency (listing by one thread and dependent loads, row after row, took 15 % of a lane's time),
 * so the list is made beside the other setup, and a warp draws its columns when its walk has ended, while others
 * still walk. */
#define GD_HUD_PATCHES 44      /* bar, arms panel, 3 + 3 + 1 + 3 + 1 large glyphs, face, 6 weapons, 4 x 6 small digits */
static_assert(GD_HUD_PATCHES * 16 <= GD_AUX2_BYTES, "the status-bar list");

/* Place `slot` of a number drawn right-aligned at `right` (engine.py:15180-15210); patch -1: no digit there. */
__device__ __forceinline__ int3 gd_hud_digit(const GdScene &sc, int value, int right, int y, bool small, int slot) {
  const int vc = value < -99 ? -99 : (value > 999 ? 999 : value);
  const int mag = vc < 0 ? -vc : vc;
  const int n = mag > 99 ? 3 : (mag > 9 ? 2 : 1);
  if (slot >= n) return make_int3(-1, 0, 0);
  const int place = n - 1 - slot;                      /* the most significant digit comes first */
  const int digit = place == 2 ? mag / 100 : (place == 1 ? mag / 10 % 10 : mag % 10);
  const int dw = small ? 4 : 14, patch = (small ? 28 : 2) + digit;
  const int4 hi = *reinterpret_cast<const int4 *>(&sc.hudInfo[patch * 4]);
  return make_int3(patch, right - (n - slot) * dw - hi.z, y - hi.w);   /* the blit subtracts the glyph offsets once more */
}

/* Threads 0 .. GD_HUD_PATCHES - 1: entries (tx | ty << 16, cw | ch << 16, sx | sy << 16, patch); cw = 0 when
 * nothing is left. */
__device__ __noinline__ void gd_hud_list(const GdScene &sc_, const int32_t *lane, int4 *entries) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const int t = threadIdx.x;
  if (t >= GD_HUD_PATCHES) return;
  const float hf = __int_as_float(lane[GD_L_HEALTH]), af = __int_as_float(lane[GD_L_ARMOR]);
  const int health = (int)(hf < 0 ? 0.0f : (hf > 999 ? 999.0f : hf));
  const int armor = (int)(af < 0 ? 0.0f : (af > 999 ? 999.0f : af));
  int3 e = make_int3(-1, 0, 0);                        /* patch, x, y */
  int number = 0, right = -1, top = 3, slot = t - 2;   /* right < 0: not a digit */
  if (t < 2) {
    e = make_int3(t, t ? 104 : 0, 0);
  } else if (t < 5) {
    const int weapon = lane[GD_L_WEAPON];
    const int ammoSlot = weapon < 2 ? -1 : (int)((0x54122100u >> (4 * (weapon > 7 ? 7 : weapon))) & 0xF);   /* -,-,1,2,2,1,4,5 */
    number = ammoSlot < 0 ? 0 : (int)__int_as_float(lane[GD_L_READY_AMMO]);
    right = 44;
  } else if (t < 8) {
    number = health; right = 90; slot = t - 5;
  } else if (t == 8) {
    e = make_int3(12, 90, 3);
  } else if (t < 12) {
    number = armor; right = 221; slot = t - 9;
  } else if (t == 12) {
    e = make_int3(12, 221, 3);
  } else if (t == 13) {
    int pain = (100 - health) >= 0 ? (100 - health) / 20 : -((health - 100 + 19) / 20);
    pain = pain < 0 ? 0 : (pain > 4 ? 4 : pain);
    int face = 13 + pain * 3 + lane[GD_L_FACE_INDEX];
    if (lane[GD_L_GRIN_TICS] > 0) face = 64 + pain;
    else if (lane[GD_L_PAIN_TICS] > 0) {
      if (lane[GD_L_FLAGS] & 2) face = 59 + pain;
      else {
        int d = lane[GD_L_PAIN_DIRECTION];
        d = d < 0 ? 0 : (d > 2 ? 2 : d);
        face = (d == 0 ? 44 : (d == 1 ? 49 : 54)) + pain;
      }
    } else if (lane[GD_L_ATTACK_HELD] >= 70) face = 49 + pain;
    if (health <= 0) face = 69;
    e = make_int3(face < 0 ? 0 : (face > 69 ? 69 : face), 143, 0);
  } else if (t < 20) {
    const int wi = t - 14;
    const bool owned = wi < 5 && ((lane[GD_L_WEAPONS_OWNED] >> (wi + 1)) & 1);
    e = make_int3(owned ? 28 + wi + 2 : 38 + wi, 111 + 12 * (wi % 3), wi < 3 ? 4 : 14);
  } else {
    const int row = (t - 20) / 6;
    slot = (t - 20) % 6;
    top = 5 + row * 6;
    if (slot < 3) { number = (int)__int_as_float(lane[GD_L_AMMO0 + row]); right = 288; }
    else { number = row == 0 ? 200 : (row == 3 ? 300 : 50); right = 314; slot -= 3; }   /* ammo maxima */
  }
  if (right >= 0) e = gd_hud_digit(sc, number, right, top, t >= 20, slot);
#ifdef GD_CHECKED
  if (e.x >= sc.hudPatches) { atomicOr(gdCheckedStatus, GD_STATUS_BAD_INDEX); e.x = -1; }
#endif
  int tx = 0, ty = 0, cw = 0, ch = 0, sx = 0, sy = 0;
  if (e.x >= 0) {
    const int4 hi = *reinterpret_cast<const int4 *>(&sc.hudInfo[e.x * 4]);
    const int x = e.y - hi.z, y = e.z - hi.w;
    sx = x < 0 ? -x : 0; sy = y < 0 ? -y : 0;
    tx = x > 0 ? x : 0; ty = y > 0 ? y : 0;
    cw = min(hi.x - sx, GD_SW - tx); ch = min(hi.y - sy, GD_HUD_H - ty);
    if (hi.x <= 0 || hi.y <= 0 || cw <= 0 || ch <= 0) { cw = 0; ch = 0; }
  }
  entries[t] = make_int4(tx | (ty << 16), cw | (ch << 16), sx | (sy << 16), e.x < 0 ? 0 : e.x);
}

/* Column x of the status bar; the list is complete. */
__device__ __noinline__ void gd_hud_column(const GdScene &sc_, const int4 *entries_, uint8_t *canvas, int x) {
  const GdScene &sc = *gd_as_shared(&sc_);
  const int4 *entries = gd_as_shared(entries_);
  unsigned long long mine = 0;                         /* entries that cross this column */
#pragma unroll 1
  for (int k = 0; k < GD_HUD_PATCHES; ++k) {
    const int4 e = entries[k];
    const int tx = e.x & 0xFFFF;
    if (x >= tx && x < tx + (e.y & 0xFFFF)) mine |= 1ull << k;
  }
#pragma unroll 1
  for (int y = 0; y < GD_HUD_H; ++y) {
    uint8_t value = 0;
    unsigned long long m = mine;
#pragma unroll 1
    while (m) {
      const int k = 63 - __clzll((long long)m);        /* topmost remaining entry */
      m &= ~(1ull << k);
      const int4 e = entries[k];
      const int ty = e.x >> 16;
      if (y < ty || y >= ty + (e.y >> 16)) continue;
      const int si = (e.w * GD_HUD_H + (e.z >> 16) + y - ty) * GD_SW + (e.z & 0xFFFF) + x - (e.x & 0xFFFF);
      const uint8_t opaque = sc.hudOpaque[si], texel = sc.hudAtlas[si];   /* both on their way at once */
      if (opaque) { value = texel; break; }
    }
    canvas[y * GD_SW + x] = value;
  }
}

#endif

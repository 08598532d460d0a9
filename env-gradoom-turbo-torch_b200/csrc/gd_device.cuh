/*
 * Device-side view of the scene blob and small exact-arithmetic helpers shared
 * by the render kernels.  Everything is integer 16.16 / 20.12 fixed point on
 * 64-bit integers or separately rounded float32 (the library is compiled with
 * -fmad=false), because the results must equal the reference's
 * (src/gradoom/engine.py:10534-15457) bit for bit.
 */
#pragma once

#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "../../include/gradoom_b200_layout.h"

typedef long long i64;

#define GD_FU 65536LL
#define GD_SW GD_SCREEN_W
#define GD_VH GD_VIEW_H
#define GD_ANG90 (1LL << 30)
#define GD_FOCAL_X (160LL * GD_FU)
#define GD_Y_ASPECT ((320LL * GD_FU * 240LL) / (200LL * 320LL))
#define GD_FOCAL_Y (160LL * GD_Y_ASPECT)
#define GD_FLOOR_VIS ((160LL * GD_FU * (8LL * GD_FU)) / GD_FOCAL_Y)
#define GD_WALL_VIS (((GD_FOCAL_Y * (320LL * 600LL) / (320LL * 240LL * 3LL)) * (8LL * GD_FU)) >> 16)
#define GD_SPRITE_MIN_DEPTH (2048LL * 4LL)
#define GD_U32MASK 0xFFFFFFFFLL

/* status bits written to the device status word */
#define GD_STATUS_EVENT_OVERFLOW 1   /* a column produced more clip events than the scratch holds */
#define GD_STATUS_THINGS_OVERFLOW 2  /* a lane lists more things than the configured maximum */
#define GD_STATUS_BAD_SECTOR 4       /* checked build: a sector index outside the scene */
#define GD_STATUS_BAD_INDEX 8        /* checked build: a wall, texture, sprite or patch index outside its table */
#define GD_STATUS_BAD_STATE 16       /* checked build: a lane or thing record with a value outside its range */

/* A map's area in GD_CELLS x GD_CELLS cells; a cell lists, in ascending order, every sector that may contain a point
 * of it (points outside belong to the nearest cell).  One 16-byte load fetches a cell. */
#define GD_CELLS 32
#define GD_CELL_SECTORS 7
struct __align__(16) GdCells {
  float x0, y0, perX, perY;       /* cell of a coordinate: (c - x0) * perX */
  float xLo, xHi, yLo, yHi;       /* no sector contains a point with x > xHi, y >= yHi, y < yLo or (all closed) x < xLo */
  unsigned short cell[GD_CELLS * GD_CELLS][1 + GD_CELL_SECTORS];   /* count (255: more than the list holds), sectors */
};

struct GdScene {
  int W, S, T, texH, texW, P, sprH, sprW, Q, wpnH, wpnW, wpnTics, nStarts, B, nbDirect, wpnAvailable, hudPatches;
  const float *walls;
  const int32_t *wsec;
  const float *wlen;
  const int32_t *sideTex;
  const float *sideOff;
  const int32_t *wvtx, *vtxOff, *vtxWalls;
  const int32_t *nbDirectTab, *nbOff, *nbIdx, *nbFlags;
  const int32_t *sbStartOff, *sbStartIdx, *sbEndOff, *sbEndIdx;
  const float *secF;
  const int32_t *secI;
  const int32_t *secOff, *secWalls, *edgeOff, *edgeWalls, *blocking;
  const int32_t *texInfo;
  const uint8_t *texAtlas, *texAtlasCol, *playpal, *colormap;
  const int32_t *sprInfo;
  const uint8_t *sprAtlas, *sprPost;
  const uint8_t *addLut, *transLut;
  const int32_t *wpnInfo;
  const uint8_t *wpnAtlas, *wpnOpaque;
  const int32_t *wpnFrameIds, *wpnFlashIds, *wpnFlashLights;
  const int32_t *hudInfo;
  const uint8_t *hudAtlas, *hudOpaque;
  const int32_t *fineSine, *fineTan;
  const float *rayOffsets, *rayCosCorr;
  const float *secBBox;
  const int32_t *maskedWalls;   /* M two-sided walls that carry a middle texture */
  const float *damageAlpha;     /* 114: damage count -> red flash alpha */
  /* sectors grouped by floor / ceiling height, nearest plane first */
  const float *groupH[2];       /* [0] ceilings ascending, [1] floors descending */
  const int32_t *groupOff[2], *groupSec[2];
  int groups[2];
  int M;
  /* projection fragments of the lines a node builder split: total count, CSR per line, 16.16 endpoints */
  int F;
  const int32_t *fragOff, *fragFixed;
  const GdCells *cells;         /* the sectors that may hold a point, by where it lies */
  /* bullet-chip decals: variants (0 = none), atlas slice height / width */
  int decals, decalH, decalW;
  const int32_t *decalInfo, *wallFine;
  const uint8_t *decalAtlas, *decalOpacity, *decalBlack;
};

/*
 * Checked build (-DGD_CHECKED, libgradoom_b200_checked.so): every index taken from
 * the scene blob, a lane record or a thing record is range-tested where it is about
 * to address memory; an index out of range is replaced by 0 (the access it would
 * have made is skipped) and a bit is set in the caller's status word.  Nothing
 * traps.  The regular build compiles the tests away.
 */
#ifdef GD_CHECKED
__device__ int *gdCheckedStatus;     /* the status word of the launch in flight (one launch at a time) */
__device__ __forceinline__ int gd_checked(int i, int n, int bit) {
  if ((unsigned)i < (unsigned)n) return i;
  atomicOr(gdCheckedStatus, bit);
  return 0;
}
#define GD_CHECK_INDEX(i, n) gd_checked((int)(i), (int)(n), GD_STATUS_BAD_INDEX)
#define GD_CHECK_SECTOR(i, n) gd_checked((int)(i), (int)(n), GD_STATUS_BAD_SECTOR)
#define GD_FLAG_STATE(bad) do { if (bad) atomicOr(gdCheckedStatus, GD_STATUS_BAD_STATE); } while (0)
#else
#define GD_CHECK_INDEX(i, n) (i)
#define GD_CHECK_SECTOR(i, n) (i)
#define GD_FLAG_STATE(bad) do { } while (0)
#endif

/* sector on one side of a wall: entry `i` of the wall-sector table, -1 = none */
__device__ __forceinline__ int gd_wsec(const GdScene &sc, int i) {
  const int s = sc.wsec[i];
#ifdef GD_CHECKED
  if (s < -1 || s >= sc.S) { atomicOr(gdCheckedStatus, GD_STATUS_BAD_SECTOR); return -1; }
#endif
  return s;
}

/* The CTA's dynamic shared memory. */
extern __shared__ __align__(16) uint8_t gd_smem[];

__device__ __forceinline__ unsigned gd_shared_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
/* The same pointer, re-derived from the shared array itself.  The pointers of the shared-memory map are generic (they
 * are read from a structure); this way the compiler knows their address space and addresses everything reached through
 * them with 32 bits and shared-space instructions. */
template <class T>
__device__ __forceinline__ T *gd_as_shared(T *p) {
  return (T *)(gd_smem + (int)(gd_shared_addr(p) - gd_shared_addr(gd_smem)));   /* static shared variables lie below */
}
__device__ __forceinline__ i64 gd_min(i64 a, i64 b) { return a < b ? a : b; }
__device__ __forceinline__ i64 gd_max(i64 a, i64 b) { return a > b ? a : b; }
__device__ __forceinline__ i64 gd_clamp(i64 v, i64 lo, i64 hi) { return v < lo ? lo : (v > hi ? hi : v); }
__device__ __forceinline__ i64 gd_wmul(i64 a, i64 b) { return (i64)((unsigned long long)a * (unsigned long long)b); }
__device__ __forceinline__ i64 gd_shl(i64 a, int k) { return (i64)((unsigned long long)a << k); }
/* float32 -> int64, round half to even */
__device__ __forceinline__ i64 gd_rint(float v) { return (i64)rintf(v); }
__device__ __forceinline__ i64 gd_pymod(i64 a, i64 m) {
  i64 r = a % m;
  return (r != 0 && ((r < 0) != (m < 0))) ? r + m : r;
}
/* the same for a texture width: a power of two needs no division */
__device__ __forceinline__ int gd_pymod_width(i64 a, int w) {
  if (w > 0 && (w & (w - 1)) == 0) return (int)(a & (i64)(w - 1));
  return (int)gd_pymod(a, w);
}

/*
 * Truncating signed 64-bit division.  The generic 64-bit divide is a long
 * software routine on the GPU; nearly every quotient on this path has operands
 * below 2^52, where a double-precision divide is within one of the exact
 * quotient and an integer remainder check makes it exact.
 */
__device__ __noinline__ i64 gd_div_generic(i64 a, i64 b) { return a / b; }

__device__ __noinline__ i64 gd_div(i64 a, i64 b) {
  unsigned long long ua = a < 0 ? 0ull - (unsigned long long)a : (unsigned long long)a;
  unsigned long long ub = b < 0 ? 0ull - (unsigned long long)b : (unsigned long long)b;
  if (((ua | ub) >> 52) != 0 || ub == 0) return gd_div_generic(a, b);
  i64 q = (i64)__ddiv_rn((double)ua, (double)ub);
  i64 r = (i64)ua - q * (i64)ub;
  if (r < 0) q -= 1;
  else if (r >= (i64)ub) q += 1;
  return ((a ^ b) < 0) ? -q : q;
}

struct GdView {
  float x, y, angle, viewZ;
  i64 vx, vy, pitchBam;
  i64 vsin, vcos;
  float fcos, fsin;
  i64 center;
  i64 upperClip, lowerClip;  /* view frustum top / bottom slopes used by the row projection */
  int flashLight;
};

/* Per-wall record of the lane being drawn, in the CTA's scratch: what the slow path of the walk, the sprites and
 * the middle textures read. */
struct __align__(8) GdWall {
  i64 visL[2], visStep[2], visSl[2];  /* wallscan light per side */
  i64 sl, sr;                         /* projected half-open span (unbounded when rejected) */
  i64 dl, dr;                         /* clipped endpoint depths, 20.12 */
  int tx[2], ty[2];                   /* view coordinates in stored endpoint order */
};

/* A segment's ends in view coordinates (20.12), and the screen columns they project to. */
struct GdEnds {
  i64 tx0, ty0, tx1, ty1, column0, column1;
  bool front;                         /* the viewer is on its front side */
};

/* What the column walk reads of a wall of the lane being drawn, kept in shared memory: the ray test's
 * lane-dependent operands, the owned columns and the sectors on its two sides.  A wall outside the
 * frustum has dn = 0 and an empty span, so no column ray ever meets it. */
struct __align__(16) GdHot {
  float segx, segy, offx, offy;   /* extent of the wall, and its start as seen from the viewer */
  float dn;                       /* offx * segy - offy * segx: the column-independent numerator of the ray distance */
  unsigned span;                  /* columns [span & 0xFFFF, span >> 16) owned by the column-ray test; 0xFFFF, 0: none */
  int secs;                       /* front sector (low 16 bits), back sector (high 16 bits, -1: none) */
  unsigned bits;                  /* GD_HOT_* and the projected span [sl, sr) clamped to -1 .. 321, stored + 1 */
};
#define GD_HOT_SL(b) ((int)((b) & 1023u) - 1)
#define GD_HOT_SR(b) ((int)(((b) >> 10) & 1023u) - 1)
#define GD_HOT_ONESIDED (1u << 20)
#define GD_HOT_FRONT (1u << 21)
#define GD_HOT_SPLIT (1u << 22)
#define GD_HOT_NEIGHBOUR (1u << 23)   /* another line between the same two sectors shares an endpoint */
#define GD_HOT_BRIDGE0 (1u << 24)     /* one-sided lines that may own the columns past its start, past its end */
#define GD_HOT_BRIDGE1 (1u << 25)
#define GD_HOT_STATIC (GD_HOT_ONESIDED | GD_HOT_SPLIT | GD_HOT_NEIGHBOUR | GD_HOT_BRIDGE0 | GD_HOT_BRIDGE1)

/* Everything of a crossing that depends on the wall and the side it is seen from alone; built by every
 * launch.  The flags assume that the sectors of the crossing are the wall's own two. */
struct __align__(16) GdSide {
  int tex[3];                     /* middle, lower, upper texture, -1: none */
  int contrast;                   /* fake contrast: +16 vertical, -16 horizontal */
  float yoff;
  unsigned flags;                 /* GD_C_ONE_SIDED .. GD_C_CEIL_BELOW, static part */
  i64 tox;                        /* texture x offset, 16.16 */
  i64 repeat;                     /* wall length, 16.16 */
  i64 pad;
};

/* flags of one crossing of a column */
#define GD_C_RASTER 1u            /* draws, marks and clips */
#define GD_C_ONE_SIDED 2u
#define GD_C_MARK_CEIL 4u
#define GD_C_MARK_FLOOR 8u
#define GD_C_LOWER 16u            /* view floor below the other sector's */
#define GD_C_UPPER 32u            /* view ceiling above the other sector's */
#define GD_C_TIER0 64u            /* the tier has rows to draw: middle, lower, upper */
#define GD_C_TIER1 128u
#define GD_C_TIER2 256u
#define GD_C_FLOOR_ABOVE 512u     /* view floor above the other sector's */
#define GD_C_CEIL_BELOW 1024u     /* view ceiling below the other sector's */
#define GD_C_PORTAL 2048u         /* a portal behind a projected solid contributes its clips */

/* One clip event of a column: what a drawn seg contributes to sprite clipping
 * and to visplane ownership. Rows are 0..208 and fit a byte. */
struct __align__(4) GdEvent {
  float dist;
  short wall;      /* wall whose depth clips sprites */
  short sector;    /* sector owning the planes marked by this event, -1 none */
  unsigned char t0a, t0b, t1a, t1b;  /* rows drawn by this event: two tier ranges */
  unsigned char silTop, silBot;      /* silhouettes: rows < silTop and rows >= silBot */
  unsigned char ceilA, ceilB, floorA, floorB;  /* plane marks */
  unsigned char pad0, pad1;
};

#define GD_MAX_EVENTS 48

/* Row projection of one (wall or fragment, plane height) pair, the form the walk reads: the row is
 * (a + x * step) >> 16 clamped to the view, with forced rows left of column `la` and from column `lb` on. */
struct __align__(16) GdRow {
  int a, step;
  unsigned lim;                   /* la | lb << 10 | GD_ROW_* */
  int vis;                        /* wallscan light of a side: origin in the side's floor row, step in its ceiling row */
};
#define GD_ROW_LEFT_TOP (1u << 20)    /* the rows forced on the left are row 0, else the bottom row */
#define GD_ROW_RIGHT_TOP (1u << 21)
#define GD_ROW_WIDE (1u << 22)        /* does not fit this form: take the full record */
#define GD_ROW_LIGHT_WIDE (1u << 23)  /* the same of the light of the side */
#define GD_ROW_PLAIN (1023u << 10)    /* no column is forced */

/* Row projection of one (wall, plane height) pair: everything of the OWallMost
 * replay that does not depend on the screen column. */
struct __align__(8) GdRowProj {
  i64 pl, pstep, cl;     /* clipped-edge projection: center + pl + (x - cl) * pstep */
  i64 opl, ostep;        /* whole-wall projection for columns outside the seg's span */
  short topA, topB;      /* columns forced to row 0 (above the view frustum) */
  short botA, botB;      /* columns forced to the bottom row */
  short collapsedX;      /* the one column exempt from both, or -1 */
  unsigned char entAbove, entBelow;
  short pad;
};

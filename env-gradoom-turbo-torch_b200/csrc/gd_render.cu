/*
 * Fused render-to-observation kernel for sm_100a.
 *
 * One persistent CTA of 320 threads draws one environment lane at a time, two
 * CTAs to an SM (four of them a lane, each a quarter of its columns, when the
 * lanes are few):
 *   1. the walls that a column ray may cross are listed and projected once per
 *      lane, and their ray-owned column spans found at the projections of their
 *      ends (by warps that try all 320 rays where an end is too close);
 *   2. thread x then walks column x front to back through the sector portals,
 *      keeping the ceiling / floor clip pair and the rows claimed so far in
 *      registers, drawing wall tiers
 *      and the visplane rows they uncover straight into the palette-indexed
 *      frame (aligned groups of four columns exchange their tier bounds with
 *      warp shuffles);
 *   3. the depth-sorted sprites are drawn against the clip events the walk
 *      recorded for the columns they may cover;
 *   4. the weapon and, on request, the status bar are composited;
 *   5. the 320x240 frame is reduced to the 84x84 grayscale observation with the
 *      exact integer area weights and written, 16 bytes per store, into the
 *      four-frame stack; the RGB24 frame is written only when asked for.
 * Only the lane record, the thing records and the stack slots have to cross
 * HBM; the indexed frame, the clip events and the CTA's tables lie in scratch,
 * most of which L2 holds (4096 lanes of the 64-sector map move about 437 MB, 202 of them
 * the stack's: 2 % of what HBM moves in that time).
 * Tensor cores are unused: nothing here is a contraction.
 *
 * What bounds it is the supply of instructions: the whole kernel is far larger
 * than the instruction caches, so a phase costs what its code costs to fetch
 * and its chains to wait for.  Measured with one 10-warp CTA per SM (frame in
 * shared memory, every rule of the walk in its loop): 5.17 ms per 4096 lanes of
 * the 64-sector map, 32.0 ms per 8192 lanes of the 256-sector map; two such
 * CTAs per SM were slower (5.95 ms: warps waiting for instructions went from
 * 0.9 to 5.0 per issue).  With the plain crossings decided apart from the full
 * set of rules and the walk's tables in 16-byte records, two CTAs per SM took
 * 3.99 and 20.2 ms; with a sixth of the code and the full searches of sprite and
 * fallback pixels gone, 3.4 and 15.2 ms; with claims drawn as runs, the repair of
 * unclaimed pixels kept to the columns near them, and shorter setups, sprites and
 * resize, 3.0 and 13.5 ms.  Drawing apart from the walk, from lists of runs, took
 * 15 to 40 % more; more warps with fewer registers 11 % more.
 *
 * The arithmetic restates src/gradoom/engine.py (file:line beside each
 * function) and must stay bit-identical to it; compile with -fmad=false.
 */
#include "gd_device.cuh"

#define GD_THREADS 320
#define GD_WARPS (GD_THREADS / 32)
#define GD_INF CUDART_INF_F

/* render flags */
#define GD_F_MASK_HUD 1     /* observation sees 32 black rows instead of the status bar */
#define GD_F_DRAW_HUD 2     /* composite the status bar (needed for RGB / unmasked obs) */
#define GD_F_STACK_ROLL 4   /* shift the stack by one slot and append */
#define GD_F_STACK_FILL 8   /* write all four slots of lanes whose mask byte is set */
#define GD_F_WRITE_OBS 16   /* write plain (n,84,84) observations to obsOut */
#define GD_F_STACK_RING 32  /* the stack is a mirrored ring of eight slots per lane (see gd_render_step_ring) */
#define GD_F_STEP_RESET 64  /* a step of every lane and a reset of the masked ones (see gd_render_step_reset) */

struct GdParams {
  GdScene sc;
  const int32_t *lanes;
  const gd_thing *things;
  int maxThings;
  int n;
  int flags;
  uint8_t *stack;            /* n x 4 x 84 x 84, or n x 8 x 84 x 84 with GD_F_STACK_RING */
  int ringHead;              /* GD_F_STACK_RING: slot 0..3 that takes the new frame (and slot + 4) */
  const uint8_t *resetMask;  /* n, for GD_F_STACK_FILL */
  const int32_t *resetLanes; /* GD_F_STEP_RESET: the records that the resets are drawn from ... */
  const gd_thing *resetThings;
  uint8_t *finalStack;       /* ... and the stacks as the step left them */
  int sliceShift;            /* a lane is drawn by 1 << sliceShift CTAs, each a slice of its columns */
  uint8_t *obsOut;           /* n x 84 x 84, optional */
  uint8_t *indexedOut;       /* n x 240 x 320, optional */
  uint8_t *rgbOut;           /* n x 240 x 320 x 3, optional */
  uint8_t *scratch;          /* ctas x perCta, the crossing records below, the lane queue (2 words, zero between launches) */
  size_t queueOffset, perCta;
  GdSide *sides;             /* 2 W crossing records of maps whose tables are not on chip, in the launch's scratch */
  /* byte offsets in shared memory; those of the last four are offsets into the CTA's scratch tables when
   * they do not fit on chip (kChip false) */
  int offSectors, offSecOff, offSecWalls, offVtx, offFrags, offActors;
  int offRows, offPrep, offPlanes, offSides;
  int secWallsN;
  int *status;
  const gd_decal *decals;    /* n x decalSlots rings of bullet chips, or null */
  int decalSlots;
  uint8_t *decalScratch;     /* ctas x gd_decal_scratch_per_cta(decalSlots) */
  /* scenes with split lines: a CTA's F fragment records, the line of each, then their F x 4 row projections when
   * those are not on chip; in the launch's own scratch like all that a CTA writes, so that launches of one renderer may overlap */
  uint8_t *frags;
  size_t fragStride;         /* from CTA to CTA */
};

#define GD_SCRATCH_EVENTS_BYTES (GD_MAX_EVENTS * GD_SW * (int)sizeof(GdEvent))
#define GD_SCRATCH_VSEC_BYTES (GD_VH * GD_SW * 2)   /* flat fallback: vertically repaired sector per pixel */
#define GD_SCRATCH_ANCHOR_BYTES (GD_VH * GD_WARPS * 4)
#define GD_SCRATCH_VSEC (GD_SCRATCH_EVENTS_BYTES + GD_SW * 4)
#define GD_SCRATCH_ANCHORS (GD_SCRATCH_VSEC + GD_SCRATCH_VSEC_BYTES)
#define GD_SCRATCH_FRAME (GD_SCRATCH_ANCHORS + GD_SCRATCH_ANCHOR_BYTES)
#define GD_SCRATCH_FIXED (GD_SCRATCH_FRAME + GD_SCREEN_H * GD_SW)
#define GD_PLANE_ENTRY_BYTES 88          /* sizeof(GdPlaneEntry), checked below */
#define GD_PLANE_BYTES 48                /* sizeof(GdPlane), checked below */
/* After the fixed part: the full wall records, the full row projections, the full span setups, and the tables of
 * the walk, which live here when they do not fit in shared memory: row projections, column operands, span setups. */
__host__ __device__ inline size_t gd_align16(size_t v) { return (v + 15) & ~(size_t)15; }
__host__ __device__ inline size_t gd_scratch_walls(int, int) { return gd_align16(GD_SCRATCH_FIXED); }
__host__ __device__ inline size_t gd_scratch_rowproj(int W, int) { return gd_scratch_walls(0, 0) + gd_align16((size_t)W * sizeof(GdWall)); }
__host__ __device__ inline size_t gd_scratch_planes(int W, int S) { return gd_scratch_rowproj(W, S) + gd_align16((size_t)W * 4 * sizeof(GdRowProj)); }
__host__ __device__ inline size_t gd_scratch_tables(int W, int S) { return gd_scratch_planes(W, S) + gd_align16((size_t)S * 2 * GD_PLANE_ENTRY_BYTES); }
__host__ __device__ inline size_t gd_table_bytes(int W, int S) {
  return (size_t)W * 4 * sizeof(GdRow) + (size_t)W * 16 + (size_t)S * 2 * GD_PLANE_BYTES;
}
__host__ __device__ inline size_t gd_scratch_per_cta(int W, int S) { return gd_scratch_tables(W, S) + gd_table_bytes(W, S); }
__host__ __device__ inline size_t gd_frag_wall_bytes(int F) { return gd_align16((size_t)F * sizeof(GdWall)); }
__host__ __device__ inline size_t gd_frag_rows(int F) { return gd_frag_wall_bytes(F) + gd_align16((size_t)F * 4); }
inline size_t gd_frag_bytes(int F, bool chip) { return gd_frag_rows(F) + (chip ? 0 : (size_t)F * 4 * sizeof(GdRow)); }

struct GdActor {
  float x, y, depth;
  i64 depthFixed, xstep, yscale, topFixed, fracBase, iscale;   /* patch row at screen row y: (fracBase + y * iscale) >> 16 */
  int left, right;
  short row0, row1;               /* rows whose patch row lies inside the patch */
  int sprite, w, h;
  short shade;
  signed char style;
  unsigned char alive;
};

/* ---- shared memory ------------------------------------------------------- */
/* The CTA's shared memory begins with these fixed areas; the walls' records follow, then the tables whose
 * sizes depend on the scene (offsets in GdParams).  The palette-indexed frame itself lives in the CTA's
 * scratch, mostly in L2: its pixels are stored once each, a warp's 32 columns of a row in one sector,
 * and the 77 KB that leaves free on chip let two lanes share an SM. */
#define GD_OFF_COLORMAP 0                                  /* 32 x 256 */
#define GD_OFF_PAL64 (GD_OFF_COLORMAP + 32 * 256)          /* 256: R | B << 16 | G << 32; then a zero: black rows */
#define GD_OFF_PAL32 (GD_OFF_PAL64 + 258 * 8)              /* 256: r | g << 8 | b << 16, for the RGB24 output */
#define GD_OFF_YSLOPE (GD_OFF_PAL32 + 256 * 4)             /* 208 */
#define GD_OFF_LANE (GD_OFF_YSLOPE + GD_VIEW_H * 4)        /* 32 */
#define GD_OFF_OWNER (GD_OFF_LANE + GD_LANE_WORDS * 4)     /* 10 words of column bits: boundary_has_projected_owner; words 16..25: the
                                                              walk may go on after leaving the map; words 32..41: some wall's
                                                              projected span starts here */
#define GD_OWNER_WORDS 48
#define GD_OFF_MISC (GD_OFF_OWNER + GD_OWNER_WORDS * 4)                   /* 16 ints: start sector, fallback queue length, its unresolved
                                                              rows' range, GdFlatBounds, counters of the fallback; 14, 15: the slice's
                                                              columns */
#define GD_OFF_MASKS (GD_OFF_MISC + 64)                    /* 7 x 320: per-column row bitmasks */
#define GD_OFF_MASKED_DIST (GD_OFF_MASKS + 7 * 320 * 4)   /* 320: nearest masked drawseg of the column ... */
#define GD_OFF_MASKED_INFO (GD_OFF_MASKED_DIST + 320 * 4)  /* ... its wall << 16 | ceiling clip << 8 | floor clip; 0xFFFF0000 | .. = none */
#define GD_OFF_CAND (GD_OFF_MASKED_INFO + 320 * 4)         /* 320 x 64 bits: things that may show in the column */
#define GD_OFF_AUX (GD_OFF_CAND + 320 * 8)                 /* 10,240 bytes for one phase at a time: listed walls, fallback queue,
                                                              chip ranks, sprite columns' events */
#define GD_AUX_BYTES (8 * 320 * 4)
#define GD_OFF_AUX2 (GD_OFF_AUX + GD_AUX_BYTES)            /* 4,096: sectors of points, status-bar list, sprite columns, chip spans */
#define GD_AUX2_BYTES 4096
#define GD_OFF_FLAT_LIST (GD_OFF_AUX2 + GD_SW * 4)         /* flat fallback, behind a word a column: three lists of columns */
static_assert(GD_SW * 4 + 3 * GD_SW * 2 <= GD_AUX2_BYTES, "the lists");
#define GD_OFF_HOT (GD_OFF_AUX2 + GD_AUX2_BYTES)           /* W wall records */
/* the resize, when all before it is done: its sums from the masks on, the result behind them */
#define GD_OFF_RESULT ((GD_OFF_MASKS + 7 * GD_SW * 8 + 15) / 16 * 16)
static_assert(GD_OFF_RESULT + GD_OBS * GD_OBS <= GD_OFF_HOT, "the sums and the result");
static_assert(GD_OFF_HOT % 16 == 0 && GD_OFF_AUX % 16 == 0 && GD_OFF_AUX2 % 16 == 0, "vector loads");
static_assert(65 * 4 <= GD_AUX2_BYTES && GD_SW * 2 <= GD_AUX2_BYTES,
              "the sectors of 64 things and the player, the sprite columns");

struct GdPlaneEntry;

struct GdShared {
  GdPlaneEntry *planeTab; /* scratch: per (sector, floor/ceiling) span setup of the lane being drawn */
  uint8_t *frame;       /* scratch: 240 x 320 */
  uint8_t *colormap;
  int32_t *lane;
  unsigned *ownerMask;
  GdWall *walls;        /* scratch: W, the listed ones filled */
  GdWall *frags;        /* scratch: F projection fragments of split lines (only their spans, depths and light) */
  unsigned *anchors;    /* scratch: flat fallback */
  unsigned *planeRows;  /* scratch: 7 x 320, rows of the planes of loose columns; where the fallback's sector table will be */
  GdActor *actors;      /* maxThings */
  unsigned long long *pal64;
  uint8_t *obs;         /* 84 x 84 */
  int *misc;
  unsigned *masks;
  unsigned *pal32;
  float *maskedDist;
  unsigned *maskedInfo;
  float *hitD, *hitA;   /* the two aux areas */
  const unsigned short *secOff, *secWalls;   /* incident walls of every sector */
};

__device__ __forceinline__ GdHot &gd_hot(int w) { return reinterpret_cast<GdHot *>(gd_smem + GD_OFF_HOT)[w]; }
__device__ __forceinline__ int gd_hot_front(int w) { return (int)(short)(gd_hot(w).secs & 0xFFFF); }
__device__ __forceinline__ int gd_hot_back(int w) { return gd_hot(w).secs >> 16; }
/* endpoint vertex of a wall: the scene's `wvtx` holds 32-bit ids in global memory, this copy is on chip */
__device__ __forceinline__ int gd_vertex(const GdScene &sc, int w, int slot) { return gd_as_shared(sc.wvtx)[w * 2 + slot]; }

#include "gd_geometry.cuh"
#include "gd_walk.cuh"
#include "gd_flats.cuh"
#include "gd_sprites.cuh"
#include "gd_decals.cuh"
#include "gd_output.cuh"

/* ---- the kernel ----------------------------------------------------------- */

/* kSplit: the scene carries projection fragments of split lines.  kChip: the walk's tables fit in shared memory
 * beside a second CTA.  kPlain: every task is one frame of a lane (the code for the other launches costs a step of 4096
 * lanes 4 %, 3015 and 3133 us, and the 256-sector map 3 %, which only the calls that want it should pay). */
template <bool kSplit, bool kChip, bool kPlain>
__global__ void __launch_bounds__(GD_THREADS, 2) gd_render_kernel(const __grid_constant__ GdParams p) {
  /* The scene descriptor, the shared-memory map and the lane's view are read by
   * the phases around the walk through references; keeping them in shared memory (one copy
   * per CTA) keeps those reads off the per-thread stack. */
  __shared__ GdScene sScene;
  __shared__ GdShared sShared;
  __shared__ GdView sView;
  const int tid = threadIdx.x;
  uint8_t *myScratch = p.scratch + (size_t)blockIdx.x * p.perCta;
  uint8_t *tables = myScratch + gd_scratch_tables(p.sc.W, p.sc.S);
  uint8_t *frame = myScratch + GD_SCRATCH_FRAME;
  if (tid == 0) {
    GdScene sc = p.sc;
    GdShared sh;
    sh.planeTab = (GdPlaneEntry *)(myScratch + gd_scratch_planes(sc.W, sc.S));
    sh.frame = frame;
    sh.colormap = gd_smem + GD_OFF_COLORMAP;
    sh.lane = (int32_t *)(gd_smem + GD_OFF_LANE);
    sh.ownerMask = (unsigned *)(gd_smem + GD_OFF_OWNER);
    sh.walls = (GdWall *)(myScratch + gd_scratch_walls(sc.W, sc.S));
    sh.frags = (GdWall *)(p.frags + blockIdx.x * p.fragStride);
    sh.anchors = (unsigned *)(myScratch + GD_SCRATCH_ANCHORS);
    sh.planeRows = (unsigned *)(myScratch + GD_SCRATCH_VSEC);
    sh.actors = (GdActor *)(gd_smem + p.offActors);
    sh.pal64 = (unsigned long long *)(gd_smem + GD_OFF_PAL64);
    sh.obs = gd_smem + GD_OFF_RESULT;
    sh.misc = (int *)(gd_smem + GD_OFF_MISC);
    sh.masks = (unsigned *)(gd_smem + GD_OFF_MASKS);
    sh.pal32 = (unsigned *)(gd_smem + GD_OFF_PAL32);
    sh.maskedDist = (float *)(gd_smem + GD_OFF_MASKED_DIST);
    sh.maskedInfo = (unsigned *)(gd_smem + GD_OFF_MASKED_INFO);
    sh.secOff = (const unsigned short *)(gd_smem + p.offSecOff);
    sh.secWalls = (const unsigned short *)(gd_smem + p.offSecWalls);
    sh.hitD = (float *)(gd_smem + GD_OFF_AUX);
    sh.hitA = (float *)(gd_smem + GD_OFF_AUX2);
    sc.wvtx = (const int32_t *)(gd_smem + p.offVtx);
    sScene = sc; sShared = sh;
#ifdef GD_CHECKED
    gdCheckedStatus = p.status;
#endif
  }
  __syncthreads();
  const GdScene &sc = sScene;
  const GdShared &sh = sShared;
  /* tables shared by every lane this CTA draws */
  for (int i = tid; i < 32 * 256 / 4; i += GD_THREADS)
    ((unsigned *)(gd_smem + GD_OFF_COLORMAP))[i] = ((const unsigned *)sc.colormap)[i];
  gd_lane_palette(sc, sh, 0);
  for (int w = tid; w < sc.W; w += GD_THREADS) {
    const int front = gd_wsec(sc, w * 2), back = gd_wsec(sc, w * 2 + 1);
    gd_hot(w).secs = (front & 0xFFFF) | (back << 16);
    const bool neighbour = sc.nbDirect ? sc.nbDirectTab[w * 4] >= 0 || sc.nbDirectTab[w * 4 + 1] >= 0 : sc.nbOff[w + 1] > sc.nbOff[w];
    gd_hot(w).bits = (back < 0 ? GD_HOT_ONESIDED : 0u) | (kSplit && sc.fragOff[w + 1] > sc.fragOff[w] ? GD_HOT_SPLIT : 0u) |
                     (neighbour ? GD_HOT_NEIGHBOUR : 0u) | (sc.sbStartOff[w + 1] > sc.sbStartOff[w] ? GD_HOT_BRIDGE0 : 0u) |
                     (sc.sbEndOff[w + 1] > sc.sbEndOff[w] ? GD_HOT_BRIDGE1 : 0u);
    ((int2 *)(gd_smem + p.offVtx))[w] = ((const int2 *)p.sc.wvtx)[w];
  }
  for (int s = tid; s < sc.S; s += GD_THREADS)
    ((float4 *)(gd_smem + p.offSectors))[s] = make_float4(sc.secF[s * 2], sc.secF[s * 2 + 1], __int_as_float(sc.secI[s * 4]), 0.0f);
  for (int s = tid; s <= sc.S; s += GD_THREADS) ((unsigned short *)(gd_smem + p.offSecOff))[s] = (unsigned short)sc.secOff[s];
  for (int i = tid; i < p.secWallsN; i += GD_THREADS)
    ((unsigned short *)(gd_smem + p.offSecWalls))[i] = (unsigned short)GD_CHECK_INDEX(sc.secWalls[i], sc.W);
  if (kChip)
#pragma unroll 1
    for (int i = tid; i < sc.W * 2; i += GD_THREADS) gd_side_setup(sc, i, ((GdSide *)(gd_smem + p.offSides))[i]);
  int *fragLine = (int *)(p.frags + blockIdx.x * p.fragStride + gd_frag_wall_bytes(sc.F));
  if (kSplit)
#pragma unroll 1
    for (int w = tid; w < sc.W; w += GD_THREADS)
      for (int f = max(sc.fragOff[w], 0); f < min(sc.fragOff[w + 1], sc.F); ++f) fragLine[f] = w;
  bool paletteBlended = false;    /* CTA-uniform: the shared palette holds a lane's screen-flash blend */
  GdEvent *events = (GdEvent *)myScratch;
  int *eventCount = (int *)(myScratch + GD_SCRATCH_EVENTS_BYTES);
  unsigned short *vsec = (unsigned short *)(myScratch + GD_SCRATCH_VSEC);
  GdRowProj *rowproj = (GdRowProj *)(myScratch + gd_scratch_rowproj(sc.W, sc.S));
  GdRow *rows = (GdRow *)(kChip ? gd_smem + p.offRows : tables + p.offRows);
  GdRow *fragRows = kChip ? rows + sc.W * 4 : (GdRow *)(p.frags + blockIdx.x * p.fragStride + gd_frag_rows(sc.F));
  float4 *prep = (float4 *)(kChip ? gd_smem + p.offPrep : tables + p.offPrep);
  GdPlane *planes = (GdPlane *)(kChip ? gd_smem + p.offPlanes : tables + p.offPlanes);

  /* Lanes differ a lot in cost (a long corridor crosses many sectors), so the
   * persistent CTAs take lanes from a shared counter instead of a fixed stride.
   * The counter pair lives behind the event scratch and is left at zero by the
   * last CTA to finish. */
  unsigned *queue = (unsigned *)(p.scratch + (size_t)p.queueOffset);
  __shared__ int nextLane;
  for (;;) {
    __syncthreads();
    if (tid == 0) nextLane = (int)atomicAdd(&queue[0], 1u);
    __syncthreads();
    /* a launch that steps and resets has both frames in one queue, the resets' first: as a launch of their own they
     * waited for the slowest lane of the step (256 environment lanes 584 us a call, now 511; 1024 lanes 1227 and 1042) */
    const int sliceShift = kPlain ? 0 : p.sliceShift;
    int l = nextLane >> sliceShift;
    const bool both = !kPlain && (p.flags & GD_F_STEP_RESET) != 0;
    if (l >= (both ? 2 * p.n : p.n)) break;
    const bool fill = both ? l < p.n : (p.flags & GD_F_STACK_FILL) != 0;
    if (both && !fill) l -= p.n;
    if (fill && p.resetMask && !p.resetMask[l]) continue;  /* uniform across the CTA */
    const gd_thing *things = (both && fill ? p.resetThings : p.things) + (size_t)l * p.maxThings;
    if (tid < GD_LANE_WORDS) sh.lane[tid] = (both && fill ? p.resetLanes : p.lanes)[(size_t)l * GD_LANE_WORDS + tid];
    if (tid < GD_OWNER_WORDS) sh.ownerMask[tid] = 0;
    if (tid == 0) {
      sh.misc[1] = sh.misc[2] = 0;
      sh.misc[14] = GD_SW * (nextLane & ((1 << sliceShift) - 1)) >> sliceShift;     /* the slice's columns */
      sh.misc[15] = sh.misc[14] + (GD_SW >> sliceShift);
    }
    /* sector of every thing and of the player (slot 64): lowest index that
     * contains the point (engine.py:9598-9617), found by warps 1 to 9
     * while thread 0 sets up the view */
    int *pointSector = (int *)sh.hitA;
    __syncthreads();
    {
      const int laneFlags = sh.lane[GD_L_FLAGS];
      const bool wantBlend = (laneFlags & 4) != 0;
      if (wantBlend || paletteBlended) gd_lane_palette(sc, sh, laneFlags);   /* read again after later barriers */
      paletteBlended = wantBlend;
    }
    int nThings = sh.lane[GD_L_THINGS];
    if (nThings > p.maxThings || nThings > 64) {
      if (tid == 0) atomicOr(p.status, GD_STATUS_THINGS_OVERFLOW);
      nThings = min(p.maxThings, 64);
    }
    if (nThings < 0) nThings = 0;
#ifdef GD_CHECKED
    {
      /* a lane whose pose is not a number, or lies far outside any map, is drawn from the map's origin instead */
      const float lx = __int_as_float(sh.lane[GD_L_X]), ly = __int_as_float(sh.lane[GD_L_Y]);
      const float lz = __int_as_float(sh.lane[GD_L_VIEW_Z]), la = __int_as_float(sh.lane[GD_L_ANGLE]);
      const bool badPose = !isfinite(lx) || !isfinite(ly) || !isfinite(lz) || !isfinite(la) || fabsf(lx) > 32768.0f ||
                           fabsf(ly) > 32768.0f;
      const int weapon = sh.lane[GD_L_WEAPON];
      __syncthreads();
      if (tid == 0) {
        GD_FLAG_STATE(badPose || weapon < 0 || weapon > 7 || sh.lane[GD_L_THINGS] < 0);
        if (badPose) {
          sh.lane[GD_L_X] = sh.lane[GD_L_Y] = sh.lane[GD_L_ANGLE] = 0;
          sh.lane[GD_L_X_FIXED] = sh.lane[GD_L_Y_FIXED] = sh.lane[GD_L_ANGLE_BAM] = 0;
          sh.lane[GD_L_VIEW_Z] = __float_as_int(41.0f);
        }
      }
      __syncthreads();
    }
#endif
    if (tid == 0) {
      gd_view_setup(sc, sh.lane, sView);
    } else if (tid >= 32) {
      /* eight threads a point: its cell of the map names the sectors to test */
#pragma unroll 1
      for (int t = (tid - 32) / GD_POINT_THREADS; t <= nThings; t += (GD_THREADS - 32) / GD_POINT_THREADS) {
        float px = __int_as_float(sh.lane[GD_L_X]), py = __int_as_float(sh.lane[GD_L_Y]);
        if (t < nThings) {
          const gd_thing &th = things[t];
          px = th.x; py = th.y;
        }
        const int s = gd_sector_of_point(sc, px, py);
        if (tid % GD_POINT_THREADS == 0) pointSector[t < nThings ? t : 64] = s;
      }
    }
    __syncthreads();
    const GdView &v = sView;
    if (tid < GD_VH) {
      /* yslope of the row (engine.py:10933-10946) */
      i64 centerRow = v.center >> 16;
      i64 den = (tid < centerRow) ? (v.center - (i64)tid * GD_FU - GD_FU / 2) : ((i64)tid * GD_FU - v.center + GD_FU / 2);
      den = gd_max(den, 1);
      i64 ys = gd_div(GD_FOCAL_Y << 16, den);
      if (den <= (GD_FOCAL_Y >> 15)) ys = (1LL << 31) - 1;
      ((unsigned *)(gd_smem + GD_OFF_YSLOPE))[tid] = (unsigned)ys;
    }
    if (kSplit)
#pragma unroll 1
      for (int f = tid; f < sc.F; f += GD_THREADS) {
        GdWall &q = sh.frags[f];
        gd_project_fragment(sc, v, f, q);
        const unsigned sl = (unsigned)gd_clamp(q.sl, 0, GD_SW), sr = (unsigned)gd_clamp(q.sr, 0, GD_SW);
        ((unsigned *)(gd_smem + p.offFrags))[f] = q.sr > q.sl ? sl | (sr << 16) : 0u;
      }
    gd_wall_list(sc, v);
    if (tid == GD_THREADS - 1) sh.misc[0] = pointSector[64] == 0x7fffffff ? 0 : pointSector[64];
    __syncthreads();
    /* the setups of the lane's walls (a thread a side), span tables and things, side by side: what bounds each is the
     * latency of its divisions */
    const short *frustumList = (const short *)(gd_smem + GD_OFF_AUX);
    const int frustumListed = sh.misc[2];
    {
      /* whole warps of one kind, the longest chains first */
      const int wallTask = (nThings + 31) & ~31, planeTask = (wallTask + frustumListed * 2 + 31) & ~31;
#pragma unroll 1
      for (int task = tid; task < planeTask + sc.S * 2; task += GD_THREADS) {
        if (task < nThings) {
          gd_actor_setup(sc, v, things[task], pointSector[task] == 0x7fffffff ? 0 : pointSector[task], sh.actors[task]);
        } else if (task >= planeTask) {
          const int idx = task - planeTask;
          gd_plane_entry_setup(sc, v, idx >> 1, (idx & 1) != 0, sh.planeTab[idx], planes[idx]);
        } else if (task >= wallTask && task < wallTask + frustumListed * 2) {
          const int i = task - wallTask, side = i >= frustumListed, w = frustumList[i - (side ? frustumListed : 0)];
          gd_project_wall(sc, v, w, side, sh.walls[w], gd_hot(w), *reinterpret_cast<int2 *>(&prep[w]));
        }
      }
    }
    __syncthreads();
    gd_wall_spans(v, sh, prep);
    __syncthreads();
    /* row projections, light and column operands of the listed walls (the walk selects no other wall) and of the
     * fragments in view */
    const int fragTasks = kSplit ? sc.F * 4 : 0;
#pragma unroll 1
    for (int idx = tid; idx < frustumListed * 4 + fragTasks; idx += GD_THREADS) {
      const bool piece = kSplit && idx >= frustumListed * 4;
      const int f = piece ? (idx - frustumListed * 4) >> 2 : 0, slot = idx & 3;
      if (piece && ((const unsigned *)(gd_smem + p.offFrags))[f] == 0u) continue;
      const int w = piece ? fragLine[f] : frustumList[idx >> 2];
      const GdWall &q = piece ? sh.frags[f] : sh.walls[w];
      const int sector = gd_wsec(sc, w * 2 + (slot >> 1)), sd = slot >> 1;
      GdRow row;
      row.a = row.step = 0; row.lim = GD_ROW_WIDE; row.vis = 0;
      if (sector >= 0) {
        GdRowProj unused;
        gd_rowproj_setup(v, q, sc.secF[sector * 2 + (slot & 1)], piece ? unused : rowproj[w * 4 + slot], row);
        /* the light of the side, modulo 2^32 as well: exact while the owned columns' values fit.  Nothing below
         * -2^30 is left to this form either: gd_shade takes the light from a base below 2^30 in 32 bits */
        const i64 step = q.visStep[sd], origin = q.visL[sd] - gd_wmul(q.visSl[sd], step);
        const i64 l0 = origin + gd_wmul(gd_max(q.sl, 0), step), l1 = origin + gd_wmul(gd_min(q.sr, GD_SW) - 1, step);
        if (gd_min(l0, l1) < -(1LL << 30) || gd_max(l0, l1) >= (1LL << 31)) row.lim |= GD_ROW_LIGHT_WIDE;
        row.vis = (int)((slot & 1) ? step : origin);
      }
      (piece ? fragRows + f * 4 : rows + w * 4)[slot] = row;
    }
#pragma unroll 1
    for (int i = tid; i < frustumListed; i += GD_THREADS) {   /* walls outside the frustum own no column */
      const int w = frustumList[i];
      prep[w] = gd_prep_setup(sh.walls[w]);
      const int xl = (int)(short)(gd_hot(w).span & 0xFFFFu);
      if (xl >= 0 && xl < GD_SW) {
        float rx, ry;
        gd_ray(v, xl, rx, ry);
        GdHit h = gd_hit_slow(sc, w, xl, rx, ry);
        if (isfinite(h.d)) atomicOr(&sh.ownerMask[xl >> 5], 1u << (xl & 31));
        if (h.proj) atomicOr(&sh.ownerMask[32 + (xl >> 5)], 1u << (xl & 31));
      }
    }
    gd_mark_afterlife_columns(sc, sh);
    if (p.flags & GD_F_DRAW_HUD) gd_hud_list(sc, sh.lane, (int4 *)sh.hitA);   /* the sectors of points have been read */
    const bool mine = kPlain || (tid >= sh.misc[14] && tid < sh.misc[15]);
    ((unsigned long long *)(gd_smem + GD_OFF_CAND))[tid] = !mine ? 0ull : gd_sprite_candidates(sc, v, sh, nThings, frustumList, frustumListed);
    __syncthreads();
    const bool open = gd_walk<kSplit, kChip>(p, sc, v, sh, frame, tables, events, eventCount, rowproj, sh.misc[0], mine);
    {
      /* a slice's walk leaves the warps half a screen on idle: they draw its status bar meanwhile (one image 222 us, now
       * 196; 30 lanes with grates 156 and 129) */
      const int x = kPlain || sliceShift == 0 ? tid : (tid + GD_SW / 2) % GD_SW;
      if ((p.flags & GD_F_DRAW_HUD) && (kPlain || (x >= sh.misc[14] && x < sh.misc[15])))
        gd_hud_column(sc, (const int4 *)sh.hitA, frame + GD_VH * GD_SW, x);
    }
    __syncthreads();
    /* Rows no seg ever claimed show the per-pixel flat fallback.  They are
     * queued (the first aux area is free once every column has finished its walk)
     * and resolved; a frame with more such pixels than the queue holds takes
     * several rounds, each pass marking what it drew as claimed. */
    bool sweepDone = false;                          /* CTA-uniform */
    for (;;) {
      const unsigned *claimed = sh.masks + tid;
#pragma unroll 1
      for (int k = 0; k < 7 && open; ++k) {
        unsigned m = gd_range_word(k, 0, GD_VH) & ~claimed[k * GD_SW];
#pragma unroll 1
        while (m) {
          int y = (k << 5) + __ffs(m) - 1;
          m &= m - 1;
          int slot = atomicAdd(&sh.misc[1], 1);
          if (slot < GD_FALLBACK_MAX) ((int *)sh.hitD)[slot] = (y << 16) | tid;
        }
      }
      __syncthreads();
      const int queued = sh.misc[1];
      if (queued == 0) break;                        /* block-uniform */
      if (!open)
#pragma unroll 1
        for (int k = 0; k < 7; ++k) sh.masks[k * GD_SW + tid] = 0xffffffffu;
      gd_fallback_pass(sc, v, sh, sh.misc[0], vsec, sweepDone);
      if (queued <= GD_FALLBACK_MAX) break;
      if (tid == 0) sh.misc[1] = 0;
      __syncthreads();
    }
    if (sc.M > 0) {
      if (mine) gd_masked_pass<kSplit>(sc, v, sh);
      __syncthreads();
    }
#ifndef GD_NO_DECALS
    if (p.decals != nullptr && sc.decals > 0)
      gd_decals(sc, v, sh, events, eventCount, p.decals + (size_t)l * p.decalSlots, p.decalSlots,
                p.decalScratch + (size_t)blockIdx.x * gd_decal_scratch_per_cta(p.decalSlots));
#endif
    gd_sprites(sc, v, sh, events, eventCount, nThings);
    __syncthreads();
    gd_weapon(sc, sh, sh.lane, sh.frame);
    __syncthreads();
    const bool wantFull = p.indexedOut != nullptr || p.rgbOut != nullptr;
    if (wantFull && !(p.flags & GD_F_DRAW_HUD)) {
#pragma unroll 1
      for (int i = tid; i < GD_HUD_H * GD_SW / 4; i += GD_THREADS) ((unsigned *)(sh.frame + GD_VH * GD_SW))[i] = 0;
      __syncthreads();
    }
    const int x0 = kPlain ? 0 : sh.misc[14], wide = GD_SW / 16 >> sliceShift;       /* the slice, in groups of sixteen columns */
    if (p.indexedOut) {
      uint4 *dst = (uint4 *)(p.indexedOut + (size_t)l * GD_SCREEN_H * GD_SW);
      const uint4 *src = (const uint4 *)sh.frame;
#pragma unroll 1
      for (int i = tid; i < GD_SCREEN_H * wide; i += GD_THREADS) {
        const int q = i / wide * (GD_SW / 16) + x0 / 16 + i % wide;
        dst[q] = src[q];
      }
    }
    if (p.rgbOut) {
      /* sixteen pixels (one 16-byte load) become three 16-byte stores (a word at a time: 43 of a lane's 442 thousand
       * cycles, now 19; 1024 lanes with RGB24 1396 and 1362 us) */
      uint4 *dst = (uint4 *)(p.rgbOut + (size_t)l * GD_SCREEN_H * GD_SW * 3);
      const uint4 *src = (const uint4 *)sh.frame;
      const unsigned *pal32 = (const unsigned *)(gd_smem + GD_OFF_PAL32);
#pragma unroll 1
      for (int i = tid; i < GD_SCREEN_H * wide; i += GD_THREADS) {
        const int q = i / wide * (GD_SW / 16) + x0 / 16 + i % wide;
        const uint4 four = src[q];
        const unsigned idx[4] = {four.x, four.y, four.z, four.w};
        unsigned out[12];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const unsigned p0 = pal32[idx[k] & 0xFF], p1 = pal32[(idx[k] >> 8) & 0xFF];
          const unsigned p2 = pal32[(idx[k] >> 16) & 0xFF], p3 = pal32[idx[k] >> 24];
          out[k * 3] = p0 | (p1 << 24);
          out[k * 3 + 1] = (p1 >> 8) | (p2 << 16);
          out[k * 3 + 2] = (p2 >> 16) | (p3 << 8);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) dst[q * 3 + k] = make_uint4(out[k * 4], out[k * 4 + 1], out[k * 4 + 2], out[k * 4 + 3]);
      }
    }
    if (p.stack || p.obsOut) {
      int srcRows = (p.flags & GD_F_MASK_HUD) ? GD_VH : GD_SCREEN_H;
      gd_resize<kPlain>(sh.frame, srcRows, sh.obs, x0, sliceShift);
      __syncthreads();
      const size_t frameBytes = GD_OBS * GD_OBS;
      uint8_t *newest = p.obsOut ? p.obsOut + (size_t)l * frameBytes : nullptr, *stack = nullptr, *final = nullptr;
      int mode = GD_PUT_NONE;
      if (p.stack && (p.flags & GD_F_STACK_RING)) {
        stack = p.stack + (size_t)l * 2 * GD_STACK * frameBytes;
        mode = fill ? GD_PUT_ALL8 : GD_PUT_RING;
      } else if (p.stack) {
        stack = p.stack + (size_t)l * GD_STACK * frameBytes;
        mode = fill ? GD_PUT_ALL : ((p.flags & GD_F_STACK_ROLL) ? GD_PUT_ROLL : GD_PUT_LAST);
        if (both && !fill) {
          final = p.finalStack + (size_t)l * GD_STACK * frameBytes;
          mode = p.resetMask[l] ? GD_PUT_FINAL_LAST : GD_PUT_ROLL_FINAL;
        }
      }
      if (kPlain || sliceShift == 0) gd_put_frame<uint4>(sh.obs, stack, final, newest, mode, p.ringHead, 0, 0);
      else gd_put_frame<uint8_t>(sh.obs, stack, final, newest, mode, p.ringHead, x0 * GD_OBS / GD_SW, GD_OBS >> sliceShift);
    }
  }
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(&queue[1], 1u) == gridDim.x - 1) {
      queue[0] = 0;
      queue[1] = 0;
      __threadfence();
    }
  }
}

#include "gd_abi.cuh"
#include "gd_state.cuh"
#include "gd_state_abi.cuh"
#include "gd_move.cuh"
#include "gd_stepper.cuh"

/* The C ABI declared in include/gradoom_b200.h: renderer objects, argument validation, launches.
 * Part of gd_render.cu (one translation unit); not meant to be included elsewhere. */
#ifndef GD_ABI_CUH
#define GD_ABI_CUH

/* ---- C ABI (declared in include/gradoom_b200.h) --------------------------- */
#include "../../include/gradoom_b200.h"

#include <new>
#include <string.h>

#define GD_HOST_CHUNKS 4
/* limits of the scratch array built into the library (gd_render_step_static) */
#define GD_STATIC_MAX_CTAS 32
#define GD_STATIC_MAX_WALLS 256
static bool gd_fits_static(const GdScene &sc) { return sc.W <= GD_STATIC_MAX_WALLS && sc.S <= GD_STATIC_MAX_WALLS; }

struct gd_renderer {
  int32_t header[GD_HDR_WORDS];
  const void *blobDev;
  int device;
  int maxThings;
  int ctas;
  size_t smemBytes;          /* dynamic shared memory per CTA */
  bool chip;                 /* the walk's tables are in it */
  GdParams base;             /* scene, table pointers and shared-memory offsets of every launch */
  /* gd_render_step_host overlaps the device->host copy of one lane chunk with
   * the drawing of the next on this side stream */
  cudaStream_t copyStream;
  cudaEvent_t chunkDone[GD_HOST_CHUNKS], copiesDone;
  /* gd_renderer_bind_decals: the lanes' decal rings and the renderer's own scratch for them */
  const gd_decal *decals;
  int decalSlots;
  uint8_t *decalScratch;
  size_t decalScratchBytes;
  size_t fragBytes;          /* a CTA's records of split lines: behind its scratch; F is not bounded, so */
  uint8_t *staticFrags;      /* those of the built-in array's CTAs are allocated with the renderer */
  size_t sidesOffset;        /* crossing records of maps whose tables are not on chip: behind the CTAs' scratch */
};

/* The crossing records of a map that reads them from scratch, before every draw of it (the others build theirs on
 * chip): a few microseconds beside draws of milliseconds, and the renderer keeps nothing of the blob's. */
__global__ void gd_side_setup_kernel(const __grid_constant__ GdScene sc, GdSide *sides) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < sc.W * 2) gd_side_setup(sc, i, sides[i]);
}

/* for blobs without GD_S_CELLS: every list is too long, no point lies past the map */
#define GD_FLOAT_INF __builtin_huge_valf()
static __device__ const GdCells gd_no_cells = {0.0f, 0.0f, 0.0f, 0.0f, -GD_FLOAT_INF, GD_FLOAT_INF, -GD_FLOAT_INF, GD_FLOAT_INF, {{255}}};

static const void *gd_section(const uint8_t *dev, const int32_t *h, int s) { return dev + h[GD_HDR_SECTION0 + s]; }

extern "C" const char *gd_error_string(int code) {
  switch (code) {
    case GD_OK: return "ok";
    case GD_ERR_NULL: return "null pointer argument";
    case GD_ERR_BLOB: return "scene blob has a bad magic, version or size";
    case GD_ERR_UNSUPPORTED: return "scene uses a feature this render path does not draw";
    case GD_ERR_SIZE: return "size argument out of range";
    case GD_ERR_ALIGN: return "device pointer is not 16-byte aligned";
    case GD_ERR_CUDA: return "CUDA runtime call failed";
    case GD_ERR_SCRATCH: return "scratch buffer is too small";
    case GD_ERR_SHARED: return "scene needs more shared memory than one SM offers";
    case GD_ERR_STATIC_LIMIT: return "scene or device index exceeds the limits of the built-in scratch array";
    case GD_ERR_DEVICE: return "the renderer's device is not the current CUDA device";
    case GD_ERR_OVERLAP: return "the stack and the final stack overlap";
    default: return "unknown error";
  }
}

/* The dynamic shared-memory limit belongs to the kernel on a device, not to one
 * renderer: every renderer raises it to the most the device allows beside the
 * kernel's static shared memory, so renderers of different scenes can live side
 * by side.  Returns that limit, or -1. */
typedef void (*gd_kernel_fn)(const GdParams);
/* the instantiations: without or with the code for split lines; tables in scratch or on chip; all kinds of launches or the
 * plain ones */
static const gd_kernel_fn gd_kernels[8] = {
    gd_render_kernel<false, false, false>, gd_render_kernel<false, false, true>, gd_render_kernel<false, true, false>,
    gd_render_kernel<false, true, true>, gd_render_kernel<true, false, false>, gd_render_kernel<true, false, true>,
    gd_render_kernel<true, true, false>, gd_render_kernel<true, true, true>};
static gd_kernel_fn gd_kernel_for(const gd_renderer *r, bool plain) {
  return gd_kernels[(r->base.sc.F > 0 ? 4 : 0) + (r->chip ? 2 : 0) + (plain ? 1 : 0)];
}

static int gd_raise_shared_limit(int maxOptin) {
  int limit = maxOptin;
  for (int k = 0; k < 8; ++k) {
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, gd_kernels[k]) != cudaSuccess) return -1;
    if (maxOptin - (int)fa.sharedSizeBytes < limit) limit = maxOptin - (int)fa.sharedSizeBytes;
  }
  for (int k = 0; k < 8; ++k)
    if (cudaFuncSetAttribute(gd_kernels[k], cudaFuncAttributeMaxDynamicSharedMemorySize, limit) != cudaSuccess) return -1;
  return limit;
}

/* Shared-memory offsets of a scene (r->base), with the walk's tables on chip or not; returns the total. */
static size_t gd_layout(gd_renderer *r, int secWallsN, bool chip) {
  GdParams &b = r->base;
  const int W = b.sc.W, S = b.sc.S, F = b.sc.F;
  size_t o = GD_OFF_HOT + (size_t)W * sizeof(GdHot);
  auto take = [&o](size_t bytes) { const size_t at = o; o += gd_align16(bytes); return (int)at; };
  b.offSectors = take((size_t)S * 16);
  b.offSecOff = take(((size_t)S + 1) * 2);
  b.offSecWalls = take((size_t)secWallsN * 2);
  b.offVtx = take((size_t)W * 8);
  b.offFrags = take((size_t)F * 4);
  b.offActors = take((size_t)(r->maxThings > 0 ? r->maxThings : 1) * sizeof(GdActor));
  if (chip) {
    b.offRows = take(((size_t)W + F) * 4 * sizeof(GdRow));
    b.offPrep = take((size_t)W * 16);
    b.offPlanes = take((size_t)S * 2 * GD_PLANE_BYTES);
    b.offSides = take((size_t)W * 2 * sizeof(GdSide));
  } else {
    b.offRows = 0;
    b.offPrep = W * 4 * (int)sizeof(GdRow);
    b.offPlanes = b.offPrep + W * 16;
    b.offSides = 0;
  }
  return o;
}

extern "C" int gd_renderer_create(const void *blob_header_host, const void *blob_dev, size_t blob_bytes, int device,
                                  int max_things, gd_renderer **out) {
  if (!blob_header_host || !blob_dev || !out) return GD_ERR_NULL;
  if (blob_bytes < GD_HDR_WORDS * 4) return GD_ERR_BLOB;
  if (((uintptr_t)blob_dev) & 15) return GD_ERR_ALIGN;
  if (max_things < 0 || max_things > 64) return GD_ERR_SIZE;
  const int32_t *h = (const int32_t *)blob_header_host;
  if (h[GD_H_MAGIC] != GD_MAGIC || h[GD_H_VERSION] != GD_VERSION || (size_t)h[GD_H_BYTES] != blob_bytes)
    return GD_ERR_BLOB;
  if (h[GD_H_UNSUPPORTED] != 0) return GD_ERR_UNSUPPORTED;
  if (h[GD_H_WALLS] <= 0 || h[GD_H_WALLS] >= 32768 || h[GD_H_SECTORS] <= 0 || h[GD_H_SECTORS] >= 32768)
    return GD_ERR_SIZE;
  gd_renderer *r = new (std::nothrow) gd_renderer;
  if (!r) return GD_ERR_CUDA;
  r->copyStream = nullptr;
  r->copiesDone = nullptr;
  r->decalScratch = nullptr;
  r->staticFrags = nullptr; r->fragBytes = 0;
  for (int c = 0; c < GD_HOST_CHUNKS; ++c) r->chunkDone[c] = nullptr;
  memcpy(r->header, h, sizeof r->header);
  r->device = device;
  r->blobDev = blob_dev;
  r->maxThings = max_things;
  const uint8_t *d = (const uint8_t *)blob_dev;
  memset(&r->base, 0, sizeof r->base);
  GdScene &sc = r->base.sc;
  sc.W = h[GD_H_WALLS]; sc.S = h[GD_H_SECTORS]; sc.T = h[GD_H_TEXTURES];
  sc.texH = h[GD_H_TEX_H]; sc.texW = h[GD_H_TEX_W];
  sc.P = h[GD_H_SPRITES]; sc.sprH = h[GD_H_SPR_H]; sc.sprW = h[GD_H_SPR_W];
  sc.Q = h[GD_H_WPN_PATCHES]; sc.wpnH = h[GD_H_WPN_H]; sc.wpnW = h[GD_H_WPN_W]; sc.wpnTics = h[GD_H_WPN_TICS];
  sc.nStarts = h[GD_H_STARTS]; sc.B = h[GD_H_BLOCKING]; sc.nbDirect = h[GD_H_NB_DIRECT];
  sc.wpnAvailable = h[GD_H_WPN_AVAILABLE]; sc.hudPatches = h[GD_H_HUD_PATCHES];
#define SECP(type, name) (const type *)gd_section(d, h, name)
  sc.walls = SECP(float, GD_S_WALLS); sc.wsec = SECP(int32_t, GD_S_WALL_SECTORS); sc.wlen = SECP(float, GD_S_WALL_LEN);
  sc.sideTex = SECP(int32_t, GD_S_SIDE_TEX); sc.sideOff = SECP(float, GD_S_SIDE_OFF);
  sc.wvtx = SECP(int32_t, GD_S_WALL_VTX); sc.vtxOff = SECP(int32_t, GD_S_VTX_OFF); sc.vtxWalls = SECP(int32_t, GD_S_VTX_WALLS);
  sc.nbDirectTab = SECP(int32_t, GD_S_NB_DIRECT); sc.nbOff = SECP(int32_t, GD_S_NB_OFF);
  sc.nbIdx = SECP(int32_t, GD_S_NB_IDX); sc.nbFlags = SECP(int32_t, GD_S_NB_FLAGS);
  sc.sbStartOff = SECP(int32_t, GD_S_SB_START_OFF); sc.sbStartIdx = SECP(int32_t, GD_S_SB_START_IDX);
  sc.sbEndOff = SECP(int32_t, GD_S_SB_END_OFF); sc.sbEndIdx = SECP(int32_t, GD_S_SB_END_IDX);
  sc.secF = SECP(float, GD_S_SECTOR_F); sc.secI = SECP(int32_t, GD_S_SECTOR_I);
  sc.secOff = SECP(int32_t, GD_S_SEC_OFF); sc.secWalls = SECP(int32_t, GD_S_SEC_WALLS);
  sc.edgeOff = SECP(int32_t, GD_S_EDGE_OFF); sc.edgeWalls = SECP(int32_t, GD_S_EDGE_WALLS);
  sc.blocking = SECP(int32_t, GD_S_BLOCKING);
  sc.texInfo = SECP(int32_t, GD_S_TEX_INFO); sc.texAtlas = SECP(uint8_t, GD_S_TEX_ATLAS);
  sc.texAtlasCol = SECP(uint8_t, GD_S_TEX_ATLAS_COL);
  sc.playpal = SECP(uint8_t, GD_S_PLAYPAL); sc.colormap = SECP(uint8_t, GD_S_COLORMAP);
  sc.sprInfo = SECP(int32_t, GD_S_SPR_INFO); sc.sprAtlas = SECP(uint8_t, GD_S_SPR_ATLAS); sc.sprPost = SECP(uint8_t, GD_S_SPR_POST);
  sc.addLut = SECP(uint8_t, GD_S_ADD_LUT); sc.transLut = SECP(uint8_t, GD_S_TRANS_LUT);
  sc.wpnInfo = SECP(int32_t, GD_S_WPN_INFO); sc.wpnAtlas = SECP(uint8_t, GD_S_WPN_ATLAS); sc.wpnOpaque = SECP(uint8_t, GD_S_WPN_OPAQUE);
  sc.wpnFrameIds = SECP(int32_t, GD_S_WPN_FRAME_IDS); sc.wpnFlashIds = SECP(int32_t, GD_S_WPN_FLASH_IDS);
  sc.wpnFlashLights = SECP(int32_t, GD_S_WPN_FLASH_LIGHTS);
  sc.hudInfo = SECP(int32_t, GD_S_HUD_INFO); sc.hudAtlas = SECP(uint8_t, GD_S_HUD_ATLAS); sc.hudOpaque = SECP(uint8_t, GD_S_HUD_OPAQUE);
  sc.fineSine = SECP(int32_t, GD_S_FINESINE); sc.fineTan = SECP(int32_t, GD_S_FINETAN);
  sc.rayOffsets = SECP(float, GD_S_RAY_OFFSETS); sc.rayCosCorr = SECP(float, GD_S_RAY_COSCORR);
  sc.secBBox = SECP(float, GD_S_SECTOR_BBOX);
  sc.maskedWalls = SECP(int32_t, GD_S_MASKED_WALLS);
  sc.damageAlpha = SECP(float, GD_S_DAMAGE_ALPHA);
  sc.groupH[1] = SECP(float, GD_S_FLOOR_GROUP_H); sc.groupOff[1] = SECP(int32_t, GD_S_FLOOR_GROUP_OFF);
  sc.groupSec[1] = SECP(int32_t, GD_S_FLOOR_GROUP_SEC); sc.groups[1] = h[GD_H_FLOOR_GROUPS];
  sc.groupH[0] = SECP(float, GD_S_CEIL_GROUP_H); sc.groupOff[0] = SECP(int32_t, GD_S_CEIL_GROUP_OFF);
  sc.groupSec[0] = SECP(int32_t, GD_S_CEIL_GROUP_SEC); sc.groups[0] = h[GD_H_CEIL_GROUPS];
  sc.M = h[GD_H_MASKED_WALLS_N];
  sc.decals = h[GD_H_DECALS]; sc.decalH = h[GD_H_DECAL_H]; sc.decalW = h[GD_H_DECAL_W];
  sc.decalInfo = SECP(int32_t, GD_S_DECAL_INFO); sc.wallFine = SECP(int32_t, GD_S_WALL_FINE);
  sc.decalAtlas = SECP(uint8_t, GD_S_DECAL_ATLAS); sc.decalOpacity = SECP(uint8_t, GD_S_DECAL_OPACITY);
  sc.decalBlack = SECP(uint8_t, GD_S_DECAL_BLACK);
  sc.F = h[GD_H_FRAGMENTS]; sc.fragOff = SECP(int32_t, GD_S_FRAG_OFF); sc.fragFixed = SECP(int32_t, GD_S_FRAG_FIXED);
  sc.cells = SECP(GdCells, GD_S_CELLS);
  r->decals = nullptr; r->decalSlots = 0; r->decalScratch = nullptr; r->decalScratchBytes = 0;
#undef SECP
  const int secWallsN = h[GD_H_SEC_WALLS_N];
  if (secWallsN < 0 || secWallsN > 65535) { delete r; return GD_ERR_SIZE; }
  int prev = 0;
  if (cudaGetDevice(&prev) != cudaSuccess || cudaSetDevice(device) != cudaSuccess) { delete r; return GD_ERR_CUDA; }
  int maxOptin = 0, perSmBytes = 0, reserved = 0, sms = 0;
  cudaDeviceGetAttribute(&maxOptin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  cudaDeviceGetAttribute(&perSmBytes, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device);
  cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, device);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  int rc = GD_OK;
  const int limit = gd_raise_shared_limit(maxOptin);
  /* what one of two CTAs on an SM may take beside the kernel's static shared memory */
  const size_t half = (size_t)(perSmBytes / 2 - reserved - (maxOptin - limit));
  r->smemBytes = gd_layout(r, secWallsN, true);
  r->chip = r->smemBytes <= half;
  if (!r->chip) r->smemBytes = gd_layout(r, secWallsN, false);
  if (limit < 0) {
    rc = GD_ERR_CUDA;
  } else if ((size_t)limit < r->smemBytes || (size_t)sc.W * 2 > GD_AUX_BYTES) {
    rc = GD_ERR_SHARED;
  } else {
    int perSm = 0, perSmPlain = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, gd_kernel_for(r, false), GD_THREADS, r->smemBytes) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSmPlain, gd_kernel_for(r, true), GD_THREADS, r->smemBytes) != cudaSuccess ||
        perSm < 1 || perSmPlain < 1)
      rc = GD_ERR_CUDA;
    else
      r->ctas = sms * (perSm < perSmPlain ? perSm : perSmPlain);  /* one persistent CTA per resident slot */
  }
  if (sc.F > 0) r->fragBytes = gd_frag_bytes(sc.F, r->chip);
  if (rc == GD_OK && sc.F > 0 && gd_fits_static(sc)) {
    void *mem = nullptr;
    if (cudaMalloc(&mem, GD_STATIC_MAX_CTAS * r->fragBytes) != cudaSuccess) rc = GD_ERR_CUDA;
    r->staticFrags = (uint8_t *)mem;
  }
  if (rc == GD_OK && h[GD_HDR_SECTION0 + GD_S_CELLS] == 0) {
    void *address = nullptr;
    if (cudaGetSymbolAddress(&address, gd_no_cells) != cudaSuccess) rc = GD_ERR_CUDA;
    sc.cells = (const GdCells *)address;
  }
  r->base.maxThings = max_things;
  r->base.secWallsN = secWallsN;
  r->base.perCta = r->base.fragStride = gd_scratch_per_cta(sc.W, sc.S) + r->fragBytes;
  r->sidesOffset = (size_t)r->ctas * r->base.perCta;
  r->base.queueOffset = r->sidesOffset + (r->chip ? 0 : (size_t)sc.W * 2 * sizeof(GdSide));
  r->copyStream = nullptr;
  r->copiesDone = nullptr;
  for (int c = 0; c < GD_HOST_CHUNKS; ++c) r->chunkDone[c] = nullptr;
  if (rc == GD_OK) {
    bool ok = cudaStreamCreateWithFlags(&r->copyStream, cudaStreamNonBlocking) == cudaSuccess &&
              cudaEventCreateWithFlags(&r->copiesDone, cudaEventDisableTiming) == cudaSuccess;
    for (int c = 0; ok && c < GD_HOST_CHUNKS; ++c)
      ok = cudaEventCreateWithFlags(&r->chunkDone[c], cudaEventDisableTiming) == cudaSuccess;
    if (!ok) rc = GD_ERR_CUDA;
  }
  cudaSetDevice(prev);
  if (rc != GD_OK) { cudaGetLastError(); gd_renderer_destroy(r); return rc; }
  *out = r;
  return GD_OK;
}

extern "C" void gd_renderer_destroy(gd_renderer *r) {
  if (!r) return;
  int prev = 0;
  bool switched = cudaGetDevice(&prev) == cudaSuccess && cudaSetDevice(r->device) == cudaSuccess;
  for (int c = 0; c < GD_HOST_CHUNKS; ++c)
    if (r->chunkDone[c]) cudaEventDestroy(r->chunkDone[c]);
  if (r->copiesDone) cudaEventDestroy(r->copiesDone);
  if (r->copyStream) cudaStreamDestroy(r->copyStream);
  if (r->decalScratch) cudaFree(r->decalScratch);
  if (r->staticFrags) cudaFree(r->staticFrags);
  if (switched) cudaSetDevice(prev);
  delete r;
}

extern "C" int gd_renderer_bind_decals(gd_renderer *r, const void *decals, int slots) {
  if (!r) return GD_ERR_NULL;
  if (!decals) { r->decals = nullptr; r->decalSlots = 0; return GD_OK; }
  if (slots < 1 || slots > GD_MAX_DECAL_SLOTS) return GD_ERR_SIZE;
  if ((uintptr_t)decals & 15) return GD_ERR_ALIGN;
  int current = -1;
  if (cudaGetDevice(&current) != cudaSuccess) return GD_ERR_CUDA;
  if (current != r->device) return GD_ERR_DEVICE;
  const size_t need = (size_t)r->ctas * gd_decal_scratch_per_cta(slots);
  if (need > r->decalScratchBytes) {
    if (r->decalScratch) cudaFree(r->decalScratch);      /* waits for work that still uses it */
    r->decalScratch = nullptr; r->decalScratchBytes = 0;
    r->decals = nullptr; r->decalSlots = 0;
    void *mem = nullptr;
    if (cudaMalloc(&mem, need) != cudaSuccess) { cudaGetLastError(); return GD_ERR_CUDA; }
    r->decalScratch = (uint8_t *)mem; r->decalScratchBytes = need;
  }
  r->decals = (const gd_decal *)decals; r->decalSlots = slots;
  return GD_OK;
}

extern "C" size_t gd_renderer_scratch_bytes(const gd_renderer *r) {
  return r ? r->base.queueOffset + 16 : 0;
}

extern "C" int gd_renderer_ctas(const gd_renderer *r) { return r ? r->ctas : 0; }
extern "C" size_t gd_renderer_shared_bytes(const gd_renderer *r) { return r ? r->smemBytes : 0; }
extern "C" size_t gd_renderer_shared_bytes_view(const gd_renderer *r) { return r ? r->smemBytes : 0; }

/* `frames` frames by up to `ctas` CTAs.  When they are so few that three of four CTAs would idle, a lane is drawn by
 * four of them, each a slice of its columns: what a lane waits for is its slowest warp, and then its sprites, unclaimed
 * pixels and resize, which a slice has a quarter of.  (64 sectors, 12 things, us a step without and with slices: 1 lane 112 and
 * 92, 16 lanes 322 and 297, 74 lanes 323 and 314.  Halves of a lane for the next 74 lanes do not pay for setting each
 * lane up twice: 100 lanes 324 and 327, 148 lanes 326 and 351.) */
static int gd_draw(const gd_renderer *r, GdParams &p, int frames, int ctas, bool slices, void *stream) {
  p.sliceShift = slices && frames * 4LL <= ctas ? 2 : 0;
  const long long tasks = ((long long)((p.flags & GD_F_STEP_RESET) ? 2 : 1) * frames) << p.sliceShift;
  const int grid = tasks < ctas ? (int)tasks : ctas;
  if (!r->chip) gd_side_setup_kernel<<<(p.sc.W * 2 + 127) / 128, 128, 0, (cudaStream_t)stream>>>(p.sc, p.sides);
  gd_kernel_for(r, !(p.flags & GD_F_STEP_RESET) && p.sliceShift == 0)<<<grid, GD_THREADS, r->smemBytes, (cudaStream_t)stream>>>(p);
  return cudaGetLastError() == cudaSuccess ? GD_OK : GD_ERR_CUDA;
}

/* gd_render_step_reset: the old frames of the lanes that are reset, before the resets' frames take their place */
__global__ void gd_final_frames_kernel(const uint8_t *mask, const uint4 *stack, uint4 *finalStack) {
  const int frame = GD_OBS * GD_OBS / 16;
  if (!mask[blockIdx.x]) return;
  stack += (size_t)blockIdx.x * GD_STACK * frame;
  finalStack += (size_t)blockIdx.x * GD_STACK * frame;
  for (int i = threadIdx.x; i < (GD_STACK - 1) * frame; i += blockDim.x) finalStack[i] = stack[frame + i];
}

static int gd_launch(const gd_renderer *r, const int32_t *lanes, const gd_thing *things, int n, int flags,
                     uint8_t *stack, const uint8_t *reset_mask, uint8_t *obs_out, uint8_t *indexed_out,
                     uint8_t *rgb_out, void *scratch, size_t scratch_bytes, int *status, void *stream,
                     int ring_head = 0, const int32_t *reset_lanes = nullptr, const gd_thing *reset_things = nullptr,
                     uint8_t *final_stack = nullptr, bool slices = true) {
  if (!r || !lanes || !scratch || !status) return GD_ERR_NULL;
  if (r->maxThings > 0 && !things) return GD_ERR_NULL;
  if (n < 0) return GD_ERR_SIZE;
  if (n == 0) return GD_OK;
  int current = -1;
  if (cudaGetDevice(&current) != cudaSuccess) return GD_ERR_CUDA;
  if (current != r->device) return GD_ERR_DEVICE;   /* the launch goes to the current device */
  if (scratch_bytes < gd_renderer_scratch_bytes(r)) return GD_ERR_SCRATCH;
  uintptr_t align = (uintptr_t)lanes | (uintptr_t)things | (uintptr_t)stack | (uintptr_t)obs_out |
                    (uintptr_t)indexed_out | (uintptr_t)rgb_out | (uintptr_t)scratch | (uintptr_t)reset_lanes |
                    (uintptr_t)reset_things | (uintptr_t)final_stack;
  if (align & 15) return GD_ERR_ALIGN;
  if ((flags & GD_F_STEP_RESET) && n > 0x3FFFFFFF) return GD_ERR_SIZE;
  GdParams p = r->base;
  p.lanes = lanes; p.things = things; p.n = n; p.flags = flags;
  p.stack = stack; p.ringHead = ring_head; p.resetMask = reset_mask; p.obsOut = obs_out; p.indexedOut = indexed_out; p.rgbOut = rgb_out;
  p.scratch = (uint8_t *)scratch; p.status = status;
  p.sides = (GdSide *)(p.scratch + r->sidesOffset);
  p.frags = p.scratch + gd_scratch_per_cta(r->base.sc.W, r->base.sc.S);
  p.decals = r->decals; p.decalSlots = r->decalSlots; p.decalScratch = r->decalScratch;
  p.resetLanes = reset_lanes; p.resetThings = reset_things; p.finalStack = final_stack;
  if (flags & GD_F_STEP_RESET) {
    gd_final_frames_kernel<<<n, 256, 0, (cudaStream_t)stream>>>(reset_mask, (const uint4 *)stack, (uint4 *)final_stack);
  }
  return gd_draw(r, p, n, r->ctas, slices, stream);
}

extern "C" int gd_render_step(const gd_renderer *r, const int32_t *lanes, const void *things, int n, int mask_hud,
                              uint8_t *stack, void *scratch, size_t scratch_bytes, int *status, void *stream) {
  if (r && n == 0) return GD_OK;   /* an empty batch needs no buffers */
  if (!stack) return GD_ERR_NULL;
  int flags = GD_F_STACK_ROLL | (mask_hud ? GD_F_MASK_HUD : GD_F_DRAW_HUD);
  return gd_launch(r, lanes, (const gd_thing *)things, n, flags, stack, nullptr, nullptr, nullptr, nullptr, scratch,
                   scratch_bytes, status, stream);
}

extern "C" int gd_render_step_ring(const gd_renderer *r, const int32_t *lanes, const void *things, int n,
                                   int mask_hud, uint8_t *ring, int head, void *scratch, size_t scratch_bytes,
                                   int *status, void *stream) {
  if (r && n == 0) return GD_OK;   /* an empty batch needs no buffers */
  if (!ring) return GD_ERR_NULL;
  if (head < 0 || head >= GD_STACK) return GD_ERR_SIZE;
  int flags = GD_F_STACK_RING | (mask_hud ? GD_F_MASK_HUD : GD_F_DRAW_HUD);
  return gd_launch(r, lanes, (const gd_thing *)things, n, flags, ring, nullptr, nullptr, nullptr, nullptr, scratch,
                   scratch_bytes, status, stream, head);
}

extern "C" int gd_render_reset_ring(const gd_renderer *r, const int32_t *lanes, const void *things, int n,
                                    int mask_hud, const uint8_t *reset_mask, uint8_t *ring, void *scratch,
                                    size_t scratch_bytes, int *status, void *stream) {
  if (r && n == 0) return GD_OK;   /* an empty batch needs no buffers */
  if (!ring || !reset_mask) return GD_ERR_NULL;
  int flags = GD_F_STACK_RING | GD_F_STACK_FILL | (mask_hud ? GD_F_MASK_HUD : GD_F_DRAW_HUD);
  return gd_launch(r, lanes, (const gd_thing *)things, n, flags, ring, reset_mask, nullptr, nullptr, nullptr, scratch,
                   scratch_bytes, status, stream);
}

extern "C" int gd_render_reset(const gd_renderer *r, const int32_t *lanes, const void *things, int n, int mask_hud,
                               const uint8_t *reset_mask, uint8_t *stack, void *scratch, size_t scratch_bytes,
                               int *status, void *stream) {
  if (r && n == 0) return GD_OK;   /* an empty batch needs no buffers */
  if (!stack || !reset_mask) return GD_ERR_NULL;
  int flags = GD_F_STACK_FILL | (mask_hud ? GD_F_MASK_HUD : GD_F_DRAW_HUD);
  return gd_launch(r, lanes, (const gd_thing *)things, n, flags, stack, reset_mask, nullptr, nullptr, nullptr, scratch,
                   scratch_bytes, status, stream);
}

extern "C" int gd_render_step_reset(const gd_renderer *r, const int32_t *lanes, const void *things, const int32_t *reset_lanes,
                                    const void *reset_things, int n, int mask_hud, const uint8_t *reset_mask, uint8_t *stack,
                                    uint8_t *final_stack, void *scratch, size_t scratch_bytes, int *status, void *stream) {
  if (r && n == 0) return GD_OK;   /* an empty batch needs no buffers */
  if (!r || !stack || !final_stack || !reset_mask || !reset_lanes) return GD_ERR_NULL;
  if (r->maxThings > 0 && !reset_things) return GD_ERR_NULL;
  if (n < 0) return GD_ERR_SIZE;
  /* a lane's step and its reset are drawn in any order and at the same time, the one into both stacks */
  const uintptr_t bytes = (uintptr_t)n * GD_STACK * GD_OBS * GD_OBS, a = (uintptr_t)stack, b = (uintptr_t)final_stack;
  if ((a < b ? b - a : a - b) < bytes) return GD_ERR_OVERLAP;
  int flags = GD_F_STEP_RESET | (mask_hud ? GD_F_MASK_HUD : GD_F_DRAW_HUD);
  return gd_launch(r, lanes, (const gd_thing *)things, n, flags, stack, reset_mask, nullptr, nullptr, nullptr, scratch,
                   scratch_bytes, status, stream, 0, reset_lanes, (const gd_thing *)reset_things, final_stack);
}

extern "C" int gd_render_frames(const gd_renderer *r, const int32_t *lanes, const void *things, int n, int mask_hud,
                                int include_hud, uint8_t *obs_out, uint8_t *indexed_out, uint8_t *rgb_out,
                                void *scratch, size_t scratch_bytes, int *status, void *stream) {
  if (r && n == 0) return GD_OK;   /* an empty batch needs no buffers */
  if (!obs_out && !indexed_out && !rgb_out) return GD_ERR_NULL;
  int flags = (mask_hud ? GD_F_MASK_HUD : 0) | ((include_hud || !mask_hud) ? GD_F_DRAW_HUD : 0);
  return gd_launch(r, lanes, (const gd_thing *)things, n, flags, nullptr, nullptr, obs_out, indexed_out, rgb_out,
                   scratch, scratch_bytes, status, stream);
}

extern "C" int gd_render_step_frames(const gd_renderer *r, const int32_t *lanes, const void *things, int n,
                                     int mask_hud, int include_hud, uint8_t *stack, uint8_t *indexed_out,
                                     uint8_t *rgb_out, void *scratch, size_t scratch_bytes, int *status,
                                     void *stream) {
  if (r && n == 0) return GD_OK;   /* an empty batch needs no buffers */
  if (!stack || (!indexed_out && !rgb_out)) return GD_ERR_NULL;
  int flags = GD_F_STACK_ROLL | (mask_hud ? GD_F_MASK_HUD : 0) | ((include_hud || !mask_hud) ? GD_F_DRAW_HUD : 0);
  return gd_launch(r, lanes, (const gd_thing *)things, n, flags, stack, nullptr, nullptr, indexed_out, rgb_out,
                   scratch, scratch_bytes, status, stream);
}

/* Host-buffer variant of gd_render_step: copies the lane and thing records to
 * the caller's device staging buffers, renders, and copies the newest frame of
 * every lane (stack slot 3) back to `obs_host`.  Everything is queued on
 * `stream`; pinned host memory keeps the copies asynchronous. */
extern "C" int gd_render_step_host(const gd_renderer *r, const int32_t *lanes_host, const void *things_host, int n,
                                   int mask_hud, int32_t *lanes_dev, void *things_dev, uint8_t *stack,
                                   uint8_t *obs_host, void *scratch, size_t scratch_bytes, int *status,
                                   void *stream) {
  if (r && n == 0) return GD_OK;   /* an empty batch needs no buffers */
  if (!r || !lanes_host || !lanes_dev || !stack || !obs_host) return GD_ERR_NULL;
  if (r->maxThings > 0 && (!things_host || !things_dev)) return GD_ERR_NULL;
  if (n < 0) return GD_ERR_SIZE;
  if (n == 0) return GD_OK;
  /* every argument is checked before the first copy is queued */
  if (!scratch || !status) return GD_ERR_NULL;
  if (scratch_bytes < gd_renderer_scratch_bytes(r)) return GD_ERR_SCRATCH;
  if (((uintptr_t)lanes_dev | (uintptr_t)things_dev | (uintptr_t)stack | (uintptr_t)scratch) & 15) return GD_ERR_ALIGN;
  {
    int current = -1;
    if (cudaGetDevice(&current) != cudaSuccess) return GD_ERR_CUDA;
    if (current != r->device) return GD_ERR_DEVICE;
  }
  cudaStream_t s = (cudaStream_t)stream;
  size_t thingStride = (size_t)(r->maxThings > 0 ? r->maxThings : 1) * sizeof(gd_thing);
  if (cudaMemcpyAsync(lanes_dev, lanes_host, (size_t)n * GD_LANE_WORDS * 4, cudaMemcpyHostToDevice, s) != cudaSuccess)
    return GD_ERR_CUDA;
  if (things_host &&
      cudaMemcpyAsync(things_dev, things_host, (size_t)n * thingStride, cudaMemcpyHostToDevice, s) != cudaSuccess)
    return GD_ERR_CUDA;
  /* Pinned (or registered) host memory is mapped into the device's address
   * space: the kernel then writes every lane's newest frame straight into it
   * while it draws the following lanes, and no copy is left to wait for. */
  {
    cudaPointerAttributes attr;
    if (cudaPointerGetAttributes(&attr, obs_host) == cudaSuccess && attr.type == cudaMemoryTypeHost &&
        attr.devicePointer != nullptr && (((uintptr_t)attr.devicePointer) & 15) == 0) {
      int flags = GD_F_STACK_ROLL | (mask_hud ? GD_F_MASK_HUD : GD_F_DRAW_HUD);
      return gd_launch(r, lanes_dev, (const gd_thing *)things_dev, n, flags, stack, nullptr,
                       (uint8_t *)attr.devicePointer, nullptr, nullptr, scratch, scratch_bytes, status, stream, 0, nullptr, nullptr,
                       nullptr, false);    /* whole frames: a slice's would cross the bus in runs of 21 bytes */
    }
    cudaGetLastError();
  }
  /* Pageable host memory: lanes are drawn in chunks; each chunk's newest frames travel to the host
   * on the side stream while the next chunk is drawn.  The caller's stream
   * waits for the last copy, so synchronising it covers the whole call. */
  const size_t frame = (size_t)GD_OBS * GD_OBS;
  const int chunks = n >= 512 * GD_HOST_CHUNKS ? GD_HOST_CHUNKS : 1;
  const int per = (n + chunks - 1) / chunks;
  for (int c = 0; c < chunks; ++c) {
    const int n0 = c * per, nc = (n0 + per <= n ? per : n - n0);
    if (nc <= 0) break;
    const gd_thing *th = things_dev ? (const gd_thing *)things_dev + (size_t)n0 * (r->maxThings > 0 ? r->maxThings : 1)
                                    : nullptr;
    uint8_t *st = stack + (size_t)n0 * GD_STACK * frame;
    int rc = gd_render_step(r, lanes_dev + (size_t)n0 * GD_LANE_WORDS, th, nc, mask_hud, st, scratch, scratch_bytes,
                            status, stream);
    if (rc != GD_OK) return rc;
    cudaStream_t cs = s;
    if (chunks > 1) {
      cs = r->copyStream;
      if (cudaEventRecord(r->chunkDone[c], s) != cudaSuccess || cudaStreamWaitEvent(cs, r->chunkDone[c], 0) != cudaSuccess)
        return GD_ERR_CUDA;
    }
    if (cudaMemcpy2DAsync(obs_host + (size_t)n0 * frame, frame, st + (GD_STACK - 1) * frame, GD_STACK * frame, frame,
                          (size_t)nc, cudaMemcpyDeviceToHost, cs) != cudaSuccess)
      return GD_ERR_CUDA;
  }
  if (chunks > 1) {
    if (cudaEventRecord(r->copiesDone, r->copyStream) != cudaSuccess ||
        cudaStreamWaitEvent(s, r->copiesDone, 0) != cudaSuccess)
      return GD_ERR_CUDA;
  }
  return GD_OK;
}

/* ---- allocation-free entry point ------------------------------------------
 * gd_render_step for hosts that are not allowed to allocate device memory at
 * all -- for instance a plugin loaded into an inference server or a game
 * process whose memory pool is owned and fully budgeted by its embedder, or
 * code that runs after the framework's allocator has been frozen.  Such a
 * caller cannot obtain the scratch buffer the other entry points ask for, so
 * this variant keeps the CTAs' scratch in a fixed array inside the
 * library image.  Every GPU that loads the library holds GD_STATIC_SCRATCH_BYTES
 * of it until the process exits.
 */
/* a scene of W walls has fewer than W sectors (three walls bound a sector, a wall bounds two) */
#define GD_STATIC_PER_CTA ((GD_SCRATCH_FIXED + GD_STATIC_MAX_WALLS * (2 * GD_PLANE_ENTRY_BYTES + 2 * GD_PLANE_BYTES + \
                            sizeof(GdWall) + 4 * sizeof(GdRowProj) + 4 * sizeof(GdRow) + 16) + 127) & ~(size_t)63)
#define GD_STATIC_SIDES (GD_STATIC_MAX_CTAS * GD_STATIC_PER_CTA)
#define GD_STATIC_QUEUE (GD_STATIC_SIDES + GD_STATIC_MAX_WALLS * 2 * sizeof(GdSide))
#define GD_STATIC_SCRATCH_BYTES (GD_STATIC_QUEUE + 16)
#define GD_STATIC_MAX_DEVICES 64

static __device__ __align__(256) unsigned char gd_static_scratch[GD_STATIC_SCRATCH_BYTES];

/* device address of the array above, looked up once per device */
static unsigned char *gd_static_scratch_ptr[GD_STATIC_MAX_DEVICES];

extern "C" size_t gd_static_scratch_bytes(void) { return GD_STATIC_SCRATCH_BYTES; }
extern "C" int gd_static_max_walls(void) { return GD_STATIC_MAX_WALLS; }

extern "C" int gd_render_step_static(const gd_renderer *r, const int32_t *lanes, const void *things, int n,
                                     int mask_hud, uint8_t *stack, int *status, void *stream) {
  if (r && n == 0) return GD_OK;   /* an empty batch needs no buffers */
  if (!r || !lanes || !stack || !status) return GD_ERR_NULL;
  if (r->maxThings > 0 && !things) return GD_ERR_NULL;
  if (n < 0) return GD_ERR_SIZE;
  if (!gd_fits_static(r->base.sc)) return GD_ERR_STATIC_LIMIT;
  if (r->device < 0 || r->device >= GD_STATIC_MAX_DEVICES) return GD_ERR_STATIC_LIMIT;
  if (n == 0) return GD_OK;
  uintptr_t align = (uintptr_t)lanes | (uintptr_t)things | (uintptr_t)stack;
  if (align & 15) return GD_ERR_ALIGN;
  int current = -1;
  if (cudaGetDevice(&current) != cudaSuccess) return GD_ERR_CUDA;
  if (current != r->device) return GD_ERR_DEVICE;  /* the renderer's device must be the current one */
  unsigned char *scratch = gd_static_scratch_ptr[current];
  if (!scratch) {
    /* In host code the array's name is only a handle: the kernel needs the
     * address the symbol has on this device. */
    void *address = nullptr;
    if (cudaGetSymbolAddress(&address, gd_static_scratch) != cudaSuccess || !address) {
      cudaGetLastError();
      return GD_ERR_CUDA;
    }
    scratch = (unsigned char *)address;
    gd_static_scratch_ptr[current] = scratch;
  }
  GdParams p = r->base;
  p.lanes = lanes; p.things = (const gd_thing *)things; p.n = n;
  p.flags = GD_F_STACK_ROLL | (mask_hud ? GD_F_MASK_HUD : GD_F_DRAW_HUD);
  p.stack = stack; p.ringHead = 0; p.resetMask = nullptr; p.obsOut = nullptr; p.indexedOut = nullptr; p.rgbOut = nullptr;
  p.scratch = scratch; p.status = status;
  p.perCta = gd_scratch_per_cta(r->base.sc.W, r->base.sc.S);
  p.frags = r->staticFrags; p.fragStride = r->fragBytes;
  /* lane queue: the last 16 bytes of the array; zero when the library is
   * loaded and left at zero by every launch */
  p.queueOffset = GD_STATIC_QUEUE;
  p.sides = (GdSide *)(scratch + GD_STATIC_SIDES);
  p.decals = r->decals; p.decalSlots = r->decalSlots; p.decalScratch = r->decalScratch;
  return gd_draw(r, p, n, r->ctas < GD_STATIC_MAX_CTAS ? r->ctas : GD_STATIC_MAX_CTAS, true, stream);
}

/* ---- diagnostic: the device's float32 libm on caller-given arguments -------------------- */
__global__ void gd_probe_libm_kernel(int function, const float *a, const float *b, float *out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float r;
  switch (function) {
    case GD_PROBE_ATAN2F: r = atan2f(a[i], b[i]); break;
    case GD_PROBE_COSF: r = cosf(a[i]); break;
    case GD_PROBE_SINF: r = sinf(a[i]); break;
    default: r = sqrtf(a[i] * a[i] + b[i] * b[i]); break;      /* GD_PROBE_HYPOT: the sprite distance as the kernel forms it */
  }
  out[i] = r;
}

extern "C" int gd_probe_libm(int function, const float *a, const float *b, float *out, int n, void *stream) {
  if (!a || !out || ((function == GD_PROBE_ATAN2F || function == GD_PROBE_HYPOT) && !b)) return GD_ERR_NULL;
  if (function < GD_PROBE_ATAN2F || function > GD_PROBE_HYPOT || n < 0) return GD_ERR_SIZE;
  if (n == 0) return GD_OK;
  gd_probe_libm_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(function, a, b, out, n);
  return cudaGetLastError() == cudaSuccess ? GD_OK : GD_ERR_CUDA;
}

#endif

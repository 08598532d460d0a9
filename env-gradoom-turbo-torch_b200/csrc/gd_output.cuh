/* Area resize to the observation, the per-lane palette.
 * Part of gd_render.cu (one translation unit); not meant to be included elsewhere. */
#ifndef GD_OUTPUT_CUH
#define GD_OUTPUT_CUH

/* ---- phase: 320x240 -> 84x84 area resize + grayscale ---------------------
 * Integer definition: src/gradoom/_triton_kernels.py:120-177.  The weights
 * (y_overlap*x_overlap)/48 factor exactly into (y_overlap/12)*(x_overlap/4): twenty source rows of 7 units each
 * become seven output rows of 20 units, and a source column of 21 units goes to output columns of 80.
 *
 * Thread x sums its column's twenty rows into seven output rows (every pixel looks its colour up once; the weights
 * are constants of the unrolled rows), then the threads sum four or five columns each into the 7 x 84 pixels.
 * What bounds it is instructions: twenty lookups and 64-bit products per output pixel, as a loop over the output,
 * took 57 of a lane's 557 thousand cycles; column sums first, 44 of 426; with the weights of a thread's pixel column found
 * once, a black palette entry in place of tests, and the next rows' loads ahead of the barriers, 33. */
#define GD_RESIZE_ROWS 20
#define GD_RESIZE_OUT 7
#define GD_RESIZE_GROUPS (GD_THREADS / GD_OBS)           /* rows of pixels that the threads sum at once */
static_assert(GD_SCREEN_H % GD_RESIZE_ROWS == 0 && GD_OFF_MASKS + GD_RESIZE_OUT * GD_SW * 8 <= GD_OFF_RESULT, "the sums lie before the result");

__device__ __noinline__ void gd_resize(const uint8_t *frame, int srcRows, uint8_t *out_) {
  uint8_t *out = gd_as_shared(out_);
  const uint2 *pal = (const uint2 *)(gd_smem + GD_OFF_PAL64);
  uint2 *sums = (uint2 *)(gd_smem + GD_OFF_MASKS);       /* [7][320]: R | B << 16, G */
  const int x = threadIdx.x;
  const uint8_t *column = frame + x;
  /* the pixel column that a thread sums, in every third row: its four or five columns and their weights */
  const int group = x / GD_OBS < GD_RESIZE_GROUPS ? x / GD_OBS : GD_RESIZE_OUT, ox = x % GD_OBS, c0 = 80 * ox / 21;
  const unsigned w0 = 21u * (c0 + 1) - 80u * ox, w3 = min(38u - w0, 21u), w4 = w0 < 17u ? 17u - w0 : 0u;
  const int last = w4 ? 4 : 3;                           /* a fifth column may lie past the edge */
  unsigned index[GD_RESIZE_ROWS];                        /* the twenty rows' pixels; the next ones travel while these are summed */
#pragma unroll
  for (int r = 0; r < GD_RESIZE_ROWS; ++r) index[r] = column[r * GD_SW];
#pragma unroll 1
  for (int y0 = 0, o0 = 0; y0 < GD_SCREEN_H; y0 += GD_RESIZE_ROWS, o0 += GD_RESIZE_OUT * GD_OBS) {
    if (y0 >= srcRows) {                                 /* masked status-bar rows: black */
#pragma unroll 1
      for (int i = x; i < GD_RESIZE_OUT * GD_OBS; i += GD_THREADS) out[o0 + i] = 0;
      continue;
    }
    unsigned rb[GD_RESIZE_OUT], g[GD_RESIZE_OUT];
#pragma unroll
    for (int o = 0; o < GD_RESIZE_OUT; ++o) rb[o] = g[o] = 0u;
#pragma unroll
    for (int r = 0; r < GD_RESIZE_ROWS; ++r) {
      const uint2 c = pal[index[r]];
      const int o = 7 * r / 20;
      const unsigned first = 7 * r + 7 <= 20 * (o + 1) ? 7u : 20u * (o + 1) - 7u * r;
      rb[o] += first * c.x; g[o] += first * c.y;
      if (first < 7u) { rb[o + 1] += (7u - first) * c.x; g[o + 1] += (7u - first) * c.y; }
    }
    {
      const int next = y0 + GD_RESIZE_ROWS;
#pragma unroll
      for (int r = 0; r < GD_RESIZE_ROWS; ++r) index[r] = next + r < srcRows ? column[(next + r) * GD_SW] : 256u;
    }
    __syncthreads();                                     /* the sums of the rows before have been read */
#pragma unroll
    for (int o = 0; o < GD_RESIZE_OUT; ++o) sums[o * GD_SW + x] = make_uint2(rb[o], g[o]);
    __syncthreads();
#pragma unroll 1
    for (int o = group; o < GD_RESIZE_OUT; o += GD_RESIZE_GROUPS) {
      const uint2 *row = sums + o * GD_SW + c0;
      const uint2 c[5] = {row[0], row[1], row[2], row[3], row[last]};
      unsigned r = w0 * (c[0].x & 0xFFFFu), b = w0 * (c[0].x >> 16), gg = w0 * c[0].y;
      r += 21u * ((c[1].x & 0xFFFFu) + (c[2].x & 0xFFFFu)); b += 21u * ((c[1].x >> 16) + (c[2].x >> 16)); gg += 21u * (c[1].y + c[2].y);
      r += w3 * (c[3].x & 0xFFFFu); b += w3 * (c[3].x >> 16); gg += w3 * c[3].y;
      r += w4 * (c[4].x & 0xFFFFu); b += w4 * (c[4].x >> 16); gg += w4 * c[4].y;
      r = (r + 800) / 1600; gg = (gg + 800) / 1600; b = (b + 800) / 1600;
      out[o0 + o * GD_OBS + ox] = (uint8_t)((r * 77 + gg * 150 + b * 29 + 128) >> 8);
    }
  }
}

/* PLAYPAL of the lane in shared memory, as R | B << 16 | G << 32 for the
 * resize and as RGB24 words: the scene's palette, or its bonus / damage blends when
 * the lane's flags ask for screen flashes (engine.py:15381-15398; float32,
 * separately rounded, truncating conversion). */
__device__ void gd_lane_palette(const GdScene &sc, const GdShared &sh, int flags) {
  const int i = threadIdx.x;
  if (i >= 256) {
    if (i == 256) sh.pal64[i] = 0;
    return;
  }
  float bonus = 0.0f, flash = 0.0f;
  const bool blend = (flags & 4) != 0;
  if (blend) {
    int damage = min((flags >> 8) & 0xFF, 113), bonusCount = (flags >> 16) & 0xFF;
    bonus = fminf((float)bonusCount * 8.0f, 128.0f) / 255.0f;
    flash = sc.damageAlpha[damage] / 255.0f;
  }
  const float gold[3] = {215.0f, 186.0f, 69.0f}, red[3] = {255.0f, 0.0f, 0.0f};
  unsigned ch[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    unsigned v = sc.playpal[i * 3 + c];
    if (blend) {
      float rgb = (float)v * (1.0f - bonus) + gold[c] * bonus;
      float out = rgb * (1.0f - flash) + red[c] * flash;
      out = fminf(fmaxf(out, 0.0f), 255.0f);
      v = (unsigned)out;
    }
    ch[c] = v;
  }
  sh.pal64[i] = (unsigned long long)(ch[0] | (ch[2] << 16)) | ((unsigned long long)ch[1] << 32);
  sh.pal32[i] = ch[0] | (ch[1] << 8) | (ch[2] << 16);
}

#endif

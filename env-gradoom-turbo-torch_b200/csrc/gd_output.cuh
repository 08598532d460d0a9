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

template <bool kWhole>
__device__ __noinline__ void gd_resize(const uint8_t *frame, int srcRows, uint8_t *out_, int firstColumn, int shift) {
  const int x0 = kWhole ? 0 : firstColumn, sliceShift = kWhole ? 0 : shift;
  uint8_t *out = gd_as_shared(out_);
  const uint2 *pal = (const uint2 *)(gd_smem + GD_OFF_PAL64);
  /* a slice's columns are dealt to as many groups of threads as there are slices, and each takes every so many-th band
   * of rows */
  const int width = GD_SW >> sliceShift, obsWidth = GD_OBS >> sliceShift, bands = 1 << sliceShift;
  const int band = threadIdx.x / width, x = threadIdx.x - band * width;
  uint2 *sums = (uint2 *)(gd_smem + GD_OFF_MASKS) + band * GD_RESIZE_OUT * width;   /* [7][width]: R | B << 16, G */
  const uint8_t *column = frame + x0 + x;
  /* the pixel column that a thread sums, in every third row: its four or five columns and their weights */
  const int group = x / obsWidth < GD_RESIZE_GROUPS ? x / obsWidth : GD_RESIZE_OUT, ox = x % obsWidth, c0 = 80 * ox / 21;
  const unsigned w0 = 21u * (c0 + 1) - 80u * ox, w3 = min(38u - w0, 21u), w4 = w0 < 17u ? 17u - w0 : 0u;
  const int last = w4 ? 4 : 3;                           /* a fifth column may lie past the edge */
  out += x0 * GD_OBS / GD_SW + ox;
  unsigned index[GD_RESIZE_ROWS];                        /* the twenty rows' pixels; the next ones travel while these are summed */
#pragma unroll
  for (int r = 0; r < GD_RESIZE_ROWS; ++r) index[r] = column[(band * GD_RESIZE_ROWS + r) * GD_SW];
#pragma unroll 1
  for (int b = band; b < GD_SCREEN_H / GD_RESIZE_ROWS; b += bands) {
    const int y0 = b * GD_RESIZE_ROWS, o0 = b * GD_RESIZE_OUT * GD_OBS;
    if (bands == 1 && y0 >= srcRows) {                   /* masked status-bar rows: black */
#pragma unroll 1
      for (int i = threadIdx.x; i < GD_RESIZE_OUT * GD_OBS; i += GD_THREADS) gd_as_shared(out_)[o0 + i] = 0;
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
      const int next = y0 + bands * GD_RESIZE_ROWS;
#pragma unroll
      for (int r = 0; r < GD_RESIZE_ROWS; ++r) index[r] = next + r < srcRows ? column[(next + r) * GD_SW] : 256u;
    }
    __syncthreads();                                     /* the sums of the rows before have been read */
#pragma unroll
    for (int o = 0; o < GD_RESIZE_OUT; ++o) sums[o * width + x] = make_uint2(rb[o], g[o]);
    __syncthreads();
#pragma unroll 1
    for (int o = group; o < GD_RESIZE_OUT; o += GD_RESIZE_GROUPS) {
      const uint2 *row = sums + o * width + c0;
      const uint2 c[5] = {row[0], row[1], row[2], row[3], row[last]};
      unsigned r = w0 * (c[0].x & 0xFFFFu), b = w0 * (c[0].x >> 16), gg = w0 * c[0].y;
      r += 21u * ((c[1].x & 0xFFFFu) + (c[2].x & 0xFFFFu)); b += 21u * ((c[1].x >> 16) + (c[2].x >> 16)); gg += 21u * (c[1].y + c[2].y);
      r += w3 * (c[3].x & 0xFFFFu); b += w3 * (c[3].x >> 16); gg += w3 * c[3].y;
      r += w4 * (c[4].x & 0xFFFFu); b += w4 * (c[4].x >> 16); gg += w4 * c[4].y;
      r = (r + 800) / 1600; gg = (gg + 800) / 1600; b = (b + 800) / 1600;
      out[o0 + o * GD_OBS] = (uint8_t)((r * 77 + gg * 150 + b * 29 + 128) >> 8);
    }
  }
}
static_assert(GD_SW / 4 == 80 && GD_OBS / 4 == 21 && GD_SCREEN_H / GD_RESIZE_ROWS % 4 == 0,
              "a quarter's columns make whole pixels, and its bands come out even");

/* What becomes of a lane's new frame: a whole frame in 16-byte vectors, a slice of it (pixel columns px0 .. px0 + px - 1) a
 * byte at a time.  A slice moves only its own bytes of the old frames, so that slices need not wait for each other. */
enum { GD_PUT_NONE, GD_PUT_ALL, GD_PUT_ALL8, GD_PUT_RING, GD_PUT_ROLL, GD_PUT_ROLL_FINAL, GD_PUT_FINAL_LAST, GD_PUT_LAST };
template <class T>
__device__ __noinline__ void gd_put_frame(const uint8_t *src_, uint8_t *stack_, uint8_t *final_, uint8_t *newest_, int mode, int head, int px0,
                                          int px) {
  const T *src = (const T *)gd_as_shared(src_);
  T *stack = (T *)stack_, *final = (T *)final_, *newest = (T *)newest_;
  const bool whole = sizeof(T) == 16;
  const int frame = GD_OBS * GD_OBS / (int)sizeof(T), count = whole ? frame : GD_OBS * px;
#pragma unroll 1
  for (int k = threadIdx.x; k < count; k += GD_THREADS) {
    const int i = whole ? k : k / px * GD_OBS + px0 + k % px;
    const T val = src[i];
    if (newest) newest[i] = val;
    if (mode == GD_PUT_ROLL || mode == GD_PUT_ROLL_FINAL) {
      const T a = stack[frame + i], b = stack[2 * frame + i], c = stack[3 * frame + i];
      stack[i] = a; stack[frame + i] = b; stack[2 * frame + i] = c; stack[3 * frame + i] = val;
      if (mode == GD_PUT_ROLL_FINAL) { final[i] = a; final[frame + i] = b; final[2 * frame + i] = c; final[3 * frame + i] = val; }
    } else if (mode == GD_PUT_RING) {
      stack[head * frame + i] = val; stack[(head + GD_STACK) * frame + i] = val;
    } else if (mode == GD_PUT_FINAL_LAST) {
      final[3 * frame + i] = val;
    } else if (mode == GD_PUT_LAST) {
      stack[3 * frame + i] = val;
    } else if (mode != GD_PUT_NONE) {
#pragma unroll 1
      for (int slot = 0; slot < (mode == GD_PUT_ALL8 ? 2 * GD_STACK : GD_STACK); ++slot) stack[slot * frame + i] = val;
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

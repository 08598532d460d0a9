/* The built-in state producer's step and reset as one launch each.
 * Part of gd_render.cu (one translation unit); not meant to be included elsewhere. */
#ifndef GD_STEPPER_CUH
#define GD_STEPPER_CUH

/* What bounds these kernels is that there are two of them: a few hundred bytes a lane move, while the same
 * work as elementwise tensor operations was 34 launches for a step and 150 for a reset.  With four lanes of the
 * 16-sector map one step_and_reset_device call took 2.12 ms for 0.2 ms of drawing; it takes 0.2 ms. */

#define GD_SIGNALS 27          /* width of the signal buffer (src/gradoom/engine.py:509-539) */
#define GD_STEPPER_VIEW_HEIGHT 41.0f

/* deterministic number in [0, 1) of a seed (modulo 2^64) and a salt */
__device__ __forceinline__ double gd_stepper_uniform(i64 seed, i64 salt) {
  unsigned long long v = ((unsigned long long)seed * 2654435761ull + (unsigned long long)salt * 40503ull + 12345ull) & 0xFFFFFFFFull;
  v ^= v >> 15;
  v = (v * 2246822519ull) & 0xFFFFFFFFull;
  v ^= v >> 13;
  v = (v * 3266489917ull) & 0xFFFFFFFFull;
  v ^= v >> 16;
  return (double)v / 4294967296.0;
}

/* One warp per lane: the button mask, the game tics, then lane 0 of the warp does the bookkeeping. */
__global__ void __launch_bounds__(GDM_BLOCK) gd_stepper_step_kernel(const GdMoveParams q, const gd_stepper_state st,
                                                                    const uint8_t *buttons, int columns, long long tick,
                                                                    float *rewards, uint8_t *terminated, uint8_t *truncated) {
  const int l = (int)(((size_t)blockIdx.x * GDM_BLOCK + threadIdx.x) >> 5), t = threadIdx.x & 31;
  if (l >= q.n) return;                                        /* whole warps leave */
  const uint32_t pressed = __ballot_sync(0xffffffffu, t < columns && buttons[(size_t)l * columns + t] != 0);
  int time;
  if (q.tics > 0) {
    int32_t p[GD_PLAYER_WORDS];
    gd_player_advance(q, l, pressed, p);
    time = p[GD_P_EPISODE_TIME];
  } else {
    time = q.lanes[(size_t)l * GD_LANE_WORDS + GD_L_EPISODE_TIME];
  }
  if (t != 0) return;
  /* an attack kills the first living thing once in a while */
  float reward = 0.0f;
  if (st.k > 0) {
    const bool lucky = gd_stepper_uniform((i64)l + tick * 7919, 5) < 0.02;
    const i64 victim = gd_clamp((i64)(gd_stepper_uniform((i64)l + tick * 104729, 6) * (double)st.k), 0, st.k - 1);
    int32_t *word = st.things + ((size_t)l * st.max_things + (size_t)victim) * 4 + 3;
    if ((pressed & 1u) && lucky && (*word & (GD_THING_ALIVE << 16))) {
      *word &= ~(GD_THING_ALIVE << 16);
      reward = 1.0f;
    }
  }
  const bool late = time >= q.episodeTimeout;
  const bool pending = st.pending[l] != 0 || late;
  rewards[l] = reward;
  terminated[l] = 0;
  truncated[l] = late;
  st.pending[l] = pending;
  float *sb = st.signals + (size_t)l * GD_SIGNALS;
  sb[0] += reward;
  sb[26] += reward;
  sb[18] += reward;
  sb[17] = (float)time;
  sb[20] = pending ? 1.0f : 0.0f;
}

/* a seeded coordinate in 16.16, away from the edges of its room */
__device__ i64 gd_stepper_coordinate(i64 seed, i64 salt, double extent, i64 room) {
  const i64 margin = 20 * GD_FU;
  i64 v = (i64)((gd_stepper_uniform(seed, salt) * (extent - 48.0) + 24.0) * 65536.0);
  const i64 jitter = (i64)(gd_stepper_uniform(seed, salt + 10) * (double)(8 * GD_FU));
  i64 rem = gd_pymod(v, room);
  if (rem < margin) v += margin - rem + jitter;
  rem = gd_pymod(v, room);
  if (rem > room - margin) v -= rem - (room - margin) + jitter;
  return v;
}

/* One thread per lane whose mask byte is set. */
__global__ void gd_stepper_reset_kernel(const gd_stepper_state st, int n, const uint8_t *mask, const long long *seeds, float room,
                                        long long roomFixed, double width, double height) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= n || !mask[l]) return;
  const i64 seed = seeds[l];
  const i64 xf = gd_stepper_coordinate(seed, 1, width, roomFixed), yf = gd_stepper_coordinate(seed, 2, height, roomFixed);
  const i64 bam = (i64)(gd_stepper_uniform(seed, 3) * 4294967296.0) & GD_U32MASK;
  const float x = (float)xf / 65536.0f, y = (float)yf / 65536.0f;
  const i64 col = gd_clamp((i64)(x / room), 0, st.cols - 1), row = gd_clamp((i64)(y / room), 0, st.rows - 1);
  const i64 sector = row * st.cols + col;
  const float floor = st.floors[sector], ceiling = st.ceilings[sector];
  const float bamToRad = (float)(2.0 * 3.14159265358979323846 / 4294967296.0);
  int32_t *lane = st.lanes + (size_t)l * GD_LANE_WORDS;
  lane[GD_L_X] = __float_as_int(x);
  lane[GD_L_Y] = __float_as_int(y);
  lane[GD_L_ANGLE] = __float_as_int((float)bam * bamToRad);
  lane[GD_L_VIEW_Z] = __float_as_int(floor + GD_STEPPER_VIEW_HEIGHT);
  lane[GD_L_X_FIXED] = (int32_t)xf;
  lane[GD_L_Y_FIXED] = (int32_t)yf;
  lane[GD_L_ANGLE_BAM] = (int32_t)(uint32_t)bam;
  lane[GD_L_EPISODE_TIME] = 1;
  lane[GD_L_FLAGS] = 0;
  lane[GD_L_BOB_FIXED] = 0;
  if (st.k > 0)
    for (int k = 0; k < st.max_things; ++k) st.things[((size_t)l * st.max_things + k) * 4 + 3] |= GD_THING_ALIVE << 16;
  int32_t *p = st.players + (size_t)l * GD_PLAYER_WORDS;
  for (int k = 0; k < GD_PLAYER_WORDS; ++k) p[k] = 0;
  p[GD_P_X_FIXED] = (int32_t)xf;
  p[GD_P_Y_FIXED] = (int32_t)yf;
  p[GD_P_ANGLE_BAM] = (int32_t)(uint32_t)bam;
  p[GD_P_Z] = p[GD_P_FLOOR_Z] = p[GD_P_PREV_FLOOR_Z] = __float_as_int(floor);
  p[GD_P_VIEW_Z] = __float_as_int(floor + GD_STEPPER_VIEW_HEIGHT);
  p[GD_P_VIEW_HEIGHT] = __float_as_int(GD_STEPPER_VIEW_HEIGHT);
  p[GD_P_CEILING_Z] = __float_as_int(ceiling);
  p[GD_P_REACTION_TIME] = 7;                                   /* the input freeze after a spawn (src/gradoom/engine.py:81, 2407) */
  p[GD_P_EPISODE_TIME] = 1;
  float *sb = st.signals + (size_t)l * GD_SIGNALS;
  for (int k = 0; k < GD_SIGNALS; ++k) sb[k] = k == 1 ? 100.0f : 0.0f;
  st.pending[l] = 0;
}

static int gd_stepper_checks(const gd_renderer *r, const gd_stepper_state *st, int n) {
  if (!r || !st || !st->lanes || !st->players || !st->signals || !st->pending || !st->floors || !st->ceilings) return GD_ERR_NULL;
  if (n < 0 || st->k < 0 || st->max_things < st->k || st->cols <= 0 || st->rows <= 0) return GD_ERR_SIZE;
  if (st->k > 0 && !st->things) return GD_ERR_NULL;
  if (((uintptr_t)st->lanes | (uintptr_t)st->players | (uintptr_t)st->things) & 15) return GD_ERR_ALIGN;
  int current = -1;
  if (cudaGetDevice(&current) != cudaSuccess) return GD_ERR_CUDA;
  return current == r->device ? GD_OK : GD_ERR_DEVICE;
}

extern "C" int gd_stepper_step(const gd_renderer *r, const gd_stepper_state *st, int n, const uint8_t *buttons, int columns,
                               int tics, int episode_timeout, long long tick, float *rewards, uint8_t *terminated,
                               uint8_t *truncated, void *stream) {
  const int rc = gd_stepper_checks(r, st, n);
  if (rc != GD_OK || n == 0) return rc;
  if (!buttons || !rewards || !terminated || !truncated) return GD_ERR_NULL;
  if (tics < 0 || columns < 1) return GD_ERR_SIZE;
  GdMoveParams q;
  gd_move_params(r, q);
  q.players = st->players; q.buttons = nullptr; q.n = n; q.tics = tics; q.episodeTimeout = episode_timeout; q.lanes = st->lanes;
  const int lanesPerBlock = GDM_BLOCK / 32;
  gd_stepper_step_kernel<<<(n + lanesPerBlock - 1) / lanesPerBlock, GDM_BLOCK, 0, (cudaStream_t)stream>>>(
      q, *st, buttons, columns, tick, rewards, terminated, truncated);
  return cudaGetLastError() == cudaSuccess ? GD_OK : GD_ERR_CUDA;
}

extern "C" int gd_stepper_reset(const gd_renderer *r, const gd_stepper_state *st, int n, const uint8_t *mask, const long long *seeds,
                                double room, void *stream) {
  const int rc = gd_stepper_checks(r, st, n);
  if (rc != GD_OK || n == 0) return rc;
  if (!mask || !seeds) return GD_ERR_NULL;
  const long long roomFixed = (long long)(room * 65536.0);
  if (roomFixed <= 0) return GD_ERR_SIZE;
  gd_stepper_reset_kernel<<<(n + 63) / 64, 64, 0, (cudaStream_t)stream>>>(*st, n, mask, seeds, (float)room, roomFixed,
                                                                          st->cols * room, st->rows * room);
  return cudaGetLastError() == cudaSuccess ? GD_OK : GD_ERR_CUDA;
}

#endif

// fs_tune.cu -- the autotuner: for one context (grid, suspension, precision),
// the fastest combination of the FCM launch variants, timed on the device with
// the context's own beads. No reference counterpart.
//
// Knobs: beads staged per pass of the FP32 spread (32 or 64; the 16^3 tile is fixed by the
// binning), beads per interpolation CTA (4, 8 or 16 warps), on FP32 grids that have a transform
// of this library (fs_lines.cuh, fs_fft.cu) that one or cuFFT, and the shape of a warp's column
// block in the FP32 spread tile (x width 2, 4 or 8: 2 x 16 x 8, 4 x 16 x 4 or 8 x 16 x 2 points). A
// knob that this suspension's solves do not read keeps its value: the spread's two in FP64, the
// interpolation's where beads are split over warps. A captured step graph bakes the launch
// shapes, so tuning invalidates it.
#include "fs_internal.cuh"

extern "C" {

fs_status fs_set_tuning(fs_ctx *c, const int *choice_h) {
  if (!c || !choice_h) return FS_ERR_INVALID_ARG;
  const int ch = choice_h[0], wpb = choice_h[1], fft = choice_h[2], cx = choice_h[3];
  if ((ch != 32 && ch != 64) || (wpb != 4 && wpb != 8 && wpb != 16) || (fft != 0 && fft != 1) ||
      (cx != 2 && cx != 4 && cx != 8))
    return FS_ERR_INVALID_ARG;
  c->tune_spread_chunk = ch;
  c->tune_spread_cols = cx;
  c->tune_interp_wpb = wpb;
  c->tune_fft32 = fft;
  graph_invalidate(c);
  return FS_OK;
}

fs_status fs_autotune(fs_ctx *c, int reps, int *choice_h, float *best_ms_h) {
  if (!c || reps < 1) return FS_ERR_INVALID_ARG;
  if (!c->have_state) return FS_ERR_STATE;
  FS_TRY(fil_forces(c, c->p.initial_friction_steps + 1));  // Y, F, TAU of the current state
  cudaEvent_t e0, e1;
  FS_CUDA(cudaEventCreate(&e0));
  FS_CUDA(cudaEventCreate(&e1));
  const bool f32 = c->precision == FS_PREC_FP32, wpb_used = fcm_interp_wpb_used(c, c->np);
  float best = 1e30f;
  int bch = c->tune_spread_chunk, bwpb = c->tune_interp_wpb, bfft = c->tune_fft32, bcx = c->tune_spread_cols;
  const int ch_lo = f32 ? 32 : bch, ch_hi = f32 ? 64 : bch, wpb_lo = wpb_used ? 4 : bwpb, wpb_hi = wpb_used ? 16 : bwpb;
  const int cx_lo = f32 ? 2 : bcx, cx_hi = f32 ? 8 : bcx;
  const bool two = f32 && c->line_tw[FS_PREC_FP32][0];
  const int fft_lo = two ? 0 : bfft, fft_hi = two ? 1 : bfft;
  fs_status st = FS_OK;
  for (int ch = ch_lo; ch <= ch_hi && st == FS_OK; ch *= 2)
    for (int wpb = wpb_lo; wpb <= wpb_hi && st == FS_OK; wpb *= 2)
      for (int fft = fft_lo; fft <= fft_hi && st == FS_OK; ++fft)
        for (int cx = cx_lo; cx <= cx_hi && st == FS_OK; cx *= 2) {
        c->tune_spread_chunk = ch;
        c->tune_spread_cols = cx;
        c->tune_interp_wpb = wpb;
        c->tune_fft32 = fft;
        st = fcm_set_stream(c, c->stream);
        if (st == FS_OK) st = fcm_mobility(c, c->Y, c->F, c->TAU, c->V, c->W, c->np);  // warm-up
        if (st != FS_OK) break;
        if (cudaEventRecord(e0, c->stream) != cudaSuccess) st = FS_ERR_CUDA;
        for (int r = 0; r < reps && st == FS_OK; ++r) st = fcm_mobility(c, c->Y, c->F, c->TAU, c->V, c->W, c->np);
        float ms = 0.f;
        if (st == FS_OK && (cudaEventRecord(e1, c->stream) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess ||
                            cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess))
          st = FS_ERR_CUDA;
        ms /= reps;
        if (st == FS_OK && ms < best) {
          best = ms;
          bch = ch;
          bwpb = wpb;
          bfft = fft;
          bcx = cx;
        }
      }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  c->tune_spread_chunk = bch;
  c->tune_interp_wpb = bwpb;
  c->tune_fft32 = bfft;
  c->tune_spread_cols = bcx;
  graph_invalidate(c);
  FS_TRY(st);
  FS_TRY(fcm_set_stream(c, c->stream));
  if (choice_h) {
    choice_h[0] = bch;
    choice_h[1] = bwpb;
    choice_h[2] = bfft;
    choice_h[3] = bcx;
  }
  if (best_ms_h) *best_ms_h = best;
  return FS_OK;
}

}  // extern "C"

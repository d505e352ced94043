// collide_lowp.cu -- the storage types' entry points by number, and the
// autotuner of the FP32-collision kernels (collide_lowp.cuh).
#include "lbmpsm_internal.cuh"

namespace lbmpsm {

cudaError_t prepare_collide_lowp(const Geom& g, int storage, int sm_count, int stages,
                                 PipeConfig* cfg) {
  if (storage == 1) return prepare_collide_f32(g, sm_count, stages, cfg);
  if (storage == 3) return prepare_collide_bf16(g, sm_count, stages, cfg);
  return prepare_collide_f16(g, sm_count, stages, cfg);
}

cudaError_t prepare_collide_multi(MultiCollide& mc, MultiMember* mem, int storage, int sm_count) {
  if (storage == 0) {
    // FP64: the members' own blocks in turn
    int total = 0;
    for (int m = 0; m < mc.nm; ++m) {
      const long long blocks = collide_f64_blocks(mem[m].p.g);
      if (total + blocks >= (1ll << 31)) return cudaErrorInvalidValue;
      mc.first[m] = total;
      total += (int)blocks;
    }
    mc.first[mc.nm] = total;
    return cudaSuccess;
  }
  if (storage == 1) return prepare_multi_f32(mc, mem, sm_count);
  if (storage == 3) return prepare_multi_bf16(mc, mem, sm_count);
  return prepare_multi_f16(mc, mem, sm_count);
}

cudaError_t launch_collide_multi(const MultiCollide& mc, int storage, int odd, cudaStream_t st) {
  if (storage == 0) return launch_collide_f64_multi(mc, odd, st);
  if (storage == 1) return launch_multi_f32(mc, odd, st);
  if (storage == 3) return launch_multi_bf16(mc, odd, st);
  return launch_multi_f16(mc, odd, st);
}

// The project's autotuner for the FP32/FP16 collide: every candidate launch
// shape -- the row pipeline with 3, 2, 4 or 5 stages, each at the blocks per
// multiprocessor its shared memory and registers allow -- runs even/odd step
// pairs on p.f (a scratch copy of the populations), timed with CUDA events on
// the stream; the fastest is kept.  The candidates are one template
// (only the stage count and the launch bounds differ), so they round alike
// and the choice changes speed only, never results.  The direct kernel rounds
// |u_s|^2 in another order and is not a candidate.
//
// A pair untimed, then one timed, or three where a pair is shorter than 200 us
// or so (a rate of 3 TB/s assumed).
static const int cand[LBMPSM_TUNE_CANDIDATES] = {3, 2, 4, 5};

int tune_shapes(const Geom& g, int storage, int sm_count, PipeConfig (&shape)[LBMPSM_TUNE_CANDIDATES]) {
  int n = 0;
  for (int k = 0; k < LBMPSM_TUNE_CANDIDATES; ++k) {
    PipeConfig& c = shape[k];
    // (a long row has one shape whatever the stages asked for; where tiles hold
    // several rows, one row a tile is the slower shape and not timed)
    if (prepare_collide_lowp(g, storage, sm_count, cand[k], &c) != cudaSuccess || c.stages != cand[k] ||
        c.k < shape[0].k)
      c = PipeConfig{};
    if (c.grid > 0) ++n;
  }
  cudaGetLastError();
  return n;
}

cudaError_t tune_collide_lowp(CollideParams p, int storage, cudaStream_t st,
                              const PipeConfig (&shape)[LBMPSM_TUNE_CANDIDATES], PipeConfig* best,
                              float* ms_out) {
  const double pair_bytes = 4.0 * p.g.Q * (storage == 1 ? 4 : 2) * (double)p.g.N;
  const int reps = pair_bytes < 3e12 * 200e-6 ? 3 : 1;
  cudaEvent_t e0, e1;
  cudaError_t e = cudaEventCreate(&e0);
  if (e != cudaSuccess) return e;
  if ((e = cudaEventCreate(&e1)) != cudaSuccess) {
    cudaEventDestroy(e0);
    return e;
  }
  float best_ms = 0.0f;
  bool have = false;
  for (int k = 0; k < LBMPSM_TUNE_CANDIDATES; ++k) {
    ms_out[k] = -1.0f;
    const PipeConfig& c = shape[k];
    if (c.grid == 0) continue;  // this shape does not fit the lattice's rows
    p.pipe = c;
    auto pair = [&]() {
      for (int odd = 0; odd < 2; ++odd)
        if (storage == 1)
          launch_collide_f32(p, odd, st);
        else if (storage == 3)
          launch_collide_bf16(p, odd, st);
        else
          launch_collide_f16(p, odd, st);
    };
    pair();
    cudaEventRecord(e0, st);
    for (int r = 0; r < reps; ++r) pair();
    cudaEventRecord(e1, st);
    if ((e = cudaEventSynchronize(e1)) != cudaSuccess) break;
    if ((e = cudaGetLastError()) != cudaSuccess) break;
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, e0, e1);
    ms_out[k] = ms / (float)reps;
    if (!have || ms_out[k] < best_ms) {
      best_ms = ms_out[k];
      *best = c;
      have = true;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return e;
}

}  // namespace lbmpsm

// kernels.h -- host-side launchers of the device kernels.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include <vector>

#include "cupic_internal.cuh"

namespace cupic {

// Raises a kernel's dynamic shared memory limit on the current device to at
// least `bytes`.  The attribute is per device, so the largest size set so
// far is kept per (kernel, device), under a lock; it only grows, so
// contexts of different sizes coexist.
cudaError_t raise_dyn_smem(const void *kernel, size_t bytes);

cudaError_t launch_init_particles(const SimArgs &a, cudaStream_t st);
cudaError_t launch_deposit(const SimArgs &a, cudaStream_t st);
cudaError_t launch_zero_next_rho(const SimArgs &a, cudaStream_t st);
cudaError_t launch_leapfrog_start(const SimArgs &a, cudaStream_t st);
cudaError_t launch_push_deposit(const SimArgs &a, cudaStream_t st);
cudaError_t launch_arrive(const SimArgs &a, cudaStream_t st);
cudaError_t launch_inject_draw(const SimArgs &a, cudaStream_t st);
// the same in two parts where a step draws few particles: all that needs no
// field, and the field's kick
bool few_draws(const SimArgs &a);
cudaError_t launch_draw_few(const SimArgs &a, cudaStream_t st);
cudaError_t launch_inject_kick(const SimArgs &a, cudaStream_t st);
cudaError_t launch_inject_append(const SimArgs &a, cudaStream_t st);
cudaError_t launch_finalize(const SimArgs &a, cudaStream_t st);
// room check, arrivals, append and bookkeeping in one launch
bool tail_applies(const SimArgs &a);
cudaError_t tail_set_smem(const SimArgs &a);
cudaError_t launch_tail(const SimArgs &a, int num_sms, cudaStream_t st);
// room check between the push and the arrivals (sets ctl->halt), and the
// move of a species' rows into a larger layout
cudaError_t launch_room(const SimArgs &a, cudaStream_t st);
cudaError_t launch_move_rows(const float4 *old, const int64_t *oseg, float4 *parts, const int64_t *nseg,
                             const int32_t *keep, int ncy, cudaStream_t st);
size_t push_smem_bytes(int nnx, int pb = 256);  // pb: threads per block (256 single context)
cudaError_t push_set_smem(size_t bytes);
// set-up on the context's stream
cudaError_t launch_uniform_layout(const SpeciesDev &S, int ncy, int capj, cudaStream_t st);
cudaError_t launch_set_time(Ctl *ctl, int64_t step, double t, double tin_e, double tin_i, cudaStream_t st);
cudaError_t launch_linear_phi(const SimArgs &a, double phi_p, double *phi64, cudaStream_t st);

int load_blocks(int64_t n, int num_sms);
cudaError_t launch_load_hist(const SimArgs &a, const double *in, int64_t n, int nb, float4 *tmp,
                             int32_t *H, unsigned *bad, cudaStream_t st);
cudaError_t launch_load_scan(int32_t *H, int nb, int ncy, int32_t *cnt, cudaStream_t st);
cudaError_t launch_load_scatter(const SimArgs &a, int sp, const float4 *tmp, int64_t n, int nb,
                                const int32_t *H, cudaStream_t st);
cudaError_t launch_pack_rows(const SimArgs &a, int sp, const int64_t *off, float4 *out32,
                             double *out64, cudaStream_t st);

size_t jacobi_smem_bytes(int rows_per_cta, int depth, int pitch);
int jacobi_strip_rows(int nnx, int urows);
cudaError_t jacobi_set_smem(size_t bytes);
cudaError_t jacobi_max_ctas(size_t smem, int *per_sm);
cudaError_t launch_jacobi(const SimArgs &a, const JacobiArgs &J, cudaStream_t st);

// the register-tile solve (tile.cuh, tile.cu)
constexpr int kTileWarps = 16;  // most warps of a CTA, of 128 registers a thread
constexpr int kTileRows = 8;    // most rows of a strip
constexpr int kTileDepth = 16;  // deepest halo
// Most CTAs of a ring layout that run as one cluster (the most a cluster may
// have).  An exchange takes them 1000 cycles instead of 3000; 64x256 at depth 8
// takes 0.189 us a sweep on 16 CTAs, 0.299 on 17 and 0.286 on 24.
constexpr int kTileCluster = 16;
// a solve of a fixed number of sweeps, one that may stop on its tolerance
// (and keeps snapshots), the precision form (and keeps its FP64 potential)
enum TileForm { kTileFixed, kTileEarly, kTileRefine };
struct TilePlan {
  TileForm form;
  int R;                   // rows of a strip
  int mode;                // 0 halo, 1 ring, 2 ragged ring
  int nbx, nby, G, K;      // blocks in x and y, their product, halo depth
  int B;                   // most rows a block owns
  int near;                // the CTAs are one cluster and trade through shared memory
  int nl, segs, warps, ip; // lanes of a strip, strips per warp, warps, exchange row pitch
  int trows, tpairs, ppairs;  // rows of the exchange image, entries of the tables of words in and out
  size_t smem, words;      // dynamic shared memory; exchange words
  double cost;             // estimated SM cycles per sweep
};
bool tile_plan(int nnx, int nny, int nbx, int nby, int K, int R, TileForm form, TilePlan *out);
std::vector<TilePlan> tile_plans(int nnx, int nny, int num_sms, TileForm form, size_t max_smem);
void tile_args(const TilePlan &t, JacobiArgs *J);
cudaError_t tile_max_ctas(const TilePlan &t, int num_sms, int *ctas);
cudaError_t launch_tile(const SimArgs &a, const JacobiArgs &J, const TilePlan &t, cudaStream_t st);
// the field of the stored potential, and the report of a solve of no sweeps
cudaError_t launch_field(const SimArgs &a, int do_field, int write_stats, cudaStream_t st);

// many contexts in one launch (batch.cu): SimArgs / JacobiArgs arrays in
// device memory, work lists of {instance, row}
cudaError_t jacobi_batch_set_smem(size_t bytes);
cudaError_t jacobi_batch_max_ctas(size_t smem, int *per_sm);
cudaError_t launch_jacobi_batch(const SimArgs *inst, const JacobiArgs *jargs, const JGroup *groups,
                                int ngroups, const int *list, int nctas, size_t smem, cudaStream_t st);
cudaError_t launch_push_deposit_batch(const SimArgs *inst, const int2 *row_work, int n, int max_nnx,
                                      int threads, cudaStream_t st);
cudaError_t launch_arrive_batch(const SimArgs *inst, const int2 *row_work, int n, cudaStream_t st);
cudaError_t launch_inject_draw_batch(const SimArgs *inst, int n, int max_inj_cap, cudaStream_t st);
cudaError_t launch_inject_append_batch(const SimArgs *inst, int n, int max_ncy, cudaStream_t st);
cudaError_t launch_room_batch(const SimArgs *inst, int n, int max_ncy, cudaStream_t st);
cudaError_t launch_finalize_batch(const SimArgs *inst, int n, cudaStream_t st);

// fault-detection self-test (jacobi.cu)
cudaError_t launch_wait_probe(const SimArgs &a, cudaStream_t st);

// precision form of the solve (refine.cu)
// gated: the kernel returns at once when the device-side stop test has passed
cudaError_t launch_r64_source(const SimArgs &a, double *b64, cudaStream_t st);
cudaError_t launch_r64_residual(const SimArgs &a, const double *phi64, const double *b64, float *rr,
                                unsigned long long *maxr, cudaStream_t st, int gated = 0);
cudaError_t launch_r64_phi32(const SimArgs &a, const double *phi64, cudaStream_t st);
cudaError_t launch_r64_update(const SimArgs &a, double *phi64, const float *dl, cudaStream_t st,
                              int gated = 0);
cudaError_t launch_r64_decide(const SimArgs &a, const unsigned long long *maxr, int sweeps, int mn,
                              int mx, double tol, int write_stats, cudaStream_t st);
cudaError_t launch_r64_field(const SimArgs &a, const double *phi64, cudaStream_t st);

}  // namespace cupic

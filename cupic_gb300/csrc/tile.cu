// tile.cu -- layouts and launch of the register-tile solve (tile.cuh), and
// the field of a potential that no solve has just swept.
#include <algorithm>

#include "cupic_internal.cuh"
#include "kernels.h"

namespace cupic {

const void *tile_kernel_halo(int r);
const void *tile_kernel_ring(int r);
const void *tile_kernel_ragged(int r);
const void *tile_kernel_halo_refine(int r);
const void *tile_kernel_ring_refine(int r);
const void *tile_kernel_ragged_refine(int r);

namespace {

const void *tile_kernel(const TilePlan &t) {
  if (t.form == kTileRefine)
    return t.mode == 0   ? tile_kernel_halo_refine(t.R)
           : t.mode == 1 ? tile_kernel_ring_refine(t.R)
                         : tile_kernel_ragged_refine(t.R);
  return t.mode == 0 ? tile_kernel_halo(t.R) : t.mode == 1 ? tile_kernel_ring(t.R) : tile_kernel_ragged(t.R);
}

// E = -grad phi (mesh.cu:413-468) of the stored potential, operation for
// operation the field of the solve; a solve of no sweeps reports that
__global__ void k_field(SimArgs a, int do_field, int write_stats) {
  if (halted(a.ctl)) return;
  const int j = blockIdx.y, nnx = a.nnx, nny = a.nny;
  const float *const q = a.phi + (size_t)j * nnx;
  if (do_field)
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nnx; i += gridDim.x * blockDim.x) {
      float2 e = make_float2(0.0f, 0.0f);
      if (j == 0) {
        e.y = __fdiv_rn(__fsub_rn(q[i], q[nnx + i]), a.ds);
      } else if (j == nny - 1) {
        e.y = __fdiv_rn(__fsub_rn(q[i - nnx], q[i]), a.ds);
      } else {
        const bool seam = i == 0 || i == nnx - 1;
        e.x = __fdiv_rn(__fsub_rn(seam ? q[nnx - 2] : q[i - 1], seam ? q[1] : q[i + 1]), a.two_ds);
        e.y = __fdiv_rn(__fsub_rn(q[i - nnx], q[i + nnx]), a.two_ds);
      }
      a.E[(size_t)j * nnx + i] = e;
    }
  if (write_stats && j == 0 && blockIdx.x == 0 && threadIdx.x == 0) {
    a.ctl->sweeps = 0;
    a.ctl->residual = __int_as_float(0x7f800000);
  }
}

}  // namespace

// The layout of nbx x nby blocks with halo depth K and strips of R rows (0:
// the fewest that need at most kTileWarps warps); false if there is none.
bool tile_plan(int nnx, int nny, int nbx, int nby, int K, int R, TileForm form, TilePlan *out) {
  const int W = nnx - 1, M = nny - 2, W4 = (W + 3) / 4;
  TilePlan t{};
  t.form = form;
  if ((long long)M * (nby + 1) >= 1ll << 31) return false;
  if (nbx < 1 || nby < 1 || K < 1 || nby > M || nbx > W4 || K > kTileDepth) return false;
  if (nby > 1 && K > M / nby) return false;  // a block trades K of its own rows
  if (nbx == 1) {
    if (W4 > 32) return false;
    t.mode = W % 4 == 0 ? 1 : 2;
    t.nl = W4;
    t.segs = 32 / W4;
  } else {
    t.mode = 0;
    if (K % 4 != 0) return false;
    int most = 0;
    for (int b = 0; b < nbx; ++b) {
      const int x0 = 4 * (b * W4 / nbx), x1 = std::min(W, 4 * ((b + 1) * W4 / nbx));
      if (x1 - x0 < K) return false;
      most = std::max(most, (x1 - x0 + 2 * K + 3) / 4);
    }
    if (most > 32) return false;
    t.nl = most;
    t.segs = 1;
  }
  t.B = (M + nby - 1) / nby;
  int rows = 0;  // most rows updated by one block
  for (int b = 0; b < nby; ++b) {
    const int r0 = 1 + (int)((long long)b * M / nby), r1 = 1 + (int)((long long)(b + 1) * M / nby);
    const int lo = nby > 1 ? std::max(1, r0 - (K - 1)) : 1, hi = nby > 1 ? std::min(nny - 2, r1 + K - 2) : nny - 2;
    rows = std::max(rows, hi - lo + 1);
    if (b == 2 && nby > 8 && M % nby == 0) break;  // all inner blocks alike
  }
  if (R == 0) R = (rows + kTileWarps * t.segs - 1) / (kTileWarps * t.segs);
  if (R < 1 || R > kTileRows) return false;
  t.R = R;
  t.warps = (rows + R * t.segs - 1) / (R * t.segs);
  if (t.warps > kTileWarps) return false;
  t.nbx = nbx;
  t.nby = nby;
  t.G = nbx * nby;
  t.K = K;
  t.ip = nbx == 1 ? 4 * W4 : 4 * W4 + 36;
  const size_t thr = 32 * (size_t)t.warps;
  t.trows = rows;
  t.near = nbx == 1 && nby > 1 && nby <= kTileCluster;
  if (t.near) {
    t.tpairs = 2 * K * 4 * t.nl;  // the rows that arrive, two exchanges in turn
    if (form == kTileEarly) t.tpairs += 2 * t.G * 32 / 2;  // and the maxima of checked blocks
  } else if (t.G > 1) {
    const int wide = nbx > 1 ? 4 * ((W4 + nbx - 1) / nbx) + 2 * K : W;
    const int own = nbx > 1 ? 4 * ((W4 + nbx - 1) / nbx) : W, side = nbx > 1 ? t.B * K : 0;
    t.tpairs = ((nby > 1 ? 2 : 0) * K * ((wide + 1) / 2) + side + 1) / 2 * 2;
    t.ppairs = (nby > 1 ? 2 : 0) * K * ((own + 1) / 2) + side;
    if (nbx > 1 && nby > 1) t.ppairs += 2 * (W % 2 ? K : K / 2) * 2 * K;  // periodic images
    t.ppairs = (t.ppairs + 1) / 2 * 2;
  }
  // strip rows in two parities, edge rows, the tile's image and the tables of
  // exchange words (even numbers of entries: what follows is 16-byte aligned),
  // two snapshots of the strips or the charges' image in their place, or the
  // FP64 potential
  t.smem = (4 * thr * 4 + 4 * 2 * 128 + (size_t)(rows + 2) * 4 * t.nl + (rows + 3) / 4 * 4) * sizeof(float) +
           (size_t)(rows + 1) / 2 * 16 +
           (size_t)(t.tpairs + t.ppairs) * sizeof(uint2) + (form == kTileEarly ? 2 * R * thr * sizeof(float4) : 0) +
           (form == kTileFixed ? (size_t)rows * 4 * t.nl * sizeof(long long) : 0) +
           (form == kTileRefine ? ((size_t)(rows + 2) * 4 * t.nl + 8) * sizeof(double) : 0);
  t.words = t.G == 1 || t.near ? 0
                     : (size_t)2 * nby * 2 * K * t.ip + (nbx > 1 ? (size_t)2 * nny * nbx * 2 * K : 0);
  if (t.words >= 1ull << 31) return false;
  // Estimated SM cycles per sweep, fitted to the times of 2900 layouts of 12
  // meshes (33x129 .. 513x2049, 200 sweeps, at 2 GHz; the cheapest estimate is
  // within 8% of the fastest layout timed on all but two of them): the
  // barrier and the two rows that every warp takes and sends through shared
  // memory, 16 issue slots a row for each warp of a scheduler (more above 5
  // rows, where registers run short, and for the selects of a ragged ring),
  // the stop test, and the share of an exchange: 640 cycles in a cluster,
  // 1160 by way of L2, more for each warp that issues it and for each pair of
  // words a thread waits for.
  // Measured slower, 512x2048, 200 sweeps: strips of 12 rows on 8 warps of 255
  // registers (half the rows through shared memory) 188 us against 170; two
  // CTAs to an SM, one sweeping while the other waits, 239 against 175.
  const double per = (t.warps + 3) / 4 * R;  // rows of a scheduler
  t.cost = 55.0 * R + 5.0 * t.warps + per * (16.0 + 6.5 * std::max(0, R - 5) + (t.mode == 2 ? 30.0 : 0.0));
  if (form == kTileEarly) t.cost += 127.0 + 3.0 * t.warps + (t.near ? 500.0 / K : 0.0);
  if (t.near)
    t.cost += (640.0 + 52.0 * t.warps) / K;
  else if (t.G > 1)
    t.cost += (1160.0 + 130.0 * t.warps + 240.0 * t.tpairs / thr) / K;
  // the precision form's FP64 work: about 9 operations a node at 2 a clock,
  // once a correction (32 sweeps)
  if (form == kTileRefine) t.cost += 4.5 * 4 * 32 * R * t.warps / 32;
  *out = t;
  return true;
}

// The layouts worth timing, cheapest estimate first.
std::vector<TilePlan> tile_plans(int nnx, int nny, int num_sms, TileForm form, size_t max_smem) {
  const int W = nnx - 1, M = nny - 2, W4 = (W + 3) / 4;
  std::vector<TilePlan> out;
  const int depths[] = {1, 2, 4, 6, 8, 12, 16};
  const int grids[] = {1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64, 96, 128, num_sms};
  for (int nbx = 1; nbx <= std::min(W4, 64); ++nbx)
    for (int g : grids) {
      const int nby = g / nbx;
      if (nby < 1 || nby > M || (nbx > 1 && g < num_sms && g % nbx)) continue;
      for (int K : depths) {
        if (nbx * nby == 1 && K > 1) continue;
        TilePlan t;
        if (!tile_plan(nnx, nny, nbx, nby, K, 0, form, &t)) continue;
        const int R0 = t.R;
        for (int R = R0; R <= kTileRows; ++R)
          if (tile_plan(nnx, nny, nbx, nby, K, R, form, &t) && t.smem <= max_smem) out.push_back(t);
      }
    }
  std::sort(out.begin(), out.end(), [](const TilePlan &a, const TilePlan &b) { return a.cost < b.cost; });
  return out;
}

void tile_args(const TilePlan &t, JacobiArgs *J) {
  J->G = t.G;
  J->rows_per_cta = t.B;
  J->depth = t.K;
  J->tile = t.R;
  J->mode = t.mode;
  J->nbx = t.nbx;
  J->nby = t.nby;
  J->nl = t.nl;
  J->segs = t.segs;
  J->warps = t.warps;
  J->ip = t.ip;
  J->near = t.near;
  J->trows = t.trows;
  J->tpairs = t.tpairs;
  J->ppairs = t.ppairs;
  J->pwords = (uint32_t)(t.words / 2);
}

// the launch of a layout: a cluster, or a cooperative grid where CTAs wait for
// one another without one
static void tile_launch(const TilePlan &t, cudaLaunchConfig_t *cfg, cudaLaunchAttribute *attr) {
  cfg->gridDim = dim3(t.G);
  cfg->blockDim = dim3(32 * t.warps);
  cfg->dynamicSmemBytes = t.smem;
  if (t.near) {
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = t.G;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
  } else {
    attr->id = cudaLaunchAttributeCooperative;
    attr->val.cooperative = 1;
  }
  cfg->attrs = attr;
  cfg->numAttrs = t.G > 1 ? 1 : 0;
}

// CTAs of this layout that the device holds at once
cudaError_t tile_max_ctas(const TilePlan &t, int num_sms, int *ctas) {
  const void *fn = tile_kernel(t);
  cudaError_t e = raise_dyn_smem(fn, t.smem);
  int n = 0;
  if (e == cudaSuccess && t.near) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    tile_launch(t, &cfg, attr);
    if (t.G > 8) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, fn, &cfg);
    *ctas = n * t.G;
  } else {
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, 32 * t.warps, t.smem);
    *ctas = n * num_sms;
  }
  return e;
}

cudaError_t launch_tile(const SimArgs &a, const JacobiArgs &J, const TilePlan &t, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  tile_launch(t, &cfg, attr);
  cfg.stream = st;
  SimArgs sa = a;
  JacobiArgs ja = J;
  void *args[] = {&sa, &ja};
  return cudaLaunchKernelExC(&cfg, tile_kernel(t), args);
}

cudaError_t launch_field(const SimArgs &a, int do_field, int write_stats, cudaStream_t st) {
  k_field<<<dim3((a.nnx + 255) / 256, do_field ? a.nny : 1), 256, 0, st>>>(a, do_field, write_stats);
  return cudaGetLastError();
}

}  // namespace cupic

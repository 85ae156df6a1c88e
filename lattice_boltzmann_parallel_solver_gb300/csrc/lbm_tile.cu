// lbm_tile.cu -- the tile kernels of one lattice, how a lattice is cut, and
// their launches.
#include "lbm_tile.h"

#include "lbm_tile.cuh"

namespace lbm {

struct TileArgs {
  KParams P;
  int tiles_x, tiles_y, ksteps;
};

// columns a region may have: the narrow form for small lattices, the wide one
// for the others (a row of either is a whole number of warps or half a warp)
template <int STORE>
constexpr int tile_columns(bool wide) {
  return (STORE == LBM_STORE_F64 || STORE == LBM_STORE_FX64 ? 16 : 32) * (wide ? 2 : 1);
}

// threads per block at most: what the body's registers allow without spills
// (128 of them in the narrow form, 80 and 64 in the wide one)
template <int STORE>
constexpr int tile_threads(bool wide) {
  return !wide ? 512 : (STORE == LBM_STORE_F64 || STORE == LBM_STORE_FX64 ? 768 : 1024);
}

template <int STORE, bool SHIFT, int WC, bool HAS_BC, bool HAS_PRESSURE>
__global__ void __launch_bounds__(tile_threads<STORE>(WC == tile_columns<STORE>(true)), 1)
    tile_kernel(const __grid_constant__ TileArgs A) {
  extern __shared__ __align__(16) unsigned char tile_shared[];
  const int bx = (int)blockIdx.x % A.tiles_x, by = (int)blockIdx.x / A.tiles_x;
  // nearly equal tiles; columns in whole units so that a pair starts at an even x
  constexpr int N = tile_npt<STORE>();
  const int units = (A.P.g.nx + N - 1) / N;
  TileRect t;
  t.x0 = (int)((int64_t)bx * units / A.tiles_x) * N;
  t.tx = min((int)((int64_t)(bx + 1) * units / A.tiles_x) * N, A.P.g.nx) - t.x0;
  t.y0 = (int)((int64_t)by * A.P.g.ny / A.tiles_y);
  t.ty = (int)((int64_t)(by + 1) * A.P.g.ny / A.tiles_y) - t.y0;
  tile_body<STORE, SHIFT, WC, HAS_BC, HAS_PRESSURE>(A.P, A.P.pop_in, A.P.pop_out, A.P.aux_in, A.P.aux_out, t, A.ksteps,
                                                A.P.seed, tile_shared);
}

using TileKernel = void (*)(const TileArgs);

template <int STORE, int WC, bool SHIFT>
static TileKernel pick(const KParams& P) {
  if (P.g.pressure) return tile_kernel<STORE, SHIFT, WC, true, true>;
  return P.g.bcmask != nullptr ? tile_kernel<STORE, SHIFT, WC, true, false>
                               : tile_kernel<STORE, SHIFT, WC, false, false>;
}
template <int STORE, bool SHIFT = false>
static TileKernel pick(const KParams& P, bool wide) {
  return wide ? pick<STORE, tile_columns<STORE>(true), SHIFT>(P) : pick<STORE, tile_columns<STORE>(false), SHIFT>(P);
}

static TileKernel kernel_of(int storage, const KParams& P, bool wide) {
  switch (storage) {
    case LBM_STORE_F64: return pick<LBM_STORE_F64>(P, wide);
    case LBM_STORE_F32: return pick<LBM_STORE_F32>(P, wide);
    case LBM_STORE_F16S: return pick<LBM_STORE_F16S>(P, wide);
    case LBM_STORE_BF16S: return pick<LBM_STORE_BF16S>(P, wide);
    case LBM_STORE_FX64: return pick<LBM_STORE_FX64>(P, wide);
    case LBM_STORE_F16R: return pick<LBM_STORE_F16S, true>(P, wide);
    case LBM_STORE_BF16R: return pick<LBM_STORE_BF16S, true>(P, wide);
    default: return nullptr;
  }
}

template <int STORE>
static size_t smem_of(int h, bool wide) {
  return wide ? TileShared<STORE, tile_columns<STORE>(true)>::bytes(h)
              : TileShared<STORE, tile_columns<STORE>(false)>::bytes(h);
}
static size_t smem_of(int storage, int h, bool wide) {
  switch (storage) {
    case LBM_STORE_F64: return smem_of<LBM_STORE_F64>(h, wide);
    case LBM_STORE_F32: return smem_of<LBM_STORE_F32>(h, wide);
    case LBM_STORE_FX64: return smem_of<LBM_STORE_FX64>(h, wide);
    default: return smem_of<LBM_STORE_F16S>(h, wide);
  }
}

// Time of a launch in microseconds, fitted to 1700 measured (storage, lattice,
// cut) points from 32x24 to 800x640 nodes within 2 to 6 percent rms without
// boundary nodes and 4 to 13 with them:
//   fixed + (trips of a block's threads over its region, summed over the steps)
//         * trip + (warps of such trips) * warp
// and of a one-step launch, one_floor + nodes / one_rate, on the same lattices.
struct TileCost {
  float fixed, trip, warp, one_floor, one_rate;  // rate: nodes per microsecond
};
static TileCost tile_cost(int storage, bool bc) {
  switch (storage) {
    case LBM_STORE_FX64:
      return bc ? TileCost{2.13f, 0.90f, 0.084f, 3.4f, 46e3f} : TileCost{1.69f, 0.61f, 0.080f, 2.2f, 62e3f};
    case LBM_STORE_F64:
      return bc ? TileCost{1.05f, 1.36f, 0.579f, 7.2f, 8.0e3f} : TileCost{2.15f, 1.01f, 0.502f, 5.9f, 8.5e3f};
    case LBM_STORE_F32:
      return bc ? TileCost{3.25f, 0.36f, 0.030f, 4.6f, 130e3f} : TileCost{2.32f, 0.28f, 0.019f, 2.5f, 92e3f};
    default:
      return bc ? TileCost{3.55f, 0.80f, 0.059f, 5.0f, 190e3f} : TileCost{2.25f, 0.49f, 0.046f, 2.4f, 150e3f};
  }
}

// Under the pressure rewrite the 64-bit tile bodies cost more than that (every row of
// a tile at column 1 or nx-2 runs it): whether the cut that these numbers choose is
// still faster than a one-step launch, by numbers fitted to the lattices that were
// tiled without the question (36 in fx64 within 4 percent rms, 31 in f64 within 10).
// f64's one-step launch, bound by its pipe, counts in whole blocks per SM.  us per
// step, tiled / one step: fx64 515x230 14.9 / 7.6, 420x180 10.5 / 7.6, 251x132 6.5 / 5.7,
// 119x168 5.5 / 5.4, 200x60 4.6 / 5.2; f64 251x132 13.4 / 10.8, 267x112 12.4 / 13.8.
static bool pressure_tile_pays(int storage, const KParams& P, int sms, int ksteps, float trips, float warps) {
  const int64_t nodes = (int64_t)P.g.nx * P.g.ny;
  if (storage == LBM_STORE_FX64)
    return (3.1f + 2.2f * trips + 0.23f * warps) / (float)ksteps < 4.9f + (float)nodes / 39.5e3f;
  const int64_t blocks = (int64_t)((P.g.nx + 255) / 256) * P.g.ny;  // of 128 threads x 2 nodes
  return (3.0f + 1.36f * trips + 0.87f * warps) / (float)ksteps < 5.8f + 4.8f * (float)((blocks + sms - 1) / sms);
}

// The cut with the least time per step: odd numbers of steps, and at most one
// tile per SM (a second wave never won in a sweep up to 1024^2: by then the
// one-step launches are bound by their arithmetic, not by their latency, and
// the halo's share of it decides).
TilePlan tile_plan(int storage, const KParams& P) {
  TilePlan best;
  int dev = 0, sms = 0, smem_max = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  best.smem_limit = smem_max;
  const TileCost c = tile_cost(storage, P.g.bcmask != nullptr || P.g.pressure);
  const int nx = P.g.nx, ny = P.g.ny;
  const bool eight = storage == LBM_STORE_F64 || storage == LBM_STORE_FX64;
  const int npt = eight || storage == LBM_STORE_F32 ? 1 : 2;
  const int units = (nx + npt - 1) / npt;
  float best_time = c.one_floor + (float)((double)nx * ny / c.one_rate);
  float best_trips = 0.0f, best_warps = 0.0f;
  for (int k = 3; k <= 7; k += 2) {
    const int margin = 2 * tile_margin_x(k, P.g.pressure != 0);
    for (int tx = 1; tx <= std::min(units, sms); ++tx) {
      const int cols = (units + tx - 1) / tx * npt;
      if (tx > 1 && cols < 4) break;
      const int w = cols + margin;
      const bool wide = w > (eight ? 16 : 32);
      const int columns = (eight ? 16 : 32) * (wide ? 2 : 1);
      if (w > columns) continue;
      // the outlet memory of a region's row is one column's
      if (P.g.outlet && w > nx) continue;
      const int ty = std::min(sms / tx, ny);
      const int h = (ny + ty - 1) / ty + 2 * (k - 1);
      const size_t smem = smem_of(storage, h, wide);
      if (smem > (size_t)smem_max) continue;
      // whole rows, whole warps
      const int row = columns / npt, most = !wide ? 512 : (eight ? 768 : 1024);
      const int threads = (std::min(most, h * row) + 63) / 64 * 64;
      float time = c.fixed, trips = 0.0f, warps = 0.0f;
      for (int s = 0; s < k; ++s) {
        const int lanes = (h - 2 * s) * row;
        const float t = (float)((lanes + threads - 1) / threads), w32 = (float)((lanes + 31) / 32);
        time += c.trip * t + c.warp * w32;
        trips += t;
        warps += w32;
      }
      if (time / (float)k < best_time) {
        best_time = time / (float)k;
        best_trips = trips;
        best_warps = warps;
        best.ksteps = k;
        best.tiles_x = tx;
        best.tiles_y = ty;
        best.threads = threads;
        best.wide = wide;
        best.smem = smem;
      }
    }
  }
  if (best.ksteps > 1 && P.g.pressure && eight &&
      !pressure_tile_pays(storage, P, std::max(1, sms), best.ksteps, best_trips, best_warps))
    best.ksteps = 1;
  return best;
}

int tile_prepare(int storage, const TilePlan& plan, const KParams& P) {
  const TileKernel k = kernel_of(storage, P, plan.wide);
  if (k == nullptr) return set_error(LBM_ERR_ARG, "unknown storage type");
  // The limit belongs to the kernel, not to this run: the same value whatever the
  // plan, so that no other thread's run finds it lowered between its launches.
  const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, plan.smem_limit);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return set_error(LBM_ERR_CUDA, cudaGetErrorString(e));
  }
  return LBM_OK;
}

int tile_launch(int storage, const TilePlan& plan, int ksteps, const KParams& P, bool overlap, cudaStream_t s) {
  TileArgs a;
  a.P = P;
  a.tiles_x = plan.tiles_x;
  a.tiles_y = plan.tiles_y;
  a.ksteps = ksteps;
  launch_step(kernel_of(storage, P, plan.wide), dim3((unsigned)(plan.tiles_x * plan.tiles_y)), plan.threads, overlap, s,
              plan.smem, a);
  count_launch();
  return check_launch("tile_kernel");
}

}  // namespace lbm

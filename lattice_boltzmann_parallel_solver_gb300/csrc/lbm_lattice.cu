// lbm_lattice.cu -- fused pull-scheme stream + boundary + collide kernel and
// the C ABI of the drop-in step and of the resident lattice.
//
// State convention.  The reference's step (lattice_boltzmann_method.py:191-228)
// maps the post-streaming state f_n to f_{n+1} = BC(stream(collide(f_n))).
// The resident state kept here is S_n = collide(f_n) with the pre-streaming
// pressure rewrite already applied (boundary_conditions.py:320-346), so one
// kernel per step reads S_{n-1} once (pull: node x takes S(x - c_i, i)),
// applies the boundary sources, forms the moments of f_n, collides and
// writes S_n once: 72 B read + 72 B written per node in float64.
//   init_kernel : S_0 = collide(f_0) from a reference-layout f_0 (rho,u passed in or recomputed)
//   the steps   : S_n from S_{n-1}
//   read_kernel : f_n = BC(stream(S_{n-1})) and its moments, in the reference layout
// The outlet (boundary_conditions.py:279-280) needs f_{n-1} at column nx-2;
// each kernel stores those three populations in aux[3][ny] for the next one.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <type_traits>
#include <vector>

#include "lbm_fused.cuh"
#include "lbm_tile.h"

namespace lbm {

// The generic one-node-per-thread code: any geometry, any storage, exact or FMA
// arithmetic.

// populations of a storage as the generic code reads and writes them: in the
// reference-shifted 16-bit storages (dev_shift) the stored deviation is taken
// from c_i = w_i + sig_i instead of w_i
template <int STORE>
__device__ __forceinline__ typename Store<STORE>::R node_ld(const KParams& P, const typename Store<STORE>::T* p, int i) {
  using R = typename Store<STORE>::R;
  const R v = Store<STORE>::ld(p, i);
  if constexpr (Store<STORE>::kShifted) return P.dev_shift ? v + (R)P.shf[1].sig[i] : v;
  else return v;
}
template <int STORE>
__device__ __forceinline__ void node_st(const KParams& P, typename Store<STORE>::T* p, typename Store<STORE>::R v, int i) {
  using R = typename Store<STORE>::R;
  if constexpr (Store<STORE>::kShifted) Store<STORE>::st(p, P.dev_shift ? v - (R)P.shf[1].sig[i] : v, i);
  else Store<STORE>::st(p, v, i);
}

// f of node (x, y) pulled from the collided populations, with its boundary sources
template <int STORE, bool EXACT>
__device__ __forceinline__ void pull_node(const KParams& P, int x, int y, typename Store<STORE>::R f[9]) {
  using St = Store<STORE>;
  using T = typename St::T;
  using R = typename St::R;
  const int nx = P.g.nx, ny = P.g.ny;
  const int64_t r0 = (int64_t)y * P.pitch;
  const typename St::A* aux_in = static_cast<const typename St::A*>(P.aux_in);
  auto ld = [&](const T* p, int i) -> R { return node_ld<STORE>(P, p, i); };
  // pull: direction i arrives from node (x - cx_i, y - cy_i), periodic
  const int xm = x == 0 ? nx - 1 : x - 1, xp = x == nx - 1 ? 0 : x + 1;
  const int ym = y == 0 ? ny - 1 : y - 1, yp = y == ny - 1 ? 0 : y + 1;
  const int64_t rm = (int64_t)ym * P.pitch, rp = (int64_t)yp * P.pitch;
  const T* pin = static_cast<const T*>(P.pop_in);
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    const int xs = cx(i) == 1 ? xm : (cx(i) == -1 ? xp : x);
    const int64_t rs = cy(i) == 1 ? rm : (cy(i) == -1 ? rp : r0);
    f[i] = ld(pin + i * P.plane + rs + xs, i);
  }
  if (P.g.bcmask != nullptr) {
    const uint32_t word = __ldg(P.g.bcmask + (int64_t)y * P.g.words + (x >> 5));
    if ((word >> (x & 31)) & 1u) {
      const uint32_t d = __ldg(P.g.desc + (int64_t)y * nx + x);
      const int ks = (d >> LBM_DESC_KSET_SHIFT) & 15, cs = (d >> LBM_DESC_CSET_SHIFT) & 15;
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        const uint32_t s = (d >> (2 * i)) & 3u;
        if (s == LBM_SRC_BOUNCE) {
          const R v = ld(pin + opp(i) * P.plane + r0 + x, opp(i));
          if (EXACT)
            f[i] = (R)__dsub_rn((double)v, P.g.kconst[ks][i]);
          else
            f[i] = v - (R)P.g.kconst[ks][i];
        } else if (s == LBM_SRC_CONST) {
          f[i] = (R)P.g.cconst[cs][i];
        } else if (s == LBM_SRC_OUTLET && outlet_slot(i) >= 0 && aux_in != nullptr) {
          f[i] = St::from_aux(aux_in[outlet_slot(i) * ny + y], i);
        }
      }
    }
  }
}

// Collides node (x, y) of f_n in place (its moments rho, ux, uy as given) and
// stores S_n and the outlet memory.
template <int STORE, bool EXACT>
__device__ __forceinline__ void collide_store(const KParams& P, int x, int y, typename Store<STORE>::R f[9],
                                              typename Store<STORE>::R rho, typename Store<STORE>::R ux,
                                              typename Store<STORE>::R uy) {
  using St = Store<STORE>;
  using T = typename St::T;
  using R = typename St::R;
  using A = typename St::A;
  const int nx = P.g.nx, ny = P.g.ny;
  const int64_t r0 = (int64_t)y * P.pitch;
  auto st = [&](T* p, R v, int i) { node_st<STORE>(P, p, v, i); };
  // outlet memory: the pre-collision populations 3,6,7 of column nx-2
  if (P.aux_out != nullptr && x == nx - 2) {
    A* aux_out = static_cast<A*>(P.aux_out);
    aux_out[0 * ny + y] = St::to_aux(f[3], 3);
    aux_out[1 * ny + y] = St::to_aux(f[6], 6);
    aux_out[2 * ny + y] = St::to_aux(f[7], 7);
  }
  // collision
  const bool pressure_src = P.g.pressure && (x == nx - 2 || x == 1);
  R pin_v[9], pout_v[9];
  if (EXACT) {
    double fd[9], feq[9], br[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) fd[i] = (double)f[i];
    collide_exact(fd, (double)rho, (double)ux, (double)uy, P.omega, feq, br);
    if (pressure_src) {
      // feq(rho_in, u(nx-2)) + (fpre - feq(rho, u))  at column 0, and the outlet analogue
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        const double neq = __dsub_rn(fd[i], feq[i]);
        pin_v[i] = (R)__dadd_rn(__dmul_rn(__dmul_rn(wd(i), P.g.rho_in), br[i]), neq);
        pout_v[i] = (R)__dadd_rn(__dmul_rn(__dmul_rn(wd(i), P.g.rho_out), br[i]), neq);
      }
    }
#pragma unroll
    for (int i = 0; i < 9; ++i) f[i] = (R)fd[i];
  } else {
    collide_fast(f, rho, ux, uy, (R)P.omega);
    if (pressure_src) {
      R br[9];
      bracket9_fast(ux, uy, br);
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        pin_v[i] = fma(wr<R>(i) * br[i], (R)P.g.rho_in - rho, f[i]);
        pout_v[i] = fma(wr<R>(i) * br[i], (R)P.g.rho_out - rho, f[i]);
      }
    }
  }

  // store S_n; columns 0 / nx-1 take the pressure rewrite from columns nx-2 / 1
  T* pout = static_cast<T*>(P.pop_out);
  const uint32_t skip = P.g.pressure ? ((x == 0 ? P.g.pin : 0u) | (x == nx - 1 ? P.g.pout : 0u)) : 0u;
#pragma unroll
  for (int i = 0; i < 9; ++i)
    if (!((skip >> i) & 1u)) st(pout + i * P.plane + r0 + x, f[i], i);
  if (pressure_src) {
    if (x == nx - 2) {
#pragma unroll
      for (int i = 0; i < 9; ++i)
        if ((P.g.pin >> i) & 1u) st(pout + i * P.plane + r0 + 0, pin_v[i], i);
    }
    if (x == 1) {
#pragma unroll
      for (int i = 0; i < 9; ++i)
        if ((P.g.pout >> i) & 1u) st(pout + i * P.plane + r0 + (nx - 1), pout_v[i], i);
    }
  }
}

// moments of f_n: exactly as compute_density / compute_velocity_field, or the FMA form
template <bool EXACT, typename R>
__device__ __forceinline__ void node_moments(const R f[9], R& rho, R& ux, R& uy) {
  if constexpr (EXACT) {
    double fd[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) fd[i] = (double)f[i];
    const double r = density9_exact(fd);
    double a, b;
    velocity_exact(fd, r, a, b);
    rho = (R)r;
    ux = (R)a;
    uy = (R)b;
  } else {
    rho = density9(f);
    velocity_fast(f, rho, ux, uy);
  }
}

// S_n from S_{n-1}, one node per thread
template <int STORE, bool EXACT>
__global__ void __launch_bounds__(256) lattice_kernel(const __grid_constant__ KParams P) {
  using R = typename Store<STORE>::R;
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= P.g.nx || y >= P.g.ny) return;
  R f[9], rho, ux, uy;
  pull_node<STORE, EXACT>(P, x, y, f);
  node_moments<EXACT>(f, rho, ux, uy);
  write_probe(P, x, y, ux, uy);
  if (P.rho_out.p != nullptr) {
    P.rho_out.p[x * P.rho_out.sx + y * P.rho_out.sy] = (double)rho;
    if (P.u_out.p != nullptr) {
      double* up = P.u_out.p + x * P.u_out.sx + y * P.u_out.sy;
      up[0] = (double)ux;
      up[P.u_out.sc] = (double)uy;
    }
  }
  collide_store<STORE, EXACT>(P, x, y, f, rho, ux, uy);
}

// The read-out goes from the resident layout (x fastest) to the reference's
// f[x][y][9] (y fastest).  On larger lattices of the 64-bit storages (read_tiled) a
// tile of kTileX x kTileY nodes passes through shared memory, so that both sides move whole runs (32 elements of
// a plane per row, 576 B of f per column of the tile; a thread that stores its
// node's 72 B itself takes a sector per population).  The shared rows are 73, 9 and
// 17 doubles long: odd, so that lanes along x hit different banks.  What is left is
// float64 arithmetic, some 40 instructions a node (conversions, exact moments with
// two divisions) on a pipe that serves 1.6 a clock per SM.  1024^2 with f, us: f64
// 130 -> 98, fx64 147 -> 128.  The float32 and 16-bit storages are bound by it
// already (128 either way, and the barrier costs small lattices 2 us), so a thread
// writes its node there.  (The first step through shared memory lost, 150 -> 164 us
// in float64: its loads wait for nobody as they are, and the barrier made the
// float64 work wait for them.)
constexpr int kTileX = 32, kTileY = 8, kTileThreads = kTileX * kTileY;
struct RefTile {
  double f[kTileX][9 * kTileY + 1];
  double rho[kTileX][kTileY + 1];
  double u[kTileX][2 * kTileY + 1];
};

// Writes the shared tile to the reference layout (N values per node); columns
// x0 .. xe - 1, rows y0 .. ny - 1 at most.
template <int N, int W>
__device__ __forceinline__ void tile_write(double* g, const double (*s)[W], int tid, int x0, int xe, int y0,
                                           int ny) {
  static_assert(W == N * kTileY + 1, "a tile column and one more");
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const int e = tid + j * kTileThreads, c = e / (N * kTileY), r = e - c * (N * kTileY);
    if (x0 + c < xe && y0 + r / N < ny) g[((int64_t)(x0 + c) * ny + y0) * N + r] = s[c][r];
  }
}

// S_0 = collide(f_0) from the reference layout, with the rho, u passed in or their moments
template <int STORE, bool EXACT>
__global__ void __launch_bounds__(256) init_kernel(const __grid_constant__ KParams P, const double* f_in,
                                                   const double* rho_in, const double* u_in) {
  using R = typename Store<STORE>::R;
  const int ny = P.g.ny, x = P.xb + blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= (P.xe > 0 ? P.xe : P.g.nx) || y >= ny) return;
  const int64_t n = (int64_t)x * ny + y;
  R f[9], rho, ux, uy;
#pragma unroll
  for (int i = 0; i < 9; ++i) f[i] = (R)f_in[9 * n + i];
  if (rho_in != nullptr) {
    rho = (R)rho_in[n];
    ux = (R)u_in[2 * n];
    uy = (R)u_in[2 * n + 1];
  } else {
    node_moments<EXACT>(f, rho, ux, uy);
  }
  collide_store<STORE, EXACT>(P, x, y, f, rho, ux, uy);
}

// Whether a read-out of `nodes` nodes goes through the tile.  Below, the barrier costs
// more than the whole runs save: us, direct / tiled, with f fx64 64^2 8.4 / 10.5, 420x180
// 17.9 / 18.1, 640x410 39.2 / 37.7, f64 200x60 5.9 / 7.5, 420x180 15.9 / 15.7; the moments
// alone f64 420x180 12.9 / 14.7, 1024^2 115.4 / 115.5, 2100x1900 435 / 433.
template <int STORE>
constexpr bool may_tile_read() { return sizeof(typename Store<STORE>::T) == 8; }
template <int STORE>
static bool read_tiled(int64_t nodes, bool with_f) {
  if (!may_tile_read<STORE>()) return false;
  return nodes >= (int64_t)1 << (!with_f ? 21 : STORE == LBM_STORE_FX64 ? 17 : 16);
}

// f_n = BC(stream(S_{n-1})) and its moments in the reference layout (each of the
// outputs may be null); the moments always follow compute_density /
// compute_velocity_field exactly.  Blocks of kTileX x kTileY threads in the tiled
// form, of node_grid otherwise.
template <int STORE, bool EXACT, bool TILED>
__global__ void __launch_bounds__(256) read_kernel(const __grid_constant__ KParams P, double* f_out, double* rho_out,
                                                   double* u_out) {
  using R = typename Store<STORE>::R;
  pdl_wait();
  const int ny = P.g.ny, xe = P.xe > 0 ? P.xe : P.g.nx;
  const int x0 = P.xb + (int)(blockIdx.x * blockDim.x), y0 = (int)(blockIdx.y * blockDim.y);
  const int c = (int)threadIdx.x, r = (int)threadIdx.y, x = x0 + c, y = y0 + r;
  R f[9], rho, ux, uy;
  const bool in = x < xe && y < ny;
  if (in) {
    pull_node<STORE, EXACT>(P, x, y, f);
    node_moments<true>(f, rho, ux, uy);
  }
  if constexpr (TILED) {
    __shared__ RefTile t;
    if (in) {
#pragma unroll
      for (int i = 0; i < 9; ++i) t.f[c][9 * r + i] = (double)f[i];
      t.rho[c][r] = (double)rho;
      t.u[c][2 * r] = (double)ux;
      t.u[c][2 * r + 1] = (double)uy;
    }
    __syncthreads();
    const int tid = r * kTileX + c;
    if (f_out != nullptr) tile_write<9>(f_out, t.f, tid, x0, xe, y0, ny);
    if (rho_out != nullptr) tile_write<1>(rho_out, t.rho, tid, x0, xe, y0, ny);
    if (u_out != nullptr) tile_write<2>(u_out, t.u, tid, x0, xe, y0, ny);
  } else if (in) {
    const int64_t n = (int64_t)x * ny + y;
    if (rho_out != nullptr) rho_out[n] = (double)rho;
    if (u_out != nullptr) {
      u_out[2 * n] = (double)ux;
      u_out[2 * n + 1] = (double)uy;
    }
    if (f_out != nullptr) {
#pragma unroll
      for (int i = 0; i < 9; ++i) f_out[9 * n + i] = (double)f[i];
    }
  }
}

// How a vectorised step's kernel applies the boundary sources: kBcNone without
// any, kBcInline inside the body, kBcPass (float32) in the first pass_rows rows of
// blocks, one thread per listed boundary node, beside the blocks of a body that
// leaves those nodes out.
enum { kBcNone = 0, kBcInline = 1, kBcPass = 2 };

// The boundary-node pass, one thread per listed boundary node: recomputes the
// node with its sources (the same body at one node per thread, so the arithmetic
// and the random bits are those of the sources inside the step).  It is bound by
// the latency of its dependent loads.
template <int STORE, int THREADS, bool HAS_PRESSURE, bool SHIFT>
__device__ __forceinline__ void pass_block(const KParams& P) {
  const int t = (int)((blockIdx.y * gridDim.x + blockIdx.x) * THREADS + threadIdx.x);
  if (t >= P.g.n_bcnodes) return;
  const int node = __ldg(P.g.bcnodes + t);
  const int y = node / P.g.nx, x = node - y * P.g.nx;
  if constexpr (STORE == LBM_STORE_FX64)
    fused_fx_body<1, true, HAS_PRESSURE>(P, P.pop_in, P.pop_out, P.aux_in, P.aux_out, x, y);
  else
    fused_v2_body<STORE, 1, true, HAS_PRESSURE, false, SHIFT>(P, P.pop_in, P.pop_out, P.aux_in, P.aux_out, x, y,
                                                              launch_seed(P), true);
}

// The pass as a launch of its own, after a boundary-free step over every node:
// it overwrites the listed nodes' outputs.
template <int STORE, int THREADS, bool HAS_PRESSURE, bool SHIFT>
__global__ void __launch_bounds__(THREADS) fixup_v2_kernel(const __grid_constant__ KParams P) {
  pdl_wait();
  pass_block<STORE, THREADS, HAS_PRESSURE, SHIFT>(P);
}

// the float32 and 16-bit storages: registers capped so that 1024 threads fit on
// an SM (float32 at 4 nodes per thread: 640); SHIFT: the reference-shifted
// 16-bit storages.  In float32 a warp whose nodes are all inside (see inside())
// takes a body without wrap, outlet memory and pressure code (4096^2: 194 ->
// 174 us); in the others, nearer to their register cap, a second body costs more
// than it saves.
template <int STORE, int NPT, int THREADS, bool SHIFT, int BC, bool HAS_PRESSURE>
__global__ void __launch_bounds__(THREADS, (STORE == LBM_STORE_F16S || STORE == LBM_STORE_BF16S ||
                                            (STORE == LBM_STORE_F32 && NPT <= 2))
                                               ? 1024 / THREADS
                                               : (STORE == LBM_STORE_F32 ? 640 / THREADS : 1))
    fused_v2_kernel(const __grid_constant__ KParams P) {
  pdl_wait();
  int y = (int)blockIdx.y;
  if constexpr (BC == kBcPass) {
    if (y < P.pass_rows) {
      pass_block<STORE, THREADS, HAS_PRESSURE, SHIFT>(P);
      return;
    }
    y -= P.pass_rows;
  }
  const int t = (int)(blockIdx.x * THREADS + threadIdx.x);
  if constexpr (STORE == LBM_STORE_F32 && BC != kBcInline) {
    const int xa = (t & ~31) * NPT;
    if (inside(P.g, BC == kBcPass, xa, xa + 32 * NPT - 1, y)) {
      fused_v2_body<STORE, NPT, false, false, false, SHIFT, false, true>(P, P.pop_in, P.pop_out, P.aux_in, P.aux_out,
                                                                         t * NPT, y, launch_seed(P));
      return;
    }
  }
  fused_v2_body<STORE, NPT, BC == kBcInline, HAS_PRESSURE, false, SHIFT, BC == kBcPass>(
      P, P.pop_in, P.pop_out, P.aux_in, P.aux_out, t * NPT, y, launch_seed(P), false,
      BC == kBcPass && pass_chunk(P.g, (int)blockIdx.x * (THREADS * NPT), THREADS * NPT, y));
}

// one node per thread: registers capped so that 1024 threads fit on an SM
template <int NPT, int THREADS, int BC, bool HAS_PRESSURE>
__global__ void __launch_bounds__(THREADS, NPT == 1 ? 1024 / THREADS : 1) fused_fx_kernel(const __grid_constant__ KParams P) {
  pdl_wait();
  fused_fx_body<NPT, BC == kBcInline, HAS_PRESSURE>(P, P.pop_in, P.pop_out, P.aux_in, P.aux_out,
                                                    (blockIdx.x * THREADS + threadIdx.x) * NPT, blockIdx.y);
}

// adds the steps of a lbm_lattice_run_opts call to its device step counter
__global__ void advance_counter_kernel(int32_t* counter, int32_t n) { *counter += n; }

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// f(storage, exact) with the storage and the arithmetic as compile-time numbers
template <typename F>
static int by_storage(int storage, bool exact, const KParams& P, F&& f) {
  if (exact && storage != LBM_STORE_F64)
    return set_error(LBM_ERR_UNSUPPORTED, "exact arithmetic needs float64 storage");
  using std::integral_constant;
  constexpr std::false_type fma{};
  switch (storage) {
    case LBM_STORE_F64:
      return exact ? f(P, integral_constant<int, LBM_STORE_F64>{}, std::true_type{})
                   : f(P, integral_constant<int, LBM_STORE_F64>{}, fma);
    case LBM_STORE_F32: return f(P, integral_constant<int, LBM_STORE_F32>{}, fma);
    case LBM_STORE_F16S: return f(P, integral_constant<int, LBM_STORE_F16S>{}, fma);
    case LBM_STORE_BF16S: return f(P, integral_constant<int, LBM_STORE_BF16S>{}, fma);
    case LBM_STORE_FX64: return f(P, integral_constant<int, LBM_STORE_FX64>{}, fma);
    case LBM_STORE_F16R:
    case LBM_STORE_BF16R: {
      KParams Q = P;
      Q.dev_shift = 1;
      return storage == LBM_STORE_F16R ? f(Q, integral_constant<int, LBM_STORE_F16S>{}, fma)
                                       : f(Q, integral_constant<int, LBM_STORE_BF16S>{}, fma);
    }
    default: return set_error(LBM_ERR_ARG, "unknown storage type");
  }
}

// one thread per node, along x
static void node_grid(int w, int ny, dim3& grid, dim3& block) {
  const int bx = w >= 128 ? 128 : (w + 31) / 32 * 32, by = std::max(1, 128 / bx);
  block = dim3((unsigned)bx, (unsigned)by);
  grid = dim3((unsigned)((w + bx - 1) / bx), (unsigned)((ny + by - 1) / by));
}

// one generic step
static int launch_node(int storage, bool exact, const KParams& P, cudaStream_t s) {
  return by_storage(storage, exact, P, [&](const KParams& Q, auto store, auto ex) {
    dim3 grid, block;
    node_grid(Q.g.nx, Q.g.ny, grid, block);
    lattice_kernel<store(), ex()><<<grid, block, 0, s>>>(Q);
    count_launch();
    return check_launch("lattice_kernel");
  });
}

static int launch_init(int storage, bool exact, const KParams& P, const double* f, const double* rho, const double* u,
                       cudaStream_t s) {
  return by_storage(storage, exact, P, [&](const KParams& Q, auto store, auto ex) {
    dim3 grid, block;
    node_grid((Q.xe > 0 ? Q.xe : Q.g.nx) - Q.xb, Q.g.ny, grid, block);
    init_kernel<store(), ex()><<<grid, block, 0, s>>>(Q, f, rho, u);
    count_launch();
    return check_launch("init_kernel");
  });
}

// `overlap`: right after the init_kernel of the same call
static int launch_read(int storage, bool exact, const KParams& P, double* f, double* rho, double* u, bool overlap,
                       cudaStream_t s) {
  return by_storage(storage, exact, P, [&](const KParams& Q, auto store, auto ex) {
    const int w = (Q.xe > 0 ? Q.xe : Q.g.nx) - Q.xb;
    dim3 grid, block;
    if constexpr (may_tile_read<store()>()) {
      if (read_tiled<store()>((int64_t)w * Q.g.ny, f != nullptr)) {
        block = dim3(kTileX, kTileY);
        grid = dim3((unsigned)((w + kTileX - 1) / kTileX), (unsigned)((Q.g.ny + kTileY - 1) / kTileY));
        launch_step(read_kernel<store(), ex(), true>, grid, block, overlap, s, 0, Q, f, rho, u);
        count_launch();
        return check_launch("read_kernel");
      }
    }
    node_grid(w, Q.g.ny, grid, block);
    launch_step(read_kernel<store(), ex(), false>, grid, block, overlap, s, 0, Q, f, rho, u);
    count_launch();
    return check_launch("read_kernel");
  });
}

constexpr int kV2Threads = 128;

// the boundary specialisations of one vectorised kernel; PASS: with kBcPass
#define LBM_LAUNCH_FORM(STORE, BC, PR, KERNEL, ...)                                                                 \
  launch_step(KERNEL<__VA_ARGS__, BC, PR>, grid, kV2Threads,                                                        \
              overlap && overlaps<STORE, KERNEL<__VA_ARGS__, BC, PR>>((int64_t)grid.x * grid.y, kV2Threads), s, 0, P)
#define LBM_LAUNCH_SPECIALISED(PASS, STORE, KERNEL, ...)                                            \
  do {                                                                                              \
    const bool pr = P.g.pressure != 0;                                                              \
    if constexpr (PASS) {                                                                           \
      if (bc == kBcPass && pr) LBM_LAUNCH_FORM(STORE, kBcPass, true, KERNEL, __VA_ARGS__);          \
      else if (bc == kBcPass) LBM_LAUNCH_FORM(STORE, kBcPass, false, KERNEL, __VA_ARGS__);          \
    }                                                                                               \
    if (bc == kBcInline && pr) LBM_LAUNCH_FORM(STORE, kBcInline, true, KERNEL, __VA_ARGS__);        \
    else if (bc == kBcInline) LBM_LAUNCH_FORM(STORE, kBcInline, false, KERNEL, __VA_ARGS__);        \
    else if (bc == kBcNone && pr) LBM_LAUNCH_FORM(STORE, kBcNone, true, KERNEL, __VA_ARGS__);       \
    else if (bc == kBcNone) LBM_LAUNCH_FORM(STORE, kBcNone, false, KERNEL, __VA_ARGS__);            \
  } while (0)

template <int NPT>
static int v2_blocks(const KParams& P) {
  return ((P.g.nx + NPT - 1) / NPT + kV2Threads - 1) / kV2Threads;
}

template <int STORE, int NPT, bool SHIFT = false>
static int launch_v2(KParams P, int bc, bool overlap, cudaStream_t s) {
  const int bx = v2_blocks<NPT>(P);
  P.pass_rows = bc == kBcPass ? (P.g.n_bcnodes + kV2Threads * bx - 1) / (kV2Threads * bx) : 0;
  const dim3 grid((unsigned)bx, (unsigned)(P.g.ny + P.pass_rows));
  LBM_LAUNCH_SPECIALISED(STORE == LBM_STORE_F32, STORE, fused_v2_kernel, STORE, NPT, kV2Threads, SHIFT);
  count_launch();
  return check_launch("fused_v2_kernel");
}

template <int NPT>
static int launch_fx(const KParams& P, int bc, bool overlap, cudaStream_t s) {
  const dim3 grid((unsigned)v2_blocks<NPT>(P), (unsigned)P.g.ny);
  LBM_LAUNCH_SPECIALISED(false, LBM_STORE_FX64, fused_fx_kernel, NPT, kV2Threads);
  count_launch();
  return check_launch("fused_fx_kernel");
}

// nodes per thread, measured on the 8192^2 cavity: float32 87.7 GLUPS at 4
// against 83.6 at 2; 16-bit 168 at 4 against 160 at 8 (512 threads per SM)
static int default_npt(int storage) {
  switch (storage) {
    case LBM_STORE_F64: return 2;
    case LBM_STORE_FX64: return 1;
    default: return 4;
  }
}

// the reference-shifted 16-bit storages run at 4 nodes per thread only
static bool ref_shifted(int storage) { return storage == LBM_STORE_F16R || storage == LBM_STORE_BF16R; }

// nodes per thread of the vectorised kernel for this lattice, 0 when it does not apply
static int v2_npt(int storage, int flags, const KParams& P) {
  if ((flags & LBM_FLAG_EXACT) || (flags & LBM_FLAG_GENERIC)) return 0;
  int npt = ref_shifted(storage) ? 0 : (flags >> LBM_FLAG_NPT_SHIFT) & 15;
  if (npt == 0) npt = default_npt(storage);
  if (!v2_fits(P, npt)) return 0;
  return npt;
}

// whether the fixed-point storage has a vectorised kernel of this node count
// (the cases of launch_fused_step; others take the generic kernel)
static bool fx_compiled(int npt) { return npt == 1 || npt == 2 || npt == 4; }

// Whether the boundary nodes may be left to the boundary-node pass: the geometry
// lists them and they are at most an eighth of the lattice; a probe keeps the
// sources inside the step, so its node is recorded once.
static bool pass_listed(int npt, int flags, const KParams& P) {
  return npt > 0 && !(flags & LBM_FLAG_BC_INLINE) && P.g.bcmask != nullptr && P.g.n_bcnodes > 0 &&
         P.probe_buf == nullptr && (int64_t)P.g.n_bcnodes * 8 <= (int64_t)P.g.nx * P.g.ny;
}

// whether a pass that is not in the body's launch is a launch of its own (else the
// sources stay inside)
constexpr int64_t kApartNodes = (int64_t)1 << 25;
static bool pass_apart(int storage, int flags, const KParams& P) {
  const int64_t nodes = (int64_t)P.g.nx * P.g.ny;
  if (flags & LBM_FLAG_BC_SPLIT) return true;
  return nodes >= (ref_shifted(storage) ? (int64_t)1 << (small_box(P.g) ? 22 : 24) : kApartNodes);
}

// Whether a run's boundary tables are read as fixed-point numbers: by the
// vectorised kernels and by the pass.  The generic kernel reads them as float64
// (before a pass that is a second launch it reads none).
static bool fx_tables(int storage, int flags, const KParams& P) {
  const int npt = v2_npt(storage, flags, P);
  return storage == LBM_STORE_FX64 && npt > 0 &&
         (fx_compiled(npt) || (pass_listed(npt, flags, P) && pass_apart(storage, flags, P)));
}

// Lattices that may take several steps per launch: those of the vectorised
// kernels at their default shape (a flag that picks a one-step kernel or where
// the boundary sources go keeps the one-step launches).  Under the pressure
// rewrite a tile's halo may hold columns 0 and nx-1 once per side only.
static bool tile_applies(int storage, int flags, const KParams& P) {
  const int one_step = LBM_FLAG_EXACT | LBM_FLAG_GENERIC | LBM_FLAG_BC_INLINE | LBM_FLAG_BC_SPLIT | (15 << LBM_FLAG_NPT_SHIFT);
  return (flags & one_step) == 0 && v2_fits(P, default_npt(storage)) && (!P.g.pressure || P.g.nx >= 16);
}

constexpr int kFixupThreads = 128;

// (always right after the step kernel of the same launch_fused)
template <int STORE, bool SHIFT = false>
static int launch_fixup(const KParams& P, cudaStream_t s) {
  const dim3 grid((unsigned)((P.g.n_bcnodes + kFixupThreads - 1) / kFixupThreads));
  if (P.g.pressure)
    launch_step(fixup_v2_kernel<STORE, kFixupThreads, true, SHIFT>, grid, kFixupThreads, true, s, 0, P);
  else
    launch_step(fixup_v2_kernel<STORE, kFixupThreads, false, SHIFT>, grid, kFixupThreads, true, s, 0, P);
  count_launch();
  return check_launch("fixup_v2_kernel");
}

static int launch_fused_step(int storage, int npt, int bc, int flags, const KParams& P, bool overlap, cudaStream_t s) {
  switch (storage * 16 + npt) {
    case LBM_STORE_F64 * 16 + 2: return launch_v2<LBM_STORE_F64, 2>(P, bc, overlap, s);
    case LBM_STORE_F64 * 16 + 4: return launch_v2<LBM_STORE_F64, 4>(P, bc, overlap, s);
    case LBM_STORE_FX64 * 16 + 1: return launch_fx<1>(P, bc, overlap, s);
    case LBM_STORE_FX64 * 16 + 2: return launch_fx<2>(P, bc, overlap, s);
    case LBM_STORE_FX64 * 16 + 4: return launch_fx<4>(P, bc, overlap, s);
    case LBM_STORE_F32 * 16 + 2: return launch_v2<LBM_STORE_F32, 2>(P, bc, overlap, s);
    case LBM_STORE_F32 * 16 + 4: return launch_v2<LBM_STORE_F32, 4>(P, bc, overlap, s);
    case LBM_STORE_F16S * 16 + 2: return launch_v2<LBM_STORE_F16S, 2>(P, bc, overlap, s);
    case LBM_STORE_F16S * 16 + 4: return launch_v2<LBM_STORE_F16S, 4>(P, bc, overlap, s);
    case LBM_STORE_F16S * 16 + 8: return launch_v2<LBM_STORE_F16S, 8>(P, bc, overlap, s);
    case LBM_STORE_BF16S * 16 + 2: return launch_v2<LBM_STORE_BF16S, 2>(P, bc, overlap, s);
    case LBM_STORE_BF16S * 16 + 4: return launch_v2<LBM_STORE_BF16S, 4>(P, bc, overlap, s);
    case LBM_STORE_BF16S * 16 + 8: return launch_v2<LBM_STORE_BF16S, 8>(P, bc, overlap, s);
    case LBM_STORE_F16R * 16 + 4: return launch_v2<LBM_STORE_F16S, 4, true>(P, bc, overlap, s);
    case LBM_STORE_BF16R * 16 + 4: return launch_v2<LBM_STORE_BF16S, 4, true>(P, bc, overlap, s);
    default: return launch_node(storage, flags & LBM_FLAG_EXACT, P, s);
  }
}

// One step.  The boundary nodes may be left to the boundary-node pass (pass_listed).
//
// float32 takes the pass in blocks of the step's own launch, at every size: its
// body is far from its register cap, and with the sources inside, the warps at a
// row's ends wait for mask, descriptor and bounced populations in turn.  Cavity,
// us per step, inside against pass: 1024^2 12.5 / 10.7, 2048^2 55.3 / 47.5, 4096^2
// 195 / 178, 8192^2 759 / 698.  In the other storages leaving the nodes out costs
// the capped body more than the pass saves (4096^2 f16 117 against 107, fx64 377
// against 367), so they keep the sources inside, and from 2^25 nodes take the pass
// as a second launch (8192^2 fx64 1437 against 1444).  The reference-shifted
// storages, whose body with sources has the most to hold under its cap, do so from
// 2^22 (f16r cavity 1500^2 19.4 inside, 20.6 as a second launch, 2049^2 42.5 / 39.3,
// 5000^2 177.5 / 164.2; walls alone 2100^2 40.1 / 37.6), from 2^24 without a frame (half
// of a side 3000x2600 56.5 / 57.8, 4500^2 139.0 / 133.6).
static int launch_fused(int storage, int flags, const KParams& P, bool overlap, cudaStream_t s) {
  const int npt = v2_npt(storage, flags, P);
  const int inside = P.g.bcmask != nullptr ? kBcInline : kBcNone;
  if (!pass_listed(npt, flags, P)) return launch_fused_step(storage, npt, inside, flags, P, overlap, s);
  if (storage == LBM_STORE_F32) {
    // the pass's rows of blocks fit the grid beside the lattice's; where boundary
    // nodes are spread over a large lattice, a second launch (5800^2, inside / same
    // launch / second launch: 396 / 438 / 353)
    const bool fits = (int64_t)P.g.ny + P.g.n_bcnodes / kV2Threads + 1 <= 65535;
    const bool large = (int64_t)P.g.nx * P.g.ny >= kApartNodes;
    if (fits && (small_box(P.g) || ((flags & LBM_FLAG_BC_SPLIT) && !large)))
      return launch_fused_step(storage, npt, kBcPass, flags, P, overlap, s);
  }
  if (!pass_apart(storage, flags, P)) return launch_fused_step(storage, npt, inside, flags, P, overlap, s);
  KParams Q = P;
  Q.g.bcmask = nullptr;
  if (int e = launch_fused_step(storage, npt, kBcNone, flags, Q, overlap, s)) return e;
  switch (storage) {
    case LBM_STORE_F64: return launch_fixup<LBM_STORE_F64>(P, s);
    case LBM_STORE_F32: return launch_fixup<LBM_STORE_F32>(P, s);
    case LBM_STORE_F16S: return launch_fixup<LBM_STORE_F16S>(P, s);
    case LBM_STORE_BF16S: return launch_fixup<LBM_STORE_BF16S>(P, s);
    case LBM_STORE_FX64: return launch_fixup<LBM_STORE_FX64>(P, s);
    case LBM_STORE_F16R: return launch_fixup<LBM_STORE_F16S, true>(P, s);
    case LBM_STORE_BF16R: return launch_fixup<LBM_STORE_BF16S, true>(P, s);
    default: return set_error(LBM_ERR_ARG, "unknown storage type");
  }
}

static size_t store_bytes(int storage) {
  switch (storage) {
    case LBM_STORE_F64:
    case LBM_STORE_FX64: return 8;
    case LBM_STORE_F32: return 4;
    case LBM_STORE_F16S:
    case LBM_STORE_BF16S:
    case LBM_STORE_F16R:
    case LBM_STORE_BF16R: return 2;
    default: return 0;
  }
}

}  // namespace lbm

using namespace lbm;

extern "C" {

size_t lbm_lattice_pop_bytes(int32_t nx, int32_t ny, int64_t pitch, int32_t storage) {
  (void)nx;
  return (size_t)9 * (size_t)ny * (size_t)pitch * store_bytes(storage);
}

int lbm_lattice_init(const lbm_geometry* g, int32_t storage, const double* f, const double* rho,
                     const double* u, double omega, void* pop_out, int64_t pitch, void* aux_out,
                     int32_t flags, void* stream) {
  KParams P;
  std::memset(&P, 0, sizeof(P));
  if (!to_geok(g, P.g)) return last_status();
  if (int e = check_omega(omega)) return e;
  if (int e = check_pitch(g->nx, pitch)) return e;
  if (f == nullptr || pop_out == nullptr) return set_error(LBM_ERR_ARG, "f and pop_out are required");
  if ((rho == nullptr) != (u == nullptr)) return set_error(LBM_ERR_ARG, "rho and u must be given together");
  if (g->outlet && aux_out == nullptr) return set_error(LBM_ERR_ARG, "the outlet needs aux_out");
  P.pop_out = pop_out;
  P.pitch = pitch;
  P.plane = pitch * g->ny;
  P.aux_out = aux_out;
  P.omega = omega;
  set_shift(P);
  return launch_init(storage, flags & LBM_FLAG_EXACT, P, f, rho, u, (cudaStream_t)stream);
}

int lbm_lattice_run(const lbm_geometry* g, int32_t storage, void* pop_a, void* pop_b, int64_t pitch,
                    void* aux_a, void* aux_b, double omega, int32_t nsteps, double* rho_out,
                    double* u_out, int32_t flags, uint32_t seed, void* stream) {
  return lbm_lattice_run_opts(g, storage, pop_a, pop_b, pitch, aux_a, aux_b, omega, nsteps, rho_out, u_out, flags,
                              seed, nullptr, stream);
}

int lbm_lattice_run_opts(const lbm_geometry* g, int32_t storage, void* pop_a, void* pop_b, int64_t pitch,
                         void* aux_a, void* aux_b, double omega, int32_t nsteps, double* rho_out,
                         double* u_out, int32_t flags, uint32_t seed, const lbm_run_options* opt,
                         void* stream) {
  KParams P;
  std::memset(&P, 0, sizeof(P));
  if (!to_geok(g, P.g)) return last_status();
  if (int e = check_omega(omega)) return e;
  if (int e = check_pitch(g->nx, pitch)) return e;
  if (pop_a == nullptr || pop_b == nullptr || pop_a == pop_b)
    return set_error(LBM_ERR_ARG, "two distinct population buffers are required");
  if (g->outlet && (aux_a == nullptr || aux_b == nullptr || aux_a == aux_b))
    return set_error(LBM_ERR_ARG, "the outlet needs two distinct aux buffers");
  if (nsteps < 0) return set_error(LBM_ERR_ARG, "nsteps must be >= 0");
  P.probe_x = P.probe_y = -1;
  if (opt != nullptr && opt->probe_buf != nullptr) {
    if (opt->probe_count == nullptr || opt->probe_cap < 0)
      return set_error(LBM_ERR_ARG, "a probe needs probe_count and probe_cap >= 0");
    if (opt->probe_x < 0 || opt->probe_x >= g->nx || opt->probe_y < 0 || opt->probe_y >= g->ny)
      return set_error(LBM_ERR_ARG, "the probe node lies outside the lattice");
    P.probe_x = opt->probe_x;
    P.probe_y = opt->probe_y;
    P.probe_cap = opt->probe_cap;
    P.probe_buf = opt->probe_buf;
    P.probe_count = opt->probe_count;
  }
  const int32_t* counter = opt != nullptr ? opt->step_counter : nullptr;
  P.pitch = pitch;
  P.plane = pitch * g->ny;
  P.omega = omega;
  set_shift(P);
  P.sr = (flags & LBM_FLAG_STOCHASTIC) != 0;
  P.qc = fx::q_consts(omega);
  P.step_dev = counter;
  // small lattices take several steps per launch; the moments of the last step
  // (rho_out, u_out) come from a one-step launch
  P.pop_in = pop_a;
  P.pop_out = pop_b;
  P.aux_in = aux_a;
  P.aux_out = aux_b;
  if (fx_tables(storage, flags, P)) set_fx_tables(P.g);
  const int tiled_steps = nsteps - (rho_out != nullptr || u_out != nullptr ? 1 : 0);
  TilePlan plan;
  if (tiled_steps >= 3 && tile_applies(storage, flags, P)) plan = tile_plan(storage, P);
  if (plan.ksteps > 1)
    if (int e = tile_prepare(storage, plan, P)) return e;
  int launches = 0;
  bool after_tile = false;
  for (int s = 0; s < nsteps; ++launches) {
    const bool even = (launches % 2) == 0;
    P.pop_in = even ? pop_a : pop_b;
    P.pop_out = even ? pop_b : pop_a;
    P.aux_in = even ? aux_a : aux_b;
    P.aux_out = even ? aux_b : aux_a;
    // an odd number of steps per launch: the buffers alternate as they would
    // step by step
    const int left = tiled_steps - s;
    const int k = plan.ksteps > 1 && left >= 3 ? std::min(plan.ksteps, left - (left % 2 == 0)) : 1;
    if (k > 1) {
      P.seed = seed + (uint32_t)s;
      if (int e = tile_launch(storage, plan, k, P, s > 0, (cudaStream_t)stream)) return e;
      s += k;
      after_tile = true;
      continue;
    }
    // with a device counter the kernels hash (seed + s + *counter) themselves
    P.seed = counter != nullptr ? seed + (uint32_t)s : hash32(seed + (uint32_t)s);
    const bool last = s == nsteps - 1;
    P.rho_out = OutView{last ? rho_out : nullptr, 1, pitch, 0};
    P.u_out = OutView{last ? u_out : nullptr, 1, pitch, pitch * g->ny};
    // tiles leave no room beside them: a float64 step that overlaps them piles its
    // blocks up on the SMs that come free first (428x129 periodic, four steps: 61.7 us, plain 49.5)
    const bool piles = after_tile && storage == LBM_STORE_F64;
    if (int e = launch_fused(storage, flags, P, s > 0 && !piles, (cudaStream_t)stream)) return e;
    after_tile = false;
    ++s;
  }
  if (counter != nullptr && nsteps > 0) {
    advance_counter_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(opt->step_counter, nsteps);
    count_launch();
    if (int e = check_launch("advance_counter_kernel")) return e;
  }
  return LBM_OK;
}

int lbm_lattice_read(const lbm_geometry* g, int32_t storage, const void* pop, int64_t pitch, const void* aux,
                     double* f_out, double* rho_out, double* u_out, void* stream) {
  KParams P;
  std::memset(&P, 0, sizeof(P));
  if (!to_geok(g, P.g)) return last_status();
  if (int e = check_pitch(g->nx, pitch)) return e;
  if (pop == nullptr) return set_error(LBM_ERR_ARG, "pop is required");
  if (g->outlet && aux == nullptr) return set_error(LBM_ERR_ARG, "the outlet needs aux");
  P.pop_in = pop;
  P.aux_in = aux;
  P.pitch = pitch;
  P.plane = pitch * g->ny;
  set_shift(P);  // omega 1: the read converts, it does not collide
  return launch_read(storage, false, P, f_out, rho_out, u_out, false, (cudaStream_t)stream);
}

size_t lbm_step_scratch_bytes(int32_t nx, int32_t ny) {
  const int64_t pitch = ((int64_t)nx + 31) / 32 * 32;
  return (size_t)(9 * pitch * ny + 3 * (int64_t)ny) * sizeof(double) + 256;
}

int lbm_step_f64(const lbm_geometry* g, const double* f, const double* rho, const double* u, double omega,
                 double* f_out, double* rho_out, double* u_out, void* scratch, int32_t flags, void* stream) {
  if (g == nullptr) return set_error(LBM_ERR_ARG, "geometry is NULL");
  if (f == nullptr || rho == nullptr || u == nullptr || f_out == nullptr || rho_out == nullptr ||
      u_out == nullptr || scratch == nullptr)
    return set_error(LBM_ERR_ARG, "f, rho, u, f_out, rho_out, u_out and scratch are required");
  const int64_t pitch = ((int64_t)g->nx + 31) / 32 * 32;
  uintptr_t base = ((uintptr_t)scratch + 255) & ~(uintptr_t)255;
  double* pop = reinterpret_cast<double*>(base);
  double* aux = pop + 9 * pitch * g->ny;
  if (int e = lbm_lattice_init(g, LBM_STORE_F64, f, rho, u, omega, pop, pitch, aux, flags, stream)) return e;
  // the read-out kernel recomputes the moments the same way in both forms
  KParams P;
  std::memset(&P, 0, sizeof(P));
  if (!to_geok(g, P.g)) return last_status();
  P.pop_in = pop;
  P.aux_in = aux;
  P.pitch = pitch;
  P.plane = pitch * g->ny;
  return launch_read(LBM_STORE_F64, flags & LBM_FLAG_EXACT, P, f_out, rho_out, u_out, true, (cudaStream_t)stream);
}

// ---- the drop-in step on host buffers, with copies and kernels overlapped ----
size_t lbm_step_host_scratch_bytes(int32_t nx, int32_t ny) {
  const int64_t pitch = ((int64_t)nx + 31) / 32 * 32, n = (int64_t)nx * ny;
  return (size_t)(24 * n + 9 * pitch * ny + 3 * (int64_t)ny) * sizeof(double) + 4 * 256;
}

int lbm_step_f64_host(const lbm_geometry* g, const double* f, const double* rho, const double* u, double omega,
                      double* f_out, double* rho_out, double* u_out, void* scratch, size_t scratch_bytes,
                      int32_t flags, int32_t slabs, void* stream) {
  if (g == nullptr) return set_error(LBM_ERR_ARG, "geometry is NULL");
  if (f == nullptr || rho == nullptr || u == nullptr || f_out == nullptr || rho_out == nullptr ||
      u_out == nullptr || scratch == nullptr)
    return set_error(LBM_ERR_ARG, "f, rho, u, f_out, rho_out, u_out and scratch are required");
  KParams G;
  std::memset(&G, 0, sizeof(G));
  if (!to_geok(g, G.g)) return last_status();
  if (int e = check_omega(omega)) return e;
  const int nx = g->nx, ny = g->ny;
  if (scratch_bytes < lbm_step_host_scratch_bytes(nx, ny)) return set_error(LBM_ERR_ARG, "scratch too small");
  const int64_t n = (int64_t)nx * ny, pitch = ((int64_t)nx + 31) / 32 * 32;
  const bool exact = (flags & LBM_FLAG_EXACT) != 0;
  // device layout: inputs f, rho, u | outputs f, rho, u | populations | outlet memory
  double* base = reinterpret_cast<double*>(((uintptr_t)scratch + 255) & ~(uintptr_t)255);
  double* fin = base;
  double* rin = fin + 9 * n;
  double* uin = rin + n;
  double* fo = uin + 2 * n;
  double* ro = fo + 9 * n;
  double* uo = ro + n;
  double* pop = reinterpret_cast<double*>(((uintptr_t)(uo + 2 * n) + 255) & ~(uintptr_t)255);
  double* aux = pop + 9 * pitch * ny;
  // default depth: one slab per 2^18 nodes, at most 32 (the copies then run
  // within a few percent of the link's two-way rate on large lattices)
  const int64_t auto_k = std::max<int64_t>(1, std::min<int64_t>(32, n >> 18));
  const int K = (int)std::max<int64_t>(1, std::min<int64_t>(slabs > 0 ? slabs : auto_k, nx));
  auto xs = [&](int k) { return (int)((int64_t)k * nx / K); };
  cudaStream_t caller = (cudaStream_t)stream, sh = nullptr, sc = nullptr, sd = nullptr;
  std::vector<cudaEvent_t> ev;
  int st = LBM_OK;
  auto cuda_ok = [&](cudaError_t e) {
    if (e != cudaSuccess && st == LBM_OK) st = set_error(LBM_ERR_CUDA, cudaGetErrorString(e));
    return st == LBM_OK;
  };
  auto event = [&]() {
    cudaEvent_t e = nullptr;
    cuda_ok(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    ev.push_back(e);
    return e;
  };
  cuda_ok(cudaStreamCreateWithFlags(&sh, cudaStreamNonBlocking));
  cuda_ok(cudaStreamCreateWithFlags(&sc, cudaStreamNonBlocking));
  cuda_ok(cudaStreamCreateWithFlags(&sd, cudaStreamNonBlocking));
  cudaEvent_t start = event();
  cuda_ok(cudaEventRecord(start, caller));
  cuda_ok(cudaStreamWaitEvent(sh, start, 0));
  cuda_ok(cudaStreamWaitEvent(sc, start, 0));
  cuda_ok(cudaStreamWaitEvent(sd, start, 0));
  std::vector<cudaEvent_t> in_ready(K), out_ready(K);
  auto upload = [&](int k) {
    if (st != LBM_OK) return;
    const int64_t a = xs(k), w = xs(k + 1) - xs(k);
    cuda_ok(cudaMemcpyAsync(fin + 9 * a * ny, f + 9 * a * ny, 9 * w * ny * sizeof(double), cudaMemcpyHostToDevice, sh));
    cuda_ok(cudaMemcpyAsync(rin + a * ny, rho + a * ny, w * ny * sizeof(double), cudaMemcpyHostToDevice, sh));
    cuda_ok(cudaMemcpyAsync(uin + 2 * a * ny, u + 2 * a * ny, 2 * w * ny * sizeof(double), cudaMemcpyHostToDevice, sh));
    in_ready[k] = event();
    cuda_ok(cudaEventRecord(in_ready[k], sh));
  };
  auto init = [&](int k) {
    if (st != LBM_OK) return;
    KParams P = G;
    P.xb = xs(k);
    P.xe = xs(k + 1);
    P.pop_out = pop;
    P.pitch = pitch;
    P.plane = pitch * ny;
    P.aux_out = aux;
    P.omega = omega;
    if (!cuda_ok(cudaStreamWaitEvent(sc, in_ready[k], 0))) return;
    const int e = launch_init(LBM_STORE_F64, exact, P, fin, rin, uin, sc);
    if (e != LBM_OK && st == LBM_OK) st = e;
  };
  auto read = [&](int k) {
    if (st != LBM_OK) return;
    KParams P = G;
    P.xb = xs(k);
    P.xe = xs(k + 1);
    P.pop_in = pop;
    P.aux_in = aux;
    P.pitch = pitch;
    P.plane = pitch * ny;
    const int e = launch_read(LBM_STORE_F64, exact, P, fo, ro, uo, false, sc);
    if (e != LBM_OK && st == LBM_OK) st = e;
    out_ready[k] = event();
    cuda_ok(cudaEventRecord(out_ready[k], sc));
  };
  auto download = [&](int k) {
    if (st != LBM_OK) return;
    const int64_t a = xs(k), w = xs(k + 1) - xs(k);
    cuda_ok(cudaStreamWaitEvent(sd, out_ready[k], 0));
    cuda_ok(cudaMemcpyAsync(f_out + 9 * a * ny, fo + 9 * a * ny, 9 * w * ny * sizeof(double), cudaMemcpyDeviceToHost, sd));
    cuda_ok(cudaMemcpyAsync(rho_out + a * ny, ro + a * ny, w * ny * sizeof(double), cudaMemcpyDeviceToHost, sd));
    cuda_ok(cudaMemcpyAsync(u_out + 2 * a * ny, uo + 2 * a * ny, 2 * w * ny * sizeof(double), cudaMemcpyDeviceToHost, sd));
  };
  // Read-out of slab k pulls from columns of slabs k-1 and k+1 (periodic in x),
  // so it follows their collisions.  The pressure rewrite writes columns 0 and
  // nx-1 from columns nx-2 and 1: with it, every collision runs first.  The
  // calls are issued interleaved (upload k, collide k, read out and download
  // k-1), which also keeps the host issuing work while copies from pageable
  // memory block it.
  if (g->pressure || K < 3) {
    for (int k = 0; k < K; ++k) {
      upload(k);
      init(k);
    }
    for (int k = 0; k < K; ++k) {
      read(k);
      download(k);
    }
  } else {
    upload(0);
    init(0);
    upload(1);
    init(1);
    for (int k = 2; k < K; ++k) {
      upload(k);
      init(k);
      read(k - 1);
      download(k - 1);
    }
    read(K - 1);
    download(K - 1);
    read(0);
    download(0);
  }
  // the caller's stream continues once every copy has landed
  cudaEvent_t done_h = event(), done_c = event(), done_d = event();
  cuda_ok(cudaEventRecord(done_h, sh));
  cuda_ok(cudaEventRecord(done_c, sc));
  cuda_ok(cudaEventRecord(done_d, sd));
  cuda_ok(cudaStreamWaitEvent(caller, done_h, 0));
  cuda_ok(cudaStreamWaitEvent(caller, done_c, 0));
  cuda_ok(cudaStreamWaitEvent(caller, done_d, 0));
  // streams and events are released once their work completes
  for (cudaEvent_t e : ev)
    if (e) cudaEventDestroy(e);
  if (sh) cudaStreamDestroy(sh);
  if (sc) cudaStreamDestroy(sc);
  if (sd) cudaStreamDestroy(sd);
  return st;
}

}  // extern "C"

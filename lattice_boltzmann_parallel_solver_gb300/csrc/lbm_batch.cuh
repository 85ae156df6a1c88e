// lbm_batch.cuh -- the batched step kernels and their launcher (many lattices
// of different sizes advanced together, one or two launches per time step).
// Three translation units instantiate the launcher: lbm_batch_inline.cu
// (boundary sources inside the step), lbm_batch_split.cu and lbm_batch_split16.cu
// (boundary-free step + boundary-node pass, the wider and the 16-bit storages).
#pragma once
#include <algorithm>
#include <cstddef>

#include "lbm_fused.cuh"

namespace lbm {

// Registers: the boundary-free 16-bit bodies and the one-node fixed-point body
// run at 1024 threads per SM (64 registers; the plain grid and the span walk
// keep little state across the body, 44 bytes of spill at 4 nodes per thread),
// the bodies with the boundary sources inside at 768; float32 at 2 nodes per
// thread without sources at 1024.
template <int STORE, int NPT, int THREADS, bool HAS_BC>
constexpr int batch_min_blocks() {
  if constexpr (STORE == LBM_STORE_F16S || STORE == LBM_STORE_BF16S || (STORE == LBM_STORE_FX64 && NPT == 1))
    return (HAS_BC ? 768 : 1024) / THREADS;
  else if constexpr (!HAS_BC && STORE == LBM_STORE_F32 && NPT <= 2)
    return 1024 / THREADS;
  else
    return 1;
}

// The entry's boundary constant tables (kconst, cconst: 2.3 KB of its 2.7 KB)
// are read only by the boundary sources; a body without them stages the 16-byte
// words before and after the tables.
constexpr int kEntryWords = (int)(sizeof(BatchEntry) / 16);
constexpr int kTablesFirst = (int)((offsetof(BatchEntry, P.g.kconst) + 15) / 16);  // first word inside the tables
constexpr int kTablesEnd = (int)(offsetof(BatchEntry, P.g.bcnodes) / 16);         // first word holding bytes after them
static_assert(offsetof(BatchEntry, P.g.cconst) == offsetof(BatchEntry, P.g.kconst) + sizeof(GeoK::kconst) &&
                  offsetof(BatchEntry, P.g.bcnodes) == offsetof(BatchEntry, P.g.cconst) + sizeof(GeoK::cconst),
              "the constant tables are contiguous, followed by bcnodes");

// stages lattice `lo`'s entry in the block's shared buffer (every thread of the
// block calls it with the same `lo`); TABLES: with the boundary constant tables
template <int THREADS, bool TABLES>
__device__ __forceinline__ void stage_entry(const BatchEntry* __restrict__ tab, int lo, unsigned char* ebuf) {
  static_assert(sizeof(BatchEntry) % 16 == 0, "entry copied in 16-byte words");
  __syncthreads();  // every thread is done with the previous entry
  const uint4* src = reinterpret_cast<const uint4*>(tab + lo);
  uint4* dst = reinterpret_cast<uint4*>(ebuf);
  constexpr int skip = TABLES ? 0 : kTablesEnd - kTablesFirst;
  for (int w = threadIdx.x; w < kEntryWords - skip; w += THREADS) {
    const int v = TABLES || w < kTablesFirst ? w : w + skip;
    dst[v] = __ldg(src + v);
  }
  __syncthreads();
}

// last index j in [0, n) with start[j] <= t (start ascending, start[0] == 0)
__device__ __forceinline__ int owner_of(const int* __restrict__ start, int n, int t) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(start + mid) <= t) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// One tile of lattice `e` (staged in shared memory) at global step g; SHIFT:
// the reference-shifted 16-bit storages.
template <int STORE, int NPT, int THREADS, bool HAS_BC, bool SHIFT, bool MERGED>
__device__ __forceinline__ void batch_tile(const BatchEntry& e, int local, int g) {
  const bool odd = (g - e.s0) & 1;
  const void* pin = odd ? e.pop_b : e.pop_a;
  void* pout = odd ? e.pop_a : e.pop_b;
  const void* ain = odd ? e.aux_b : e.aux_a;
  void* aout = odd ? e.aux_a : e.aux_b;
  const uint32_t seed = hash32(e.P.seed + (uint32_t)(g - e.s0));
  // with the sources inside the step, lattices without the pressure rewrite
  // take the body without it; the boundary-free body leaves the rewrite to
  // the boundary-node pass
  const bool pressure = HAS_BC && e.P.g.pressure != 0;
  // the boundary-free body applies the plain inlet / outlet columns itself
  // (EDGES), the boundary-node pass the other boundary nodes
  auto step_chunk = [&](int x0, int y, bool special) {
    if constexpr (STORE == LBM_STORE_FX64) {
      if (pressure) fused_fx_body<NPT, HAS_BC, HAS_BC, !HAS_BC, MERGED>(e.P, pin, pout, ain, aout, x0, y, special);
      else fused_fx_body<NPT, HAS_BC, false, !HAS_BC, MERGED>(e.P, pin, pout, ain, aout, x0, y, special);
    } else {
      if (pressure) fused_v2_body<STORE, NPT, HAS_BC, HAS_BC, !HAS_BC, SHIFT, MERGED>(e.P, pin, pout, ain, aout, x0, y, seed, false, special);
      else fused_v2_body<STORE, NPT, HAS_BC, false, !HAS_BC, SHIFT, MERGED>(e.P, pin, pout, ain, aout, x0, y, seed, false, special);
    }
  };
  if constexpr (HAS_BC) {
    // row-segment tiles (small batches): `rows` rows of one segment of
    // THREADS chunks; the row is uniform over the block, so its addressing
    // runs in the uniform datapath (on a lone 420x180 lattice 15 % faster
    // than runs across row ends)
    const int yb = local / e.xblocks, xb = local - yb * e.xblocks;
    const int x0 = (xb * THREADS + (int)threadIdx.x) * NPT;
    const int y1 = min((yb + 1) * e.rows, e.P.g.ny);
    for (int y = yb * e.rows; y < y1; ++y) step_chunk(x0, y, false);
  } else {
    // runs of THREADS consecutive chunks, chunks numbered row by row: no
    // idle lanes at row ends.  The lanes of a run past the lattice's last
    // chunk stay idle (x0 = nx).  The body takes x0 and y per thread: at a
    // row end inside a warp the x neighbours come by direct loads.
    for (int r = 0; r < e.rows; ++r) {
      const int c = (local * e.rows + r) * THREADS + (int)threadIdx.x;
      const int cpr = e.cpr;
      int y = (int)__umulhi((uint32_t)c, e.cpr_magic);
      int xc = c - y * cpr;
      if (xc >= cpr) {
        xc -= cpr;
        ++y;
      }
      int x0 = xc * NPT;
      if (y >= e.P.g.ny) {
        y = e.P.g.ny - 1;
        x0 = e.P.g.nx;
      }
      bool special = false;
      if constexpr (MERGED) {
        // the warp's chunks: 32 in a row from its first one, or some row end
        const int xa = __shfl_sync(0xffffffffu, x0, 0), ya = __shfl_sync(0xffffffffu, y, 0);
        special = pass_chunk(e.P.g, xa, 32 * NPT, ya);
      }
      step_chunk(x0, y, special);
    }
  }
}

constexpr int kStartSmem = 512;

// owner_of for a whole block: the start list is copied into shared memory
// (one round trip) and searched there when it has at most kStartSmem entries
template <int THREADS>
__device__ __forceinline__ int owner_of_staged(const int* __restrict__ start, int n, int t) {
  __shared__ int sstart[kStartSmem];
  if (n > kStartSmem) return owner_of(start, n, t);
  for (int j = (int)threadIdx.x; j < n; j += THREADS) sstart[j] = __ldg(start + j);
  __syncthreads();
  int a = 0, b = n - 1;
  while (a < b) {
    const int mid = (a + b + 1) >> 1;
    if (sstart[mid] <= t) a = mid;
    else b = mid - 1;
  }
  return a;
}

// The boundary-node pass of a batch, in the first bc_chunks blocks of a launch
// whose other blocks leave the pass nodes out (MERGED), or in a second launch
// that overwrites their outputs.  One thread per pass node recomputes that node
// with its sources and, under the pressure rewrite, with the rewrite (the body at
// one node per thread, the same arithmetic and random bits as the in-step
// sources).  A lattice's pass nodes are its listed
// boundary nodes other than the plain edge nodes (the boundary-free body applies
// those itself), then, under the pressure rewrite, columns 1 and nx-2 of every
// row (those not listed already), whose nodes write the rewritten populations of
// columns nx-1 and 0.  Block b takes chunk b of the chunk list: lattice j owns
// chunks [bc_start[j], bc_start[j + 1]) of THREADS pass nodes.

// Where a batch applies its boundary sources, by its nodes in total (us per
// step, inside the tiles / pass in the same launch / pass as a second launch):
//   below kBatchPassNodes inside the tiles (six 108x110 channels and the like; a
//     caller with 16-bit storages asks for it up to 2^18: 151k nodes 5.7 / 6.0)
//   from there in the same launch: six 420x180 channels fx64 21.0 / 17.3 / 24.6,
//     f16 11.6 / 8.9 / 9.8; 1.0M nodes fx64 42.4 / 34.5 / 42.4, f16 19.2 / 13.4 / 14.8
//   A launch of its own overwrites what a body free of the pass's tests stored; it
//     pays on larger batches: the 16-bit storages from 2^20 nodes (1.5M nodes f16
//     31.3 / 22.5 / 19.8, 4.8M 72 / 55 / 50), fx64 from 2^22 (2.2M channels 78 /
//     66.2 / 68.1, 4.8M 168 / 140.8 / 138.6, 20M 570 / 563 / 539), f32 from 2^23
//     (4.8M 94 / 84.6 / 84.9, 12M 182 / 178.6 / 169.8); f64 never (2.2M 297 / 262.7
//     / 270.0, 40M 4826 / 4831 / 4836).
//   Where some lattice has a wide box (small_box), whose chunks test and store node
//     by node beside the pass: inside below 2^20 nodes; from 2^21 f32 and fx64 in a
//     launch of its own (all such / every second one: f32 1.1M 21.2 / 24.3 / 23.4 and
//     23.2 / 22.5 / 23.3, 2.2M 39.1 / 47.7 / 43.3 and 40.2 / 43.4 / 43.4, 20M 268 /
//     340 / 275; fx64 1.6M 55.1 / 55.7 / 56.0, 2.2M 69.5 / 70.0 / 68.3, 20M 548 / 593 /
//     539); f64, bound by its arithmetic, in the same launch (4.8M 670 / 593 / 599).
//   Without pass nodes the body is free of the tests as well (periodic, same launch's
//     body / free one: fx64 20M 560 / 532, f32 12M 172 / 161, f16 0.9M 11.9 / 10.7).
constexpr int64_t kBatchPassNodes = (int64_t)1 << 17, kBatchSplitNodes = (int64_t)1 << 20;

// A batch's boundary-node plan, from lbm_batch_build to lbm_batch_run: the chunks of
// pass nodes, whether some lattice has a wide box, and the size class of the nodes in
// total (0 below 2^20, k below 2^(20 + k), 7 above).
constexpr int kPlanWide = 1 << 27, kPlanSizeShift = 28;
inline int plan_size(int64_t nodes) {
  int k = 0;
  while (k < 7 && nodes >= kBatchSplitNodes << k) ++k;
  return k;
}
// first size class whose pass is a launch of its own (8: none)
template <int STORE>
constexpr int apart_from(bool wide) {
  if (Store<STORE>::kShifted) return 1;
  if (STORE == LBM_STORE_F64) return 8;
  return wide ? 2 : (STORE == LBM_STORE_FX64 ? 3 : 4);
}

inline int64_t pass_nodes(const GeoK& g) {
  return (g.bcmask != nullptr ? (int64_t)(g.n_bcnodes - g.n_bcnodes_edge) : 0) + (g.pressure ? 2 * (int64_t)g.ny : 0);
}

template <int STORE, int THREADS, bool SHIFT>
__device__ __forceinline__ void batch_pass(const BatchEntry* __restrict__ tab, const int* __restrict__ bc_start,
                                           int n_inst, const int* __restrict__ gbase, int k, unsigned char* ebuf) {
  const BatchEntry& e = *reinterpret_cast<const BatchEntry*>(ebuf);
  const int g = *gbase + k;
  const int j = owner_of_staged<THREADS>(bc_start, n_inst, (int)blockIdx.x);
  stage_entry<THREADS, true>(tab, j, ebuf);
  pdl_wait();  // the table and the global step are not written during a run
  if (g < e.s0 || g >= e.s_end) return;
  const int t = ((int)blockIdx.x - __ldg(bc_start + j)) * THREADS + (int)threadIdx.x;
  const int nx = e.P.g.nx;
  const int listed = e.P.g.bcmask != nullptr ? e.P.g.n_bcnodes - e.P.g.n_bcnodes_edge : 0;
  int x, y;
  if (t < listed) {
    const int node = __ldg(e.P.g.bcnodes + t);
    y = node / nx;
    x = node - y * nx;
  } else {
    // a pressure column node: (1, y) for even q, (nx-2, y) for odd q
    const int q = t - listed;
    if (!e.P.g.pressure || q >= 2 * e.P.g.ny) return;
    y = q >> 1;
    x = (q & 1) ? nx - 2 : 1;
    if ((q & 1) && nx - 2 == 1) return;  // one column: its even entry covers it
    if (e.P.g.bcmask != nullptr && ((__ldg(e.P.g.bcmask + y * e.P.g.words + (x >> 5)) >> (x & 31)) & 1u) &&
        !plain_edge_node(e.P, x, y))
      return;  // listed already
  }
  const bool odd = (g - e.s0) & 1;
  const void* pin = odd ? e.pop_b : e.pop_a;
  void* pout = odd ? e.pop_a : e.pop_b;
  const void* ain = odd ? e.aux_b : e.aux_a;
  void* aout = odd ? e.aux_a : e.aux_b;
  if constexpr (STORE == LBM_STORE_FX64) {
    if (e.P.g.pressure) fused_fx_body<1, true, true>(e.P, pin, pout, ain, aout, x, y);
    else fused_fx_body<1, true, false>(e.P, pin, pout, ain, aout, x, y);
  } else {
    const uint32_t seed = hash32(e.P.seed + (uint32_t)(g - e.s0));
    const bool in_list = t < listed;
    if (e.P.g.pressure)
      fused_v2_body<STORE, 1, true, true, false, SHIFT>(e.P, pin, pout, ain, aout, x, y, seed, in_list);
    else
      fused_v2_body<STORE, 1, true, false, false, SHIFT>(e.P, pin, pout, ain, aout, x, y, seed, in_list);
  }
}

// The persistent form: block b walks the contiguous span of tiles
// [b T / B, (b + 1) T / B) (T tiles, B blocks), so consecutive tiles mostly
// belong to one lattice: the owner search and the entry staging happen once per
// lattice the span touches, not once per tile, and the spans differ by at most
// one tile (no tail of partly filled waves).
template <int STORE, int NPT, int THREADS, bool HAS_BC, bool SHIFT, bool MERGED>
__global__ void __launch_bounds__(THREADS, batch_min_blocks<STORE, NPT, THREADS, HAS_BC>())
    batch_kernel(const BatchEntry* __restrict__ tab, const int* __restrict__ tile_start, int n_inst,
                 int total_tiles, const int* __restrict__ bc_start, int bc_chunks, const int* __restrict__ gbase,
                 int k) {
  // the current lattice's entry, staged in shared memory: the body reads its
  // parameters many times per tile, and in global memory the streaming
  // population traffic would evict them from L1
  __shared__ __align__(16) unsigned char ebuf[sizeof(BatchEntry)];
  const BatchEntry& e = *reinterpret_cast<const BatchEntry*>(ebuf);
  if (MERGED && (int)blockIdx.x < bc_chunks) {
    batch_pass<STORE, THREADS, SHIFT>(tab, bc_start, n_inst, gbase, k, ebuf);
    return;
  }
  const int blocks = (int)gridDim.x - bc_chunks, b = (int)blockIdx.x - bc_chunks;
  const int per = total_tiles / blocks, extra = total_tiles % blocks;
  const int t0 = b * per + min(b, extra), t1 = t0 + per + (b < extra ? 1 : 0);
  if (t0 >= t1) {
    pdl_wait();
    return;
  }
  const int g = *gbase + k;
  int lo = owner_of(tile_start, n_inst, t0);
  int first = __ldg(tile_start + lo);
  int next = lo + 1 < n_inst ? __ldg(tile_start + lo + 1) : total_tiles;
  stage_entry<THREADS, HAS_BC>(tab, lo, ebuf);
  pdl_wait();  // the table and the global step are not written during a run
  for (int tile = t0; tile < t1; ++tile) {
    if (tile >= next) {
      do {
        ++lo;
        first = next;
        next = lo + 1 < n_inst ? __ldg(tile_start + lo + 1) : total_tiles;
      } while (tile >= next);
      stage_entry<THREADS, HAS_BC>(tab, lo, ebuf);
    }
    if (g >= e.s0 && g < e.s_end) batch_tile<STORE, NPT, THREADS, HAS_BC, SHIFT, MERGED>(e, tile - first, g);
  }
}

// The plain-grid form (one tile per block).  The block copies the lattices' tile
// starts into shared memory (one round trip) and finds its lattice there, instead
// of a search through global memory (a dependent L2 round trip per halving).
template <int STORE, int NPT, int THREADS, bool HAS_BC, bool SHIFT, bool MERGED>
__global__ void __launch_bounds__(THREADS, batch_min_blocks<STORE, NPT, THREADS, HAS_BC>())
    batch_grid_kernel(const BatchEntry* __restrict__ tab, const int* __restrict__ tile_start, int n_inst,
                      const int* __restrict__ bc_start, int bc_chunks, const int* __restrict__ gbase, int k) {
  __shared__ __align__(16) unsigned char ebuf[sizeof(BatchEntry)];
  const BatchEntry& e = *reinterpret_cast<const BatchEntry*>(ebuf);
  if (MERGED && (int)blockIdx.x < bc_chunks) {
    batch_pass<STORE, THREADS, SHIFT>(tab, bc_start, n_inst, gbase, k, ebuf);
    return;
  }
  const int tile = (int)blockIdx.x - bc_chunks;
  const int lo = owner_of_staged<THREADS>(tile_start, n_inst, tile);
  stage_entry<THREADS, HAS_BC>(tab, lo, ebuf);
  const int g = *gbase + k;
  pdl_wait();  // the table and the global step are not written during a run
  if (g < e.s0 || g >= e.s_end) return;
  batch_tile<STORE, NPT, THREADS, HAS_BC, SHIFT, MERGED>(e, tile - __ldg(tile_start + lo), g);
}

// the pass as a launch of its own (64 registers; the fixed-point body would spill)
template <int STORE, int THREADS, bool SHIFT>
__global__ void __launch_bounds__(THREADS, STORE == LBM_STORE_FX64 ? 1 : 1024 / THREADS)
    batch_fixup_kernel(const BatchEntry* __restrict__ tab, const int* __restrict__ bc_start, int n_inst,
                       const int* __restrict__ gbase, int k) {
  __shared__ __align__(16) unsigned char ebuf[sizeof(BatchEntry)];
  batch_pass<STORE, THREADS, SHIFT>(tab, bc_start, n_inst, gbase, k, ebuf);
}

// one copy per translation unit (each unit launches its own)
static __global__ void batch_advance_kernel(int* gbase, int k) { *gbase += k; }

template <int STORE, int NPT, int THREADS, bool HAS_BC, bool SHIFT, bool MERGED>
inline int launch_batch_form(const void* table, int n, int tiles, int bc_chunks, int* gbase, int nsteps, int blocks,
                        cudaStream_t s) {
  // the entries with float64 boundary constants, then with fixed-point ones
  const BatchEntry* tab = static_cast<const BatchEntry*>(table) + (STORE == LBM_STORE_FX64 ? n : 0);
  const int* start = reinterpret_cast<const int*>(static_cast<const char*>(table) + 2 * (size_t)n * sizeof(BatchEntry));
  const int* bc_start = start + n;
  if (blocks <= 0) {
    // resident blocks of this kernel on the whole GPU, queried on the first
    // call (make that call outside stream capture) and reused afterwards
    static int fill = 0;
    if (fill == 0) {
      int per_sm = 0, sms = 0, dev = 0;
      cudaGetDevice(&dev);
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_kernel<STORE, NPT, THREADS, HAS_BC, SHIFT, MERGED>,
                                                    THREADS, 0);
      fill = std::max(1, sms * std::max(1, per_sm));
    }
    blocks = fill;
  }
  // a grid of more than half the tile count is a plain grid of one tile per
  // block; otherwise persistent blocks walk contiguous spans of tiles
  const bool plain = (int64_t)blocks * 2 > (int64_t)tiles;
  blocks = std::min(blocks, std::max(1, tiles));
  const int pass = MERGED ? bc_chunks : 0;
  const bool overlap =
      plain && tiles > 0
          ? overlaps<STORE, batch_grid_kernel<STORE, NPT, THREADS, HAS_BC, SHIFT, MERGED>>((int64_t)pass + tiles, THREADS)
          : overlaps<STORE, batch_kernel<STORE, NPT, THREADS, HAS_BC, SHIFT, MERGED>>((int64_t)pass + blocks, THREADS);
  for (int k = 0; k < nsteps; ++k) {
    if (plain && tiles > 0) {
      launch_step(batch_grid_kernel<STORE, NPT, THREADS, HAS_BC, SHIFT, MERGED>, dim3((unsigned)(pass + tiles)), THREADS,
                  k > 0 && overlap, s, 0, tab, start, n, bc_start, pass, (const int*)gbase, k);
      count_launch();
      if (int e = check_launch("batch_grid_kernel")) return e;
    } else {
      launch_step(batch_kernel<STORE, NPT, THREADS, HAS_BC, SHIFT, MERGED>, dim3((unsigned)(pass + blocks)), THREADS,
                  k > 0 && overlap, s, 0, tab, start, n, tiles, bc_start, pass, (const int*)gbase, k);
      count_launch();
      if (int e = check_launch("batch_kernel")) return e;
    }
    if (!HAS_BC && !MERGED && bc_chunks > 0) {
      launch_step(batch_fixup_kernel<STORE, THREADS, SHIFT>, dim3((unsigned)bc_chunks), THREADS, true, s, 0, tab, bc_start,
                  n, (const int*)gbase, k);
      count_launch();
      if (int e = check_launch("batch_fixup_kernel")) return e;
    }
  }
  batch_advance_kernel<<<1, 1, 0, s>>>(gbase, nsteps);
  count_launch();
  return check_launch("batch_advance_kernel");
}


template <int STORE, int NPT, int THREADS, bool HAS_BC, bool SHIFT = false>
inline int launch_batch(const void* table, int n, int tiles, int bc_chunks, int* gbase, int nsteps, int blocks,
                        cudaStream_t s) {
  if constexpr (HAS_BC) {
    return launch_batch_form<STORE, NPT, THREADS, true, SHIFT, false>(table, n, tiles, 0, gbase, nsteps, blocks, s);
  } else {
    const int chunks = bc_chunks & (kPlanWide - 1), size = bc_chunks >> kPlanSizeShift;
    if constexpr (apart_from<STORE>(true) < 8)
      if (chunks == 0 || size >= apart_from<STORE>((bc_chunks & kPlanWide) != 0))
        return launch_batch_form<STORE, NPT, THREADS, false, SHIFT, false>(table, n, tiles, chunks, gbase, nsteps, blocks, s);
    return launch_batch_form<STORE, NPT, THREADS, false, SHIFT, true>(table, n, tiles, chunks, gbase, nsteps, blocks, s);
  }
}

// dispatch over (storage, npt, threads) to launch_batch<..., HAS_BC>; split16: the
// 16-bit storages (a translation unit of their own)
int batch_launch_inline(const void* table, int n, int tiles, int bc_chunks, int storage, int npt, int threads,
                        int* gbase, int nsteps, int blocks, cudaStream_t s);
int batch_launch_split(const void* table, int n, int tiles, int bc_chunks, int storage, int npt, int threads,
                       int* gbase, int nsteps, int blocks, cudaStream_t s);
int batch_launch_split16(const void* table, int n, int tiles, int bc_chunks, int storage, int npt, int threads,
                         int* gbase, int nsteps, int blocks, cudaStream_t s);

#define LBM_BATCH_DISPATCH_WIDE(HAS_BC)   \
  LBM_BATCH_NPT(LBM_STORE_F64, 2, HAS_BC)  \
  LBM_BATCH_NPT(LBM_STORE_F64, 4, HAS_BC)  \
  LBM_BATCH_NPT(LBM_STORE_FX64, 1, HAS_BC) \
  LBM_BATCH_NPT(LBM_STORE_FX64, 2, HAS_BC) \
  LBM_BATCH_NPT(LBM_STORE_F32, 2, HAS_BC)  \
  LBM_BATCH_NPT(LBM_STORE_F32, 4, HAS_BC)
#define LBM_BATCH_DISPATCH_16(HAS_BC)                      \
  LBM_BATCH_NPT(LBM_STORE_F16S, 2, HAS_BC)                 \
  LBM_BATCH_NPT(LBM_STORE_F16S, 4, HAS_BC)                 \
  LBM_BATCH_NPT(LBM_STORE_F16S, 8, HAS_BC)                 \
  LBM_BATCH_NPT(LBM_STORE_BF16S, 2, HAS_BC)                \
  LBM_BATCH_NPT(LBM_STORE_BF16S, 4, HAS_BC)                \
  LBM_BATCH_NPT(LBM_STORE_BF16S, 8, HAS_BC)                \
  LBM_BATCH_REF(LBM_STORE_F16R, LBM_STORE_F16S, 2, HAS_BC)   \
  LBM_BATCH_REF(LBM_STORE_F16R, LBM_STORE_F16S, 4, HAS_BC)   \
  LBM_BATCH_REF(LBM_STORE_BF16R, LBM_STORE_BF16S, 2, HAS_BC) \
  LBM_BATCH_REF(LBM_STORE_BF16R, LBM_STORE_BF16S, 4, HAS_BC)
inline int no_batch_kernel() {
  return set_error(LBM_ERR_UNSUPPORTED, "no batched kernel for this storage / npt / threads");
}
#define LBM_BATCH_CASE(ST, NP, TH, HAS_BC)               \
  if (storage == ST && npt == NP && threads == TH)       \
    return launch_batch<ST, NP, TH, HAS_BC>(table, n, tiles, bc_chunks, gbase, nsteps, blocks, s);
// the reference-shifted storages: 128 threads only
#define LBM_BATCH_REF(ST, BASE, NP, HAS_BC)                  \
  if (storage == ST && npt == NP && threads == 128)          \
    return launch_batch<BASE, NP, 128, HAS_BC, true>(table, n, tiles, bc_chunks, gbase, nsteps, blocks, s);
#define LBM_BATCH_NPT(ST, NP, HAS_BC) \
  LBM_BATCH_CASE(ST, NP, 64, HAS_BC) LBM_BATCH_CASE(ST, NP, 128, HAS_BC) LBM_BATCH_CASE(ST, NP, 256, HAS_BC)

}  // namespace lbm

// lbm_tile.cuh -- several fused steps per launch on one tile of a lattice.
//
// A one-step launch takes 2.2 us (periodic) to 5 us (boundary nodes) whatever
// the lattice's size: launch, load and store latency, and the chain of
// dependent operations of one node.  A lattice of up to a few hundred thousand
// nodes is bound by them.  Here each block takes a tile of the lattice through
// K steps: it pulls the tile and a halo of K - 1 nodes from L2, keeps the
// populations of the steps between in shared memory, where the computed region
// shrinks by one node per side and step, and writes the tile back at step K.
// Neighbouring blocks compute the overlap twice instead of waiting for one
// another, so no block ever waits for a block.  What bounds it now is latency on
// the smallest lattices (64^2 fx64: 1.1 us a step, of which one node's chain 0.6 and
// the launch's 1.7 us over five steps 0.3) and the issue rate above (half of the issue
// slots used on 420x180).
//
// Measured, us per step, one-step launches -> this: 64^2 fx64 2.2 -> 1.25
// (1.1 in runs of 2000), f64 6.5 -> 3.0, f32 2.5 -> 0.85, f16 2.4 -> 1.05; 420x180
// channel fx64 5.8 -> 3.9, f64 16.3 -> 14.4, f32 5.1 -> 2.5, f16 5.5 -> 2.8; 512^2 cavity
// f32 6.3 -> 3.7, f16 5.8 -> 4.8; 800x640 cavity f16 8.6 -> 7.2.
//
// Arithmetic, boundary sources, outlet memory, pressure rewrite, probe and
// random bits are those of fused_v2_body / fused_fx_body, node for node: the
// results are the same bits as K one-step launches.
#pragma once
#include <type_traits>

#include "lbm_fused.cuh"

namespace lbm {

// One tile's place in the lattice: nodes [x0, x0 + tx) x [y0, y0 + ty) are
// written at the last step.
struct TileRect {
  int x0, y0, tx, ty;
};

// nodes per thread: the 16-bit storages collide two nodes per instruction
template <int STORE>
constexpr int tile_npt() {
  return Store<STORE>::kShifted ? 2 : 1;
}

// halo columns of the first step: one per further step, and two more under the
// pressure rewrite, which moves values by two columns once on their way round
// the periodic boundary (column nx-2 to 0, column 1 to nx-1)
__host__ __device__ constexpr int tile_margin_x(int ksteps, bool pressure) { return ksteps - 1 + (pressure ? 2 : 0); }

// Shared memory of a region of h rows of at most WC columns.  Two buffers of
// rows, each row its nine populations one after another with the pitch WC (a
// compile-time number, so that every access of a node is one address and an
// immediate offset), with 16 spare bytes before and after them for a pair at
// the region's edge; the constants of the boundary sources in working values;
// the outlet memory of two steps; the wrapped rows; the descriptors.
template <int STORE, int WC>
struct TileShared {
  using T = typename Store<STORE>::T;
  using A = typename Store<STORE>::A;
  using V = std::conditional_t<STORE == LBM_STORE_FX64, T, typename Store<STORE>::R>;
  static constexpr int kRow = 9 * WC;  // elements per row
  __host__ __device__ static constexpr size_t pops(int h) { return 32 + 2 * (size_t)h * kRow * sizeof(T); }
  __host__ __device__ static constexpr size_t consts() { return 2 * 9 * LBM_MAX_SETS * sizeof(V); }
  __host__ __device__ static constexpr size_t aux(int h) { return (6 * (size_t)h * sizeof(A) + 15) / 16 * 16; }
  __host__ __device__ static constexpr size_t bytes(int h) {
    return pops(h) + consts() + aux(h) + (size_t)(h + 2) * 4 + (size_t)h * WC * 4;
  }
};

__device__ __forceinline__ int wrap(int v, int n) {
  v %= n;
  return v < 0 ? v + n : v;
}

template <int STORE, bool SHIFT, int WC, bool HAS_BC, bool HAS_PRESSURE>
__device__ __forceinline__ void tile_body(const KParams& P, const void* pop_in_v, void* pop_out_v,
                                          const void* aux_in_v, void* aux_out_v, const TileRect t, int ksteps,
                                          uint32_t seed0, unsigned char* smem) {
  using St = Store<STORE>;
  using T = typename St::T;
  using R = typename St::R;
  using A = typename St::A;
  using Sh = TileShared<STORE, WC>;
  // working values: the stored integers (fixed point), the stored scaled
  // deviations (16-bit storages), f otherwise
  using V = typename Sh::V;
  constexpr bool SH = St::kShifted;
  constexpr bool FX = STORE == LBM_STORE_FX64;
  constexpr int NPT = tile_npt<STORE>();
  constexpr int kUnits = WC / NPT;  // threads per row
  constexpr int kRow = Sh::kRow;
  constexpr R kS = [] {
    if constexpr (SH) return (R)St::kDev;
    else return R(1);
  }();
  const int nx = P.g.nx, ny = P.g.ny;
  const int pitch = (int)P.pitch, plane = (int)P.plane;
  const int mx = tile_margin_x(ksteps, HAS_PRESSURE), my = ksteps - 1;
  const int w = (t.tx + 2 * mx + NPT - 1) / NPT * NPT, h = t.ty + 2 * my;

  T* const pops = reinterpret_cast<T*>(smem + 16);
  unsigned char* sp = smem + Sh::pops(h);
  V* const skc = reinterpret_cast<V*>(sp);  // moving-wall terms, then fixed populations
  V* const scc = skc + 9 * LBM_MAX_SETS;
  sp += Sh::consts();
  A* const saux = reinterpret_cast<A*>(sp);
  sp += Sh::aux(h);
  int* const sgy = reinterpret_cast<int*>(sp) + 1;  // [-1, h]
  uint32_t* const sdesc = reinterpret_cast<uint32_t*>(sgy + h + 1);
  const int tid = (int)threadIdx.x, nthr = (int)blockDim.x;

  const ShiftK& shk = P.shf[STORE == LBM_STORE_F16S ? 0 : 1];
  auto work_of_raw = [&](T v, int i) -> V {
    if constexpr (FX) return v;
    else if constexpr (SH) return St::dev(v);
    else return St::to_r(v, i);
  };
  auto sig = [&](int i) -> R {
    if constexpr (SHIFT) return shk.sig[i];
    else return R(0);
  };
  // a population given in float64 (inlet, constants) or read from the outlet memory
  auto work_of_f = [&](R fv, int i) -> V {
    if constexpr (FX) return fx::to_fx(fv, wd(i));
    else if constexpr (SHIFT) return fma(fv - wr<R>(i), kS, -sig(i));
    else return SH ? (fv - wr<R>(i)) * kS : fv;
  };
  auto work_of_aux = [&](A a, int i) -> V {
    if constexpr (FX) return a;
    else return work_of_f(a, i);
  };
  auto aux_of_work = [&](V v, int i) -> A {
    if constexpr (FX) return v;
    else if constexpr (SHIFT) return fma(v + sig(i), R(1) / kS, wr<R>(i));
    else return SH ? fma(v, R(1) / kS, wr<R>(i)) : v;
  };

  // a thread keeps its columns through all steps: lx ... lx + NPT - 1 of the region
  const int lx = (tid % kUnits) * NPT, row0 = tid / kUnits, rows_at_once = nthr / kUnits;
  int xs[NPT + 2];  // wrapped columns lx - 1 ... lx + NPT
#pragma unroll
  for (int k = 0; k < NPT + 2; ++k) xs[k] = wrap(t.x0 - mx + lx - 1 + k, nx);
  for (int j = tid; j < h + 2; j += nthr) sgy[j - 1] = wrap(t.y0 - my + j - 1, ny);
  bool any_bc = false;
  if (HAS_BC && P.g.bcmask != nullptr) {
    // descriptors (mask and descriptor load together; the descriptor counts
    // where the mask's bit is set), and the source constants in working values
    if (lx < w) {
      for (int ly = row0; ly < h; ly += rows_at_once) {
        const int y = wrap(t.y0 - my + ly, ny);
#pragma unroll
        for (int k = 0; k < NPT; ++k) {
          const int x = xs[k + 1];
          const uint32_t m = __ldg(P.g.bcmask + y * P.g.words + (x >> 5)), dd = __ldg(P.g.desc + y * nx + x);
          const uint32_t d = (m >> (x & 31)) & 1u ? dd : 0u;
          sdesc[ly * WC + lx + k] = d;
          any_bc |= (d & 0x3FFFFu) != 0u;
        }
      }
    }
    for (int j = tid; j < 9 * LBM_MAX_SETS; j += nthr) {
      const int set = j / 9, i = j - 9 * set;
      if constexpr (FX) {  // fixed point already (set_fx_tables)
        skc[j] = __double_as_longlong(P.g.kconst[set][i]);
        scc[j] = __double_as_longlong(P.g.cconst[set][i]);
      } else {
        skc[j] = (R)P.g.kconst[set][i] * kS;
        scc[j] = work_of_f((R)P.g.cconst[set][i], i);
      }
    }
    // tiles away from every boundary skip the sources altogether
    any_bc = __syncthreads_or(any_bc);
  } else {
    __syncthreads();
  }
  // everything above reads the geometry only; the populations, the outlet
  // memory, the step counter and the probe's count are the previous launch's
  pdl_wait();

  const T* const pin = static_cast<const T*>(pop_in_v);
  T* const pout = static_cast<T*>(pop_out_v);
  const A* const aux_in = static_cast<const A*>(aux_in_v);
  A* const aux_out = static_cast<A*>(aux_out_v);
  if (P.step_dev != nullptr) seed0 += (uint32_t)*static_cast<const volatile int32_t*>(P.step_dev);
  bool own_col[NPT], aux_col = false;
  int probe_row[NPT], probe0 = 0;  // the probe's row in the region in its column's thread
#pragma unroll
  for (int k = 0; k < NPT; ++k) {
    own_col[k] = (unsigned)(lx + k - mx) < (unsigned)t.tx;
    aux_col |= aux_out != nullptr && xs[k + 1] == nx - 2;
    const bool here = P.probe_buf != nullptr && own_col[k] && xs[k + 1] == P.probe_x &&
                      (unsigned)(P.probe_y - t.y0) < (unsigned)t.ty;
    probe_row[k] = here ? P.probe_y - t.y0 + my : -1;
    if (here) probe0 = *static_cast<const volatile int*>(P.probe_count);
  }
  const bool sr = SH && P.sr;
  const bool pressure = HAS_PRESSURE && P.g.pressure != 0;
  const R omega = (R)P.omega;
  auto to_store = [&](V v, int i, uint32_t rbits) -> T {
    if constexpr (FX) return v;
    else if constexpr (SH) return sr ? St::dev_sr(v, rbits) : St::dev_rn(v);
    else return St::from_r(v, i);
  };
  // offset of the population that direction i pulls, from the node's own
  // population 0 in the shared buffer
  auto pull = [](int i) constexpr { return (i - 9 * cy(i)) * WC - cx(i); };

  const T* src = pops + h * kRow;
  T* dst = pops;
  for (int s = 0; s < ksteps; ++s) {
    const bool first = s == 0, last = s == ksteps - 1;
    // region of this step: one node less per side (whole pairs of columns)
    const int lo = s / NPT * NPT, ylo = last ? my : s;
    const bool act = last ? lx + NPT > mx && lx < mx + t.tx : lx >= lo && lx < w - lo;
    const uint32_t seed = SH ? hash32(seed0 + (uint32_t)s) : 0u;
    for (int ly = act ? ylo + row0 : h; ly < h - ylo; ly += rows_at_once) {
      const int at = ly * kRow + lx;  // the node's population 0
      int y = 0;
      if (first || last || SH) y = sgy[ly];
      uint32_t d[NPT] = {};
      uint32_t dany = 0u;
      if (HAS_BC && any_bc) {
#pragma unroll
        for (int k = 0; k < NPT; ++k) {
          d[k] = sdesc[ly * WC + lx + k];
          dany |= d[k] & 0x3FFFFu;
        }
      }
      V f[9][NPT];
      if (first) {
        const int r0 = y * pitch, rm = sgy[ly - 1] * pitch, rp = sgy[ly + 1] * pitch;
#pragma unroll
        for (int i = 0; i < 9; ++i) {
          const int row = cy(i) == 1 ? rm : (cy(i) == -1 ? rp : r0);
#pragma unroll
          for (int k = 0; k < NPT; ++k) {
            int p = i * plane + row + xs[k + 1 - cx(i)];
            // bounce-back reads the node's own opposite population instead
            if (HAS_BC && ((d[k] >> (2 * i)) & 3u) == LBM_SRC_BOUNCE) p = opp(i) * plane + r0 + xs[k + 1];
            f[i][k] = work_of_raw(pin[p], i);
          }
        }
      } else if (HAS_BC && dany != 0u) {
#pragma unroll
        for (int i = 0; i < 9; ++i) {
#pragma unroll
          for (int k = 0; k < NPT; ++k)
            f[i][k] = work_of_raw(
                src[at + k + (((d[k] >> (2 * i)) & 3u) == LBM_SRC_BOUNCE ? opp(i) * WC : pull(i))], i);
        }
      } else {
#pragma unroll
        for (int i = 0; i < 9; ++i) {
          const T* p = src + at + pull(i);
          if constexpr (NPT == 2) {
            if (cx(i) == 0) {
              T pr[2];
              memcpy(pr, __builtin_assume_aligned(p, 4), 4);
              f[i][0] = work_of_raw(pr[0], i);
              f[i][1] = work_of_raw(pr[1], i);
              continue;
            }
          }
#pragma unroll
          for (int k = 0; k < NPT; ++k) f[i][k] = work_of_raw(p[k], i);
        }
      }

      if (HAS_BC && dany != 0u) {
#pragma unroll
        for (int k = 0; k < NPT; ++k) {
          const V* kc = skc + 9 * ((d[k] >> LBM_DESC_KSET_SHIFT) & 15u);
#pragma unroll
          for (int i = 0; i < 9; ++i) {
            if (((d[k] >> (2 * i)) & 3u) != LBM_SRC_BOUNCE) continue;
            f[i][k] -= kc[i];
            if constexpr (SHIFT) f[i][k] += sig(opp(i)) - sig(i);
          }
          if ((d[k] & 0x2AAAAu) == 0u) continue;  // no fixed population, no outlet
          const V* cc = scc + 9 * ((d[k] >> LBM_DESC_CSET_SHIFT) & 15u);
          const int yy = sgy[ly];
#pragma unroll
          for (int i = 0; i < 9; ++i) {
            const uint32_t sc = (d[k] >> (2 * i)) & 3u;
            if (sc == LBM_SRC_CONST)
              f[i][k] = cc[i];
            else if (sc == LBM_SRC_OUTLET && outlet_slot(i) >= 0 && aux_in != nullptr)
              f[i][k] = work_of_aux(first ? aux_in[outlet_slot(i) * ny + yy]
                                          : saux[((s + 1) & 1) * 3 * h + outlet_slot(i) * h + ly], i);
          }
        }
      }

      // outlet memory of the next step: full populations (integers in fixed point)
      if (aux_col) {
#pragma unroll
        for (int k = 0; k < NPT; ++k) {
          if (xs[k + 1] != nx - 2) continue;
          const A a3 = aux_of_work(f[3][k], 3), a6 = aux_of_work(f[6][k], 6), a7 = aux_of_work(f[7][k], 7);
          if (!last) {
            A* a = saux + (s & 1) * 3 * h + ly;
            a[0] = a3;
            a[h] = a6;
            a[2 * h] = a7;
          } else if (own_col[k]) {
            aux_out[y] = a3;
            aux_out[ny + y] = a6;
            aux_out[2 * ny + y] = a7;
          }
        }
      }

      // collision; velocity at the probe's node, pressure rewrite
      auto probe = [&](double ux, double uy) {
        const int q = probe0 + s;
        if (q < P.probe_cap) {
          P.probe_buf[2 * q] = ux;
          P.probe_buf[2 * q + 1] = uy;
        }
        if (last) *P.probe_count = q + 1;
      };
      auto probed = [&](int k) { return ly == probe_row[k]; };
      auto pressure_node = [&](int k) { return pressure && (xs[k + 1] == nx - 2 || xs[k + 1] == 1); };
      auto rho_target = [&](int k) { return xs[k + 1] == nx - 2 ? P.g.rho_in : P.g.rho_out; };
      // the rewritten populations pv of column 0 (from column nx-2) or nx-1 (from column 1)
      auto rewrite = [&](int k, const V pv[9]) {
        const bool in = xs[k + 1] == nx - 2;
        const uint32_t dirs = in ? P.g.pin : P.g.pout;
        const int dcol = in ? 0 : nx - 1, dlx = lx + k + (in ? 2 : -2);
        if (last ? !own_col[k] : (unsigned)dlx >= (unsigned)w) return;
        uint32_t hp = sr ? mix32((uint32_t)(y * nx + dcol) * 0x9E3779B1u ^ seed ^ 0x5bd1e995u) : 0u;
#pragma unroll
        for (int i = 0; i < 9; ++i) {
          if ((dirs >> i) & 1u) {
            const T v = to_store(pv[i], i, hp);
            if (last) pout[i * plane + y * pitch + dcol] = v;
            else dst[ly * kRow + i * WC + dlx] = v;
          }
          hp = hp * 0x2C1B3C6Du + 0x297A2D39u;
        }
      };
      auto float_extras = [&](int k, R rho, R ux, R uy, const R g[9]) {
        if constexpr (!FX) {
          if (probed(k)) probe((double)ux, (double)uy);
          if (pressure_node(k)) {
            R br[9], pv[9];
            bracket9_fast(ux, uy, br);
            const R rb = (R)rho_target(k) * kS - rho;
#pragma unroll
            for (int i = 0; i < 9; ++i) pv[i] = fma(wr<R>(i) * br[i], rb, g[i]);
            rewrite(k, pv);
          }
        }
      };
      if constexpr (FX) {
        int64_t g[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) g[i] = f[i][0];
        if (probed(0)) {
          double e[9], ux, uy;
#pragma unroll
          for (int i = 0; i < 9; ++i) e[i] = fx::from_fx(g[i], wd(i));
          velocity_fast(e, density9(e), ux, uy);
          probe(ux, uy);
        }
        if (pressure_node(0)) {
          int64_t q[9];
          V pv[9];
          fx_pressure_node(g, q, P, xs[1] == nx - 2);
#pragma unroll
          for (int i = 0; i < 9; ++i) pv[i] = q[i];
          rewrite(0, pv);
        } else {
          fx_collide_node(g, P.qc, P.omega);
        }
#pragma unroll
        for (int i = 0; i < 9; ++i) f[i][0] = g[i];
      } else if constexpr (SH) {
        float2 g2[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) g2[i] = make_float2(f[i][0], f[i][NPT - 1]);
        float2 sum, rho, ux, uy;
        collide_pair<SHIFT>(g2, sum, rho, ux, uy, omega, kS, shk);
        R ga[9], gb[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) {
          ga[i] = g2[i].x;
          gb[i] = g2[i].y;
          f[i][0] = ga[i];
          f[i][NPT - 1] = gb[i];
        }
        float_extras(0, rho.x, ux.x, uy.x, ga);
        float_extras(NPT - 1, rho.y, ux.y, uy.y, gb);
      } else {
        R g[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) g[i] = f[i][0];
        R rho, ux, uy;
        collide_node(g, rho, ux, uy, omega);
        float_extras(0, rho, ux, uy, g);
#pragma unroll
        for (int i = 0; i < 9; ++i) f[i][0] = g[i];
      }

      // stored numbers, then to the tile or to the shared buffer
      T out[9][NPT];
      if constexpr (SH) {
        uint32_t hk[NPT];
#pragma unroll
        for (int k = 0; k < NPT; ++k) hk[k] = sr ? mix32((uint32_t)(y * nx + xs[k + 1]) * 0x9E3779B1u ^ seed) : 0u;
#pragma unroll
        for (int i = 0; i < 9; ++i) {
#pragma unroll
          for (int k = 0; k < NPT; ++k) {
            out[i][k] = to_store(f[i][k], i, hk[k]);
            hk[k] = hk[k] * 0x2C1B3C6Du + 0x297A2D39u;
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < 9; ++i) out[i][0] = to_store(f[i][0], i, 0u);
      }
      // column 0 / nx-1 leave the rewritten directions to column nx-2 / 1 (inside
      // a region where that one is computed)
      uint32_t skip[NPT];
#pragma unroll
      for (int k = 0; k < NPT; ++k) {
        skip[k] = 0u;
        if (pressure && xs[k + 1] == 0 && (last || lx + k - 2 >= lo)) skip[k] |= P.g.pin;
        if (pressure && xs[k + 1] == nx - 1 && (last || lx + k + 2 < w - lo)) skip[k] |= P.g.pout;
      }
      if (!last) {
        if constexpr (NPT == 2) {
          if (!HAS_PRESSURE || (skip[0] | skip[1]) == 0u) {
#pragma unroll
            for (int i = 0; i < 9; ++i) memcpy(__builtin_assume_aligned(dst + at + i * WC, 4), out[i], 4);
            continue;
          }
        }
#pragma unroll
        for (int i = 0; i < 9; ++i) {
#pragma unroll
          for (int k = 0; k < NPT; ++k)
            if (!HAS_PRESSURE || !((skip[k] >> i) & 1u)) dst[at + i * WC + k] = out[i][k];
        }
      } else {
        T* const po = pout + y * pitch;
        if constexpr (NPT == 2) {
          if (own_col[0] && own_col[1] && (xs[1] & 1) == 0 && (!HAS_PRESSURE || (skip[0] | skip[1]) == 0u)) {
#pragma unroll
            for (int i = 0; i < 9; ++i) memcpy(__builtin_assume_aligned(po + i * plane + xs[1], 4), out[i], 4);
            continue;
          }
        }
#pragma unroll
        for (int i = 0; i < 9; ++i) {
#pragma unroll
          for (int k = 0; k < NPT; ++k)
            if (own_col[k] && (!HAS_PRESSURE || !((skip[k] >> i) & 1u))) po[i * plane + xs[k + 1]] = out[i][k];
        }
      }
    }
    if (!last) {
      __syncthreads();
      src = dst;
      dst = pops + ((s + 1) & 1) * h * kRow;
    }
  }
}

}  // namespace lbm

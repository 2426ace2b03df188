// kernels_mixed.cu -- mixed-precision kernels of the explicit MPM step.
//
// Arithmetic in FP32 with FP64 where it carries the result:
//   * positions and displacements are stored and advanced in FP64;
//   * the shape functions use a local coordinate computed in FP64 (x and the
//     cell centroid are FP64) and then rounded;
//   * P2G forms each particle's contributions in FP32 and sums them per cell
//     slot in FP64 (one FP64 add per value costs less than a compensated FP32
//     sum), the node adds its (at most eight) cell partials in FP64 and divides
//     momentum by mass in FP64;
//   * the MohrCoulomb elastic predictor and yield check run in FP32 (stress
//     invariants in FP64, see mc_invariants); plastic returns, points at the
//     apex and separated points run in FP64 in a dense second kernel (an FP32
//     return cancels when it removes most of the trial stress and near the
//     apex, and plastic points are few and scattered, so batching them keeps
//     the elastic lanes of a warp from waiting on the return iterations);
//     the plastic deviatoric strain is kept in FP64;
//   * F, volume and density are stored as deviations (H = F - I,
//     P = V / V0 - 1) so that FP32 keeps the 1e-9 per-step increments.
// Same step structure as the FP64 path (kernels_fp64.cu): counting sort,
// per-cell P2G, node gather and update, G2P + stress + locate.
#define MPM_MC_RECIPROCALS  // see mpm_math.cuh
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "mpm_bulk.cuh"
#include "mpm_device.cuh"
#include "mpm_grid.cuh"
#include "mpm_kernels.h"
#include "mpm_launch.cuh"
#include "mpm_return.cuh"
#include "mpm_state.cuh"

#ifndef MPM_MIXED_G2P_MIN_BLOCKS
// 72 registers, hardly a spill on a grid: 2M particles in 3D 6 / 7 / 8 blocks 135 /
// 129 / 142 us (8 spill); no difference in 2D.
#define MPM_MIXED_G2P_MIN_BLOCKS 7
#endif
#ifndef MPM_MIXED_G2P_GENERAL_MIN_BLOCKS
#define MPM_MIXED_G2P_GENERAL_MIN_BLOCKS 6  // 80 registers; spills on a general mesh, more with fewer
#endif
#ifndef MPM_MIXED_AFFINE_G2P_MIN_BLOCKS
#define MPM_MIXED_AFFINE_G2P_MIN_BLOCKS 4  // the nodal velocities stay in registers for B
#endif
#ifndef MPM_MC_RETURN_MIN_BLOCKS
#define MPM_MC_RETURN_MIN_BLOCKS 4  // pass-loop return, 1M column at step 2000: 2 / 3 / 4 / 6 blocks -> FP64 0.362 / 0.320 / 0.323 / 0.403 ms, mixed 0.370 / 0.318 / 0.311 / 0.384 ms
#endif
// Blocks per SM of the persistent step kernel (3D, 2D).  Measured with 20
// steps per launch, ms per step on the 4M-particle column / the 512-slope
// ensemble: 4 blocks 1.303 / 3.018, 6 blocks 1.128 / 2.382, 8 blocks 1.161 /
// 2.047 (per-pass launches: 0.748 / 1.555).
#ifndef MPM_MIXED_NODES_MIN_BLOCKS
// 256-thread blocks, 32 registers; 6 and 4 blocks (40 / 64 registers), 4M column:
// 0.048 / 0.054 ms against 0.049 ms
#define MPM_MIXED_NODES_MIN_BLOCKS 8
#endif
#ifndef MPM_PERSISTENT_MIN_BLOCKS_3D
#define MPM_PERSISTENT_MIN_BLOCKS_3D 6
#endif
#ifndef MPM_PERSISTENT_MIN_BLOCKS_2D
#define MPM_PERSISTENT_MIN_BLOCKS_2D 8
#endif
#ifndef MPM_MIXED_P2G_TILE_MIN_BLOCKS
// 48 registers, small spills: 0.32 -> 0.26 ms (4M, 3D); against 4 and 6 (64 / 40
// registers) with the body force at the node: 128-thread tiles 0.193 vs 0.206 / 0.203
// ms, 256-thread tiles 0.216 vs 0.237 / 0.227 ms.
#define MPM_MIXED_P2G_TILE_MIN_BLOCKS 5
#endif

namespace mpm_b200 {
namespace {

template <int DIM>
__device__ __forceinline__ float pmf(const DevState& s, int f, int64_t p) {
  return s.pm[(int64_t)f * s.np + p];
}
template <int DIM>
__device__ __forceinline__ void set_pmf(const DevState& s, int f, int64_t p, float v) {
  s.pm[(int64_t)f * s.np + p] = v;
}

// The nodal velocity (and, with ACC, acceleration) of node n from its
// nfv record (nfv_stride floats: 3D v0 v1 v2 a0 | a1 a2 - -, 2D v0 v1 a0 a1).
template <int DIM, bool ACC>
__device__ __forceinline__ void load_nfv(const float* nfv, int64_t n, float* v, float* a) {
  const float4* q = reinterpret_cast<const float4*>(nfv + n * nfv_stride(DIM));
  const float4 h0 = q[0];
  v[0] = h0.x;
  v[1] = h0.y;
  if constexpr (DIM == 3) {
    v[2] = h0.z;
    if constexpr (ACC) {
      const float4 h1 = q[1];
      a[0] = h0.w;
      a[1] = h1.x;
      a[2] = h1.y;
    }
  } else if constexpr (ACC) {
    a[0] = h0.z;
    a[1] = h0.w;
  }
}
template <int DIM>
__device__ __forceinline__ void store_nfv(float* nfv, int64_t n, const float* v, const float* a) {
  float4* q = reinterpret_cast<float4*>(nfv + n * nfv_stride(DIM));
  if constexpr (DIM == 3) {
    q[0] = make_float4(v[0], v[1], v[2], a[0]);
    q[1] = make_float4(a[1], a[2], 0.f, 0.f);
  } else {
    q[0] = make_float4(v[0], v[1], a[0], a[1]);
  }
}

// local coordinate in FP64, rounded to FP32 for the shape functions.  In a box
// cell the product with the tabulated 2 / len takes the place of the quotient:
// two FP64 roundings instead of one before the FP32 one.
template <int DIM>
__device__ __forceinline__ void box_xi_f32(const DevState& s, const int* ijk, const double* x,
                                           float* xf, float* ihl) {
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    const AxisCell& g = s.axcell[d][ijk[d]];
    const double h = __ldg(&g.ihl);
    xf[d] = (float)((x[d] - __ldg(&g.centroid)) * h);
    ihl[d] = (float)h;
  }
}
template <int DIM, bool BOX>
__device__ __forceinline__ void xi_f32(const DevState& s, int c, const double* x, float* xf) {
  if constexpr (BOX) {
    int ijk[3] = {0, 0, 0};
    float ihl[DIM];
    cell_ijk<DIM>(s, c, ijk);
    box_xi_f32<DIM>(s, ijk, x, xf, ihl);
    return;
  }
  double xi[DIM];
  particle_xi<DIM, BOX>(s, c, x, xi);
#pragma unroll
  for (int d = 0; d < DIM; ++d) xf[d] = (float)xi[d];
}

// node ids and nodal coordinates relative to node 0 of the cell (FP32); the
// coordinates are not needed (nor set) for the box cells of a tensor-product
// grid
template <int DIM, bool BOX>
__device__ __forceinline__ void cell_nodes_rel(const DevState& s, int c, int* nid, float* Xr) {
  constexpr int NV = Elem<DIM>::NV;
  if constexpr (BOX) {
    grid_cell_nodes<DIM>(s, c, nid);
    return;
  }
  double X[NV * DIM];
  cell_nodes_coords<DIM>(s, c, nid, X);
#pragma unroll
  for (int n = 0; n < NV; ++n)
#pragma unroll
    for (int d = 0; d < DIM; ++d) Xr[n * DIM + d] = (float)(X[n * DIM + d] - X[d]);
}

// ---------------------------------------------------------------- P2G tiles
// The FP64 path's cell tiles (k_p2g_tiles) in FP32: staged local coordinates
// (the FP64 local coordinate rounded), mass, velocity, the stress times the
// particle's -V0 (1 + P)
// and, off a tensor-product grid, J^-1; per (cell, slot) thread 1 + 2 DIM
// FP64 sums (mass, momentum, internal force; the body force is formed by the
// node update) of the FP32 contributions of the cell's particles in id order,
// stored as FP32 partials.  AFF: the mass-momentum mapping velocity v + M r of
// the affine (1: M = B D^-1) or Taylor (2: M = B) updates, with M formed in
// FP64 by the staging thread and the branch vectors r taken from FP64
// positions relative to the cell's first node, both rounded to FP32.
//
// A particle's row is one run of 16-byte vectors, so that a (cell, slot)
// thread reads it in four accesses (3D, all values) where one array per value
// took thirteen; the run is an odd number of vectors long, so that the eight
// threads of a store phase meet different banks.
template <int DIM, int MODE, bool BOX, int AFF = 0>
struct MTileRows {
  static constexpr bool MM = MODE != 1, FORCES = MODE != 0;
  static constexpr int XI = 0, M = DIM;  // the mass (times 1/8, 1/4 in 2D) only with mass and momentum
  static constexpr int V = M + (MM ? 1 : 0);
  static constexpr int S = V + (MM ? DIM : 0);  // stress times -V0 (1 + P)
  static constexpr int INV = S + (FORCES ? PF<DIM>::NS : 0);
  static constexpr int XP = INV + (FORCES && !BOX ? DIM * DIM : 0);  // x - node 0
  static constexpr int MV = XP + (MM && AFF ? DIM : 0);              // mapping matrix
  static constexpr int N = MV + (MM && AFF ? DIM * DIM : 0);
  static constexpr int N4 = (N + 3) / 4;    // 16-byte vectors of a row
  static constexpr int STRIDE = N4 | 1;     // and from row to row
};

// On box cells the tile may also take 128 threads (a launch-shape choice);
// the blocks per SM scale so that the registers per thread stay the same.
// The mapping-velocity tiles (128 threads) form the FP64 matrix when they
// stage a row and take up to 128 registers.
template <bool BOX, int T, int AFF = 0>
constexpr int mixed_tile_min_blocks() {
  return AFF ? 4 : BOX ? MPM_MIXED_P2G_TILE_MIN_BLOCKS * 256 / T : MPM_MIXED_P2G_TILE_MIN_BLOCKS;
}

// One tile (block-sized group of cells, tile index bx) of the P2G pass; the
// block's threads are the tile's (cell, slot) pairs.
//
// A tile of up to 1.25 T particles (a cell's usual 2 per axis and some more,
// as a moving body has them) is staged at once: every thread reads the ids of
// one or two places of the sorted order, ranks each among the ids of its cell
// in shared memory while the particle's fields are on their way, and writes
// the row where the cell's ascending ids put it.  Fuller tiles sort each
// cell's ids in global memory and stage T rows at a time  Measured: 101
// -> 94 us at 2M particles in 3D, 71 -> 64 us at 1.3M in 2D (256-thread tiles).
template <int DIM, int MODE, bool BOX, int T, int AFF = 0>
__device__ __forceinline__ void p2g_tile_mixed(const DevState& s, int64_t bx) {
  constexpr int NV = Elem<DIM>::NV;
  constexpr int CB = T / NV;
  constexpr int CAP = T + T / 4;  // rows staged at once
  constexpr int NVAL = mixed_nval(DIM);
  constexpr int MASS = 0, MOM = 1, FINT = 1 + DIM;
  using RW = MTileRows<DIM, MODE, BOX, AFF>;
  constexpr bool MM = RW::MM, FORCES = RW::FORCES;
  __shared__ float4 rows[CAP * RW::STRIDE];
  __shared__ int32_t ids[CAP], cstart[CB + 1];
  const int t = threadIdx.x;
  const int64_t c0 = bx * CB;
  if (c0 >= s.ncells) return;
  const int64_t c1 = c0 + CB < s.ncells ? c0 + CB : s.ncells;
  const int q_begin = s.start[c0], count = s.start[c1] - q_begin;
  if (count == 0) return;  // no particles in the tile (the whole block)
  const int cl = t / NV, k = t % NV;
  const int64_t c = c0 + cl;
  const bool mine = c < c1;
  // the cell's rows, counted from the tile's first
  const int a0 = mine ? s.start[c] - q_begin : 0;
  const int a1 = mine ? s.start[c + 1] - q_begin : 0;
  // One staged particle row.
  auto stage = [&](int r, int64_t p, int pc) {
    float v[RW::N4 * 4];
#pragma unroll
    for (int q = RW::N; q < RW::N4 * 4; ++q) v[q] = 0.f;
    double x[DIM];
    load_x<DIM>(s, p, x);
    xi_f32<DIM, BOX>(s, pc, x, &v[RW::XI]);
    if constexpr (MM) {
      v[RW::M] = (1.f / NV) * pmf<DIM>(s, PM<DIM>::MASS, p);
#pragma unroll
      for (int d = 0; d < DIM; ++d) v[RW::V + d] = pmf<DIM>(s, PM<DIM>::V + d, p);
    }
    if constexpr (MM && AFF) {
      double X[NV * DIM], xid[DIM], Mv[DIM * DIM];
      if constexpr (BOX) {
        int ijk[3] = {0, 0, 0};
        cell_ijk<DIM>(s, pc, ijk);
#pragma unroll
        for (int d = 0; d < DIM; ++d) X[d] = __ldg(&s.axis[d][ijk[d]]);
      } else {
        int nid[NV];
        cell_nodes_coords<DIM>(s, pc, nid, X);
      }
      particle_xi<DIM, BOX>(s, pc, x, xid);
      mapping_velocity_matrix<DIM, AFF, BOX>(s, p, pc, x, xid, Mv);
#pragma unroll
      for (int d = 0; d < DIM; ++d) v[RW::XP + d] = (float)(x[d] - X[d]);
#pragma unroll
      for (int q = 0; q < DIM * DIM; ++q) v[RW::MV + q] = (float)Mv[q];
    }
    if constexpr (FORCES) {
      const float sc = -(pmf<DIM>(s, PM<DIM>::V0, p) * (1.f + pmf<DIM>(s, PM<DIM>::JP, p)));
#pragma unroll
      for (int q = 0; q < PF<DIM>::NS; ++q) v[RW::S + q] = sc * pmf<DIM>(s, PM<DIM>::S + q, p);
      if constexpr (!BOX) {
        int nid[NV];
        float Xr[NV * DIM];
        cell_nodes_rel<DIM, false>(s, pc, nid, Xr);
        const CellMap<DIM, false, float> m = cell_map<DIM, false>(s, pc, &v[RW::XI], Xr);
#pragma unroll
        for (int q = 0; q < DIM * DIM; ++q) v[RW::INV + q] = m.inv[q];
      }
    }
#pragma unroll
    for (int q = 0; q < RW::N4; ++q)
      rows[r * RW::STRIDE + q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
  };
  // the slot's signs, and on a box its gradient factors +-(1 / NV) 2 / len
  float sg[DIM], kd[DIM];
  sg[0] = off_i(k) ? 1.f : -1.f;
  sg[1] = off_j(k) ? 1.f : -1.f;
  if constexpr (DIM == 3) sg[2] = off_k(k) ? 1.f : -1.f;
  if constexpr (BOX && FORCES) {
    if (a1 > a0) {
      const CellMap<DIM, BOX, float> m = cell_map<DIM, true, float>(s, (int)c, nullptr, nullptr);
#pragma unroll
      for (int d = 0; d < DIM; ++d) kd[d] = sg[d] * (1.f / NV) * m.ihl[d];
    }
  } else {
#pragma unroll
    for (int d = 0; d < DIM; ++d) kd[d] = sg[d] * (1.f / NV);
  }
  float xkr[DIM];  // this slot's node relative to the cell's first node (AFF)
  if constexpr (MM && AFF && BOX) {
    int ijk[3] = {0, 0, 0};
    if (a1 > a0) cell_ijk<DIM>(s, (int)c, ijk);
#pragma unroll
    for (int d = 0; d < DIM; ++d)
      xkr[d] = sg[d] > 0.f ? (float)(__ldg(&s.axis[d][ijk[d] + 1]) - __ldg(&s.axis[d][ijk[d]])) : 0.f;
  } else if constexpr (MM && AFF) {
    int nid[NV];
    double X[NV * DIM];
    if (a1 > a0) cell_nodes_coords<DIM>(s, (int)c, nid, X);
#pragma unroll
    for (int d = 0; d < DIM; ++d) xkr[d] = a1 > a0 ? (float)(X[k * DIM + d] - X[d]) : 0.f;
  }
  double acc[NVAL];
#pragma unroll
  for (int v = 0; v < NVAL; ++v) acc[v] = 0.;
  // this slot's contributions of staged row r: NV N_k is the product of the
  // factors 1 +- xi and its derivatives those of the others
  auto add = [&](int r) {
    float v[RW::N4 * 4];
#pragma unroll
    for (int q = 0; q < RW::N4; ++q) {
      const float4 w = rows[r * RW::STRIDE + q];
      v[4 * q] = w.x;
      v[4 * q + 1] = w.y;
      v[4 * q + 2] = w.z;
      v[4 * q + 3] = w.w;
    }
    float f[DIM], G[DIM], N;
#pragma unroll
    for (int d = 0; d < DIM; ++d) f[d] = fmaf(sg[d], v[RW::XI + d], 1.f);
    if constexpr (DIM == 2) {
      N = f[0] * f[1];
      G[0] = kd[0] * f[1];
      G[1] = kd[1] * f[0];
    } else {
      const float xy = f[0] * f[1];
      N = xy * f[2];
      G[0] = kd[0] * (f[1] * f[2]);
      G[1] = kd[1] * (f[0] * f[2]);
      G[2] = kd[2] * xy;
    }
    if constexpr (MM) {
      const float mN = v[RW::M] * N;
      acc[MASS] += (double)mN;
      float mv[DIM];
#pragma unroll
      for (int d = 0; d < DIM; ++d) mv[d] = v[RW::V + d];
      if constexpr (AFF) {
        float br[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) br[d] = xkr[d] - v[RW::XP + d];
#pragma unroll
        for (int a = 0; a < DIM; ++a) {
          float sum = v[RW::MV + a * DIM + 0] * br[0];
#pragma unroll
          for (int b = 1; b < DIM; ++b) sum = sum + v[RW::MV + a * DIM + b] * br[b];
          mv[a] += sum;
        }
      }
#pragma unroll
      for (int d = 0; d < DIM; ++d) acc[MOM + d] += (double)(mN * mv[d]);
    }
    if constexpr (FORCES) {
      const float* sig = &v[RW::S];
      float Dn[DIM];
      if constexpr (BOX) {
#pragma unroll
        for (int d = 0; d < DIM; ++d) Dn[d] = G[d];
      } else {
        CellMap<DIM, false, float> m2;
#pragma unroll
        for (int q = 0; q < DIM * DIM; ++q) m2.inv[q] = v[RW::INV + q];
        m2.grad(G, Dn);
      }
      float fi[DIM];
      if constexpr (DIM == 2) {
        fi[0] = fmaf(Dn[1], sig[3], __fmul_rn(Dn[0], sig[0]));
        fi[1] = fmaf(Dn[0], sig[3], __fmul_rn(Dn[1], sig[1]));
      } else {
        fi[0] = fmaf(Dn[2], sig[5], fmaf(Dn[1], sig[3], __fmul_rn(Dn[0], sig[0])));
        fi[1] = fmaf(Dn[2], sig[4], fmaf(Dn[0], sig[3], __fmul_rn(Dn[1], sig[1])));
        fi[2] = fmaf(Dn[0], sig[5], fmaf(Dn[1], sig[4], __fmul_rn(Dn[2], sig[2])));
      }
#pragma unroll
      for (int d = 0; d < DIM; ++d) acc[FINT + d] += (double)fi[d];
    }
  };
  if (count <= CAP) {
    int32_t id[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int r = t + u * T;
      if (r < count) ids[r] = id[u] = s.order[q_begin + r];
    }
    if (k == 0) cstart[cl] = mine ? a0 : count;
    if (t == 0) cstart[CB] = count;
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (t + u * T < count) {
        const int pc = s.cell[id[u]];
        const int b = cstart[pc - c0], e = cstart[pc - c0 + 1];
        int r = b;
        for (int j = b; j < e; ++j) r += ids[j] < id[u] ? 1 : 0;
        stage(r, id[u], pc);
      }
    }
    __syncthreads();
    for (int j = a0; j < a1; ++j) add(j);
  } else {
    sort_cell_ids<NV>(s.order + q_begin + a0, a1 - a0, k);
    for (int q0 = 0; q0 < count; q0 += T) {
      if (q0 != 0) __syncthreads();  // the previous chunk is consumed
      if (q0 + t < count) {
        const int64_t p = s.order[q_begin + q0 + t];
        stage(t, p, s.cell[p]);
      }
      __syncthreads();
      const int j0 = a0 > q0 ? a0 : q0;
      const int j1 = a1 < q0 + T ? a1 : q0 + T;
      for (int j = j0; j < j1; ++j) add(j - q0);
    }
  }
  if (!mine || a1 == a0) return;  // empty cells keep no partials
  float* out = s.partials_f + ((int64_t)c * NV + k) * NVAL;
  float row[NVAL];  // the padding stays zero
#pragma unroll
  for (int v = 0; v < NVAL; ++v) row[v] = (float)acc[v];
  if constexpr (MM && FORCES)
    store_partial_row<NVAL, 0, NVAL>(out, row);
  else if constexpr (MM)
    store_partial_row<NVAL, MASS, FINT>(out, row);
  else
    store_partial_row<NVAL, FINT, NVAL - FINT>(out, row + FINT);
}

template <int DIM, int MODE, bool BOX, int T = p2g_tile_t<BOX>(), int AFF = 0>
__global__ void __launch_bounds__(T, (mixed_tile_min_blocks<BOX, T, AFF>()))
    k_p2g_tiles_mixed(DevState s, bool dependent) {
  if (dependent) after_previous();
  p2g_tile_mixed<DIM, MODE, BOX, T, AFF>(s, blockIdx.x);
}

// ---------------------------------------------------------------- node update
// The cell partials of a node (ascending cell id) added in FP64.
template <int DIM, int V0, int NVS>
__device__ __forceinline__ bool gather_node_mixed(const DevState& s, int64_t node, double* sum) {
  constexpr int NV = Elem<DIM>::NV;
  constexpr int NVAL = mixed_nval(DIM);
#pragma unroll
  for (int v = 0; v < NVS; ++v) sum[v] = 0.;
  bool active = false;
  auto add = [&](int c, int slot) {
    float src[NVS];
    load_partial_row<float, NVAL, V0, NVS>(s.partials_f + ((int64_t)c * NV + slot) * NVAL, src);
#pragma unroll
    for (int v = 0; v < NVS; ++v) sum[v] += (double)src[v];
    active = true;
  };
  if (s.structured) {
    constexpr int NC = DIM == 2 ? 4 : 8;
    int cid[NC], slot[NC], count[NC];
    grid_node_cells<DIM>(s, (int)node, cid, slot, count);
#pragma unroll
    for (int q = 0; q < NC; ++q)
      if (count[q] > 0) add(cid[q], slot[q]);
  } else {
    for (int e = s.nc_off[node]; e < s.nc_off[node + 1]; ++e)
      if (s.cnt[s.nc_cell[e]] > 0) add(s.nc_cell[e], s.nc_slot[e]);
  }
  return active;
}

// node.tcc:309-345 in FP64 on the gathered sums
template <int DIM>
__device__ __forceinline__ void node_accel_update_d(const DevState& s, double m, const double* fe,
                                                    const double* fi, double* vel, double* acc,
                                                    int bci, double dt, double damping) {
  if (!(m > 1.0E-15)) return;
  double uf[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) uf[d] = fe[d] + fi[d];
  double ss = uf[0] * uf[0];
#pragma unroll
  for (int d = 1; d < DIM; ++d) ss = ss + uf[d] * uf[d];
  const double nrm = sqrt(ss);
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    const double sg = (vel[d] > 0.) ? 1. : ((vel[d] < 0.) ? -1. : 0.);
    acc[d] = (uf[d] - damping * nrm * sg) / m;
  }
  if (bci >= 0) {
    const NodeBC& bc = s.bcs[bci];
    if (bc.friction) apply_friction_constraints<DIM>(bc, vel, acc, dt);
    apply_acceleration_constraints<DIM>(bc, acc);
  }
#pragma unroll
  for (int d = 0; d < DIM; ++d) vel[d] += acc[d] * dt;
  if (bci >= 0) apply_velocity_constraints<DIM>(s.bcs[bci], vel, acc);
#pragma unroll
  for (int d = 0; d < DIM; ++d)
    if (fabs(vel[d]) < 1.0E-15) vel[d] = 0.;
#pragma unroll
  for (int d = 0; d < DIM; ++d)
    if (fabs(acc[d]) < 1.0E-15) acc[d] = 0.;
}

// 8 blocks per SM: 0.111 -> 0.108 ms per 1M-node launch (more warps in flight
// on the scattered partial loads, despite small spills)
// The body force of a node is gravity times its mass (particle.tcc:893-898
// summed over the node's particles: sum_p g m_p N_p = g sum_p m_p N_p), formed
// here in FP64 from the gathered mass instead of carried in the partials.
template <int DIM, int MODE>
__device__ __forceinline__ void node_update_mixed(const DevState& s, double dt, double damping,
                                                  const double* g, int64_t n) {
  if (n >= s.nn) return;
  constexpr int NVAL = mixed_nval(DIM);
  double sum[NVAL];
  constexpr int V0 = MODE == 2 ? 1 + DIM : 0;  // MODE 2: the internal force and the padding
  constexpr int NVS = MODE == 0 ? 1 + DIM : (MODE == 1 ? NVAL : NVAL - (1 + DIM));
  if (!gather_node_mixed<DIM, V0, NVS>(s, n, sum)) return;
  const int bci = s.bc_index[n];
  double vel[DIM], acc[DIM];
  if constexpr (MODE == 2) {
    double mm[1];
    gather_node_mixed<DIM, 0, 1>(s, n, mm);
    float vf[DIM], af[DIM];
    load_nfv<DIM, true>(s.nfv, n, vf, af);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      vel[d] = (double)vf[d];
      acc[d] = (double)af[d];
    }
    double fe[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) fe[d] = g[d] * mm[0];
    node_accel_update_d<DIM>(s, mm[0], fe, &sum[0], vel, acc, bci, dt, damping);
  } else {
    const double m = sum[0];
#pragma unroll
    for (int d = 0; d < DIM; ++d) vel[d] = acc[d] = 0.;
    if (m > 1.E-16) {
#pragma unroll
      for (int d = 0; d < DIM; ++d) vel[d] = sum[1 + d] / m;  // FP64 mass division
#pragma unroll
      for (int d = 0; d < DIM; ++d)
        if (fabs(vel[d]) < 1.E-15) vel[d] = 0.;
    }
    if (bci >= 0) apply_velocity_constraints<DIM>(s.bcs[bci], vel, acc);
    if constexpr (MODE == 1) {
      double fe[DIM];
#pragma unroll
      for (int d = 0; d < DIM; ++d) fe[d] = g[d] * m;
      node_accel_update_d<DIM>(s, m, fe, &sum[1 + DIM], vel, acc, bci, dt, damping);
    }
  }
  float vf[DIM], af[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    vf[d] = (float)vel[d];
    af[d] = (float)acc[d];
  }
  store_nfv<DIM>(s.nfv, n, vf, af);
}

template <int DIM, int MODE>
__global__ void __launch_bounds__(256, MPM_MIXED_NODES_MIN_BLOCKS) k_nodes_mixed(DevState s, double dt, double damping, double g0,
                                                        double g1, double g2) {
  after_previous();
  if (MODE != 2 && blockIdx.x == 0 && threadIdx.x == 0) *s.nplastic = *s.nplastic_heavy = 0;
  const double g[3] = {g0, g1, g2};
  node_update_mixed<DIM, MODE>(s, dt, damping, g, (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}

// ------------------------------------------------------- stress and strain
// MohrCoulomb elastic predictor and yield check in FP32 (invariants in FP64):
// true with out and svf updated when the trial stress is elastic and away
// from the apex of the yield surface (deviatoric trial stress above 1e-2 of
// the stress magnitude); false for every other point (plastic, apex,
// separated), which the caller defers to the FP64 return of
// k_mc_return_mixed with its inputs unchanged.
__device__ __forceinline__ bool mc_elastic_mixed(const MaterialT<float>& mf, const float* sig,
                                                 const float* de, float rho, float* svf, float* out) {
  float trial[6];
  {
    float t[6];
    de_mul(mf, de, t);
#pragma unroll
    for (int i = 0; i < 6; ++i) trial[i] = sig[i] + t[i];
  }
  float smax = 0.f;
#pragma unroll
  for (int i = 0; i < 6; ++i) smax = fmaxf(smax, fabsf(trial[i]));
  const float rho_dev = sqrtf(2.f * mu_j2(trial));
  if (rho_dev <= 1e-2f * smax) return false;
  float sv[SV_N];
#pragma unroll
  for (int k = 0; k < SVF_N; ++k) sv[k] = svf[k];
  sv[SV_PD] = 0.f;
  double pd_unused = 0.0;
  if (mc_stress<float, double, true>(mf, sig, de, rho, sv, pd_unused, out) != MC_OK ||
      sv[SV_YIELD] != 0.f)
    return false;
#pragma unroll
  for (int k = 0; k < SVF_N; ++k) svf[k] = sv[k];
  return true;
}

// One particle's mixed-precision fields in global memory (MGlobalRow) or in
// the block's shared-memory staging (MSmemRow, MSTAGE_T particles per row):
// m(f) the FP32 field f of PM, svf(k) the FP32 MohrCoulomb state, pd() the
// FP64 plastic deviatoric strain (read only by the deferred returns, which
// work in global memory).
template <int DIM>
struct MGlobalRow {
  const DevState& s;
  int64_t p;
  __device__ __forceinline__ int64_t index() const { return p; }
  __device__ __forceinline__ float& m(int f) const { return s.pm[(int64_t)f * s.np + p]; }
  __device__ __forceinline__ float& svf(int k) const { return s.svf[(int64_t)k * s.np + p]; }
  __device__ __forceinline__ double& pd() const { return s.pf[(int64_t)PDX<DIM>::PDS * s.np + p]; }
  __device__ __forceinline__ int mat() const { return s.mat[p]; }
};
constexpr int MSTAGE_T = 128;  // particles per staged block (= PAD_PARTICLES)
struct MSmemRow {
  float* mrows;  // [PM field][MSTAGE_T]
  float* svr;    // [SVF_N][MSTAGE_T]
  int t;
  int mi;
  int64_t p;
  __device__ __forceinline__ int64_t index() const { return p; }
  __device__ __forceinline__ float& m(int f) const { return mrows[f * MSTAGE_T + t]; }
  __device__ __forceinline__ float& svf(int k) const { return svr[k * MSTAGE_T + t]; }
  __device__ __forceinline__ int mat() const { return mi; }
};

// Velocity gradient of a particle, L[a][b] = dv_a/dx_b = sum_i v_ia dN_i/dx_b,
// and the divergence with the cell's centroid gradients (the volume update's,
// particle.tcc:819-876).
template <int DIM>
struct VelGrad {
  float L[DIM * DIM];
  float divc;
};

// From the nodal velocities and D = dN/dx at the particle.
template <int DIM>
__device__ __forceinline__ VelGrad<DIM> velocity_gradient(const DevState& s, int c, const int* nid,
                                                          const float* D) {
  constexpr int NV = Elem<DIM>::NV;
  const float* Dc = s.dndx_cf + (int64_t)c * NV * DIM;
  VelGrad<DIM> g;
#pragma unroll
  for (int a = 0; a < DIM * DIM; ++a) g.L[a] = 0.f;
  float src[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) src[d] = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    float vel[DIM];
    load_nfv<DIM, false>(s.nfv, nid[i], vel, nullptr);
#pragma unroll
    for (int a = 0; a < DIM; ++a) {
#pragma unroll
      for (int q = 0; q < DIM; ++q) g.L[a * DIM + q] += vel[a] * D[i * DIM + q];
      src[a] += __ldg(&Dc[i * DIM + a]) * vel[a];
    }
  }
  g.divc = src[0];
#pragma unroll
  for (int d = 1; d < DIM; ++d) g.divc += src[d];
  return g;
}

// Nodal velocity (and, with ACC, acceleration) interpolated to a particle of
// box cell ijk at local coordinates xi and, with GRAD, the velocity gradient
// there, in one visit of the cell's nodes.  On a box the interpolation is a
// sequence of linear ones along x, y and z and the gradient the interpolated
// differences: about 130 FP32 operations in 3D where the sums over N_i and
// dN_i/dx take about 300 and, for the gradient, a second visit; the centroid
// gradients are the mean differences, so the per-cell table (96 bytes a cell)
// is not read.  Differences come first, so the gradient's rounding error is
// relative to the differences and not to the velocities  Measured with the
// division-free locate and the spills that went with both: staged G2P 200 -> 138
// us at 2M particles in 3D (2.6 -> 3.7 TB/s of state), 95 -> 77 us at 1.3M in 2D.
template <int DIM, bool ACC, bool GRAD>
__device__ __forceinline__ void gather_box(const DevState& s, const int* ijk, const float* xi,
                                           const float* ihl, float* nvel, float* nacc,
                                           VelGrad<DIM>* grad) {
  float f[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) f[d] = fmaf(0.5f, xi[d], 0.5f);
  const int nx = s.gcells[0] + 1;
  const int base = DIM == 2 ? ijk[0] + nx * ijk[1] : ijk[0] + nx * ijk[1] + (int)s.div_nxy.d * ijk[2];
  constexpr int KN = DIM == 3 ? 2 : 1;
  float vy[KN][DIM], ay[KN][DIM];  // interpolated along x and y, per layer
  float gx[KN][DIM], gy[KN][DIM];  // their differences along x and y
  float cx = 0.f, cy = 0.f, cz = 0.f;  // sums of the edge differences, component by axis
  float vz[4];                     // the lower layer's z velocities
#pragma unroll
  for (int k = 0; k < KN; ++k) {
    float vx[2][DIM], ax[2][DIM], dx[2][DIM], ya[2], yb[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int n = base + j * nx + k * (int)s.div_nxy.d;
      float va[DIM], vb[DIM], aa[DIM], ab[DIM];
      load_nfv<DIM, ACC>(s.nfv, n, va, aa);
      load_nfv<DIM, ACC>(s.nfv, n + 1, vb, ab);
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        dx[j][d] = vb[d] - va[d];
        vx[j][d] = fmaf(f[0], dx[j][d], va[d]);
        if constexpr (ACC) ax[j][d] = fmaf(f[0], ab[d] - aa[d], aa[d]);
      }
      if constexpr (GRAD) {
        cx += dx[j][0];
        ya[j] = va[1];
        yb[j] = vb[1];
        if constexpr (DIM == 3) {
          if (k == 0) {
            vz[2 * j] = va[2];
            vz[2 * j + 1] = vb[2];
          } else {
            cz += (va[2] - vz[2 * j]) + (vb[2] - vz[2 * j + 1]);
          }
        }
      }
    }
    if constexpr (GRAD) cy += (ya[1] - ya[0]) + (yb[1] - yb[0]);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      gy[k][d] = vx[1][d] - vx[0][d];
      vy[k][d] = fmaf(f[1], gy[k][d], vx[0][d]);
      if constexpr (ACC) ay[k][d] = fmaf(f[1], ax[1][d] - ax[0][d], ax[0][d]);
      if constexpr (GRAD) gx[k][d] = fmaf(f[1], dx[1][d] - dx[0][d], dx[0][d]);
    }
  }
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    if constexpr (DIM == 2) {
      nvel[d] = vy[0][d];
      if constexpr (ACC) nacc[d] = ay[0][d];
      if constexpr (GRAD) {
        grad->L[d * 2 + 0] = gx[0][d] * (0.5f * ihl[0]);
        grad->L[d * 2 + 1] = gy[0][d] * (0.5f * ihl[1]);
      }
    } else {
      const float gz = vy[KN - 1][d] - vy[0][d];
      nvel[d] = fmaf(f[DIM - 1], gz, vy[0][d]);
      if constexpr (ACC) nacc[d] = fmaf(f[DIM - 1], ay[KN - 1][d] - ay[0][d], ay[0][d]);
      if constexpr (GRAD) {
        grad->L[d * 3 + 0] = fmaf(f[DIM - 1], gx[KN - 1][d] - gx[0][d], gx[0][d]) * (0.5f * ihl[0]);
        grad->L[d * 3 + 1] = fmaf(f[DIM - 1], gy[KN - 1][d] - gy[0][d], gy[0][d]) * (0.5f * ihl[1]);
        grad->L[d * 3 + 2] = gz * (0.5f * ihl[DIM - 1]);
      }
    }
  }
  if constexpr (GRAD) {
    grad->divc = fmaf(cy, ihl[1], cx * ihl[0]);
    if constexpr (DIM == 3) grad->divc = fmaf(cz, ihl[DIM - 1], grad->divc);
    grad->divc *= DIM == 2 ? 0.25f : 0.125f;
  }
}

// mpm_scheme.tcc:75-103 in FP32 on the deviation variables (H, P).  Products
// that are used more than once are rounded (__fmul_rn) and the other sums of
// products fused by hand, so that the per-pass and the persistent kernels round
// alike whatever the compiler makes of the code around them.
template <int DIM, class Row>
__device__ __forceinline__ void stress_update_mixed(const DevState& s, const Row& r,
                                                    const VelGrad<DIM>& g, float dt) {
  constexpr int NS = PF<DIM>::NS;
  float Hi[DIM * DIM];
#pragma unroll
  for (int a = 0; a < DIM * DIM; ++a) Hi[a] = __fmul_rn(g.L[a], dt);
  float sr[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int d = 0; d < DIM; ++d) sr[d] = g.L[d * DIM + d];
  sr[3] = g.L[1] + g.L[DIM];
  if constexpr (DIM == 3) {
    sr[4] = g.L[5] + g.L[7];
    sr[5] = g.L[2] + g.L[6];
  }
  // F_inc = I + Hi with the reference's 1e-15 snapping (particle.tcc:1619-1626)
#pragma unroll
  for (int a = 0; a < DIM * DIM; ++a)
    if (fabsf(Hi[a]) < 1.E-15f) Hi[a] = 0.f;
#pragma unroll
  for (int k = 0; k < 6; ++k)
    if (fabsf(sr[k]) < 1.E-15f) sr[k] = 0.f;
  float dstrain[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) dstrain[k] = __fmul_rn(sr[k], dt);
  const float dvol = __fmul_rn(dt, g.divc);
  if constexpr (DIM == 2) {
    const int map[3] = {0, 1, 3};
#pragma unroll
    for (int k = 0; k < 3; ++k) r.m(PM<2>::E + k) += dstrain[map[k]];
  } else {
#pragma unroll
    for (int k = 0; k < 6; ++k) r.m(PM<3>::E + k) += dstrain[k];
  }
  // V *= (1 + dvol), rho /= (1 + dvol) as P = V / V0 - 1 (particle.tcc:598-605)
  const float P = r.m(PM<DIM>::JP);
  const float Pn = fmaf(P, dvol, P + dvol);
  r.m(PM<DIM>::JP) = Pn;
  const float rho = r.m(PM<DIM>::RHO0) / (1.f + Pn);
  float sig[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int k = 0; k < NS; ++k) sig[k] = r.m(PM<DIM>::S + k);
  const int mi = r.mat();
  float out[6];
  bool deferred = false;
  if (s.mats_f[mi].type == 0) {
    float t[6];
    de_mul(s.mats_f[mi], dstrain, t);
#pragma unroll
    for (int i = 0; i < 6; ++i) out[i] = sig[i] + t[i];
  } else {
    float svf[SVF_N];
#pragma unroll
    for (int k = 0; k < SVF_N; ++k) svf[k] = r.svf(k);
    if (mc_elastic_mixed(s.mats_f[mi], sig, dstrain, rho, svf, out)) {
      const int first = s.mats_f[mi].softening ? 0 : SV_EPS;  // phi..tc change only with softening
      r.svf(SV_YIELD) = svf[SV_YIELD];
#pragma unroll
      for (int k = 1; k < SVF_N; ++k)
        if (k >= first) r.svf(k) = svf[k];
    } else {
      // plastic, apex or separated: the FP64 update of k_mc_return_mixed
      deferred = true;
      const unsigned i = defer_slot_by_cost(s, r.index());
      s.plist[i] = (int32_t)r.index();
#pragma unroll
      for (int k = 0; k < 6; ++k) s.pbuf_f[(int64_t)k * s.np + i] = dstrain[k];
      s.pbuf_f[(int64_t)6 * s.np + i] = rho;
    }
  }
  if (!deferred) {
#pragma unroll
    for (int k = 0; k < NS; ++k) r.m(PM<DIM>::S + k) = out[k];
  }
  // F = F_inc F as H = H + Hi + Hi H
  if constexpr (DIM == 2) {
    float H[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) H[k] = r.m(PM<2>::H + k);
    const float n00 = H[0] + Hi[0] + fmaf(Hi[1], H[2], __fmul_rn(Hi[0], H[0]));
    const float n01 = H[1] + Hi[1] + fmaf(Hi[1], H[3], __fmul_rn(Hi[0], H[1]));
    const float n10 = H[2] + Hi[2] + fmaf(Hi[3], H[2], __fmul_rn(Hi[2], H[0]));
    const float n11 = H[3] + Hi[3] + fmaf(Hi[3], H[3], __fmul_rn(Hi[2], H[1]));
    r.m(PM<2>::H + 0) = n00;
    r.m(PM<2>::H + 1) = n01;
    r.m(PM<2>::H + 2) = n10;
    r.m(PM<2>::H + 3) = n11;
  } else {
    float H[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) H[k] = r.m(PM<3>::H + k);
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int q = 0; q < 3; ++q)
        r.m(PM<3>::H + a * 3 + q) =
            H[a * 3 + q] + Hi[a * 3 + q] +
            fmaf(Hi[a * 3 + 2], H[2 * 3 + q],
                 fmaf(Hi[a * 3 + 1], H[1 * 3 + q], __fmul_rn(Hi[a * 3 + 0], H[0 * 3 + q])));
  }
}

template <int DIM, bool BOX>
__device__ __forceinline__ void dn_dx_all_f(const DevState& s, int c, const float* xi,
                                            const float* Xr, float* D) {
  constexpr int NV = Elem<DIM>::NV;
  const CellMap<DIM, BOX, float> map = cell_map<DIM, BOX>(s, c, xi, Xr);
  float G[NV * DIM];
  grad_shapefn<DIM>(xi, G);
#pragma unroll
  for (int n = 0; n < NV; ++n) map.grad(&G[n * DIM], &D[n * DIM]);
}

// The nodal velocity, acceleration (ACC) and velocity gradient (GRAD) at a
// particle at x in cell c.
template <int DIM, bool ACC, bool GRAD, bool BOX>
__device__ __forceinline__ void gather_particle(const DevState& s, int c, const double* x,
                                                float* nvel, float* nacc, VelGrad<DIM>* grad) {
  if constexpr (BOX) {
    int ijk[3] = {0, 0, 0};
    float xi[DIM], ihl[DIM];
    cell_ijk<DIM>(s, c, ijk);
    box_xi_f32<DIM>(s, ijk, x, xi, ihl);
    gather_box<DIM, ACC, GRAD>(s, ijk, xi, ihl, nvel, nacc, grad);
  } else {
    constexpr int NV = Elem<DIM>::NV;
    float xi[DIM], N[NV], Xr[NV * DIM];
    int nid[NV];
    xi_f32<DIM, false>(s, c, x, xi);
    shapefn<DIM>(xi, N);
    cell_nodes_rel<DIM, false>(s, c, nid, Xr);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      nvel[d] = 0.f;
      if constexpr (ACC) nacc[d] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      float vn[DIM], an[DIM];
      load_nfv<DIM, ACC>(s.nfv, nid[i], vn, an);
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        nvel[d] += N[i] * vn[d];
        if constexpr (ACC) nacc[d] += N[i] * an[d];
      }
    }
    if constexpr (GRAD) {
      float D[NV * DIM];
      dn_dx_all_f<DIM, false>(s, c, xi, Xr, D);
      *grad = velocity_gradient<DIM>(s, c, nid, D);
    }
  }
}

template <int DIM, bool BOX>
__global__ void __launch_bounds__(128) k_stress_mixed(DevState s, float dt) {
  after_previous();
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= s.np) return;
  const int c = s.cell[p];
  if (c < 0) return;
  double x[DIM];
  load_x<DIM>(s, p, x);
  float nvel[DIM];
  VelGrad<DIM> grad;
  gather_particle<DIM, false, true, BOX>(s, c, x, nvel, nullptr, &grad);
  stress_update_mixed<DIM>(s, MGlobalRow<DIM>{s, p}, grad, dt);
}

template <bool BOX>
constexpr int mixed_g2p_min_blocks() {
  return BOX ? MPM_MIXED_G2P_MIN_BLOCKS : MPM_MIXED_G2P_GENERAL_MIN_BLOCKS;
}

// --------------------------------------------------------------------- G2P
// MUSL (mpm_scheme_musl.tcc:20-35): the kinematics without committing the
// positions -- the updated ones go to xnext (k_commit_locate_mixed commits them
// after the second mapping and the stress update), no locate here.
template <int DIM, bool STRESS, bool FLIP, bool BOX, bool MUSL = false>
__global__ void __launch_bounds__(128, mixed_g2p_min_blocks<BOX>())
    k_g2p_mixed(DevState s, double dt, float beta) {
  after_previous();
  static_assert(!(MUSL && STRESS), "MUSL updates the stress after its second mapping");
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= s.np) return;
  const int c = s.cell[p];
  if (c < 0) return;
  const int64_t np = s.np;
  double x[DIM];
  load_x<DIM>(s, p, x);
  float nvel[DIM], nacc[DIM];
  VelGrad<DIM> grad;
  gather_particle<DIM, FLIP, STRESS, BOX>(s, c, x, nvel, nacc, &grad);
  const float dtf = (float)dt;
  float v[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) v[d] = pmf<DIM>(s, PM<DIM>::V + d, p);
  if constexpr (FLIP) {
#pragma unroll
    for (int d = 0; d < DIM; ++d) v[d] = fmaf(nacc[d], dtf, v[d]);
#pragma unroll
    for (int d = 0; d < DIM; ++d) v[d] = fmaf(beta, v[d], __fmul_rn(1.f - beta, nvel[d]));
  } else {
#pragma unroll
    for (int d = 0; d < DIM; ++d) v[d] = nvel[d];
  }
  double xn[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    const double dx = __dmul_rn((double)nvel[d], dt);  // FP64 position / displacement update
    xn[d] = x[d] + dx;
    if constexpr (MUSL)
      s.xnext[(int64_t)d * np + p] = xn[d];
    else
      s.pf[(int64_t)(PDX<DIM>::X + d) * np + p] = xn[d];
    s.pf[(int64_t)(PDX<DIM>::U + d) * np + p] += dx;
  }
  const int pv = s.pvc[p];
  if (pv >= 0) {
    const ParticleVC& r = s.pvcs[pv];
#pragma unroll
    for (int d = 0; d < DIM; ++d)
      if (r.mask & (1u << d)) v[d] = (float)r.value[d];
  }
#pragma unroll
  for (int d = 0; d < DIM; ++d) set_pmf<DIM>(s, PM<DIM>::V + d, p, v[d]);
  if constexpr (MUSL) return;
  if constexpr (STRESS) stress_update_mixed<DIM>(s, MGlobalRow<DIM>{s, p}, grad, dtf);
  settle_particle<DIM, BOX>(s, p, xn, c);
}

// G2P of the velocity updates that carry a mapping matrix (particle.tcc:
// 1071-1139, 1663-1730), k_g2p<DIM, STRESS, VU, BOX> of the FP64 path with the
// nodal values in FP32: the matrix B at the step-start position -- affine
// sum_i N_i v_i r_i^T (APIC, ASFLIP; r_i = node i - x from FP64 positions) or
// the velocity gradient sum_i v_i dN_i/dx^T (TPIC), entries below 1e-15 set to
// zero, kept in FP64 -- then APIC and TPIC take the PIC update and ASFLIP the
// FLIP/PIC blend for the velocity and the separable blend for the position.
template <int DIM, bool STRESS, int VU, bool BOX>
__global__ void __launch_bounds__(128, BOX ? 6 : MPM_MIXED_AFFINE_G2P_MIN_BLOCKS)
    k_g2p_mixed_affine(DevState s, double dt, float beta) {
  after_previous();
  static_assert(VU >= 2, "the mapping-matrix updates");
  constexpr int NV = Elem<DIM>::NV;
  constexpr bool ASFLIP = VU == 2, TPIC = VU == 3;  // 4 APIC
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= s.np) return;
  const int c = s.cell[p];
  if (c < 0) return;
  const int64_t np = s.np;
  const float dtf = (float)dt;
  double x[DIM];
  load_x<DIM>(s, p, x);
  int nid[NV];
  float nvel[DIM], nacc[DIM], B[DIM * DIM];
  VelGrad<DIM> grad;
  if constexpr (BOX) {
    // B = sum_i N_i v_i r_i^T of a box cell is the velocity gradient with column b
    // times (1 - xi_b^2) (len_b / 2)^2, so one interpolating visit of the nodes
    // serves all: 246k particles in 3D 55 -> 40 us, and the P2G that divides by the
    // diagonal shape tensor 38 -> 31
    int ijk[3] = {0, 0, 0};
    float xi[DIM], ihl[DIM];
    cell_ijk<DIM>(s, c, ijk);
    box_xi_f32<DIM>(s, ijk, x, xi, ihl);
    gather_box<DIM, ASFLIP, true>(s, ijk, xi, ihl, nvel, nacc, &grad);
#pragma unroll
    for (int b = 0; b < DIM; ++b) {
      const float w = TPIC ? 1.f : (1.f - xi[b]) * (1.f + xi[b]) / (ihl[b] * ihl[b]);
#pragma unroll
      for (int a = 0; a < DIM; ++a) B[a * DIM + b] = grad.L[a * DIM + b] * w;
    }
    if constexpr (ASFLIP) grid_cell_nodes<DIM>(s, c, nid);
  } else {
    float xi[DIM], N[NV], Xr[NV * DIM], xr[DIM];
    xi_f32<DIM, BOX>(s, c, x, xi);
    shapefn<DIM>(xi, N);
    {
      // the branch vectors r_i = X_i - x as (X_i - X_0) - (x - X_0) in FP32
      double X[NV * DIM];
      cell_nodes_coords<DIM>(s, c, nid, X);
#pragma unroll
      for (int n = 0; n < NV; ++n)
#pragma unroll
        for (int d = 0; d < DIM; ++d) Xr[n * DIM + d] = (float)(X[n * DIM + d] - X[d]);
#pragma unroll
      for (int d = 0; d < DIM; ++d) xr[d] = (float)(x[d] - X[d]);
    }
    float vn[NV][DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) nvel[d] = nacc[d] = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      float an[DIM];
      load_nfv<DIM, ASFLIP>(s.nfv, nid[i], vn[i], an);
#pragma unroll
      for (int d = 0; d < DIM; ++d) nvel[d] += N[i] * vn[i][d];
      if constexpr (ASFLIP) {
#pragma unroll
        for (int d = 0; d < DIM; ++d) nacc[d] += N[i] * an[d];
      }
    }
    float D[NV * DIM];
    if constexpr (TPIC || ASFLIP || STRESS) {
      dn_dx_all_f<DIM, BOX>(s, c, xi, Xr, D);
      grad = velocity_gradient<DIM>(s, c, nid, D);
    }
#pragma unroll
    for (int q = 0; q < DIM * DIM; ++q) B[q] = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      float r[DIM];
#pragma unroll
      for (int d = 0; d < DIM; ++d) r[d] = Xr[i * DIM + d] - xr[d];
#pragma unroll
      for (int a = 0; a < DIM; ++a)
#pragma unroll
        for (int b = 0; b < DIM; ++b) {
          if constexpr (TPIC)
            B[a * DIM + b] += vn[i][a] * D[i * DIM + b];
          else
            B[a * DIM + b] += (N[i] * vn[i][a]) * r[b];
        }
    }
  }
#pragma unroll
  for (int q = 0; q < DIM * DIM; ++q) {
    if (fabsf(B[q]) < 1.E-15f) B[q] = 0.f;
    s.mapb[(int64_t)q * np + p] = (double)B[q];
  }
  float v[DIM], sep[DIM];  // sep: the velocity that moves the particle
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    v[d] = pmf<DIM>(s, PM<DIM>::V + d, p);
    sep[d] = nvel[d];
  }
  if constexpr (ASFLIP) {
    // beta (particle.tcc:1711-1730): 0 next to a velocity-constrained node or
    // when the deformation gradient increment compresses
    float bp = 1.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int bci = s.bc_index[nid[i]];
      if (bci >= 0 && s.bcs[bci].vel_mask != 0) bp = 0.f;
    }
    // det(I + A) < 1 with A = sum_i v_i dN_i/dx^T dt: the test is on
    // det(I + A) - 1 = tr A + (sum of A's principal 2x2 minors) + det A, which
    // FP32 resolves down to A's own rounding (1 + A in FP32 would lose every
    // increment below 6e-8 and flip the sign of J - 1 against the FP64 run)
    float A[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int a = 0; a < DIM; ++a)
#pragma unroll
      for (int b = 0; b < DIM; ++b) A[a * 3 + b] = grad.L[a * DIM + b] * dtf;
#pragma unroll
    for (int q = 0; q < 9; ++q)
      if (fabsf(A[q]) < 1.E-15f) A[q] = 0.f;  // the snaps of F's entries at 1e-15
    const float tr = A[0] + A[4] + A[8];
    const float m2 = (A[0] * A[4] - A[1] * A[3]) + (A[0] * A[8] - A[2] * A[6]) + (A[4] * A[8] - A[5] * A[7]);
    const float d3 = A[0] * (A[4] * A[8] - A[5] * A[7]) - A[1] * (A[3] * A[8] - A[5] * A[6]) +
                     A[2] * (A[3] * A[7] - A[4] * A[6]);
    if (tr + m2 + d3 < 0.f) bp = 0.f;
    // particle.tcc:1096-1110: FLIP/PIC blend for the velocity, the separable
    // blend for the position
    float flip[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) flip[d] = v[d] + nacc[d] * dtf;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      sep[d] = bp * beta * flip[d] + (1.f - bp * beta) * nvel[d];
      v[d] = beta * flip[d] + (1.f - beta) * nvel[d];
    }
  } else {
#pragma unroll
    for (int d = 0; d < DIM; ++d) v[d] = nvel[d];
  }
  double xn[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    const double dx = (double)sep[d] * dt;  // FP64 position / displacement update
    xn[d] = x[d] + dx;
    s.pf[(int64_t)(PDX<DIM>::X + d) * np + p] = xn[d];
    s.pf[(int64_t)(PDX<DIM>::U + d) * np + p] += dx;
  }
  const int pv = s.pvc[p];
  if (pv >= 0) {
    const ParticleVC& r = s.pvcs[pv];
#pragma unroll
    for (int d = 0; d < DIM; ++d)
      if (r.mask & (1u << d)) v[d] = (float)r.value[d];
  }
#pragma unroll
  for (int d = 0; d < DIM; ++d) set_pmf<DIM>(s, PM<DIM>::V + d, p, v[d]);
  if constexpr (STRESS) stress_update_mixed<DIM>(s, MGlobalRow<DIM>{s, p}, grad, dtf);
  settle_particle<DIM, BOX>(s, p, xn, c);
}

// MUSL end of step: the new positions (FP64) replace the old, then locate
template <int DIM, bool BOX>
__global__ void __launch_bounds__(128) k_commit_locate_mixed(DevState s) {
  after_previous();
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= s.np) return;
  const int c = s.cell[p];
  if (c < 0) return;
  const int64_t np = s.np;
  double xn[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    xn[d] = s.xnext[(int64_t)d * np + p];
    s.pf[(int64_t)(PDX<DIM>::X + d) * np + p] = xn[d];
  }
  settle_particle<DIM, BOX>(s, p, xn, c);
}

// USL G2P + stress update + locate with the block's particle slices staged in
// shared memory by the bulk-copy engine (as k_g2p_staged of the FP64 path):
// phase A x, u (FP64), v (FP32), cell, material, velocity-constraint slot;
// phase B stress .. P (FP32), MohrCoulomb state (FP32).  The arithmetic is
// k_g2p_mixed<DIM, true, FLIP, BOX>'s.
static_assert(MSTAGE_T == PAD_PARTICLES, "staged slices are whole padded blocks");
template <int DIM>
constexpr size_t mixed_staged_smem_bytes(bool mc) {
  return (size_t)2 * DIM * MSTAGE_T * 8 + (size_t)(PM<DIM>::MASS + (mc ? SVF_N : 0)) * MSTAGE_T * 4 +
         MSTAGE_T * (4 + 2 + 2);
}

// One block of MSTAGE_T particles (block index bx) with the staging buffers
// smem, the two initialised copy barriers bar in the phase of the given
// parity, and the block's timed-out flag.
// WRITES_DONE: wait for the block's stores to complete (a later pass of the
// same launch reads them), else only until they have read shared memory.
template <int DIM, bool FLIP, bool BOX, bool WRITES_DONE = false>
__device__ __forceinline__ void g2p_staged_block_mixed(const DevState& s, double dt, float beta,
                                                       int64_t bx, unsigned char* smem, uint64_t* bar,
                                                       unsigned parity, int& timed_out) {
  constexpr int T = MSTAGE_T;
  constexpr int XROWS = 2 * DIM;       // x, u
  constexpr int MROWS = PM<DIM>::MASS;  // v .. P
  const bool mc = s.svf != nullptr;
  double* xr = reinterpret_cast<double*>(smem);
  float* mr = reinterpret_cast<float*>(xr + XROWS * T);
  float* svr = mr + MROWS * T;
  int32_t* scell = reinterpret_cast<int32_t*>(svr + (mc ? SVF_N * T : 0));
  uint16_t* smat = reinterpret_cast<uint16_t*>(scell + T);
  int16_t* spvc = reinterpret_cast<int16_t*>(smat + T);
  const int t = threadIdx.x;
  const int64_t p0 = bx * T;
  const int64_t np = s.np;
  if (t == 0) timed_out = 0;
  __syncthreads();
  if (t == 0) {
    bulk::mbar_arrive_expect_tx(&bar[0], 2 * DIM * T * 8 + DIM * T * 4 + T * (4 + 2 + 2));
    for (int f = 0; f < XROWS; ++f) bulk::load(xr + f * T, s.pf + f * np + p0, T * 8, &bar[0]);
    for (int f = PM<DIM>::V; f < PM<DIM>::V + DIM; ++f)
      bulk::load(mr + f * T, s.pm + f * np + p0, T * 4, &bar[0]);
    bulk::load(scell, s.cell + p0, T * 4, &bar[0]);
    bulk::load(smat, s.mat + p0, T * 2, &bar[0]);
    bulk::load(spvc, s.pvc + p0, T * 2, &bar[0]);
    bulk::mbar_arrive_expect_tx(&bar[1], (MROWS - DIM + (mc ? SVF_N : 0)) * T * 4);
    for (int f = PM<DIM>::V + DIM; f < MROWS; ++f)
      bulk::load(mr + f * T, s.pm + f * np + p0, T * 4, &bar[1]);
    if (mc)
      for (int k = 0; k < SVF_N; ++k) bulk::load(svr + k * T, s.svf + k * np + p0, T * 4, &bar[1]);
  }
  // the test hook waits for the next phase, which no copy completes
  const bool okA = bulk::mbar_wait(&bar[0], parity) &&
                   !(s.test_wait_timeout && !bulk::mbar_wait(&bar[0], parity ^ 1u, 16));
  const int c = okA ? scell[t] : -1;
  const int64_t p = p0 + t;
  const MSmemRow r{mr, svr, t, okA ? (int)smat[t] : 0, p0 + t};
  double xn[DIM];
  const bool active = c >= 0;
  VelGrad<DIM> grad;
  if (active) {
    double x[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) x[d] = xr[(PDX<DIM>::X + d) * T + t];
    // the velocity gradient (and, on a box, the visit of the nodes for it) comes
    // here, while the second phase's copies are in flight
    float nvel[DIM], nacc[DIM];
    gather_particle<DIM, FLIP, true, BOX>(s, c, x, nvel, nacc, &grad);
    const float dtf = (float)dt;
    float v[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) v[d] = r.m(PM<DIM>::V + d);
    if constexpr (FLIP) {
#pragma unroll
      for (int d = 0; d < DIM; ++d) v[d] = fmaf(nacc[d], dtf, v[d]);
#pragma unroll
      for (int d = 0; d < DIM; ++d) v[d] = fmaf(beta, v[d], __fmul_rn(1.f - beta, nvel[d]));
    } else {
#pragma unroll
      for (int d = 0; d < DIM; ++d) v[d] = nvel[d];
    }
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      const double dx = __dmul_rn((double)nvel[d], dt);  // FP64 position / displacement update
      xn[d] = x[d] + dx;
      xr[(PDX<DIM>::X + d) * T + t] = xn[d];
      xr[(PDX<DIM>::U + d) * T + t] += dx;
    }
    const int pv = spvc[t];
    if (pv >= 0) {
      const ParticleVC& vc = s.pvcs[pv];
#pragma unroll
      for (int d = 0; d < DIM; ++d)
        if (vc.mask & (1u << d)) v[d] = (float)vc.value[d];
    }
#pragma unroll
    for (int d = 0; d < DIM; ++d) r.m(PM<DIM>::V + d) = v[d];
  }
  const bool okB = okA && bulk::mbar_wait(&bar[1], parity);
  if (!okA || !okB) timed_out = 1;
  if (active && okB) stress_update_mixed<DIM>(s, r, grad, (float)dt);
  bulk::fence_shared_to_async();
  __syncthreads();
  if (timed_out) {
    if (t == 0) {
      raise_err(s, ERR_TIMEOUT);
      bulk::mbar_wait(&bar[0], parity);
      bulk::mbar_wait(&bar[1], parity);
    }
    return;
  }
  if (t == 0) {
    for (int f = 0; f < XROWS; ++f) bulk::store(s.pf + f * np + p0, xr + f * T, T * 8);
    for (int f = 0; f < MROWS; ++f)  // the initial volume and density never change
      if (f != PM<DIM>::V0 && f != PM<DIM>::RHO0) bulk::store(s.pm + f * np + p0, mr + f * T, T * 4);
    if (mc)  // phi, psi, cohesion and tension cutoff change only with softening
      for (int k = 0; k < SVF_N; ++k)
        if (s.any_softening || k == SV_YIELD || k >= SV_EPS)
          bulk::store(s.svf + k * np + p0, svr + k * T, T * 4);
    bulk::store_commit();
  }
  if (active) settle_particle<DIM, BOX>(s, p, xn, c);
  if (t == 0) {
    if constexpr (WRITES_DONE)
      bulk::store_wait_all();
    else
      bulk::store_wait_read();
  }
}

template <int DIM, bool FLIP, bool BOX>
__global__ void __launch_bounds__(MSTAGE_T, mixed_g2p_min_blocks<BOX>())
    k_g2p_mixed_staged(DevState s, double dt, float beta) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t bar[2];
  __shared__ int timed_out;
  if (threadIdx.x == 0) {
    bulk::mbar_init(&bar[0], 1);
    bulk::mbar_init(&bar[1], 1);
    bulk::fence_barrier_init();
  }
  after_previous();
  g2p_staged_block_mixed<DIM, FLIP, BOX>(s, dt, beta, blockIdx.x, smem, bar, 0u, timed_out);
}

template <auto Kernel>
void prefer_shared_memory() {
  static unsigned done = 0;  // one bit per device
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 32 && !(done & (1u << dev))) {
    cudaFuncSetAttribute(Kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                         (int)cudaSharedmemCarveoutMaxShared);
    done |= 1u << dev;
  }
}

// The MohrCoulomb updates deferred by stress_update_mixed, one thread per
// listed particle (the light entries, then the heavy ones): the full FP64
// update (mohr_coulomb.tcc:348-513, as mc_return's passes) from the FP32
// stress and state before the step's update, rounded back to FP32; the number
// of corrections is kept for the next step's grouping.
// The FP64 returns of listed entries begin, begin + stride, ...
template <int DIM>
__device__ __forceinline__ void mc_return_mixed_range(const DevState& s, unsigned begin, unsigned stride) {
  const unsigned nl = *s.nplastic, n = nl + *s.nplastic_heavy;
  const int64_t np = s.np;
  for (unsigned t = begin; t < n; t += stride) {
    const unsigned i = list_slot(s, t, nl);
    const int64_t p = s.plist[i];
    const MGlobalRow<DIM> r{s, p};
    const int mi = s.mat[p];
    float sig[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, de[6], svf[SVF_N], out[6];
#pragma unroll
    for (int k = 0; k < PF<DIM>::NS; ++k) sig[k] = r.m(PM<DIM>::S + k);
#pragma unroll
    for (int k = 0; k < 6; ++k) de[k] = s.pbuf_f[(int64_t)k * np + i];
    const float rho = s.pbuf_f[(int64_t)6 * np + i];
#pragma unroll
    for (int k = 0; k < SVF_N; ++k) svf[k] = r.svf(k);
    double sd[6], ded[6], svd[SV_N], od[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      sd[k] = (double)sig[k];
      ded[k] = (double)de[k];
    }
#pragma unroll
    for (int k = 0; k < SVF_N; ++k) svd[k] = (double)svf[k];
    svd[SV_PD] = r.pd();
    int nc = 0;
    mc_return<double>(s.mats[mi], sd, ded, (double)rho, svd, od, &nc);
    s.rpass[p] = (uint8_t)(nc < 255 ? nc : 255);
#pragma unroll
    for (int k = 0; k < 6; ++k) out[k] = (float)od[k];
#pragma unroll
    for (int k = 0; k < SVF_N; ++k) svf[k] = (float)svd[k];
    r.pd() = svd[SV_PD];
    const int first = s.mats_f[mi].softening ? 0 : SV_EPS;  // phi..tc change only with softening
    r.svf(SV_YIELD) = svf[SV_YIELD];
#pragma unroll
    for (int k = 1; k < SVF_N; ++k)
      if (k >= first) r.svf(k) = svf[k];
#pragma unroll
    for (int k = 0; k < PF<DIM>::NS; ++k) r.m(PM<DIM>::S + k) = out[k];
  }
}

template <int DIM>
__global__ void __launch_bounds__(128, MPM_MC_RETURN_MIN_BLOCKS) k_mc_return_mixed(DevState s) {
  after_previous();
  mc_return_mixed_range<DIM>(s, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

inline unsigned nblk(int64_t n, int threads) { return (unsigned)((n + threads - 1) / threads); }

// ------------------------------------------------------ persistent steps
// The exclusive scan of the counts of chunk `chunk` (SCAN_BLOCK cells; T
// threads, SCAN_BLOCK / T consecutive cells each) into start, and the chunk's
// total into bsum[chunk].
template <int T>
__device__ __forceinline__ void scan_chunk(const int32_t* cnt, int32_t* start, int32_t* bsum,
                                           int64_t n, int64_t chunk, int32_t* red) {
  constexpr int PER = SCAN_BLOCK / T;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int64_t base = chunk * SCAN_BLOCK + (int64_t)t * PER;
  int32_t v[PER], run = 0;
#pragma unroll
  for (int i = 0; i < PER; ++i) v[i] = base + i < n ? cnt[base + i] : 0;
#pragma unroll
  for (int i = 0; i < PER; ++i) run += v[i];
  int32_t x = run;  // inclusive scan of the thread totals within the warp
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int32_t y = __shfl_up_sync(0xffffffffu, x, off);
    if (lane >= off) x += y;
  }
  if (lane == 31) red[w] = x;
  __syncthreads();
  int32_t prefix = x - run;
  for (int k = 0; k < w; ++k) prefix += red[k];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    if (base + i < n) start[base + i] = prefix;
    prefix += v[i];
  }
  if (t == T - 1) bsum[chunk] = prefix;
  __syncthreads();  // red is reused by the next chunk
}

// The total of bsum[0, count) by the block's T threads (every thread gets it).
template <int T>
__device__ __forceinline__ int32_t block_total(const int32_t* bsum, int64_t count, int32_t* red) {
  int32_t x = 0;
  for (int64_t j = threadIdx.x; j < count; j += T) x += bsum[j];
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  int32_t total = 0;
#pragma unroll
  for (int k = 0; k < T / 32; ++k) total += red[k];
  __syncthreads();
  return total;
}

// K whole mixed USL steps on a tensor-product grid in one cooperative launch.
// Each pass is the body of the corresponding one-pass kernel of step_mixed,
// over block-sized pieces (cell tiles, particle blocks, node blocks) taken
// grid-stride, so the results are bit for bit those of the per-pass launches
// (the P2G tiles have 128 threads; each cell's particle ids are sorted before
// they are added, so the slot order the counting sort leaves does not matter):
//   count | scan chunks | chunk prefixes | fill | P2G | nodes |
//   G2P + stress (and the next step's counts zeroed) | returns
template <int DIM, bool FLIP>
__global__ void __launch_bounds__(MSTAGE_T, DIM == 2 ? MPM_PERSISTENT_MIN_BLOCKS_2D : MPM_PERSISTENT_MIN_BLOCKS_3D)
    k_steps_persistent_mixed(DevState s, StepArgs a, PersistentArgs q) {
  constexpr int T = MSTAGE_T;
  constexpr int NV = Elem<DIM>::NV;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t bar[2];
  __shared__ int timed_out, go;
  __shared__ int32_t red[T / 32];
  const int t = threadIdx.x;
  const unsigned G = gridDim.x;
  const int64_t np = s.np, nc = s.ncells;
  const int64_t pblocks = (np + T - 1) / T, tiles = (nc + T / NV - 1) / (T / NV);
  const int64_t nodeblocks = (s.nn + T - 1) / T, chunks = (nc + SCAN_BLOCK - 1) / SCAN_BLOCK;
  const unsigned gi = blockIdx.x * T + t, gs = G * T;  // grid-stride start and stride
  __shared__ long long step0;
  unsigned gen = 0;
  if (t == 0) {
    bulk::mbar_init(&bar[0], 1);
    bulk::mbar_init(&bar[1], 1);
    bulk::fence_barrier_init();
    gen = ld_acquire_gpu(&q.barrier[1]);
    step0 = *q.step;  // block 0 advances it only after the last barrier
  }
  for (int64_t i = gi; i < nc; i += gs) s.cnt[i] = 0;
  if (!grid_barrier(s, q.barrier, G, gen, go)) return;
  unsigned parity = 0;
  for (int64_t k = 0; k < q.nsteps; ++k) {
    double gm = 1.0;  // the host's ramp, the same operations
    if (q.ramp > 0.0) gm = fmin(1.0, static_cast<double>(step0 + k) * a.dt / q.ramp);
    const double g[3] = {gm * q.gravity[0], gm * q.gravity[1], gm * q.gravity[2]};
    // counting sort
    if (blockIdx.x == 0 && t == 0) {
      if (s.svf) *s.nplastic = *s.nplastic_heavy = 0;
    }
    for (int64_t b = blockIdx.x; b < pblocks; b += G) count_particle(s, b * T + t);
    if (!grid_barrier(s, q.barrier, G, gen, go)) return;
    for (int64_t b = blockIdx.x; b < chunks; b += G) scan_chunk<T>(s.cnt, s.start, s.bsum, nc, b, red);
    if (!grid_barrier(s, q.barrier, G, gen, go)) return;
    for (int64_t b = blockIdx.x; b < chunks; b += G) {
      const int32_t prefix = block_total<T>(s.bsum, b, red);
      for (int64_t i = b * SCAN_BLOCK + t; i < nc && i < (b + 1) * SCAN_BLOCK; i += T) s.start[i] += prefix;
      if (b == chunks - 1 && t == 0) s.start[nc] = prefix + s.bsum[b];
    }
    if (!grid_barrier(s, q.barrier, G, gen, go)) return;
    for (int64_t b = blockIdx.x; b < pblocks; b += G) fill_particle(s, b * T + t);
    if (!grid_barrier(s, q.barrier, G, gen, go)) return;
    // P2G of mass, momentum and forces
    for (int64_t b = blockIdx.x; b < tiles; b += G) {
      p2g_tile_mixed<DIM, 2, true, T>(s, b);
      __syncthreads();  // the tile's staged rows are consumed
    }
    if (!grid_barrier(s, q.barrier, G, gen, go)) return;
    for (int64_t b = blockIdx.x; b < nodeblocks; b += G) node_update_mixed<DIM, 1>(s, a.dt, a.damping, g, b * T + t);
    if (!grid_barrier(s, q.barrier, G, gen, go)) return;
    // G2P with the stress update; the counts are free once the nodes are done
    for (int64_t b = blockIdx.x; b < pblocks; b += G) {
      g2p_staged_block_mixed<DIM, FLIP, true, true>(s, a.dt, (float)a.beta, b, smem, bar, parity,
                                                    timed_out);
      parity ^= 1u;
      __syncthreads();  // the block's staging buffers are free again
    }
    for (int64_t i = gi; i < nc; i += gs) s.cnt[i] = 0;
    if (!grid_barrier(s, q.barrier, G, gen, go)) return;
    if (s.svf) {
      mc_return_mixed_range<DIM>(s, gi, gs);
      if (!grid_barrier(s, q.barrier, G, gen, go)) return;
    }
  }
  if (blockIdx.x == 0 && t == 0) *q.step = step0 + q.nsteps;
}

template <int DIM, bool FLIP>
cudaError_t launch_persistent(const DevState& s, const StepArgs& a, const PersistentArgs& q,
                              cudaStream_t st) {
  auto kernel = k_steps_persistent_mixed<DIM, FLIP>;
  const size_t sm = mixed_staged_smem_bytes<DIM>(s.svf != nullptr);
  prefer_shared_memory<k_steps_persistent_mixed<DIM, FLIP>>();
  int dev = 0, sms = 0, per_sm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, MSTAGE_T, sm);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorCooperativeLaunchTooLarge;
  e = cudaMemsetAsync(q.barrier, 0, 2 * sizeof(unsigned), st);
  if (e != cudaSuccess) return e;
  DevState sv = s;
  StepArgs av = a;
  PersistentArgs qv = q;
  void* args[] = {&sv, &av, &qv};
  return cudaLaunchCooperativeKernel((const void*)kernel, dim3((unsigned)(per_sm * sms)), dim3(MSTAGE_T),
                                     args, sm, st);
}

// The plastic returns of a step.
template <int DIM>
void returns_mixed(const DevState& s, const StepArgs& a, cudaStream_t st, Profiler& pr) {
  if (!s.svf) return;
  const unsigned all = nblk(s.np, 128), cap = 148u * (unsigned)return_blocks(a);
  pr.begin(K_MC_RETURN, st);
  // A plain launch: the return keeps part of its state in local memory and needs
  // the L1 that the staged G2P gave to shared memory.  Blocks that an SM takes
  // on while G2P's last ones run keep that split to their end: a flowing 0.8M-
  // particle step took 323 us with a dependent launch here, 263 with this one.
  k_mc_return_mixed<DIM><<<all < cap ? all : cap, 128, 0, st>>>(s);
  pr.end(K_MC_RETURN, st);
}

template <int DIM, bool BOX>
void step_mixed(const DevState& s, const StepArgs& a, cudaStream_t st, Profiler& pr) {
  const int64_t np = s.np, nn = s.nn;
  if (np == 0) return;
  const unsigned nt = (unsigned)node_block(a);
  const unsigned pb = nblk(np, 128), nb = nblk(nn, nt);
  // P2G cell tiles of the step's launch shape
  auto p2g = [&](auto mode) {
    constexpr int MODE = decltype(mode)::value;
    auto launch = [&](auto kernel, int threads) {
      const unsigned tiles = nblk(s.ncells, threads / Elem<DIM>::NV);
      const bool dependent = p2g_dependent(a, tiles);
      launch_kernel(dependent, kernel, tiles, threads, 0, st, s, dependent);
    };
    if constexpr (MODE != 1) {  // the mass-momentum mapping velocity (128-thread tiles)
      if (a.vupd == 2 || a.vupd == 4) return launch(k_p2g_tiles_mixed<DIM, MODE, BOX, 128, 1>, 128);
      if (a.vupd == 3) return launch(k_p2g_tiles_mixed<DIM, MODE, BOX, 128, 2>, 128);
    }
    if (BOX && tile_threads(a, BOX, DIM, s, true) == 128)
      launch(k_p2g_tiles_mixed<DIM, MODE, BOX, 128>, 128);
    else
      launch(k_p2g_tiles_mixed<DIM, MODE, BOX>, p2g_tile_t<BOX>());
  };
  // G2P of the mapping-matrix updates (ASFLIP 2, TPIC 3, APIC 4)
  auto g2p_affine = [&](auto stress) {
    constexpr bool STRESS = decltype(stress)::value;
    const float b = (float)a.beta;
    if (a.vupd == 2)
      launch_dependent(k_g2p_mixed_affine<DIM, STRESS, 2, BOX>, pb, 128, 0, st, s, a.dt, b);
    else if (a.vupd == 3)
      launch_dependent(k_g2p_mixed_affine<DIM, STRESS, 3, BOX>, pb, 128, 0, st, s, a.dt, b);
    else
      launch_dependent(k_g2p_mixed_affine<DIM, STRESS, 4, BOX>, pb, 128, 0, st, s, a.dt, b);
  };
  auto mc_returns = [&]() {
    if (!a.defer_returns) returns_mixed<DIM>(s, a, st, pr);
  };
  if (a.scheme == 1 && a.phase == 2) goto usl_second_half;
  if (a.returns_first) {
    check_cuda(fork_side(a, st), "returns beside the sort: fork");
    returns_mixed<DIM>(s, a, a.side, pr);
  }
  pr.begin(K_SORT, st, sort_kernels(s));
  counting_sort(s, st, 1);
  pr.end(K_SORT, st);
  if (a.returns_first) check_cuda(join_side(a, st), "returns beside the sort: join");
  if (a.scheme == 2) {  // MUSL (mpm_scheme_musl.tcc:20-35)
    pr.begin(K_P2G, st);
    p2g(std::integral_constant<int, 2>{});
    pr.end(K_P2G, st);
    pr.begin(K_NODES_VEL, st);
    launch_dependent(k_nodes_mixed<DIM, 1>, nb, nt, 0, st, s, a.dt, a.damping, a.g[0], a.g[1], a.g[2]);
    pr.end(K_NODES_VEL, st);
    pr.begin(K_G2P, st);
    if (a.flip)
      launch_dependent(k_g2p_mixed<DIM, false, true, BOX, true>, pb, 128, 0, st, s, a.dt, (float)a.beta);
    else
      launch_dependent(k_g2p_mixed<DIM, false, false, BOX, true>, pb, 128, 0, st, s, a.dt, (float)a.beta);
    pr.end(K_G2P, st);
    // mass and momentum again with the updated velocities, nodal velocity,
    // then the stress update at the step's positions
    pr.begin(K_P2G_FORCES, st);
    p2g(std::integral_constant<int, 0>{});
    pr.end(K_P2G_FORCES, st);
    pr.begin(K_NODES_ACC, st);
    launch_dependent(k_nodes_mixed<DIM, 0>, nb, nt, 0, st, s, a.dt, a.damping, a.g[0], a.g[1], a.g[2]);
    pr.end(K_NODES_ACC, st);
    pr.begin(K_STRESS, st);
    launch_dependent(k_stress_mixed<DIM, BOX>, pb, 128, 0, st, s, (float)a.dt);
    pr.end(K_STRESS, st);
    mc_returns();
    pr.begin(K_LOCATE, st);
    launch_dependent(k_commit_locate_mixed<DIM, BOX>, pb, 128, 0, st, s);
    pr.end(K_LOCATE, st);
  } else if (a.scheme == 1) {  // USL
    pr.begin(K_P2G, st);
    p2g(std::integral_constant<int, 2>{});
    pr.end(K_P2G, st);
    if (a.phase == 1) return;
  usl_second_half:
    pr.begin(K_NODES_VEL, st);
    launch_dependent(k_nodes_mixed<DIM, 1>, nb, nt, 0, st, s, a.dt, a.damping, a.g[0], a.g[1], a.g[2]);
    pr.end(K_NODES_VEL, st);
    pr.begin(K_G2P, st);
    const size_t sm = mixed_staged_smem_bytes<DIM>(s.svf != nullptr);
    if (a.vupd >= 2) {
      g2p_affine(std::true_type{});
    } else if (a.flip) {
      prefer_shared_memory<k_g2p_mixed_staged<DIM, true, BOX>>();
      launch_dependent(k_g2p_mixed_staged<DIM, true, BOX>, pb, MSTAGE_T, sm, st, s, a.dt, (float)a.beta);
    } else {
      prefer_shared_memory<k_g2p_mixed_staged<DIM, false, BOX>>();
      launch_dependent(k_g2p_mixed_staged<DIM, false, BOX>, pb, MSTAGE_T, sm, st, s, a.dt, (float)a.beta);
    }
    pr.end(K_G2P, st);
    mc_returns();
  } else {  // USF
    pr.begin(K_P2G, st);
    p2g(std::integral_constant<int, 0>{});
    pr.end(K_P2G, st);
    pr.begin(K_NODES_VEL, st);
    launch_dependent(k_nodes_mixed<DIM, 0>, nb, nt, 0, st, s, a.dt, a.damping, a.g[0], a.g[1], a.g[2]);
    pr.end(K_NODES_VEL, st);
    pr.begin(K_STRESS, st);
    launch_dependent(k_stress_mixed<DIM, BOX>, pb, 128, 0, st, s, (float)a.dt);
    pr.end(K_STRESS, st);
    mc_returns();
    pr.begin(K_P2G_FORCES, st);
    p2g(std::integral_constant<int, 1>{});
    pr.end(K_P2G_FORCES, st);
    pr.begin(K_NODES_ACC, st);
    launch_dependent(k_nodes_mixed<DIM, 2>, nb, nt, 0, st, s, a.dt, a.damping, a.g[0], a.g[1], a.g[2]);
    pr.end(K_NODES_ACC, st);
    pr.begin(K_G2P, st);
    if (a.vupd >= 2)
      g2p_affine(std::false_type{});
    else if (a.flip)
      launch_dependent(k_g2p_mixed<DIM, false, true, BOX>, pb, 128, 0, st, s, a.dt, (float)a.beta);
    else
      launch_dependent(k_g2p_mixed<DIM, false, false, BOX>, pb, 128, 0, st, s, a.dt, (float)a.beta);
    pr.end(K_G2P, st);
  }
  if (!BOX) {  // on a grid every particle settled itself
    pr.begin(K_LOCATE, st);
    launch_locate_fallback(DIM, s, a.remove_lost, st);
    pr.end(K_LOCATE, st);
  }
}

}  // namespace

cudaError_t launch_steps_persistent_mixed(int dim, const DevState& s, const StepArgs& a,
                                          const PersistentArgs& q, cudaStream_t st) {
  if (s.np == 0 || q.nsteps <= 0) return cudaSuccess;
  if (dim == 2)
    return a.flip ? launch_persistent<2, true>(s, a, q, st) : launch_persistent<2, false>(s, a, q, st);
  return a.flip ? launch_persistent<3, true>(s, a, q, st) : launch_persistent<3, false>(s, a, q, st);
}

void launch_returns_mixed(int dim, const DevState& s, const StepArgs& a, cudaStream_t st, Profiler& prof) {
  dim == 2 ? returns_mixed<2>(s, a, st, prof) : returns_mixed<3>(s, a, st, prof);
}

void launch_step_mixed(int dim, const DevState& s, const StepArgs& a, cudaStream_t st,
                       Profiler& prof) {
  // the particle kernels are compiled for tensor-product grids (box cells)
  // and for general meshes
  if (dim == 2)
    s.structured ? step_mixed<2, true>(s, a, st, prof) : step_mixed<2, false>(s, a, st, prof);
  else
    s.structured ? step_mixed<3, true>(s, a, st, prof) : step_mixed<3, false>(s, a, st, prof);
}

}  // namespace mpm_b200

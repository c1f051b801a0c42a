// The residual of the time loop in two launches per RK3 stage.  A block owns
// a tile of consecutive cells (Hilbert order: compact) and keeps what its
// cells share in shared memory:
//   k_tile_gradient  states of the tile's vertices (a2), then every cell's
//                    gradient, limiter, interface states and viscous terms
//                    (a3-a6, a9);
//   k_tile_residual  viscous quantities of the tile's vertices (a10), then
//                    fluxes of the tile's edges (a7), then every cell's
//                    residual and stage update (a8, a13).
// The separate kernels (kernels.cuh) write vertex states, vertex viscous
// terms, fluxes and edge viscous terms to global memory and read them back,
// and need five launches; here they stay on chip, at the price of computing
// the vertices and edges on a tile's rim once per tile that touches them.
// The first stage's last block folds the residual norm, the last stage's
// last block ends the step and sets the next one's dt, so a step is six
// launches instead of twenty.  Per entity the arithmetic is that of
// kernels.cuh, in the same order: the same bits.
// What bounds a step of a small mesh is the latency of these kernels (index
// chains, then FP64 chains of some 35 cycles an operation), hence four blocks
// of 128 per SM: with 128 registers a thread nothing spills (five blocks of 96
// registers: 95 against 80 us per step at 74,528 triangles, three: 120).
// Measured on B200, us per step, before / now: 20,400 triangles 142 / 67,
// 58,140 quadrilaterals 172 / 93.
#pragma once

#include "step.cuh"

namespace o2f {

constexpr int kTileMax = 128;                 // cells of a tile at most
constexpr size_t kTileSmemMax = 160 * 1024;   // dynamic shared memory the tile kernels are allowed

// Tiles of the mesh (device arrays).  Local indices refer to a tile's lists.
struct TileDev {
  int n;                 // tiles
  int cells;             // cells per tile = threads per block
  int max_verts, max_edges;
  const int32_t* voff;   // [n+1] into verts
  const int32_t* verts;  // vertices of each tile's cells, ascending
  const int32_t* eoff;   // [n+1] into edges
  const int32_t* edges;  // edges of each tile's cells, ascending
  const ushort2* edge_v; // local vertices of each listed edge (ev order)
  const ushort2* cell_v; // [4*nc] slot-major: local vertices of the slot's edge (ev order)
  const uint16_t* cell_e;  // [4*nc] slot-major: local index of the slot's edge
};

// cell_gradient_body's vertex states by tile position.
template <typename T>
struct TileVertexStates {
  const ushort2* __restrict__ cell_v;  // at slot 0 of the cell
  int64_t nc;
  const Vec4<T>* s;
  using Index = ushort2;
  __device__ __forceinline__ Index index(int k, int) const { return cell_v[(int64_t)k * nc]; }
  __device__ __forceinline__ Vec4<T> first(Index i) const { return s[i.x]; }
  __device__ __forceinline__ Vec4<T> second(Index i) const { return s[i.y]; }
};

// cell_residual_from's edges by tile position.
template <typename T>
struct TileFluxes {
  const uint16_t* __restrict__ cell_e;  // at slot 0 of the cell
  int64_t nc;
  const Vec4<T>*g, *f, *t;
  const T* ty;
  __device__ __forceinline__ int at(int k, int) const { return cell_e[(int64_t)k * nc]; }
  __device__ __forceinline__ T length(int i) const { return g[i].c; }
  __device__ __forceinline__ Vec4<T> geom(int i) const { return g[i]; }
  __device__ __forceinline__ Vec4<T> flux(int i) const { return f[i]; }
  __device__ __forceinline__ Vec4<T> visc(int i) const { return t[i]; }
  __device__ __forceinline__ T visc_y(int i) const { return ty[i]; }
};

// Launch of a tile kernel that may start before the one ahead of it has ended.
template <typename... P, typename... A>
inline cudaError_t tile_launch(void (*kernel)(P...), const TileDev& td, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(td.n);
  cfg.blockDim = dim3(td.cells);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

template <typename T>
inline size_t tile_gradient_smem(const TileDev& td) {
  return sizeof(Vec4<T>) * td.max_verts;
}
template <typename T>
inline size_t tile_residual_smem(const TileDev& td) {
  return (sizeof(Vec4<T>) + sizeof(T)) * td.max_verts + (3 * sizeof(Vec4<T>) + sizeof(T)) * td.max_edges;
}

// Programmatic dependent launch: the next kernel of the step may start as
// soon as this one's blocks have all started, and does what depends on the
// mesh alone (index chains, geometry into L1) before step_inputs() waits for
// this one's results.  What the step's kernels write (states, interface
// states, viscous terms, residuals) is therefore not constant while a kernel
// that reads it runs: neither the tile kernels nor the device functions they
// share with the separate kernels take it as __restrict__, which would let its
// loads go round the coherent path, or ahead of the wait.  The mesh's arrays
// are constant and do.
__device__ __forceinline__ void step_inputs() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void warm_l1(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// One tile's gradients.  vq_out (may be null): the vertex states, also to
// global memory (a vertex of several tiles gets the same value from each).
template <typename T>
__device__ __forceinline__ void tile_gradient(int tile, const TileDev& td, const Topo& t, const Geom<T>& g,
                                              const Vec4<T>* U, const Phys& ph, const Work<T>& w,
                                              Vec4<T>* vq_out, Vec4<T>* s_vq, const int* gate) {
  const int v0 = td.voff[tile], nv = td.voff[tile + 1] - v0;
  const int64_t c = (int64_t)tile * td.cells + threadIdx.x;
  const bool mine = threadIdx.x < td.cells && c < t.nc;
  int v = 0;
  VertexFan<T> fan;
  if (threadIdx.x < nv) {
    v = td.verts[v0 + threadIdx.x];
    fan = vertex_fan<T>(v, t.voff, t.vcid, g.vw, t.vbc);
  }
  if (mine) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int s = t.slot[(int64_t)k * t.nc + c];
      if (s < 0) continue;
      const int e = s >> 1;
      warm_l1(t.ec + e);
      warm_l1(t.ebc + e);
      warm_l1(g.egeom + e);
      warm_l1(g.ectr + e);
      warm_l1(td.cell_v + (int64_t)k * t.nc + c);
    }
    warm_l1(g.cgeom + c);
  }
  step_inputs();
  if (gated(gate)) return;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    if (i >= blockDim.x) {
      v = td.verts[v0 + i];
      fan = vertex_fan<T>(v, t.voff, t.vcid, g.vw, t.vbc);
    }
    const Vec4<T> q = vertex_state_of<T>(fan, t.vcid, g.vw, U, ph);
    s_vq[i] = q;
    if (vq_out) vq_out[v] = q;
  }
  __syncthreads();
  if (mine)
    cell_gradient_from<T, false>(c, t.nc, t.slot, g, TileVertexStates<T>{td.cell_v + c, t.nc, s_vq}, t.ec, t.ebc, U,
                                 ph, w.eL, w.eR, w.ctq, w.ctqy, nullptr);
}

// One tile's vertex viscous quantities and edge fluxes, into shared memory;
// false when the loop has stopped.  ed: the accessor of cell c.
template <typename T>
__device__ __forceinline__ bool tile_fluxes(int tile, const TileDev& td, const Topo& t, const Geom<T>& g,
                                            const Phys& ph, const Work<T>& w, int64_t c, unsigned char* smem,
                                            const int* gate, TileFluxes<T>& ed) {
  Vec4<T>* s_vt = reinterpret_cast<Vec4<T>*>(smem);
  Vec4<T>* s_g = s_vt + td.max_verts;
  Vec4<T>* s_f = s_g + td.max_edges;
  Vec4<T>* s_t = s_f + td.max_edges;
  T* s_ty = reinterpret_cast<T*>(s_t + td.max_edges);
  T* s_vy = s_ty + td.max_edges;
  ed = TileFluxes<T>{td.cell_e + c, t.nc, s_g, s_f, s_t, s_ty};
  const int v0 = td.voff[tile], nv = td.voff[tile + 1] - v0;
  const int e0 = td.eoff[tile], ne = td.eoff[tile + 1] - e0;
  VertexFan<T> fan;
  if (threadIdx.x < nv) fan = vertex_fan<T>(td.verts[v0 + threadIdx.x], t.voff, t.vcid, g.vw, t.vbc);
  for (int i = threadIdx.x; i < ne; i += blockDim.x) {
    const int e = td.edges[e0 + i];
    s_g[i] = g.egeom[e];
    warm_l1(t.ebc + e);
    warm_l1(td.edge_v + e0 + i);
  }
  if (threadIdx.x < td.cells && c < t.nc) {
    warm_l1(g.cgeom + c);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      warm_l1(t.slot + (int64_t)k * t.nc + c);
      warm_l1(td.cell_e + (int64_t)k * t.nc + c);
    }
  }
  step_inputs();
  if (gated(gate)) return false;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    if (i >= blockDim.x) fan = vertex_fan<T>(td.verts[v0 + i], t.voff, t.vcid, g.vw, t.vbc);
    T qy;
    s_vt[i] = vertex_visc_of<T>(fan, t.vcid, g.vw, w.ctq, w.ctqy, qy);
    s_vy[i] = qy;
  }
  for (int i = threadIdx.x; i < ne; i += blockDim.x) {
    const int e = td.edges[e0 + i];
    s_f[i] = hllc_flux(w.eL[e], w.eR[e], s_g[i].a, s_g[i].b, (T)ph.gamma);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < ne; i += blockDim.x) {
    const ushort2 vv = td.edge_v[e0 + i];
    T qy;
    s_t[i] = edge_visc_value<T>(s_vt[vv.x], s_vy[vv.x], s_vt[vv.y], s_vy[vv.y], t.ebc[td.edges[e0 + i]], qy);
    s_ty[i] = qy;
  }
  __syncthreads();
  return true;
}

// What a stage's residual kernel adds up: kStage 1 the norm partials (r2 per
// cell), kStage 3 the wave speeds of the new states.
template <int kStage>
__device__ __forceinline__ void stage_sums(double r2, double wave, double* part, StepState* st) {
  __shared__ double smem[32];
  if (kStage == 1) {
    const double s = block_sum(r2, smem);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
  }
  if (kStage == 3) wave_speed_commit(wave, st);
}

// End of a step, start of the next: its wave speeds have been taken.
__device__ __forceinline__ void step_turn(StepState* st) {
  step_end_at(st);
  step_begin_at(st);
  if (!st->stop) step_dt_next(st);
}

// End of a tile kernel of stage 1 or 3: the last block runs the step control.
// All threads of all running blocks call it.
template <int kStage>
__device__ __forceinline__ void tile_stage_end(int tiles, double* part, double* hist, StepState* st) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&st->ticket, 1u) == (unsigned int)tiles - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (kStage == 1) {
    step_norm_block<true>(part, tiles, hist, st);
  } else if (threadIdx.x == 0) {
    step_turn(st);
  }
  if (threadIdx.x == 0) st->ticket = 0u;
}

template <typename T>
__global__ void __launch_bounds__(kTileMax, 4) k_tile_gradient(TileDev td, Topo t, Geom<T> g, const Vec4<T>* U,
                                                             Phys ph, Work<T> w, Vec4<T>* vq_out, const int* gate) {
  extern __shared__ __align__(32) unsigned char tile_sm[];
  tile_gradient<T>(blockIdx.x, td, t, g, U, ph, w, vq_out, reinterpret_cast<Vec4<T>*>(tile_sm), gate);
}

// FP64: residual and update of the state.
template <int kStage>
__global__ void __launch_bounds__(kTileMax, 4) k_tile_residual(TileDev td, Topo t, Geom<double> g, Phys ph,
                                                             Work<double> w, Vec4<double>* U,
                                                             Vec4<double>* Uold, RkStage rk, double* part,
                                                             double* hist, StepState* st) {
  extern __shared__ __align__(32) unsigned char tile_sm[];
  const int64_t c = (int64_t)blockIdx.x * td.cells + threadIdx.x;
  const bool mine = threadIdx.x < td.cells && c < t.nc;
  TileFluxes<double> ed;
  if (!tile_fluxes<double>(blockIdx.x, td, t, g, ph, w, c, tile_sm, &st->stop, ed)) return;
  double r2 = 0.0, wave = 0.0;
  if (mine) {
    Vec4<double> u;
    r2 = cell_residual_from<double, true>(c, t.nc, t.slot, g.cgeom, ed, U, Uold, kStage == 2 ? nullptr : w.R, rk, &u);
    if (kStage == 3) wave_speed_cell(u, ph.gamma, wave);
  }
  stage_sums<kStage>(r2, wave, part, st);
  if (kStage != 2) tile_stage_end<kStage>(td.n, part, hist, st);
}

// The cell phase of the separate kernels in the time loop.  On the large
// meshes that use them, step control in the last block costs more (every
// block waits for its ticket at its end) than launches of its own
// (k_step_norm, k_step_turn).
template <int kStage>
__global__ void __launch_bounds__(kBlock) k_cell_residual_stage(int64_t nc, const int32_t* __restrict__ slot,
                                                                Geom<double> g, Phys ph, Work<double> w,
                                                                Vec4<double>* __restrict__ U,
                                                                Vec4<double>* __restrict__ Uold, RkStage rk,
                                                                double* part, StepState* st) {
  if (gated(&st->stop)) return;
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  double r2 = 0.0, wave = 0.0;
  if (c < nc) {
    Vec4<double> u;
    r2 = cell_residual_from<double, true>(c, nc, slot, g.cgeom, EdgeFluxes<double>{g.egeom, w.F, w.etq, w.etqy}, U, Uold,
                                          kStage == 2 ? nullptr : w.R, rk, &u);
    if (kStage == 3) wave_speed_cell(u, ph.gamma, wave);
  }
  stage_sums<kStage>(r2, wave, part, st);
}

}  // namespace o2f

// imex_kernels.cuh -- the per-step kernels of the IMEX_SfloW2D time step.
//
//   k_mask      check_solve: wet/source seed, n_RK=2 four-neighbour dilation in
//               shared memory, inlet-interior removal (src/solver_2d.f90:666-857)
//   k_flux      one tile per block: physical states of the tile and a 2-cell
//               halo in shared memory, MUSCL faces with the reference's
//               boundary/inlet rules, local speeds, Kurganov-Tadmor fluxes,
//               divergence, explicit terms and the CFL minimum
//               (timestep + RK stage 1: src/solver_2d.f90:872-1005,2614-3918)
//   k_stage2    RK stage 2: semi-implicit terms, Newton with line search and
//               complex-step Jacobian, assembly checks
//               (src/solver_2d.f90:1105-1628, 1660-2365)
//   k_erosion   the erosion/deposition update per cell
//               (src/solver_2d.f90:2380-2595)
//
// Data layout: structure-of-arrays planes, plane v of q at q + v*plane,
// element (j,k) (0-based) at k*pitch + j.
#pragma once

#include <type_traits>

#include <cuda.h>   // CUtensorMap (the type only; maps are encoded by the host)

#include "imex_device.cuh"
#include "imex_mlp.cuh"

namespace imex {
inline namespace IMEX_TU_NS {

constexpr int HALO = 2;

// A tile of TXv x TYv cells: its shared-memory extent with the 2-cell halo,
// its interface counts and the threads of a flux block (one per cell, plus
// one warp, so that every cell keeps its own thread between the x and y
// phases of k_flux).
template <int TXv, int TYv>
struct TileShape {
  static constexpr int TX = TXv, TY = TYv;
  static constexpr int SW = TX + 2 * HALO;    // shared tile width
  static constexpr int SH = TY + 2 * HALO;    // shared tile height
  static constexpr int NXI = (TX + 1) * TY;   // x-interfaces per tile
  static constexpr int NYI = TX * (TY + 1);   // y-interfaces per tile
  static constexpr int THREADS = TX * TY + 32;
};
using Shape32x8 = TileShape<32, 8>;    // the single-grid path's tiles
using Shape16x16 = TileShape<16, 16>;
using Shape32x4 = TileShape<32, 4>;

constexpr int TX = Shape32x8::TX;
constexpr int TY = Shape32x8::TY;
constexpr int SW = Shape32x8::SW;
constexpr int SH = Shape32x8::SH;
constexpr int FLUX_THREADS = Shape32x8::THREADS;
constexpr int NXI = Shape32x8::NXI;
constexpr int NYI = Shape32x8::NYI;

// Minimum resident blocks per SM asked of ptxas for the per-cell kernels
// (their register budget); tuning knobs, set with -D at build time.
#ifndef IMEX_EROSION_MINB
#define IMEX_EROSION_MINB 8
#endif

// Device clock shared by the step kernels (graph-replayable).
struct DevClock {
  double t, dt, dt_old, dt_old_old, t_end, t_output;
  unsigned long long dtmin_bits;  // running CFL minimum (positive doubles)
  unsigned int error_mask;
  int pad_;
  unsigned long long first_error;  // (cell index << 8) | code, min over cells
  unsigned long long newton_cells, newton_iters, lnsrch_trials, newton_maxit;
  unsigned long long hist[16];
  unsigned long long solve_cells;
  unsigned long long n_listed;       // solve cells written to NewtonWork's `cells`, or
                                     // 2^62: not listed in this step
  unsigned long long steps;
  unsigned int nw_count[4];  // cells appended to the stage-2 Newton lists
                             // ([3]: the warm-start list)
  unsigned long long harvest_n;      // training pairs written so far
  unsigned long long warm_fallback;  // warm starts redone from q_si
  unsigned int nw_fb;                // cells in the warm-start fallback list
  int use_list;                      // k_stage2's form (stage2_form)
};

IMEX_HD double x_stag(const DevParams& P, int J) { return P.x0 + (double)(J - 1) * P.dx; }
IMEX_HD double y_stag(const DevParams& P, int K) { return P.y0 + (double)(K - 1) * P.dy; }
IMEX_HD double x_comp(const DevParams& P, int J) { return 0.5 * (x_stag(P, J) + x_stag(P, J + 1)); }
IMEX_HD double y_comp(const DevParams& P, int K) { return 0.5 * (y_stag(P, K) + y_stag(P, K + 1)); }

__device__ __forceinline__ void record_error(DevClock* clk, int code, long long cell) {
  atomicOr(&clk->error_mask, 1u << code);
  unsigned long long key = ((unsigned long long)cell << 8) | (unsigned long long)code;
  atomicMin(&clk->first_error, key);
}

__device__ const RingCell* find_ring(const RingCell* ring, int n, long long idx) {
  int lo = 0, hi = n - 1;
  while (lo <= hi) {
    int mid = (lo + hi) >> 1;
    long long v = ring[mid].idx;
    if (v == idx) return &ring[mid];
    if (v < idx) lo = mid + 1; else hi = mid - 1;
  }
  return nullptr;
}

// ================================================================= k_mask
// check_solve(.FALSE.) for n_RK = 2 on the tile whose first cell is
// (j0, k0): the wet/source seed of the tile and a 2-cell halo, two 4-point
// dilations, the border rows and the inlet-interior removal.  Returns, to
// every thread of the block, whether any cell of the tile is solved.  With `cells`
// the solve cells are also appended there (a tile of one cell per thread), until
// they are half the grid's: stage 2 takes the list of sparse steps only
// (DENSE_MIN_GRID).
template <class TS>
__device__ __forceinline__ bool mask_tile(const DevParams& P, const double* __restrict__ q1,
                                          const double* __restrict__ release_time,
                                          const uint8_t* __restrict__ cellinfo, double t,
                                          uint8_t* __restrict__ mask, DevClock* clkw,
                                          int solve_all, int j0, int k0,
                                          uint8_t (*s0)[TS::SW], uint8_t (*s1)[TS::SW],
                                          uint32_t* __restrict__ cells = nullptr) {
  constexpr int SWt = TS::SW, SHt = TS::SH, TXt = TS::TX, TYt = TS::TY;
  const int nx = P.nx, ny = P.ny;
  __shared__ bool list;
  unsigned long long listed = 0;   // loaded here, looked at behind the tile's loads
  if (cells && threadIdx.x == 0) listed = *(volatile unsigned long long*)&clkw->n_listed;
  for (int e = threadIdx.x; e < SWt * SHt; e += blockDim.x) {
    int lx = e % SWt, ly = e / SWt;
    int j = j0 + lx - HALO, k = k0 + ly - HALO;
    uint8_t m = 0;
    if (j >= 0 && j < nx && k >= 0 && k < ny) {
      bool border = (j == 0 || j == nx - 1 || k == 0 || k == ny - 1);
      if (border || solve_all) {
        m = 1;
      } else {
        size_t c = (size_t)k * P.pitch + j;
        bool rel = P.has_release_time ? (release_time[c] <= t) : (0.0 <= t);
        if (q1[c] > 0.0 && rel) m = 1;
        if (P.radial_source_flag && (cellinfo[(size_t)k * nx + j] & CI_SRC_MASK) == 2) m = 1;
      }
    }
    s0[ly][lx] = m;
  }
  if (threadIdx.x == 0) list = 2 * listed < (unsigned long long)nx * ny;
  __syncthreads();
  // first dilation on the tile plus a 1-cell ring
  for (int e = threadIdx.x; e < SWt * SHt; e += blockDim.x) {
    int lx = e % SWt, ly = e / SWt;
    int j = j0 + lx - HALO, k = k0 + ly - HALO;
    uint8_t m = s0[ly][lx];
    if (lx >= 1 && lx < SWt - 1 && ly >= 1 && ly < SHt - 1 && j >= 1 && j < nx - 1 && k >= 1 &&
        k < ny - 1)
      m = m | s0[ly][lx - 1] | s0[ly][lx + 1] | s0[ly - 1][lx] | s0[ly + 1][lx];
    s1[ly][lx] = m;
  }
  __syncthreads();
  int cnt = 0;
  for (int e = threadIdx.x; e < TXt * TYt; e += blockDim.x) {
    int lx = e % TXt + HALO, ly = e / TXt + HALO;
    int j = j0 + lx - HALO, k = k0 + ly - HALO;
    if (j >= nx || k >= ny) continue;
    uint8_t m = s1[ly][lx];
    if (j >= 1 && j < nx - 1 && k >= 1 && k < ny - 1)
      m = m | s1[ly][lx - 1] | s1[ly][lx + 1] | s1[ly - 1][lx] | s1[ly + 1][lx];
    if (P.radial_source_flag && (cellinfo[(size_t)k * nx + j] & CI_SRC_MASK) == 1) m = 0;
    mask[(size_t)k * P.pitch + j] = m;
    cnt += m;
  }
  const bool solve = cnt != 0;
  // the block's solve cells, in one atomic add: those to one address are served
  // one by one, and an add per warp bound the kernel (0.099 ms on 2048^2 solve
  // cells, 0.065 now)
  __shared__ int warp_cnt[8];
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  if ((threadIdx.x & 31) == 0) warp_cnt[threadIdx.x >> 5] = cnt;
  __syncthreads();
  int total = 0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) total += warp_cnt[w];
  if (threadIdx.x == 0 && total) atomicAdd(&clkw->solve_cells, (unsigned long long)total);
  if (cells && list && total) {
    __shared__ unsigned first;
    if (threadIdx.x == 0)
      first = (unsigned)atomicAdd(&clkw->n_listed, (unsigned long long)total);
    __syncthreads();
    const unsigned m = __ballot_sync(0xffffffffu, solve);
    unsigned slot = first + __popc(m & ((1u << (threadIdx.x & 31)) - 1u));
    for (int w = 0; w < (int)(threadIdx.x >> 5); ++w) slot += warp_cnt[w];
    if (solve)
      cells[slot] = (uint32_t)((k0 + threadIdx.x / TXt) * P.pitch + j0 + threadIdx.x % TXt);
  }
  return total != 0;
}

__global__ void __launch_bounds__(256) k_mask(const __grid_constant__ DevParams Pp, const double* __restrict__ q1,
                                              const double* __restrict__ release_time,
                                              const uint8_t* __restrict__ cellinfo,
                                              const DevClock* clk, uint8_t* __restrict__ mask,
                                              DevClock* clkw, int solve_all,
                                              uint32_t* __restrict__ cells) {
  static_assert(TX * TY == 256, "one cell per thread");
  __shared__ uint8_t s0[SH][SW];
  __shared__ uint8_t s1[SH][SW];
  mask_tile<Shape32x8>(Pp, q1, release_time, cellinfo, clk->t, mask, clkw, solve_all,
                       blockIdx.x * TX, blockIdx.y * TY, s0, s1, cells);
}

// ------------------------------------------------------ TMA tile loads
// One bulk tensor copy per tile (cp.async.bulk.tensor, this GPU's memory
// only, no multicast) completing on a shared-memory mbarrier.  The wait is
// bounded: past the limit the caller records IMEX_ETIMEOUT (never expected).
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}
// makes the barrier's initialisation visible to the copy engine's proxy
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y,
                                            int z, unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, uint32_t phase) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(phase)
      : "memory");
  return ok != 0;
}
constexpr int TMA_WAIT_LIMIT = 1 << 22;   // try_wait polls (seconds at most)
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long* bar, uint32_t phase) {
  for (int it = 0; it < TMA_WAIT_LIMIT; ++it)
    if (mbar_try_wait(bar, phase)) return true;
  return false;
}

// k_mask over the tile rows [ty0, ty0 + gridDim.y): one band of a step whose
// state arrives from the host band by band (imex_gpu_advance_host).
__global__ void __launch_bounds__(256) k_mask_rows(const __grid_constant__ DevParams Pp,
                                                   const double* __restrict__ q1,
                                                   const double* __restrict__ release_time,
                                                   const uint8_t* __restrict__ cellinfo,
                                                   const DevClock* clk, uint8_t* __restrict__ mask,
                                                   DevClock* clkw, int ty0) {
  __shared__ uint8_t s0[SH][SW];
  __shared__ uint8_t s1[SH][SW];
  mask_tile<Shape32x8>(Pp, q1, release_time, cellinfo, clk->t, mask, clkw, 0, blockIdx.x * TX,
                       (blockIdx.y + ty0) * TY, s0, s1);
}

// ================================================================== faces
// Shared tile of physical states: qps[v][ly][lx]; info_s[ly][lx] holds the
// cellinfo bits plus bit 7 = solve mask.
template <int NS, class TS = Shape32x8>
struct Tile {
  double qp[6 + NS][TS::SH][TS::SW];
  uint8_t info[TS::SH][TS::SW];
};

IMEX_NOINL double limit_call(double v1, double v2, double v3, double z1, double z2, double z3,
                             int lim, double theta) {
  return limit(v1, v2, v3, z1, z2, z3, lim, theta);
}

// The face values of variable i of one cell in one direction, W/E (dir 1) or
// S/N (dir 2), by all of the reference's rules.
// `stage` selects the RK-stage arrays' view of never-solved inlet-interior
// neighbours (all zero) instead of the module qp view (zero with T_ambient).
// Few cells come here (border, inlet), but a block waits for them, so the
// variables of a cell are separate tasks (special_faces below).
template <int NS, class TS>
IMEX_NOINL void special_face(const DevParams& P, const Tile<NS, TS>& T, int lx, int ly, int j, int k,
                             int dir, bool stage, const RingCell* ring, const InletRamp& ramp,
                             int var, double& Fm, double& Fp) {
  constexpr int NV = 4 + NS, NP = 6 + NS;
  const uint8_t inf = T.info[ly][lx];
  const int scell = inf & CI_SRC_MASK;
  const bool rad = P.radial_source_flag != 0;
  const bool sE = inf & CI_E, sW = inf & CI_W, sS = inf & CI_S, sN = inf & CI_N;
  const int J = j + 1, K = k + 1;  // Fortran indices
  const int n = (dir == 1) ? P.nx : P.ny;
  const int I = (dir == 1) ? J : K;
  const double dh = (dir == 1) ? P.dx2 : P.dy2;
  const double one_by_d = (dir == 1) ? P.one_by_dx : P.one_by_dy;
  auto comp = [&](int m) { return (dir == 1) ? x_comp(P, m) : y_comp(P, m); };
  auto stag = [&](int m) { return (dir == 1) ? x_stag(P, m) : y_stag(P, m); };
  const int* flagm = (dir == 1) ? P.bcW_flag : P.bcS_flag;
  const int* flagp = (dir == 1) ? P.bcE_flag : P.bcN_flag;
  const double* valm = (dir == 1) ? P.bcW_val : P.bcS_val;
  const double* valp = (dir == 1) ? P.bcE_val : P.bcN_val;
  // inlet-ring corrections apply to the x direction through sE/sW and to the
  // y direction through sS/sN; border inlet cells (lateral source) use the
  // inlet state as the Dirichlet value in x only.
  const bool ring_m = rad && scell == 2 && ((dir == 1) ? (!sE && sW) : (sS));
  const bool ring_p = rad && scell == 2 && ((dir == 1) ? sE : (!sS && sN));
  const bool border_src = (dir == 1) && scell == 2;
  double sb[NP];
#pragma unroll
  for (int i = 0; i < NP; ++i) sb[i] = 0.0;
  if (rad && scell == 2) {
    const RingCell* rc = find_ring(ring, P.n_ring, (long long)k * P.nx + j);
    if (rc) {
      int w = sE ? 0 : (sW ? 1 : (sS ? 2 : 3));
      eval_source_bdry<NS>(P, ramp, rc->vx[w], rc->vy[w], sb);
    }
  }
  auto sbv = [&](int i) {
    double r = sb[0];
#pragma unroll
    for (int m = 1; m < NP; ++m)
      if (m == i) r = sb[m];
    return r;
  };
  // stencil abscissae after the n_vars loop
  double z1, z2 = comp(I), z3;
  if (I == 1) {
    z1 = stag(1);
    z3 = comp(2);
  } else if (I == n) {
    z1 = comp(n - 1);
    z3 = stag(n + 1);
  } else {
    z1 = ring_m ? stag(I) : comp(I - 1);
    z3 = ring_p ? stag(I + 1) : comp(I + 1);
  }
  const double rc_d = P.reconstr_coeff * dh;
  const int ox = (dir == 1) ? 1 : 0, oy = 1 - ox;
  const bool hide = stage && rad;
  const bool hide_m = hide && (T.info[ly - oy][lx - ox] & CI_SRC_MASK) == 1;
  const bool hide_c = hide && scell == 1;
  const bool hide_p = hide && (T.info[ly + oy][lx + ox] & CI_SRC_MASK) == 1;
  // u and v at a border face come from that face's h, hu and hv: those first
  const bool from_q = var >= NV && (I == 1 || I == n);
  double fh = 0.0, fq = 0.0;
#pragma unroll 1
  for (int t = from_q ? 0 : 2; t < 3; ++t) {
    const int i = (t == 0) ? 0 : ((t == 1) ? 1 + var - NV : var);
    const double v2 = hide_c ? 0.0 : T.qp[i][ly][lx];
    double v1 = hide_m ? 0.0 : T.qp[i][ly - oy][lx - ox];
    double v3 = hide_p ? 0.0 : T.qp[i][ly + oy][lx + ox];
    double zz3 = z3, slope = 0.0, vf = 0.0;
    bool given = false;
    if (i < NV) {
      if (I == 1) {
        if (border_src) {
          v1 = sbv(i);
        } else if (flagm[i] == 0) {
          v1 = valm[i];
        } else {
          slope = (flagm[i] == 1) ? valm[i] : (v3 - v2) * one_by_d;
          given = true;
        }
      } else if (I == n) {
        if (border_src) {
          v3 = sbv(i);
        } else if (flagp[i] == 0) {
          v3 = valp[i];
        } else {
          slope = (flagp[i] == 1) ? valp[i] : (v2 - v1) * one_by_d;
          given = true;
        }
      } else {
        if (ring_m) v1 = sbv(i);
        if (ring_p) v3 = sbv(i);
      }
    } else {
      // u and v with the limiters of hu and hv
      if (dir == 1 && i == NV + 1 && rad && scell == 2 && I > 1 && I < n && !sE && sN && !sS &&
          K > 1 && K < P.ny)
        zz3 = y_stag(P, K + 1);  // x_stencil(3)=y_stag(k+1), src/solver_2d.f90:3616
      if (from_q) vf = (fh <= 0.0) ? 0.0 : fq / fh;
      if (I == 1) {
        v1 = vf;
      } else if (I == n) {
        v3 = vf;
      } else {
        if (ring_m) v1 = sbv(i);
        if (ring_p) v3 = sbv(i);
      }
    }
    if (!given) slope = limit_call(v1, v2, v3, z1, z2, zz3, P.limiter[i], P.theta);
    const double dq = rc_d * slope;
    double fm = v2 - dq, fp = v2 + dq;
    if (i < NV) {
      const int ivel = (dir == 1) ? 1 : 2;  // hu clamp in x, hv clamp in y
      if (I == 1) {
        if (border_src) fm = sbv(i);
        else if (flagm[i] == 0) fm = valm[i];
        else if (i == ivel) fm = fmin_f(fm, 0.0);
      }
      if (I == n) {
        if (border_src) fp = sbv(i);
        else if (flagp[i] == 0) fp = valp[i];
        else if (i == ivel) fp = fmax_f(fp, 0.0);
      }
    } else {
      if (I == 1) fm = vf;
      else if (I == n) fp = vf;
    }
    fq = (I == 1) ? fm : fp;
    if (t == 0) fh = fq;
    Fm = fm;
    Fp = fp;
  }
  if (I > 1 && I < n) {
    if (ring_p) Fp = sbv(var);
    else if (ring_m) Fm = sbv(var);
  }
}

// All face values of one cell, one after the other: F[0..NP) the minus face,
// F[NP..2NP) the plus one.
template <int NS, class TS>
IMEX_NOINL void cell_faces(const DevParams& P, const Tile<NS, TS>& T, int lx, int ly, int j, int k,
                           int dir, bool stage, const RingCell* ring, const InletRamp& ramp,
                           double* F) {
  constexpr int NP = 6 + NS;
#pragma unroll 1
  for (int i = 0; i < NP; ++i) {
    double fm, fp;
    special_face<NS, TS>(P, T, lx, ly, j, k, dir, stage, ring, ramp, i, fm, fp);
    F[i] = fm;
    F[NP + i] = fp;
  }
}

// Limited MUSCL increments of one direction, precomputed once per cell for
// the cells whose faces need none of cell_faces' special rules: not on the
// domain border in that direction, not an inlet cell, no inlet-interior
// neighbour in that direction (so the stage and timestep views agree).
// There the faces are qp -/+ rc_d*limit(...) for every variable, exactly the
// operations of cell_faces.  Indexed [ly - 1][lx - 1] of the shared tile:
// x faces use rows 2..9 and columns 1..34, y faces rows 1..10, columns 2..33.
template <int NS, class TS = Shape32x8>
struct SlopeTile {
  double dq[6 + NS][TS::TY + 2][TS::TX + 2];
  // 0: no faces kept; 1: increments in dq; FACES0 + s: both faces in slot s of
  // the special faces (see special_faces)
  uint8_t ok[TS::TY + 2][TS::TX + 2];
};
constexpr int FACES0 = 2;

// limit() for one variable on any spacing and limiter (the increments below
// that their inlined form does not cover).
IMEX_NOINL double slope_general(const DevParams& P, double v1, double v2, double v3, double dz,
                                bool uniform, double z1, double z2, double z3, int lim) {
  return (uniform && lim == 1) ? minmod_uniform(v1, v2, v3, dz, z1, z2, z3, P.theta)
                               : limit(v1, v2, v3, z1, z2, z3, lim, P.theta);
}

// What bounds this is instruction issue: one division per cell and direction
// (Recip) serves all variables.  Minmod on equal spacings with finite differences of
// ordinary size is inlined per variable; the other limiters and unequal (rounded)
// spacings take a rolled loop, one to three divisions per cell; infinities, NaN,
// tiny and huge differences are a call.
template <int NS, class TS>
__device__ __forceinline__ void precompute_slopes(const DevParams& P, const Tile<NS, TS>& T,
                                                  SlopeTile<NS, TS>& D, int dir, int j0, int k0,
                                                  int* n_special, uint16_t* special, int cap) {
  constexpr int NP = 6 + NS, TX = TS::TX, TY = TS::TY, SW = TS::SW;
  constexpr int QV = TS::SW * TS::SH, DV = (TY + 2) * (TX + 2);   // doubles per variable
  const bool rad = P.radial_source_flag != 0;
  const int n = (dir == 1) ? P.nx : P.ny;
  const int off = (dir == 1) ? 1 : SW;
  const double rc_d = P.reconstr_coeff * ((dir == 1) ? P.dx2 : P.dy2);
  const int count = (dir == 1) ? (TX + 2) * TY : TX * (TY + 2);
  for (int e = threadIdx.x; e < count; e += blockDim.x) {
    const int lx = (dir == 1) ? 1 + e % (TX + 2) : HALO + e % TX;
    const int ly = (dir == 1) ? HALO + e / (TX + 2) : 1 + e / TX;
    const int j = j0 + lx - HALO, k = k0 + ly - HALO;
    uint8_t ok = 0;
    const int I = (dir == 1) ? j + 1 : k + 1;
    const int di = (ly - 1) * (TX + 2) + lx - 1;
    if (j >= 0 && j < P.nx && k >= 0 && k < P.ny && n > 1) {
      const uint8_t* inf = &T.info[ly][lx];
      const uint8_t i2 = inf[0], i1 = inf[-off], i3 = inf[off];
      // an active interface on either side: the cell or a neighbour is solved
      const bool used = ((i1 | i2 | i3) & 128) != 0;
      const bool inner_near = rad && ((i1 & CI_SRC_MASK) == 1 || (i3 & CI_SRC_MASK) == 1);
      const bool plain = I > 1 && I < n && !(rad && (i2 & CI_SRC_MASK) != 0) && !inner_near;
      if (used && !plain && !(rad && (i2 & CI_SRC_MASK) == 1)) {
        // a slot for its faces, two (stage and timestep views) beside the inlet interior
        const int need = inner_near ? 2 : 1;
        const int s = atomicAdd(n_special, need);
        if (s + need <= cap) {
          special[s] = (uint16_t)(di << 1);
          if (need == 2) special[s + 1] = (uint16_t)((di << 1) | 1);
          ok = (uint8_t)(FACES0 + s);
        } else {
          for (int m = s; m < cap; ++m) special[m] = 0xffff;
        }
      } else if (used && plain) {
        const double z1 = (dir == 1) ? x_comp(P, I - 1) : y_comp(P, I - 1);
        const double z2 = (dir == 1) ? x_comp(P, I) : y_comp(P, I);
        const double z3 = (dir == 1) ? x_comp(P, I + 1) : y_comp(P, I + 1);
        const double dz = z3 - z2, dz1 = z2 - z1;
        const bool uniform = (dz == dz1) && (z3 > z2) && (z2 > z1);
        bool gen = true;
        const Recip R3 = recip_pos(dz, gen);
        const bool fast = gen && dz >= 1e-10 && dz1 >= 1e-10;
        const double* v = &T.qp[0][ly][lx];
        double* dq = &D.dq[0][0][0] + di;
        const float big = __int_as_float(0x65700000);
        if (uniform && P.all_minmod) {
#pragma unroll 3
          for (int i = 0; i < NP; ++i) {
            const double v1 = v[i * QV - off], v2 = v[i * QV], v3 = v[i * QV + off];
            // 0 for differences of opposite sign or a zero one, else the smaller
            // difference's slope (minmod_uniform)
            const double d3 = v3 - v2, d1 = v2 - v1;
            const bool zero = d3 == 0.0 || d1 == 0.0;
            const bool opp = (__double2hiint(d3) ^ __double2hiint(d1)) < 0;
            bool in = fast && hi_mag(d3) < big && hi_mag(d1) < big;
            double lim = 0.0;
            if (!(in && (zero || opp))) {
              lim = quot(R3, (fabs(d1) < fabs(d3)) ? d1 : d3, in);
              if (!in) lim = slope_general(P, v1, v2, v3, dz, true, z1, z2, z3, 1);
            }
            dq[i * DV] = rc_d * lim;
          }
        } else {
          const Recip R1 = recip_pos(dz1, gen), R13 = recip_pos(z3 - z1, gen);
#pragma unroll 1
          for (int i = 0; i < NP; ++i) {
            const double v1 = v[i * QV - off], v2 = v[i * QV], v3 = v[i * QV + off];
            const int l = P.limiter[i];
            const double d3 = v3 - v2, d1 = v2 - v1;
            bool in = gen && l >= 1 && l <= 4 && hi_mag(d3) < big && hi_mag(d1) < big;
            const double a = quot(R3, d3, in), b = quot(R1, d1, in);
            double lim;
            if (l == 1) {
              lim = minmod(a, b);
            } else if (l == 2) {
              lim = maxmod(minmod(a, 2.0 * b), minmod(2.0 * a, b));
            } else {
              const double c = quot(R13, v3 - v1, in);
              lim = minmod(c, ((l == 3) ? P.theta : 2.0) * minmod(a, b));
            }
            if (!in) lim = slope_general(P, v1, v2, v3, dz, uniform, z1, z2, z3, l);
            dq[i * DV] = rc_d * lim;
          }
        }
        ok = 1;
      }
    }
    (&D.ok[0][0])[di] = ok;
  }
}

// Both face states of an interface by the reference's full rules: Q[0..NP) on
// the side of cell a (left/lower), Q[NP..2NP) on b's.
template <int NS, class TS>
IMEX_NOINL void interface_states(const DevParams& P, const Tile<NS, TS>& T, int dir, int la_x,
                                 int la_y, int ja, int ka, bool stage, const RingCell* ring,
                                 const InletRamp& ramp, double* Q) {
  constexpr int NP = 6 + NS;
  const int ox = (dir == 1) ? 1 : 0, oy = 1 - ox;
  const int lb_x = la_x + ox, lb_y = la_y + oy, jb = ja + ox, kb = ka + oy;
  const int n = (dir == 1) ? P.nx : P.ny, ia0 = (dir == 1) ? ja : ka;
  const bool a_in = ia0 >= 0, b_in = ia0 + 1 < n;
  const bool rad = P.radial_source_flag != 0;
  const uint8_t ia = a_in ? T.info[la_y][la_x] : 0, ib = b_in ? T.info[lb_y][lb_x] : 0;
  const bool a_int = rad && a_in && (ia & CI_SRC_MASK) == 1;
  const bool b_int = rad && b_in && (ib & CI_SRC_MASK) == 1;
  // reconstruction of the sides that need it
  const bool comp_a = a_in && (!b_in || !a_int);
  const bool comp_b = b_in && (!a_in || !b_int);
  double F[2 * NP];
#pragma unroll 1
  for (int side = 0; side < 2; ++side) {
    if (!(side == 0 ? comp_a : comp_b)) continue;
    cell_faces<NS, TS>(P, T, side ? lb_x : la_x, side ? lb_y : la_y, side ? jb : ja,
                       side ? kb : ka, dir, stage, ring, ramp, F);
    // a's plus face, b's minus face
#pragma unroll 1
    for (int i = 0; i < NP; ++i) Q[side * NP + i] = F[side ? i : NP + i];
  }
  // -1: keep; 0: zero; 1: the other side's state
  int fix_a = -1, fix_b = -1;
  if (!a_in) {  // domain boundary on the minus side: both states from b's minus face
    fix_a = 1;
  } else if (!b_in) {
    fix_b = 1;
  } else {
    // never solved: only the ring copy of src/solver_2d.f90:3768-3771 fills it
    if (a_int)
      fix_a = comp_b && (ib & CI_SRC_MASK) == 2 &&
              ((dir == 1) ? (ib & CI_W) && !(ib & CI_E) : (ib & CI_S) != 0);
    if (b_int)
      fix_b = comp_a && (ia & CI_SRC_MASK) == 2 &&
              ((dir == 1) ? (ia & CI_E) != 0 : (ia & CI_N) && !(ia & CI_S));
  }
#pragma unroll 1
  for (int i = 0; i < NP; ++i) {
    if (fix_a >= 0) Q[i] = fix_a ? Q[NP + i] : 0.0;
    if (fix_b >= 0) Q[NP + i] = fix_b ? Q[i] : 0.0;
  }
}

// One interface by the reference's own sequence: the KT flux H (n_vars) and
// max(|a+|,|a-|) for the CFL.
template <int NS, class TS>
IMEX_FLAT void interface_flux(const DevParams& P, const Tile<NS, TS>& T, int dir, int la_x,
                              int la_y, int ja, int ka, double gcf, bool stage,
                              const RingCell* ring, const InletRamp& ramp, double* H,
                              double& amax_flux) {
  constexpr int NV = 4 + NS, NP = 6 + NS;
  double Q[2 * NP], QL[NP], QR[NP];
  interface_states<NS, TS>(P, T, dir, la_x, la_y, ja, ka, stage, ring, ramp, Q);
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    QL[i] = Q[i];
    QR[i] = Q[NP + i];
  }
  double cL[NV], cR[NV];
  Mixt mL, mR;
  face_qc_mixt<NS>(P, QL, cL, mL);
  face_qc_mixt<NS>(P, QR, cR, mR);
  double lmin, lmax, rmin, rmax;
  local_speeds<NS>(P, QL, mL, gcf, dir, lmin, lmax);
  local_speeds<NS>(P, QR, mR, gcf, dir, rmin, rmax);
  double aN = fmin_f(fmin_f(lmin, rmin), 0.0);
  double aP = fmax_f(fmax_f(lmax, rmax), 0.0);
  amax_flux = fmax_f(aP, -aN);
  double fL[NV], fR[NV];
  eval_fluxes<NS>(P, cL, QL, mL, gcf, dir, fL);
  eval_fluxes<NS>(P, cR, QR, mR, gcf, dir, fR);
  if (aN == aP) {
#pragma unroll
    for (int i = 0; i < NV; ++i) H[i] = 0.0;
  } else {
    double coef = (aP * aN) / (aP - aN);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      double avg = (aP * fL[i] - aN * fR[i]) / (aP - aN);
      H[i] = avg + coef * (cR[i] - cL[i]);
    }
  }
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < NS; ++i) s += H[4 + i];
  if (dir == 1) {
    if (s / H[0] >= 1.0) {
      double r = 0.0;
#pragma unroll
      for (int i = 0; i < NS; ++i) r += H[4 + i] / H[0];
#pragma unroll
      for (int i = 0; i < NS; ++i) H[4 + i] = H[4 + i] / r;
    }
    if (QL[1] == 0.0 && QR[1] == 0.0) {
      H[0] = 0.0;
#pragma unroll
      for (int i = 3; i < NV; ++i) H[i] = 0.0;
    }
  } else {
    if (s / H[0] > 1.0) {
      double r = s / H[0];
#pragma unroll
      for (int i = 0; i < NS; ++i) H[4 + i] = H[4 + i] / r;
    }
    if (cL[2] == 0.0 && cR[2] == 0.0) {
      H[0] = 0.0;
#pragma unroll
      for (int i = 3; i < NV; ++i) H[i] = 0.0;
    }
  }
}

// ================================================================= k_flux
// Shared memory: Tile<NS> + slopes + one direction's interface fluxes and
// CFL speeds at a time (the x ones are reduced into each cell's registers
// before the y phase overwrites them).
template <int NS, class TS = Shape32x8>
struct FluxShared {
  Tile<NS, TS> tile;
  union {
    SlopeTile<NS, TS> slopes;
    // the tile's conserved variables as one TMA box (k_flux_tma), read
    // before the slopes are first written
    alignas(128) double stage[4 + NS][TS::SH][TS::SW];
  };
  // by interface number: x faces (TX+1 per row), then, in their place, y faces
  static constexpr int NI = TS::NXI > TS::NYI ? TS::NXI : TS::NYI;
  double H[4 + NS][NI];
  double A[NI];
  double dtmin[TS::THREADS / 32];
  unsigned long long tma_bar;   // mbarrier of the TMA box
  InletRamp ramp;               // set in tiles that see an inlet ring cell
  // cells whose faces special_faces computes: how many per direction, and
  // which (slope index * 2 + timestep view)
  static constexpr int FACES = ((4 + NS) * NI) / (2 * (6 + NS)) < 128
                                   ? ((4 + NS) * NI) / (2 * (6 + NS)) : 128;
  int n_special[2];
  uint16_t special[FACES];
};
static_assert(Shape32x8::THREADS == 288, "k_flux blocks of 288 threads for 32x8 tiles");

// Blocks of k_flux per SM: 3 where three blocks' shared memory fits the SM
// (228 KB, 1 KB reserved per block; n_s <= 3), else 2.  At n_s = 3 three
// blocks at 72 registers measured 9.5 ms per step at 4096^2 against 10.9 at
// two blocks of 96.
// Other tile shapes keep the register budget of three 288-thread blocks
// (864 threads per SM) and fit as many blocks as shared memory allows.
template <int NS, class TS = Shape32x8>
__host__ __device__ constexpr int flux_min_blocks() {
#ifdef IMEX_FLUX_MINB
  return IMEX_FLUX_MINB;
#else
  return std::is_same<TS, Shape32x8>::value
             ? ((3 * (sizeof(FluxShared<NS, TS>) + 1024) <= 228 * 1024) ? 3 : 2)
             : ((864 / TS::THREADS) < (int)(228 * 1024 / (sizeof(FluxShared<NS, TS>) + 1024))
                    ? (864 / TS::THREADS)
                    : (int)(228 * 1024 / (sizeof(FluxShared<NS, TS>) + 1024)));
#endif
}

// k_cfl_tiles: the tile and both directions' CFL speeds.
template <int NS>
struct CflShared {
  Tile<NS> tile;
  double ax[TY][TX + 1];
  double ay[TY + 1][TX];
  double dtmin[FLUX_THREADS / 32];
  InletRamp ramp;
};

// One side of a plain interface: the conserved variables c of the face state
// (normal and tangential momentum in cn, ct), its flux's velocity and pressure
// term and its characteristic speeds.  The operations are those of
// face_qc_mixt, local_speeds and eval_fluxes in both directions (in y the
// normal momentum is hv and the celerity is sqrt((gcf*g')*h)); quotients by h
// and by rho_m share a division (Recip).  A face that needs anything else (h not
// above EPS by being NaN, a quotient out of Recip's range, solids above the
// mixture's mass flux) clears ok.
template <int NS>
struct FaceSide {
  double m, cn, ct, en, cs[NS];   // conserved variables
  double vel, pres, lo, hi;       // flux velocity, pressure term, speeds
};
template <int NS>
IMEX_FLAT void face_side(const DevParams& P, double h, double qn, double qt, double T,
                         const double* qs, double un, double ut, double gcf, int dir,
                         FaceSide<NS>& f, bool& ok) {
  if (!(h > EPS)) {
    ok = ok & (h <= EPS) & (0.0 * h * gcf == 0.0);   // NaN and infinite values
    f.m = f.cn = f.ct = f.en = 0.0;
#pragma unroll
    for (int i = 0; i < NS; ++i) f.cs[i] = 0.0;
    // red_grav is 0: the celerity sqrt(0*h*gcf) is 0 (or takes the other branch)
    f.vel = f.pres = 0.0;
    f.lo = f.hi = un;
    return;
  }
  double at = 0.0, al[NS];
  if (P.alpha_flag) {
#pragma unroll
    for (int i = 0; i < NS; ++i) al[i] = qs[i];
  } else if (NS == 1) {
    al[0] = qs[0] / h;
  } else {
    const Recip Rh = recip_pos(h, ok);
#pragma unroll
    for (int i = 0; i < NS; ++i) al[i] = quot(Rh, qs[i], ok);
  }
#pragma unroll
  for (int i = 0; i < NS; ++i) at += al[i];
#pragma unroll
  for (int i = 0; i < NS; ++i) al[i] = al[i] * P.rho_s[i];
  const double rho_a = P.pres / (P.sp_gas_const_a * T);
  const double rho_c = ((((1.0 - 0.0) - at) - 0.0) * rho_a + 0.0) / ((1.0 - 0.0) - at);
  const double alc = 1.0 - at;
  double sar = 0.0;
#pragma unroll
  for (int i = 0; i < NS; ++i) sar += al[i];
  const double rho_m = alc * rho_c + sar;
  const Recip Rm = recip_pos(rho_m, ok);
  const double rg = quot(Rm, rho_m - P.rho_a_amb, ok) * P.grav;
  const double inv = Rm.y;
  const double xc = alc * rho_c * inv;
  const double cpc = (xc > EPS) ? ((xc - 0.0) * P.sp_heat_a + 0.0) / xc : P.sp_heat_a;
  double dot = 0.0;
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    al[i] = al[i] * inv;
    dot += al[i] * P.sp_heat_s[i];
  }
  const double cpm = dot + xc * cpc;
  f.m = rho_m * h;
  f.cn = rho_m * qn;
  f.ct = rho_m * qt;
  f.en = P.energy_flag ? h * rho_m * (cpm * T + 0.5 * (un * un + ut * ut)) : h * rho_m * cpm * T;
#pragma unroll
  for (int i = 0; i < NS; ++i) f.cs[i] = al[i] * f.m;
  f.vel = un;
  if (rg * h < 0.0) {
    f.lo = f.hi = un;
  } else {
    const double c = sqrt((dir == 1) ? rg * h * gcf : gcf * rg * h);
    f.lo = un - c;
    f.hi = un + c;
  }
  f.pres = 0.5 * rho_m * gcf * rg * (h * h);
  // the solids' flux cap (s/flux > 1, rounded, is s > flux for flux > 0)
  const double f0 = un * f.m;
  double fs = 0.0;
#pragma unroll
  for (int i = 0; i < NS; ++i) fs += un * f.cs[i];
  ok = ok & !(f0 > 0.0 && !(fs <= f0));
}

// A divergent solids' flux cap of the KT flux in S.H: s/H0 >= 1 in x, > 1 in y.
template <int NS, class TS>
IMEX_NOINL void cap_solids(FluxShared<NS, TS>& S, int dir, int e) {
  const double H0 = S.H[0][e];
  double s = 0.0, r = 0.0;
#pragma unroll 1
  for (int i = 0; i < NS; ++i) s += S.H[4 + i][e];
  const double q = s / H0;
  if (!((dir == 1) ? q >= 1.0 : q > 1.0)) return;
  if (dir == 1) {
#pragma unroll 1
    for (int i = 0; i < NS; ++i) r += S.H[4 + i][e] / H0;
  } else {
    r = q;
  }
#pragma unroll 1
  for (int i = 0; i < NS; ++i) S.H[4 + i][e] = S.H[4 + i][e] / r;
}

// The faces of the tile's special cells (domain border, inlet ring and beside
// the inlet), one thread per cell and variable, into the space of the
// interface fluxes: slot s holds the minus face at 2*NP*s and the plus face NP
// further.  One thread per interface used to do this for all variables of both
// its cells in turn while the block waited: 42 of the 78 us that a corner
// tile of a 200^2 grid took, 130 of 245 us beside an inlet.
template <int NS, class TS>
__device__ __forceinline__ void special_faces(const DevParams& P, FluxShared<NS, TS>& S, int n,
                                              int dir, int j0, int k0,
                                              const RingCell* __restrict__ ring) {
  constexpr int NP = 6 + NS, W = TS::TX + 2;
  double* F = &S.H[0][0];
  for (int t = threadIdx.x; t < n * NP; t += blockDim.x) {
    const int slot = t / NP, var = t - slot * NP;
    const unsigned c = S.special[slot];
    if (c == 0xffffu) continue;
    const int di = c >> 1, lx = di % W + 1, ly = di / W + 1;
    double fm, fp;
    special_face<NS, TS>(P, S.tile, lx, ly, j0 + lx - HALO, k0 + ly - HALO, dir, (c & 1) == 0, ring,
                         S.ramp, var, fm, fp);
    F[slot * 2 * NP + var] = fm;
    F[slot * 2 * NP + NP + var] = fp;
  }
}

// Where an interface takes one side's face state from.
enum FaceFrom { FACE_CELL, FACE_SLOT, FACE_OTHER, FACE_ZERO, FACE_NONE };

// One side of an interface: the source of the face state of cell (x, y) of the
// tile, `other` the cell across, in the stage or the timestep view.
__device__ __forceinline__ FaceFrom face_from(bool rad, bool in, bool other_in, uint8_t inf,
                                              uint8_t other_inf, uint8_t ok, int side, int dir) {
  if (!in) return FACE_OTHER;            // domain boundary: both states from the inner cell
  if (rad && (inf & CI_SRC_MASK) == 1) {
    if (!other_in) return FACE_NONE;
    // never solved: only the ring copy of src/solver_2d.f90:3768-3771 fills it
    const bool ring = (other_inf & CI_SRC_MASK) == 2;
    bool copy;
    if (side == 0)   // a is inside: b's inlet lies on its minus side
      copy = (dir == 1) ? (other_inf & CI_W) && !(other_inf & CI_E) : (other_inf & CI_S) != 0;
    else
      copy = (dir == 1) ? (other_inf & CI_E) != 0 : (other_inf & CI_N) && !(other_inf & CI_S);
    return (ring && copy) ? FACE_OTHER : FACE_ZERO;
  }
  return ok == 1 ? FACE_CELL : (ok >= FACES0 ? FACE_SLOT : FACE_NONE);
}

// The KT flux of an interface (mass, normal and tangential momentum, energy,
// solids) and its largest speed; false when the reference's own sequence is
// needed (interface_special).  Plain interfaces take their faces from the cells'
// values and increments (ia, ib: the cells in the tile, da, db: in the
// slopes), the others as fromL/fromR say (slots sL, sR).
// Before, four fifths of an interface's instructions were index arithmetic,
// spills and the boundary and inlet rules inlined into it; now those rules
// are separate tasks, the direction is an index, and the two sides' fluxes are
// formed from c, the velocity and the pressure term when they are combined:
// 1.04 against 2.01 ms for k_flux_tma<3> on 2048^2 cells.
template <int NS, class TS>
IMEX_FLAT bool interface_kt(const DevParams& P, const FluxShared<NS, TS>& S, int dir, FaceFrom fromL,
                            FaceFrom fromR, int sL, int sR, int ia, int ib, int da, int db,
                            double gcf, double* H, double& amax, bool& still) {
  constexpr int NV = 4 + NS, NP = 6 + NS, QV = TS::SW * TS::SH, DV = (TS::TY + 2) * (TS::TX + 2);
  const double* q = &S.tile.qp[0][0][0];
  const double* d = &S.slopes.dq[0][0][0];
  const double* F = &S.H[0][0];
  const int vn = dir, vt = 3 - dir, wn = NV + dir - 1, wt = NV + 2 - dir;
  bool ok = true;
  FaceSide<NS> L, R;
  double qnL, qnR;
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    // the cell, its increment or slot, and which face of it: its own side's, or
    // (FACE_OTHER) the one the other side uses
    const FaceFrom own = side ? fromR : fromL;
    const bool swap = own == FACE_OTHER;
    const FaceFrom from = swap ? (side ? fromL : fromR) : own;
    const bool minus = (side == 1) != swap;
    const int c = minus ? ib : ia, g = minus ? db : da, slot = minus ? sR : sL;
    double h, qn, qt, T, un, ut, qs[NS];
    if (from == FACE_CELL) {
      auto face = [&](int v) {
        const double a = q[v * QV + c], b = d[v * DV + g];
        return minus ? a - b : a + b;
      };
      h = face(0);
      qn = face(vn);
      qt = face(vt);
      T = face(3);
#pragma unroll
      for (int i = 0; i < NS; ++i) qs[i] = face(4 + i);
      un = face(wn);
      ut = face(wt);
    } else {
      const bool zero = from != FACE_SLOT;
      const double* f = F + slot * 2 * NP + (minus ? 0 : NP);
      auto face = [&](int v) { return zero ? 0.0 : f[v]; };
      h = face(0);
      qn = face(vn);
      qt = face(vt);
      T = face(3);
#pragma unroll
      for (int i = 0; i < NS; ++i) qs[i] = face(4 + i);
      un = face(wn);
      ut = face(wt);
    }
    (side ? qnR : qnL) = qn;
    face_side<NS>(P, h, qn, qt, T, qs, un, ut, gcf, dir, side ? R : L, ok);
  }
  const double aN = fmin_f(fmin_f(L.lo, R.lo), 0.0);
  const double aP = fmax_f(fmax_f(L.hi, R.hi), 0.0);
  const double gap = aP - aN;
  if (aN == aP) {
#pragma unroll
    for (int i = 0; i < NV; ++i) H[i] = 0.0;
  } else {
    const Recip Rg = recip_pos(gap, ok);
    const double coef = quot(Rg, aP * aN, ok);
    // products rounded on their own in the contracted build too: a multiply-add
    // would round the two sides of the average differently, and the radial
    // current amplifies that (relative L1 at step 500, when this was written, 2.2e-12
    // with multiply-adds and 1.6e-12 without; 1.0e-12 now)
    auto kt = [&](double fl, double fr, double cl, double cr) {
      return quot(Rg, __dmul_rn(aP, fl) - __dmul_rn(aN, fr), ok) + __dmul_rn(coef, cr - cl);
    };
    H[0] = kt(L.vel * L.m, R.vel * R.m, L.m, R.m);
    H[1] = kt(L.vel * L.cn + L.pres, R.vel * R.cn + R.pres, L.cn, R.cn);
    H[2] = kt(L.vel * L.ct, R.vel * R.ct, L.ct, R.ct);
    H[3] = P.energy_flag ? kt(L.vel * (L.en + L.pres), R.vel * (R.en + R.pres), L.en, R.en)
                         : kt(L.vel * L.en, R.vel * R.en, L.en, R.en);
#pragma unroll
    for (int i = 0; i < NS; ++i) H[4 + i] = kt(L.vel * L.cs[i], R.vel * R.cs[i], L.cs[i], R.cs[i]);
  }
  amax = fmax_f(aP, -aN);
  still = (dir == 1) ? (qnL == 0.0 && qnR == 0.0) : (L.cn == 0.0 && R.cn == 0.0);
  return ok;
}

// An interface by the reference's own sequence (flux caps of a face state,
// quotients outside Recip's range, NaN and infinite states).
template <int NS, class TS>
IMEX_NOINL void interface_special(const DevParams& P, FluxShared<NS, TS>& S, int dir, int e, int ax,
                                  int ay, int ja, int ka, double gcf, bool again,
                                  const RingCell* __restrict__ ring) {
  constexpr int NV = 4 + NS;
  double amax = 0.0;
#pragma unroll 1
  for (int pass = 0; pass < (again ? 2 : 1); ++pass) {
    double H[NV];
    interface_flux<NS, TS>(P, S.tile, dir, ax, ay, ja, ka, gcf, pass == 0, ring, S.ramp, H, amax);
    if (pass == 0) {
#pragma unroll
      for (int i = 0; i < NV; ++i) S.H[i][e] = H[i];
    }
  }
  S.A[e] = amax;
}

// Stage 1 and the CFL minimum on the tile whose first cell is (j0, k0).
template <int NS, class TS>
__device__ __forceinline__ void flux_tile(const DevParams& P, const double* __restrict__ q,
                                          const uint8_t* __restrict__ mask,
                                          const uint8_t* __restrict__ cellinfo,
                                          const double* __restrict__ Bx,
                                          const double* __restrict__ By,
                                          const double* __restrict__ Bxx,
                                          const double* __restrict__ Bxy,
                                          const double* __restrict__ Byy,
                                          const double* __restrict__ gc,
                                          const double* __restrict__ dgc,
                                          const double* __restrict__ gcsx,
                                          const double* __restrict__ gcsy,
                                          const RingCell* __restrict__ ring, DevClock* clk,
                                          double* __restrict__ X, int j0, int k0,
                                          FluxShared<NS, TS>& S,
                                          const CUtensorMap* qmap = nullptr) {
  constexpr int NV = 4 + NS, NP = 6 + NS;
  constexpr int TX = TS::TX, TY = TS::TY, SW = TS::SW, SH = TS::SH, NXI = TS::NXI,
                NYI = TS::NYI;
  const int nx = P.nx, ny = P.ny;
  const double time = clk->t;
  // any solve cell in the tile?
  int any = 0;
  for (int e = threadIdx.x; e < TX * TY; e += blockDim.x) {
    int j = j0 + e % TX, k = k0 + e / TX;
    if (j < nx && k < ny && mask[(size_t)k * P.pitch + j]) any = 1;
  }
  if (!__syncthreads_or(any)) return;
  // With a tensor map of q, the tile's n_v planes (halo included, zeros
  // outside the grid) arrive as one TMA box in the staging area
  const bool staged = qmap != nullptr;
  if (staged) {
    static_assert(sizeof(S.stage) == (size_t)(4 + NS) * SH * SW * sizeof(double), "box size");
    if (threadIdx.x == 0) {
      mbar_init(&S.tma_bar, 1);
      fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      mbar_expect_tx(&S.tma_bar, (uint32_t)sizeof(S.stage));
      // x = j0 - 2 is even: 16-byte aligned for 8-byte elements
      tma_load_3d(&S.stage[0][0][0], qmap, j0 - HALO, k0 - HALO, 0, &S.tma_bar);
    }
    const bool arrived = mbar_wait_bounded(&S.tma_bar, 0);
    if (__syncthreads_or(!arrived)) {
      // never expected: record it, wait (bounded) for the copy, and leave
      if (threadIdx.x == 0) record_error(clk, 7, (long long)k0 * nx + j0);
      mbar_wait_bounded(&S.tma_bar, 0);
      return;
    }
  }
  if (threadIdx.x == 0) S.n_special[0] = S.n_special[1] = 0;
  // physical states of the tile + halo
  bool ring_cell = false;
  for (int e = threadIdx.x; e < SW * SH; e += blockDim.x) {
    int lx = e % SW, ly = e / SW;
    int j = j0 + lx - HALO, k = k0 + ly - HALO;
    double qc[NV], qpv[NP];
    uint8_t inf = 0;
    if (j >= 0 && j < nx && k >= 0 && k < ny) {
      size_t c = (size_t)k * P.pitch + j;
      inf = P.has_cellinfo ? cellinfo[(size_t)k * nx + j] : 0;
      if (mask[c]) inf |= 128;
      if (P.radial_source_flag && (inf & CI_SRC_MASK) == 1) {
        // inlet interior: never solved, holds its allocation value
#pragma unroll
        for (int i = 0; i < NP; ++i) qpv[i] = 0.0;
        qpv[3] = P.T_ambient;
      } else {
#pragma unroll
        for (int i = 0; i < NV; ++i) qc[i] = staged ? S.stage[i][ly][lx] : q[c + (size_t)i * P.plane];
        cell_qp<NS>(P, qc, qpv);
      }
    } else {
#pragma unroll
      for (int i = 0; i < NP; ++i) qpv[i] = 0.0;
    }
#pragma unroll
    for (int i = 0; i < NP; ++i) S.tile.qp[i][ly][lx] = qpv[i];
    S.tile.info[ly][lx] = inf;
    ring_cell |= (inf & CI_SRC_MASK) == 2;
  }
  // the inlet's time ramp once per block (used after the slopes' barrier)
  if (__syncthreads_or(P.radial_source_flag && ring_cell) && threadIdx.x == 0)
    inlet_ramp(P, time, S.ramp);
  // interfaces: x faces, then y faces, one interface per thread; each
  // direction's slopes are precomputed once per cell first.
  // This thread's cell (one per thread): the x part of the divergence and
  // the x CFL dt, taken before the y phase reuses the flux arrays
  double dX[NV], dtx = P.max_dt;
#pragma unroll 1
  for (int dir = 1; dir <= 2; ++dir) {
    precompute_slopes<NS, TS>(P, S.tile, S.slopes, dir, j0, k0, &S.n_special[dir - 1], S.special,
                              FluxShared<NS, TS>::FACES);
    __syncthreads();
    const int n_special = min(S.n_special[dir - 1], FluxShared<NS, TS>::FACES);
    if (n_special) {
      special_faces<NS, TS>(P, S, n_special, dir, j0, k0, ring);
      __syncthreads();
    }
    const int count = (dir == 1) ? NXI : NYI, off = (dir == 1) ? 1 : SW,
              doff = (dir == 1) ? 1 : TX + 2;
    static_assert(NXI <= TS::THREADS && NYI <= TS::THREADS, "one interface per thread");
    // this thread's interface.  x: between cells j0+jj-1 and j0+jj of row
    // k0+kk; y: between rows k0+kk-1 and k0+kk of column j0+jj
    const int e = threadIdx.x;
    const int jj = (dir == 1) ? e % (TX + 1) : e % TX, kk = (dir == 1) ? e / (TX + 1) : e / TX;
    const int ja = (dir == 1) ? j0 + jj - 1 : j0 + jj, ka = (dir == 1) ? k0 + kk : k0 + kk - 1;
    const int ax = ja - j0 + HALO, ay = ka - k0 + HALO;
    // a direction of one cell has no fluxes and no speeds: the reference
    // skips its speeds, fluxes and divergence term (src/solver_2d.f90:
    // 2667-2681, 3946-4001), and its zero-initialised speed arrays give no
    // CFL limit there
    const bool exists = e < count && ((dir == 1) ? !(ka >= ny || ja + 1 > nx || nx == 1)
                                                 : !(ja >= nx || ka + 1 > ny || ny == 1));
    // cells outside the grid have info 0
    const uint8_t* inf = &S.tile.info[exists ? ay : 0][exists ? ax : 0];
    const bool active = exists && ((inf[0] | inf[off]) & 128);
    double H[NV], amax = 0.0, gcf = 1.0;
    bool still = false, again = false, slow = false, slow2 = false;
    if (active) {
      if (P.slope_correction_flag)
        gcf = (dir == 1) ? gcsx[(size_t)ka * (nx + 1) + (ja + 1)] : gcsy[(size_t)(ka + 1) * nx + ja];
      const int ia = ay * SW + ax, da = (ay - 1) * (TX + 2) + ax - 1;
      const uint8_t* sok = &S.slopes.ok[0][0];
      const uint8_t oa = sok[da], ob = sok[da + doff];
      FaceFrom fl = FACE_CELL, fr = FACE_CELL;
      bool la = false, lb = false;   // the side's cell has a slot for the timestep view
      if (!(oa == 1 && ob == 1)) {
        const bool rad = P.radial_source_flag != 0;
        const int n = (dir == 1) ? nx : ny, i0 = (dir == 1) ? ja : ka;
        const bool a_in = i0 >= 0, b_in = i0 + 1 < n;
        fl = face_from(rad, a_in, b_in, inf[0], inf[off], oa, 0, dir);
        fr = face_from(rad, b_in, a_in, inf[off], inf[0], ob, 1, dir);
        slow = fl == FACE_NONE || fr == FACE_NONE;
        // the fluxes from the stage view; the CFL speeds from the timestep
        // view (a second pass) when an inlet-interior cell is in the stencil
        if (rad)
          for (int m = -1; m <= 2; ++m)
            if (i0 + m >= 0 && i0 + m < n && (inf[m * off] & CI_SRC_MASK) == 1) again = true;
        la = again && a_in && i0 > 0 && (inf[-off] & CI_SRC_MASK) == 1;
        la = la || (again && b_in && (inf[off] & CI_SRC_MASK) == 1);
        lb = again && a_in && (inf[0] & CI_SRC_MASK) == 1;
        lb = lb || (again && i0 + 2 < n && (inf[2 * off] & CI_SRC_MASK) == 1);
      }
      if (!slow) {
        slow = !interface_kt<NS, TS>(P, S, dir, fl, fr, oa - FACES0, ob - FACES0, ia, ia + off, da,
                                     da + doff, gcf, H, amax, still);
        if (again) {
          double H2[NV];
          bool still2;
          slow2 = !interface_kt<NS, TS>(P, S, dir, fl, fr, oa - FACES0 + la, ob - FACES0 + lb, ia,
                                        ia + off, da, da + doff, gcf, H2, amax, still2);
        }
      }
    }
    // the special faces lie where the fluxes go
    if (n_special) __syncthreads();
    if (slow || slow2) {
      interface_special<NS, TS>(P, S, dir, e, ax, ay, ja, ka, gcf, again, ring);
    } else if (e < count) {
      S.A[e] = amax;
      if (active) {
        const int vt = 3 - dir;
        S.H[0][e] = H[0];
        (&S.H[0][0])[dir * FluxShared<NS, TS>::NI + e] = H[1];
        (&S.H[0][0])[vt * FluxShared<NS, TS>::NI + e] = H[2];
#pragma unroll
        for (int i = 3; i < NV; ++i) S.H[i][e] = H[i];
        // the cap on s/H0 needs |s| >= |H0| (rounded quotients are monotone)
        double s = 0.0;
#pragma unroll
        for (int i = 0; i < NS; ++i) s += H[4 + i];
        if (fabs(s) >= fabs(H[0]) && s != 0.0) cap_solids<NS, TS>(S, dir, e);
        if (still) {
          S.H[0][e] = 0.0;
#pragma unroll
          for (int i = 3; i < NV; ++i) S.H[i][e] = 0.0;
        }
      }
    }
    __syncthreads();
    if (dir == 1 && threadIdx.x < TX * TY) {
      const int e = threadIdx.x % TX + (threadIdx.x / TX) * (TX + 1);
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        double d = 0.0;
        if (nx > 1) d = d + (S.H[i][e + 1] - S.H[i][e]) * P.one_by_dx;
        dX[i] = d;
      }
      const double max_a = fmax_f(S.A[e], S.A[e + 1]);
      dtx = (max_a > 0.0) ? P.cfl * P.dx / max_a : P.max_dt;
    }
  }
  // cells: divergence, explicit terms, CFL
  double dtl = P.max_dt;
  for (int e = threadIdx.x; e < TX * TY; e += blockDim.x) {
    int jj = e % TX, kk = e / TX;
    int j = j0 + jj, k = k0 + kk;
    if (j >= nx || k >= ny) continue;
    int lx = jj + HALO, ly = kk + HALO;
    if (!(S.tile.info[ly][lx] & 128)) continue;
    size_t c = (size_t)k * P.pitch + j;
    double qpv[NP], ex[NV];
#pragma unroll
    for (int i = 0; i < NP; ++i) qpv[i] = S.tile.qp[i][ly][lx];
    double bx = Bx[c], by = By[c];
    double bxx = 0.0, bxy = 0.0, byy = 0.0, gcf = 1.0, dg = 0.0;
    if (P.curvature_term_flag) {
      bxx = Bxx[c];
      bxy = Bxy[c];
      byy = Byy[c];
    }
    if (P.slope_correction_flag) {
      gcf = gc[c];
      dg = dgc[c];
    }
    eval_expl_terms<NS>(P, bx, by, bxx, bxy, byy, gcf, dg, qpv, ex);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      double d = dX[i];
      if (ny > 1) d = d + (S.H[i][e + TX] - S.H[i][e]) * P.one_by_dy;
      X[c + (size_t)i * P.plane] = d - ex[i];
    }
    const double max_a = fmax_f(S.A[e], S.A[e + TX]);
    double dty = (max_a > 0.0) ? P.cfl * P.dy / max_a : dtl;
    dtl = fmin_f(dtl, fmin_f(dtx, dty));
  }
  // block minimum, then a global atomic min on the bits of the positive double
  for (int off = 16; off > 0; off >>= 1) dtl = fmin_f(dtl, __shfl_down_sync(0xffffffffu, dtl, off));
  if ((threadIdx.x & 31) == 0) S.dtmin[threadIdx.x >> 5] = dtl;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = S.dtmin[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = fmin_f(m, S.dtmin[w]);
    // a speed of +inf gives a cell dt of +0.0, which the reference's MIN
    // keeps; the block minimum is never negative and NaN is filtered by
    // fmin_f, so the ordered-bits atomicMin sees only non-negative doubles
    if (m >= 0.0 && m < P.max_dt)
      atomicMin(&clk->dtmin_bits, (unsigned long long)__double_as_longlong(m));
  }
}

template <int NS>
__global__ void __launch_bounds__(FLUX_THREADS, flux_min_blocks<NS>())
    k_flux(const __grid_constant__ DevParams Pp, const double* __restrict__ q, const uint8_t* __restrict__ mask,
           const uint8_t* __restrict__ cellinfo, const double* __restrict__ Bx,
           const double* __restrict__ By, const double* __restrict__ Bxx,
           const double* __restrict__ Bxy, const double* __restrict__ Byy,
           const double* __restrict__ gc, const double* __restrict__ dgc,
           const double* __restrict__ gcsx, const double* __restrict__ gcsy,
           const RingCell* __restrict__ ring, DevClock* clk, double* __restrict__ X) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  FluxShared<NS>& S = *reinterpret_cast<FluxShared<NS>*>(smem_raw);
  flux_tile<NS, Shape32x8>(Pp, q, mask, cellinfo, Bx, By, Bxx, Bxy, Byy, gc, dgc, gcsx, gcsy, ring,
                           clk, X, blockIdx.x * TX, blockIdx.y * TY, S);
}

// k_flux with the tile's q planes loaded by one TMA box (qmap: a tensor map
// of q, dims {nx, ny, n_v}, box {SW, SH, n_v}, zero fill outside the grid).
template <int NS>
__global__ void __launch_bounds__(FLUX_THREADS, flux_min_blocks<NS>())
    k_flux_tma(const __grid_constant__ DevParams Pp, const __grid_constant__ CUtensorMap qmap,
               const double* __restrict__ q, const uint8_t* __restrict__ mask,
               const uint8_t* __restrict__ cellinfo, const double* __restrict__ Bx,
               const double* __restrict__ By, const double* __restrict__ Bxx,
               const double* __restrict__ Bxy, const double* __restrict__ Byy,
               const double* __restrict__ gc, const double* __restrict__ dgc,
               const double* __restrict__ gcsx, const double* __restrict__ gcsy,
               const RingCell* __restrict__ ring, DevClock* clk, double* __restrict__ X) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  FluxShared<NS>& S = *reinterpret_cast<FluxShared<NS>*>(smem_raw);
  flux_tile<NS, Shape32x8>(Pp, q, mask, cellinfo, Bx, By, Bxx, Bxy, Byy, gc, dgc, gcsx, gcsy, ring,
                           clk, X, blockIdx.x * TX, blockIdx.y * TY, S, &qmap);
}

// k_flux_tma over the tile rows [ty0, ty0 + gridDim.y) (imex_gpu_advance_host).
template <int NS>
__global__ void __launch_bounds__(FLUX_THREADS, flux_min_blocks<NS>())
    k_flux_tma_rows(const __grid_constant__ DevParams Pp, const __grid_constant__ CUtensorMap qmap,
                    const double* __restrict__ q, const uint8_t* __restrict__ mask,
                    const uint8_t* __restrict__ cellinfo, const double* __restrict__ Bx,
                    const double* __restrict__ By, const double* __restrict__ Bxx,
                    const double* __restrict__ Bxy, const double* __restrict__ Byy,
                    const double* __restrict__ gc, const double* __restrict__ dgc,
                    const double* __restrict__ gcsx, const double* __restrict__ gcsy,
                    const RingCell* __restrict__ ring, DevClock* clk, double* __restrict__ X,
                    int ty0) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  FluxShared<NS>& S = *reinterpret_cast<FluxShared<NS>*>(smem_raw);
  flux_tile<NS, Shape32x8>(Pp, q, mask, cellinfo, Bx, By, Bxx, Bxy, Byy, gc, dgc, gcsx, gcsy, ring,
                           clk, X, blockIdx.x * TX, (blockIdx.y + ty0) * TY, S, &qmap);
}

// k_flux over the tile rows [ty0, ty0 + gridDim.y) (imex_gpu_advance_host).
template <int NS>
__global__ void __launch_bounds__(FLUX_THREADS, flux_min_blocks<NS>())
    k_flux_rows(const __grid_constant__ DevParams Pp, const double* __restrict__ q,
                const uint8_t* __restrict__ mask, const uint8_t* __restrict__ cellinfo,
                const double* __restrict__ Bx, const double* __restrict__ By,
                const double* __restrict__ Bxx, const double* __restrict__ Bxy,
                const double* __restrict__ Byy, const double* __restrict__ gc,
                const double* __restrict__ dgc, const double* __restrict__ gcsx,
                const double* __restrict__ gcsy, const RingCell* __restrict__ ring, DevClock* clk,
                double* __restrict__ X, int ty0) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  FluxShared<NS>& S = *reinterpret_cast<FluxShared<NS>*>(smem_raw);
  flux_tile<NS, Shape32x8>(Pp, q, mask, cellinfo, Bx, By, Bxx, Bxy, Byy, gc, dgc, gcsx, gcsy, ring,
                           clk, X, blockIdx.x * TX, (blockIdx.y + ty0) * TY, S);
}

// =============================================================== Newton
// solve_rk_step (src/solver_2d.f90:1660-1994) for a_diag = 1 (stage 2 of the
// n_RK = 2 tableau): newton_begin (scaling and start), then newton_step per
// iteration.
constexpr int NEWTON_MAX_IT = 100;
constexpr double NEWTON_TOLF = 1.0e-10, NEWTON_STPMX = 100.0;

#ifndef IMEX_EVAL_FN
#define IMEX_EVAL_FN IMEX_FLAT
#endif
// Per-cell vectors that are only read during the solve (the old state, Rj, the
// scaling) have a stride ST: 1 in registers, or the block size in shared memory
// (NewtonShared).
// The residual of qj with its implicit terms, and half its squared norm.
template <int NS, int ST>
IMEX_EVAL_FN void newton_residual(const double* qj, const double* qj_old, const double* Rj,
                                  double nh2, double nh3, double dt, double* f, double& scal_f) {
  constexpr int NV = 4 + NS;
  double d = 0.0;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    double nh = (i == 1) ? nh2 : ((i == 2) ? nh3 : 0.0);
    double R = Rj[i * ST] - 1.0 * nh;
    double fi = qj[i] - qj_old[i * ST] + dt * R;
    const double fs = 1.0 * fi;
    f[i] = fs;
    d += fs * fs;
  }
  scal_f = 0.5 * d;
}
// The implicit terms of a state outside friction_real's and
// friction_jacobian's range.
template <int NS>
IMEX_FLAT void friction_any(const DevParams& P, double bx, double by, const double* qj, double& nh2,
                            double& nh3) {
  double t[4 + NS], nh[2];
#pragma unroll
  for (int i = 0; i < 4 + NS; ++i) t[i] = qj[i];
  implicit_terms_any<NS>(P, bx, by, t, nh);
  nh2 = nh[0];
  nh3 = nh[1];
}
template <int NS, int ST>
IMEX_EVAL_FN void eval_f(const DevParams& P, const double* qj, const double* qj_old,
                       const double* Rj, double bx, double by, double dt, double* f,
                       double& scal_f) {
  double nh2, nh3;
  if (!friction_real<NS>(P, bx, by, qj, nh2, nh3)) friction_any<NS>(P, bx, by, qj, nh2, nh3);
  newton_residual<NS, ST>(qj, qj_old, Rj, nh2, nh3, dt, f, scal_f);
}

// Jacobian columns 2,3 by complex step (src/solver_2d.f90:2300-2365) and the
// Newton direction: explicit rows diagonal, 2x2 Cramer on rows/cols 2,3
// (src/solver_2d.f90:1879-1901).
template <int NS>
IMEX_FLAT void newton_direction(const DevParams& P, double bx, double by, double dt,
                                              const double* qj_org, const double* qj_rel,
                                              const double* rt, double* dd, double* J2,
                                              double* J3) {
  constexpr int NV = 4 + NS;
  CPrefix<NS> pre;
  {
    cplx qc[NV];
#pragma unroll
    for (int m = 0; m < NV; ++m) qc[m] = mulr(C(qj_rel[m], 0.0), qj_org[m]);
    implicit_prefix_c<NS>(P, qc, pre);
  }
  auto column = [&](int col) {
    cplx qc[NV];
#pragma unroll
    for (int m = 0; m < NV; ++m) qc[m] = mulr(C(qj_rel[m], (m == col) ? P.hstep : 0.0), qj_org[m]);
    cplx nh2, nh3;
    implicit_terms_c<NS>(P, bx, by, qc, pre, nh2, nh3);
#pragma unroll
    for (int r = 0; r < NV; ++r) {
      double nim = (r == 1) ? nh2.im : ((r == 2) ? nh3.im : 0.0);
      double jac = 1.0 * nim * P.one_by_h;
      double l0 = (r == col) ? 1.0 * (col == 1 ? qj_org[1] : qj_org[2]) : 0.0;
      double v = l0 - dt * 1.0 * jac;
      if (col == 1) J2[r] = v;
      else J3[r] = v;
    }
  };
#pragma unroll 1
  for (int col = 1; col <= 2; ++col) column(col);
  double d1[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) d1[i] = (i == 1 || i == 2) ? 0.0 : rt[i] / (1.0 * qj_org[i]);
  double d2a = rt[1], d2b = rt[2];
  {
    double s = 0.0, s2 = 0.0;
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (i != 1 && i != 2) s += d1[i] * 0.0;
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (i != 1 && i != 2) s2 += d1[i] * 0.0;
    d2a = d2a - s;
    d2b = d2b - s2;
  }
  double s11 = J2[1], s21 = J2[2], s12 = J3[1], s22 = J3[2];
  double inv_det = 1.0 / (s11 * s22 - s21 * s12);
  double sol0 = (d2a * s22 - d2b * s12) * inv_det;
  double sol1 = (s11 * d2b - s21 * d2a) * inv_det;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    if (i == 1) dd[i] = -sol0 + 0.0;
    else if (i == 2) dd[i] = -sol1 + 0.0;
    else dd[i] = 0.0 + (-d1[i]);
  }
}

// The direction and the gradient J^T rt by the general expressions, as a call:
// in holds qj_org, qj_rel and rt, out receives dd and grad.
template <int NS>
IMEX_NOINL void newton_direction_any(const DevParams& P, double bx, double by, double dt,
                                     const double* in, double* out) {
  constexpr int NV = 4 + NS;
  double J2[NV], J3[NV];
  newton_direction<NS>(P, bx, by, dt, in, in + NV, in + 2 * NV, out, J2, J3);
#pragma unroll
  for (int c = 0; c < NV; ++c) {
    double s = 0.0;
#pragma unroll
    for (int r = 0; r < NV; ++r) {
      double L;
      if (c == 1) L = J2[r];
      else if (c == 2) L = J3[r];
      else L = (r == c) ? 1.0 * in[c] : 0.0;
      s += in[2 * NV + r] * L;
    }
    out[NV + c] = s;
  }
}

// dd and grad from the friction's imaginary parts nim (friction_jacobian) where
// `ok` says they hold; with a finite rt of ordinary size the zero rows of
// the Jacobian add exact zeros and are left out.  Otherwise the general call.
template <int NS, int ST>
IMEX_FLAT void newton_dir_grad(const DevParams& P, double bx, double by, double dt,
                               const double* qj_org, const double* qj_rel, const double* rt,
                               bool ok, const double* nim, double* dd, double* grad) {
  constexpr int NV = 4 + NS;
#pragma unroll
  for (int i = 0; i < NV; ++i) ok = ok & below_huge(rt[i]) & below_huge(qj_org[i * ST]);
  if (ok && dt > 0.0 && dt < 1e300) {
    const double s11 = 1.0 * qj_org[1 * ST] - dt * 1.0 * (1.0 * nim[0] * P.one_by_h);
    const double s21 = 0.0 - dt * 1.0 * (1.0 * nim[1] * P.one_by_h);
    const double s12 = 0.0 - dt * 1.0 * (1.0 * nim[2] * P.one_by_h);
    const double s22 = 1.0 * qj_org[2 * ST] - dt * 1.0 * (1.0 * nim[3] * P.one_by_h);
    const double inv_det = 1.0 / (s11 * s22 - s21 * s12);
    const double sol0 = (rt[1] * s22 - rt[2] * s12) * inv_det;
    const double sol1 = (s11 * rt[2] - s21 * rt[1]) * inv_det;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (i == 1 || i == 2) continue;
      dd[i] = 0.0 + (-(rt[i] / (1.0 * qj_org[i * ST])));
      grad[i] = 0.0 + rt[i] * (1.0 * qj_org[i * ST]);
    }
    dd[1] = -sol0 + 0.0;
    dd[2] = -sol1 + 0.0;
    grad[1] = (0.0 + rt[1] * s11) + rt[2] * s21;
    grad[2] = (0.0 + rt[1] * s12) + rt[2] * s22;
    return;
  }
  double in[3 * NV], out[2 * NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    in[i] = qj_org[i * ST];
    in[NV + i] = qj_rel[i];
    in[2 * NV + i] = rt[i];
  }
  newton_direction_any<NS>(P, bx, by, dt, in, out);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    dd[i] = out[i];
    grad[i] = out[NV + i];
  }
}

// Scaling (src/solver_2d.f90:1786-1798).
template <int NS>
__device__ __forceinline__ void newton_scale(const double* qj, double* qj_org) {
  constexpr int NV = 4 + NS;
#pragma unroll
  for (int i = 0; i < NV; ++i) qj_org[i] = fmax_f(fabs(qj[i]), 1.0e-3);
}

// Before the first iteration: the scaling of the start g, and qj_rel = g/qj_org.
// The reference's residual test before the first Jacobian is taken at g; where the
// scaling is exact (g = qj_rel*qj_org, as it is for |g| >= 1e-3) the first
// newton_step takes it with its Jacobian (need_rt), else it is taken here.  True: g
// already meets TOLF (nl_iter = 1); the iterate qj_rel*qj_org is then g.
template <int NS, int ST>
IMEX_FLAT bool newton_begin(const DevParams& P, const double* g, const double* qj_old,
                            const double* Rj, double bx, double by, double dt, double* qj_org,
                            double* qj_rel, double* rt, double& scal_f, bool& need_rt) {
  constexpr int NV = 4 + NS;
  bool same = true;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const double org = fmax_f(fabs(g[i]), 1.0e-3);
    qj_org[i * ST] = org;
    // g/|g| is +-1
    const double x =
        (fabs(g[i]) >= 1.0e-3 && below_huge(g[i])) ? copysign(1.0, g[i]) : g[i] / org;
    same = same && x * org == g[i];
    qj_rel[i] = x;
    rt[i] = 0.0;
  }
  scal_f = 0.0;
  need_rt = same;
  if (same) return false;
  double nh2, nh3;
  friction_any<NS>(P, bx, by, g, nh2, nh3);
  newton_residual<NS, ST>(g, qj_old, Rj, nh2, nh3, dt, rt, scal_f);
  double mx = fabs(rt[0]);
#pragma unroll
  for (int i = 1; i < NV; ++i) mx = fmax_f(mx, fabs(rt[i]));
  if (!(mx < NEWTON_TOLF)) return false;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    qj_org[i * ST] = 1.0;
    qj_rel[i] = g[i];
  }
  return true;
}

// One Newton iteration (src/solver_2d.f90:1815-1824, 1879-1988); qj_rel
// receives the iterate (times qj_org), rt its residual.  Iteration 1 is a full
// step; the later ones search along it with lnsrch (:2019-2224).  The
// reference evaluates the residual at the start of every iteration; it
// equals the one left by the previous iteration, so it is taken only in iteration 1
// (need_rt) and where the previous iteration's line search put the old
// iterate back (alam < alamin or the trial cap), leaving the residual of
// its last trial: `stale` marks that case (the loop only continues after such a
// restore when the relative step is NaN).  Every backtrack after the first
// halves alam: the cubic model's value is clamped to <= alam/2 and then maxed with
// alam/2.  The trials are capped at 4096; the cap exits like alam < alamin.
// All iterations share this code, so that a warp in its second or third
// iteration finds it in the instruction cache.  With *defer set, a cell whose
// state needs the general direction is left as it is, with *defer still set
// (cleared otherwise).
template <int NS, int ST, bool STOP = true>
IMEX_FLAT bool newton_step(const DevParams& P, bool first, bool need_rt, const double* qj_old,
                           const double* Rj, const double* qj_org, double bx, double by, double dt,
                           double* qj_rel, double* rt, double& scal_f, unsigned& trials,
                           bool& stale, bool* defer = nullptr) {
  constexpr int NV = 4 + NS;
  double dd[NV], slope = 0.0;
  {
    double x[NV], grad[NV], nh2, nh3, nim[4];
#pragma unroll
    for (int i = 0; i < NV; ++i) x[i] = qj_rel[i] * qj_org[i * ST];
    const bool ok = friction_jacobian<NS, STOP>(P, bx, by, x, P.hstep * qj_org[1 * ST],
                                                P.hstep * qj_org[2 * ST], nh2, nh3, nim);
    if (defer && *defer) {
      *defer = !ok;
      if (!ok) return false;
    }
    if (need_rt || stale) {
      stale = false;
      if (!ok) friction_any<NS>(P, bx, by, x, nh2, nh3);
      newton_residual<NS, ST>(x, qj_old, Rj, nh2, nh3, dt, rt, scal_f);
      double mx = fabs(rt[0]);
#pragma unroll
      for (int i = 1; i < NV; ++i) mx = fmax_f(mx, fabs(rt[i]));
      if (mx < NEWTON_TOLF) return true;
    }
    newton_dir_grad<NS, ST>(P, bx, by, dt, qj_org, qj_rel, rt, ok, nim, dd, grad);
    // NORM2(dd) > stpmax = STPMX*MAX(NORM2(qj_rel), NV) scales the step.  The
    // scaled sum below ends with scale = MAX|dd| and ssq <= NV (each term at
    // most 1) up to a few roundings, so its result is below 3*MAX|dd| for
    // NV <= 8; when that bound is already below stpmax (finite), or below
    // STPMX*NV, the norms are not evaluated.  A NaN component gives a NaN norm
    // and no scaling either way.
    static_assert(NV <= 8, "the norm bound 3*MAX|dd| holds for up to 8 components");
    double dmax = 0.0;
#pragma unroll
    for (int i = 0; i < NV; ++i) dmax = fmax_f(dmax, fabs(dd[i]));
    if (!first && !(3.0 * dmax < NEWTON_STPMX * (double)NV)) {
      double sdot = 0.0;
#pragma unroll
      for (int i = 0; i < NV; ++i) sdot += qj_rel[i] * qj_rel[i];
      const double stpmax = NEWTON_STPMX * fmax_f(sqrt(sdot), (double)NV);
      if (!(3.0 * dmax < stpmax)) {
        double scale = 0.0, ssq = 0.0;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          if (dd[i] != 0.0) {
            double ax = fabs(dd[i]);
            if (scale < ax) {
              double val = scale / ax;
              ssq = 1.0 + ssq * val * val;
              scale = ax;
            } else {
              double val = ax / scale;
              ssq = ssq + val * val;
            }
          }
        }
        double dabs = scale * sqrt(ssq);
        if (dabs > stpmax) {
#pragma unroll
          for (int i = 0; i < NV; ++i) dd[i] = dd[i] * stpmax / dabs;
        }
      }
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) slope += grad[i] * dd[i];
  }
  // qj_rel keeps the old iterate until the end of the search
  bool xfin = true, fin = true;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    xfin = xfin & isfinite(qj_rel[i]);
    fin = fin & isfinite(dd[i]);
  }
  const double scal_f_old = scal_f;
  double alamin = 1.0, alam = 1.0;
  bool keep = true;   // the old iterate stays
  if (!first) {
    // MAX of |dd_i|/MAX(|x_i|, 1): one division for the largest |dd|, and one
    // for each other that could still exceed it (|dd_i| bounds its quotient)
    double mx = 0.0;
    bool all = !(xfin && fin);
    if (!all) {
      double top = 0.0, d = 1.0;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const double a = fabs(dd[i]);
        if (i == 0 || a > top) {
          top = a;
          d = fmax_f(fabs(qj_rel[i]), 1.0);
        }
      }
      mx = (d == 1.0) ? top : top / d;
#pragma unroll
      for (int i = 0; i < NV; ++i) all |= fabs(dd[i]) > mx;
    }
    if (all) {
#pragma unroll 1
      for (int i = 0; i < NV; ++i) {
        double a = dd[0], x = qj_rel[0];
#pragma unroll
        for (int m = 1; m < NV; ++m)
          if (m == i) {
            a = dd[m];
            x = qj_rel[m];
          }
        const double r = fabs(a) / fmax_f(fabs(x), 1.0);
        mx = (i == 0) ? r : fmax_f(mx, r);
      }
    }
    alamin = EPS / mx;
  }
  if (alamin != 0.0) {
    // Rows other than 2, 3 carry no implicit term: eval_f's sum of f^2
    // taken over them alone, in eval_f's order, cannot exceed the full sum
    // (rounded addition of a term >= 0 never decreases a sum, and rounding
    // is monotone).  When that partial half-sum already exceeds
    // 0.9*scal_f_old the trial fails whatever the implicit terms are, and
    // the implicit terms are not evaluated.  Only for trials whose failure
    // is all that matters: not trial 0 and not alam = 1 (their scal_f sets
    // the next alam), and with a finite old iterate (then the residual left
    // by the last trial is never read: a search that puts the old iterate
    // back ends the iteration as converged).
    //
    // After the first backtrack every alam is half the previous one,
    // whatever a trial's outcome, so two consecutive trials' partial sums
    // are evaluated side by side (independent chains) and their outcomes
    // then taken in order, as one trial after the other.  Once a trial leaves
    // all those rows' iterates where they were (x + alam*dd rounds to x, as
    // it then does for every smaller alam), the partial sum no longer changes:
    // the remaining trials fail with it and are only counted.
    auto partial_half_sum = [&](double al, bool& still) {
      double d = 0.0;
      still = true;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        if (i == 1 || i == 2) continue;
        const double xo = qj_rel[i], xt = xo + al * dd[i];
        still = still & (xt == xo);
        const double qt = xt * qj_org[i * ST];
        const double R = Rj[i * ST] - 1.0 * 0.0;
        const double fi = qt - qj_old[i * ST] + dt * R;
        const double f = 1.0 * fi;
        d += f * f;
      }
      return 0.5 * d;
    };
    const double sf_thr = 0.9 * scal_f_old;
    int trial = 0;
    bool capped = true;   // the loop ran out of its 4096 trials
    while (trial < 4096) {
      if (trial > 0 && alam != 1.0 && xfin) {
        const double alam_b = 0.5 * alam;
        bool still_a, still_b;
        const double ha = partial_half_sum(alam, still_a);
        const double hb = partial_half_sum(alam_b, still_b);
        if (ha > sf_thr) {            // trial `trial` fails
          ++trials;
          if (alam < alamin) {
            capped = false;
            stale = true;
            break;
          }
          alam = alam_b;
          if (++trial >= 4096) break;
          if (alam != 1.0 && hb > sf_thr) {   // and so does the next one
            bool out = false;
            do {                              // (and, still_b, all after it)
              ++trials;
              if (alam < alamin) {
                capped = false;
                stale = true;
                out = true;
                break;
              }
              alam = 0.5 * alam;
              ++trial;
            } while (still_b && trial < 4096);
            if (out) break;
            continue;
          }
        }
      }
      // a trial with the full residual
      double qt[NV];
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const double xt = qj_rel[i] + alam * dd[i];
        qt[i] = xt * qj_org[i * ST];
      }
      eval_f<NS, ST>(P, qt, qj_old, Rj, bx, by, dt, rt, scal_f);
      capped = false;
      if (first) break;
      ++trials;
      if (scal_f <= sf_thr) break;
      if (alam < alamin) {
        stale = true;
        break;
      }
      capped = true;
      if (alam == 1.0) {
        double tmplam = -slope / (2.0 * (scal_f - scal_f_old - slope));
        alam = fmax_f(tmplam, 0.5 * alam);
      } else {
        alam = 0.5 * alam;
      }
      ++trial;
    }
    // alam < alamin or the trial cap: the old iterate is put back
    keep = stale || capped;
    if (keep) {
      scal_f = scal_f_old;
      stale = true;
    }
  }
  // the exit tests (src/solver_2d.f90:1964-1988): MAX|rt| < TOLF, or
  // MAX over i of |x_i - x_old_i|/MAX(|x_i|, 1) < EPS.  MAX skips NaN
  // quotients (all NaN: NaN, and the test fails), so the second holds when
  // some quotient is a number and every such quotient is below EPS; each
  // comparison of a rounded quotient is taken without the division where
  // its answer is certain (rel_change_below).
  bool any = false, below = true;
  double mx = fabs(rt[0]);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    if (i > 0) mx = fmax_f(mx, fabs(rt[i]));
    const double xo = qj_rel[i], x = keep ? xo : xo + alam * dd[i];
    qj_rel[i] = x;
    const double d = fabs(x - xo), s = fmax_f(fabs(x), 1.0);
    if (isnan(d) || (isinf(d) && isinf(s))) continue;   // the quotient is NaN
    any = true;
    below = below & rel_change_below(d, s, EPS);
  }
  return mx < NEWTON_TOLF || (any && below);
}

// ============================================================ mass exchange
template <int NS>
IMEX_FLAT void mass_exchange(const DevParams& P, const double* qpj, double bx, double by,
                              const double* erod, double dtl, double* ers, double* dep,
                              double& cpe, double& cpl, double* eqns, double& topo,
                              bool& dep_neg) {
  constexpr int NV = 4 + NS;
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    ers[i] = 0.0;
    dep[i] = 0.0;
  }
  cpe = 0.0;
  cpl = 0.0;
#pragma unroll
  for (int i = 0; i < NV; ++i) eqns[i] = 0.0;
  topo = 0.0;
  if (qpj[0] <= EPS) return;
  const double alpha_max = 0.6, hind_exp = 4.65;
  double r_h = qpj[0], r_u = qpj[NV], r_v = qpj[NV + 1];
  double al[NS];
#pragma unroll
  for (int i = 0; i < NS; ++i) al[i] = P.alpha_flag ? qpj[4 + i] : qpj[4 + i] / qpj[0];
  double at = 0.0;
#pragma unroll
  for (int i = 0; i < NS; ++i) at += al[i];
  double r_w = P.slope_correction_flag ? (r_u * bx + r_v * by) : 0.0;
  double mv2 = r_u * r_u + r_v * r_v + r_w * r_w;
  double mv = sqrt(mv2);
  double tse;
  if (P.erosion_coeff > 0.0) {
    double te = P.erosion_coeff * mv * r_h * (1.0 - at);
    tse = te * (1.0 - P.erodible_porosity);
#pragma unroll
    for (int i = 0; i < NS; ++i) ers[i] = P.erodible_fract[i] * tse;
  }
#pragma unroll
  for (int i = 0; i < NS; ++i) ers[i] = fmax_f(0.0, fmin_f(ers[i], erod[i] / dtl));
  tse = 0.0;
#pragma unroll
  for (int i = 0; i < NS; ++i) tse += ers[i];
  double te = tse / (1.0 - P.erodible_porosity);
  cpe = te * P.erodible_porosity;
  if (at <= P.alphastot_min) return;
  double r_T = qpj[3];
  Mixt m = mixt_var<NS>(P, qpj);
  double spc = sp_heat_c_of<NS>(P, qpj, m.rho_m);
  double ikv = 1.0 / P.kin_visc_c;
  double hind = -1.0;   // the hindered-settling factor, the same for every class
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    if (al[i] > 0.0 && P.settling_flag) {
      double sv = settling_velocity(P, P.diam_s[i], P.rho_s[i], m.rho_c, ikv);
      dep[i] = al[i] * sv * 1.0;
      if (hind < 0.0) hind = ipow(1.0 - fmin_f(1.0, at / alpha_max), hind_exp);
      dep[i] = dep[i] * hind;
      dep[i] = fmin_f(dep[i], r_h * al[i] / dtl);
      if (dep[i] < 0.0) dep_neg = true;
    }
  }
  double sdep = 0.0;
#pragma unroll
  for (int i = 0; i < NS; ++i) sdep += dep[i];
  cpl = 0.0;
  cpl = cpl + P.coeff_porosity * sdep;
  double sal = 0.0;
#pragma unroll
  for (int i = 0; i < NS; ++i) sal += al[i];
  cpl = fmin_f(cpl, r_h * fmax_f(0.0, P.maximum_solid_packing - sal) / dtl);
  cpl = fmin_f(cpl, (r_h * (1.0 - sal) - P.coeff_porosity * (r_h * sal - dtl * sdep)) / dtl);
  double T_erod = P.erodible_deposit_flag ? r_T : P.T_erodible;
  double air_entr = 0.0;
  if (P.entrainment_flag && r_h > 0.0 && m.Ri > 0.0) {
    double entr_coeff = 0.075 / sqrt(1.0 + 718.0 * ipow(m.Ri, 2.4));
    air_entr = entr_coeff * sqrt(mv2);
  }
  double dep_tot = 0.0, ers_tot = 0.0, rdt = 0.0, ret = 0.0;
#pragma unroll
  for (int i = 0; i < NS; ++i) dep_tot += dep[i];
#pragma unroll
  for (int i = 0; i < NS; ++i) ers_tot += ers[i];
#pragma unroll
  for (int i = 0; i < NS; ++i) rdt += P.rho_s[i] * dep[i];
#pragma unroll
  for (int i = 0; i < NS; ++i) ret += P.rho_s[i] * ers[i];
  eqns[0] = P.rho_a_amb * air_entr + ret - rdt + P.rho_c_sub * cpe - m.rho_c * cpl;
  eqns[1] = -(r_u * (rdt + m.rho_c * cpl));
  eqns[2] = -(r_v * (rdt + m.rho_c * cpl));
  double sdh = 0.0, seh = 0.0;
#pragma unroll
  for (int i = 0; i < NS; ++i) sdh += P.rho_s[i] * P.sp_heat_s[i] * dep[i];
#pragma unroll
  for (int i = 0; i < NS; ++i) seh += P.rho_s[i] * P.sp_heat_s[i] * ers[i];
  if (P.energy_flag)
    eqns[3] = -(r_T * (sdh + m.rho_c * spc * cpl)) - 0.5 * mv2 * (rdt + m.rho_c * cpl) +
              T_erod * (seh + P.rho_c_sub * spc * cpe) +
              P.T_ambient * P.sp_heat_a * P.rho_a_amb * air_entr;
  else
    eqns[3] = -(r_T * (sdh + m.rho_c * spc * cpl)) + T_erod * (seh + P.rho_c_sub * spc * cpe) +
              P.T_ambient * P.sp_heat_a * P.rho_a_amb * air_entr;
#pragma unroll
  for (int i = 0; i < NS; ++i) eqns[4 + i] = P.rho_s[i] * (ers[i] - dep[i]);
  topo = (dep_tot - ers_tot) / (1.0 - P.erodible_porosity);
}

// update_erosion_deposition_cell for one cell (src/solver_2d.f90:2431-2588).
template <int NS>
__device__ bool erosion_cell(const DevParams& P, double* qc, double bx, double by,
                             double* erod, double* depo, double* eros, double* Bc,
                             double dtl) {
  constexpr int NV = 4 + NS, NP = 6 + NS;
  double qpv[NP];
  cell_qp<NS>(P, qc, qpv);
  double ers[NS], dep[NS], cpe, cpl, eqns[NV], topo;
  bool bad = false;
  mass_exchange<NS>(P, qpv, bx, by, erod, dtl, ers, dep, cpe, cpl, eqns, topo, bad);
#pragma unroll
  for (int i = 0; i < NV; ++i) qc[i] = qc[i] + dtl * eqns[i];
#pragma unroll
  for (int i = 0; i < NS; ++i) qc[4 + i] = fmax_f(0.0, qc[4 + i]);
#pragma unroll
  for (int i = 0; i < NS; ++i) depo[i] = depo[i] + dtl * dep[i];
#pragma unroll
  for (int i = 0; i < NS; ++i) eros[i] = eros[i] + dtl * ers[i];
#pragma unroll
  for (int i = 0; i < NS; ++i) erod[i] = erod[i] - dtl * ers[i];
  if (P.erodible_deposit_flag) {
#pragma unroll
    for (int i = 0; i < NS; ++i) erod[i] = erod[i] + dtl * dep[i];
  }
  if (P.topo_change_flag) *Bc = *Bc + dtl * topo;
#pragma unroll
  for (int i = 0; i < NS; ++i) bad |= (qc[4 + i] < 0.0);
  if (qc[0] <= 0.0) {
    if (qc[0] > -1.0e-10) {
#pragma unroll
      for (int i = 0; i < NV; ++i) qc[i] = 0.0;
    } else {
      bad = true;
    }
  }
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < NS; ++i) s += qc[4 + i];
  if (s > qc[0]) {
    if (qc[0] < 1.0e-10) {
      double s2 = 0.0;
#pragma unroll
      for (int i = 0; i < NS; ++i) s2 += qc[4 + i];
#pragma unroll
      for (int i = 0; i < NS; ++i) qc[4 + i] = qc[4 + i] / s2 * qc[0];
    } else {
      bad = true;
    }
  }
  double red_grav = 0.0;
  if (qc[0] > 0.0) {
    qc_to_qp<NS>(P, qc, qpv);
    red_grav = mixt_var<NS>(P, qpv).red_grav;
  }
  if (red_grav <= 0.0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) qc[i] = 0.0;
  }
  return bad;
}

// =============================================================== stage 2
// RK stage 2 (src/solver_2d.f90:1105-1628):
//   k_stage2         q_fv, semi-implicit terms, q_si, Rj_not_impl, the Newton
//                    solve, sign guard, assemble_sol checks and fixes, q
//                    written: one thread per cell, its vectors in shared memory
//   k_stage2_rest    on large grids, the cells that k_stage2 left iterating
//                    when few lanes of their warp were, compacted in a list
// With the learned start or its harvest stage 2 is cut where those need it:
// k_stage2_first (up to the solve), the network, k_stage2_solve, k_stage2_post (sign guard
// and assembly).
// Between kernels a cell's Newton state (qj_rel, the residual, its norm) is
// kept in the NewtonWork planes; the iterate is carried bit for bit, so a
// cell's arithmetic is that of one uninterrupted solve_rk_step.
struct NewtonWork {
  double* qsi;    // nv planes: q_si, the Newton initial guess (scaling source)
  double* Rj;     // nv planes: Rj_not_impl
  double* x;      // nv planes: qj_rel while iterating, the final qj when done
  double* rt;     // nv planes: residual
  double* sf;     // 1 plane: 0.5*|residual|^2
  uint8_t* status;  // 1 plane: bit 0 the cell went through Newton, bit 1 its
                    // residual must be evaluated again (see newton_step); listed
                    // cells: iterations taken in the upper bits
  uint32_t* list;   // cells (k*pitch + j) still iterating
  uint32_t* cells;  // the mask's solve cells (k*pitch + j) on grids of DENSE_MIN_GRID cells, else null
  // learned warm start (warm != 0): the Newton cells of the step, their
  // network inputs and the network's momentum guesses
  int warm;
  uint32_t* wlist;    // Newton cells, in append order
  uint32_t* flist;    // warm starts to redo from q_si (k_stage2_fallback)
  float* feat;        // WARM_IN floats per wlist entry
  double* guess;      // 2 planes: proposed q(2), q(3)
  // training pairs (harvest != 0): inputs and targets of every `stride`-th
  // Newton cell, up to `cap` pairs
  int harvest;
  unsigned int hstride;
  unsigned long long hcap;
  float* hx;
  float* hy;
};

// Network inputs of one Newton cell: class-count independent quantities of
// q_si, the old state, the explicit tendency, dt and the slope.  Targets:
// the change of the two momentum components over the Newton solve, per unit
// of q(1).
constexpr int WARM_IN = 12, WARM_OUT = 2;

template <int NS>
__device__ __forceinline__ void warm_features(const double* qsi, const double* q0,
                                              const double* Rj, double dt, double bx,
                                              double by, float* f) {
  const double m = qsi[0], im = 1.0 / m;
  double xs = 0.0;
#pragma unroll
  for (int i = 0; i < NS; ++i) xs += qsi[4 + i];
  f[0] = (float)log10(fmax(m, 1.0e-12));
  f[1] = (float)(qsi[1] * im);
  f[2] = (float)(qsi[2] * im);
  f[3] = (float)(q0[1] * im);
  f[4] = (float)(q0[2] * im);
  f[5] = (float)(dt * Rj[1] * im);
  f[6] = (float)(dt * Rj[2] * im);
  f[7] = (float)(qsi[3] * im * 1.0e-6);
  f[8] = (float)(xs * im);
  f[9] = (float)log10(dt);
  f[10] = (float)bx;
  f[11] = (float)by;
}

struct WarmNorm {
  float x_mean[WARM_IN], x_std[WARM_IN], y_mean[WARM_OUT], y_std[WARM_OUT];
};

constexpr int STAGE2_THREADS = 128;

__device__ __forceinline__ unsigned int list_append(bool add, uint32_t c, uint32_t* list,
                                                    unsigned int* count) {
  const unsigned m = __ballot_sync(0xffffffffu, add);
  if (!m) return 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(m) - 1;
  unsigned int base = 0;
  if (lane == leader) base = atomicAdd(count, (unsigned int)__popc(m));
  base = __shfl_sync(0xffffffffu, base, leader);
  const unsigned int slot = base + __popc(m & ((1u << lane) - 1u));
  if (add) list[slot] = c;
  return add ? slot : 0xffffffffu;
}

// Newton statistics of a block (or warp), summed in shared memory and added to
// the clock at its end by threads t = 0..: one global atomic per warp and
// counter queued a few million of them on one address at 4096^2.
struct NewtonStats {
  unsigned hist[16];
  unsigned long long cells, iters, trials, maxit;
};
__device__ __forceinline__ void stat_reset(NewtonStats& S, int t) {   // a barrier must follow
  if (t < 16) S.hist[t] = 0;
  if (t == 16) S.cells = S.iters = S.trials = S.maxit = 0;
}
// One warp's cells: `cell` took part, finished after `iters` iterations (0: not
// finished here), with `trials` line-search trials.
__device__ __forceinline__ void stat_add(NewtonStats& S, bool cell, int iters, unsigned trials) {
  const int bin = iters > 0 ? (iters < 16 ? iters - 1 : 15) : -1;
  const unsigned peers = __match_any_sync(0xffffffffu, bin);
  if (bin >= 0 && (threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&S.hist[bin], __popc(peers));
  const unsigned n = __popc(__ballot_sync(0xffffffffu, cell));
  const unsigned full = __popc(__ballot_sync(0xffffffffu, iters >= NEWTON_MAX_IT));
  const unsigned it = __reduce_add_sync(0xffffffffu, (unsigned)iters);
  const unsigned tr = __reduce_add_sync(0xffffffffu, trials);
  if ((threadIdx.x & 31) == 0) {
    if (n) atomicAdd(&S.cells, (unsigned long long)n);
    if (it) atomicAdd(&S.iters, (unsigned long long)it);
    if (tr) atomicAdd(&S.trials, (unsigned long long)tr);
    if (full) atomicAdd(&S.maxit, (unsigned long long)full);
  }
}
__device__ __forceinline__ void stat_flush(const NewtonStats& S, DevClock* clk, int t) {   // after a barrier
  if (t < 16 && S.hist[t]) atomicAdd(&clk->hist[t], (unsigned long long)S.hist[t]);
  if (t == 16 && S.cells) atomicAdd(&clk->newton_cells, S.cells);
  if (t == 17 && S.iters) atomicAdd(&clk->newton_iters, S.iters);
  if (t == 18 && S.trials) atomicAdd(&clk->lnsrch_trials, S.trials);
  if (t == 19 && S.maxit) atomicAdd(&clk->newton_maxit, S.maxit);
}

template <int NS>
__device__ __forceinline__ bool all_finite(const double* v) {
  bool ok = true;
#pragma unroll
  for (int i = 0; i < 4 + NS; ++i) ok &= isfinite(v[i]);
  return ok;
}

// Newton iterations `it`.. of a cell until it ends (100 at most); returns the
// last iteration's number, `done` whether it converged.
template <int NS, int ST>
IMEX_FLAT int newton_finish(const DevParams& P, int it, bool need_rt, const double* qj_old,
                            const double* Rj, const double* qj_org, double bx, double by, double dt,
                            double* qj_rel, double* rt, double& scal_f, unsigned& trials,
                            bool& stale, bool& done) {
  done = false;
#pragma unroll 1
  for (; it <= NEWTON_MAX_IT; ++it) {
    done = newton_step<NS, ST>(P, it == 1, need_rt, qj_old, Rj, qj_org, bx, by, dt, qj_rel, rt,
                               scal_f, trials, stale);
    need_rt = false;
    if (done) break;
  }
  return it > NEWTON_MAX_IT ? NEWTON_MAX_IT : it;
}

// Fallback of a warm start that failed (no convergence in 100 iterations, or
// a non-finite result): the plain solve_rk_step from q_si.  Returns its
// iteration count; qj receives its result.  Run by k_stage2_fallback only.
template <int NS>
__device__ __forceinline__ int newton_plain(const DevParams& P, const NewtonWork& W, size_t c,
                                         const double* q0, const double* Rj, double bx,
                                         double by, double dt, double* qj,
                                         unsigned long long& trials) {
  constexpr int NV = 4 + NS;
  const size_t N = (size_t)P.plane;
  double qj_org[NV], qj_rel[NV], rt[NV], scal_f;
  bool need_rt, stale = false, done;
  int it = 1;
  unsigned tr = 0;
#pragma unroll
  for (int i = 0; i < NV; ++i) qj[i] = W.qsi[c + i * N];
  if (!newton_begin<NS, 1>(P, qj, q0, Rj, bx, by, dt, qj_org, qj_rel, rt, scal_f, need_rt))
    it = newton_finish<NS, 1>(P, 1, need_rt, q0, Rj, qj_org, bx, by, dt, qj_rel, rt, scal_f, tr,
                              stale, done);
#pragma unroll
  for (int i = 0; i < NV; ++i) qj[i] = qj_rel[i] * qj_org[i];
  trials += tr;
  return it;
}

// Stage 2 before the Newton solve of the cell with old state q0 and stage-1
// tendency Xc: q_fv, the semi-implicit terms, q_si and Rj_not_impl.  False: no
// solve (q_fv(1) <= 0), qsi receives q_fv.
template <int NS>
IMEX_FLAT bool stage2_start(const DevParams& P, const double* q0, const double* Xc, size_t c,
                            const double* __restrict__ Bx, const double* __restrict__ By,
                            const double* __restrict__ Bxx, const double* __restrict__ Bxy,
                            const double* __restrict__ Byy, const double* __restrict__ gc,
                            double dt, double* qsi, double* Rj, double& bx, double& by) {
  constexpr int NV = 4 + NS, NP = 6 + NS;
  double qfv[NV];
  // q_fv = q0 - dt*(MATMUL(divFlux-expl, a_tilde) - MATMUL(NH+SI_NH, a_dirk))
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    double sa = (0.0 + Xc[i] * 1.0) + (0.0 - 0.0) * 0.0;
    double sb = (0.0 + (0.0 + 0.0) * 0.0) + (0.0 + 0.0) * 0.0;
    qfv[i] = q0[i] - dt * (sa - sb);
    qsi[i] = qfv[i];
    Rj[i] = 0.0;
  }
  bx = by = 0.0;
  if (!(qfv[0] > 0.0)) return false;
  double qpv[NP];
  qc_to_qp<NS>(P, qfv, qpv);
  bx = Bx[c];
  by = By[c];
  double bxx = 0.0, bxy = 0.0, byy = 0.0, gcf = 1.0;
  if (P.curvature_term_flag) {
    bxx = Bxx[c];
    bxy = Bxy[c];
    byy = Byy[c];
  }
  if (P.slope_correction_flag) gcf = gc[c];
  double si2, si3;
  semi_impl_terms<NS>(P, bx, by, bxx, bxy, byy, gcf, qpv, si2, si3);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const double SI = (i == 1) ? si2 : ((i == 2) ? si3 : 0.0);
    qsi[i] = qfv[i] + dt * 1.0 * SI;
  }
  if (qfv[1] * qfv[1] + qfv[2] * qfv[2] == 0.0) {
    qsi[1] = 0.0;
    qsi[2] = 0.0;
  } else if (qsi[1] * qfv[1] < 0.0 || qsi[2] * qfv[2] < 0.0) {
    qsi[1] = 0.0;
    qsi[2] = 0.0;
  } else {
    double Sm = sqrt(qsi[1] * qsi[1] + qsi[2] * qsi[2]);
    double Fm = sqrt(qfv[1] * qfv[1] + qfv[2] * qfv[2]);
    qsi[1] = Sm * qfv[1] / Fm;
    qsi[2] = Sm * qfv[2] / Fm;
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    // rows other than 2, 3: qsi = qfv + dt*0 (or +0 for qfv = -0), so
    // for finite qfv and a finite dt > 0 the difference is +0 and so
    // is the quotient
    double SI;
    if (i != 1 && i != 2 && isfinite(qfv[i]) && dt > 0.0 && dt < 1e300) SI = 0.0;
    else SI = (qsi[i] - qfv[i]) / (dt * 1.0);
    double sa = 0.0 + Xc[i] * 1.0;
    double sb = 0.0 + (0.0 + 0.0) * 0.0;
    Rj[i] = (sa - sb) - 1.0 * SI;
  }
  return true;
}

// Sign guard after Newton (src/solver_2d.f90:1238-1255) and assemble_sol
// (src/solver_2d.f90:1339-1626) of one cell: qc the solve's result (newton: it
// went through Newton from q_si's momenta qs1, qs2), written to q.
template <int NS>
IMEX_FLAT void stage2_assemble(const DevParams& P, double* qc, bool newton, double qs1, double qs2,
                               double* __restrict__ q, const uint8_t* __restrict__ cellinfo,
                               DevClock* clk, int j, int k) {
  constexpr int NV = 4 + NS, NP = 6 + NS;
  const int nx = P.nx, ny = P.ny;
  const size_t N = (size_t)P.plane;
  const size_t c = (size_t)k * P.pitch + j;
  if (newton) {
    if (ny == 1) qc[2] = 0.0;
    if (nx == 1) qc[1] = 0.0;
    if (qs1 * qs1 + qs2 * qs2 == 0.0) {
      qc[1] = 0.0;
      qc[2] = 0.0;
    } else if (qc[1] * qs1 <= 0.0 && qc[2] * qs2 <= 0.0) {
      qc[1] = 0.0;
      qc[2] = 0.0;
    } else {
      double Sm = sqrt(qc[1] * qc[1] + qc[2] * qc[2]);
      double Fm = sqrt(qs1 * qs1 + qs2 * qs2);
      qc[1] = Sm * qs1 / Fm;
      qc[2] = Sm * qs2 / Fm;
    }
  }
  const long long cell = (long long)k * nx + j;
  bool anynan = false;
#pragma unroll
  for (int i = 0; i < NV; ++i) anynan |= isnan(qc[i]);
  if (anynan) record_error(clk, 1, cell);
  if (qc[0] < EPS) {
    if (qc[0] > -1.0e-7) {
#pragma unroll
      for (int i = 0; i < NV; ++i) qc[i] = 0.0;
    } else {
      record_error(clk, 2, cell);
    }
  }
  bool anyneg = false, anybad = false;
#pragma unroll
  for (int i = 0; i < NS; ++i) anyneg |= (qc[4 + i] < 0.0);
  if (anyneg) {
#pragma unroll
    for (int i = 0; i < NS; ++i) anybad |= (qc[4 + i] <= -1.0e-7);
    if (anybad) {
      record_error(clk, 3, cell);
    } else {
#pragma unroll
      for (int i = 0; i < NS; ++i)
        if (qc[4 + i] > -1.0e-7) qc[4 + i] = 0.0;
    }
  }
  double qpv[NP];
  qc_to_qp<NS>(P, qc, qpv);
  if (qpv[3] < 273.0) record_error(clk, 4, cell);
  double ssum = 0.0;
#pragma unroll
  for (int i = 0; i < NS; ++i) ssum += qc[4 + i];
  if (ssum > qc[0]) {
    if ((ssum - qc[0]) / qc[0] < 1.0e-10 || qc[0] < EPS) {
      double s = 0.0;
#pragma unroll
      for (int i = 0; i < NS; ++i) s += qc[4 + i];
#pragma unroll
      for (int i = 0; i < NS; ++i) qc[4 + i] = qc[4 + i] / s * qc[0];
    } else {
      record_error(clk, 5, cell);
    }
  }
  if (P.has_cellinfo && (cellinfo[cell] & CI_NODATA)) {
#pragma unroll
    for (int i = 0; i < NV; ++i) qc[i] = 0.0;
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) q[c + i * N] = qc[i];
}

// The vectors that live through a cell's solve, one column per thread.  In
// registers they and the solve's temporaries spilled (at 80 registers 300
// local accesses per cell, whose lines reached DRAM: 588 MB written by the
// former first pass for 237 MB of results).
template <int NS, int T>
struct NewtonShared {
  double q0[4 + NS][T], Rj[4 + NS][T], org[4 + NS][T];
  double qs[2][T];   // q_si's momenta
  NewtonStats st;
};

// Steps that solve at least this many cells, and half of the grid or more, leave
// some cells to the compacted list of k_stage2_rest (LIST): those that the lean
// Jacobian does not cover (the rest's code evicts the others', see k_stage2), and
// a warp's last few iterating lanes.  The line lies between the states that gain
// and those that lose (ms per step with the list / without): a layer of 600^2 cells
// 0.487 / 0.462, 720^2 0.659 / 0.643, 900^2 0.979 / 0.978, 1024^2 1.230 / 1.251,
// 2048^2 4.57 / 4.85; a layer on a slope after 60 steps, 700^2 0.589 / 0.600, 850^2
// 0.797 / 0.852; a dam break of 2048^2 cells, most of them in one iteration, 2.01 /
// 1.75.  Steps that solve less than half of the grid never take it: a radial
// current of 1600^2 cells 0.733 / 0.530, a slope of 2048^2 1.33 / 1.12.
constexpr unsigned long long LIST_MIN_CELLS = 1 << 18;
// On grids of at least this many cells (more than the 512 threads per SM that
// k_stage2 has in flight) the mask pass lists its solve cells, and a step
// that solves less than half of the grid takes stage 2 over that list: blocks
// of solve cells only, in place of grid rows that the current covers in part.
// A block lasts as long as its slowest cell, up to ten iterations, so that
// the number of blocks decides.  Stage 2 of the radial current of 1024^2 cells
// after 1000 steps (84367 solve cells, 2952 of 8192 grid blocks touched): 0.277 ms
// against 0.431 over the grid, after 300 steps (28143) 0.270 against 0.301; a
// slope of 512^2 (45728) 0.116 against 0.132.  The list costs the mask pass
// 0.003 ms on 1024^2 cells.
constexpr unsigned long long DENSE_MIN_GRID = 148 * 512;
// Lanes still iterating at or below which a warp leaves them to the list: going on
// costs the whole warp an iteration, the list about sixty loads and stores per
// cell (2: 2.05 ms, 6: 2.27 ms, 12: 2.29 ms in the first example above).
#ifndef IMEX_REST_LANES
#define IMEX_REST_LANES 2
#endif

// Stage 2 of one lane's cell (j, k) (the lane takes part in the warp's votes and
// list appends whether or not it has a solve cell).  LIST: see LIST_MIN_CELLS; both
// forms in one kernel, chosen per step, spilled twice as much and were slower
// than either (2.11 ms, 0.045 ms against 0.042 on 100x68 cells).
template <int NS, int T, bool LIST>
__device__ __forceinline__ void stage2_lane(
    const DevParams& P, NewtonShared<NS, T>& S, double* __restrict__ q, const double* __restrict__ X,
    const uint8_t* __restrict__ mask, const uint8_t* __restrict__ cellinfo,
    const double* __restrict__ Bx, const double* __restrict__ By, const double* __restrict__ Bxx,
    const double* __restrict__ Bxy, const double* __restrict__ Byy, const double* __restrict__ gc,
    const NewtonWork& W, DevClock* clk, double dt, bool valid, int j, int k) {
  constexpr int NV = 4 + NS, ST = T;
  const size_t N = (size_t)P.plane;
  const size_t c = valid ? (size_t)k * P.pitch + j : 0;
  const bool solve = valid && mask[c];
  if (!__syncthreads_or(solve)) return;
  double* q0 = &S.q0[0][threadIdx.x];
  double* Rj = &S.Rj[0][threadIdx.x];
  double* org = &S.org[0][threadIdx.x];
  double rel[NV], rt[NV], scal_f = 0.0, bx = 0.0, by = 0.0;
  bool newton = false, go = false, need_rt = false, stale = false;
  int it = 0;   // iterations taken
  unsigned trials = 0;
  if (solve) {
    double qsi[NV];
    {
      double qo[NV], Xc[NV], R[NV];
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        qo[i] = q[c + i * N];
        Xc[i] = X[c + i * N];
      }
      newton = stage2_start<NS>(P, qo, Xc, c, Bx, By, Bxx, Bxy, Byy, gc, dt, qsi, R, bx, by);
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        q0[i * ST] = qo[i];
        Rj[i * ST] = R[i];
      }
    }
    if (newton) {
      S.qs[0][threadIdx.x] = qsi[1];
      S.qs[1][threadIdx.x] = qsi[2];
      go = !newton_begin<NS, ST>(P, qsi, q0, Rj, bx, by, dt, org, rel, rt, scal_f, need_rt);
    } else {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        org[i * ST] = 1.0;
        rel[i] = qsi[i];
      }
    }
  }
  bool listed = false;
#pragma unroll 1
  for (int n = 1; n <= NEWTON_MAX_IT; ++n) {   // n: this iteration, the same in all lanes
    // the block's warps go through the iterations together: they then fetch the
    // same instructions at the same time
    if (!__syncthreads_or(go)) break;
    if (LIST && n > 2 && n <= 60 && __popc(__ballot_sync(0xffffffffu, go)) <= IMEX_REST_LANES) {
      listed = listed || go;
      go = false;
    }
    if (go) {
      bool defer = LIST && n <= 60;
      go = !newton_step<NS, ST, !LIST>(P, n == 1, need_rt, q0, Rj, org, bx, by, dt, rel, rt, scal_f,
                                trials, stale, LIST ? &defer : nullptr);
      if (defer) {
        // the list takes it from here (its first residual too, if still to do)
        listed = true;
        go = false;
        stale = stale || need_rt;
      } else {
        it = n;
      }
      need_rt = false;
    }
  }
  stat_add(S.st, newton, newton && !listed ? max(it, 1) : 0, trials);
  if (LIST) {
    list_append(listed, (uint32_t)c, W.list, &clk->nw_count[0]);
    if (listed) {
      // q_si's momenta and, for the other rows, their scaling (all >= 1e-3, so
      // the scaling of these values is itself)
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        W.qsi[c + i * N] = (i == 1 || i == 2) ? S.qs[i - 1][threadIdx.x] : org[i * ST];
        W.Rj[c + i * N] = Rj[i * ST];
        W.x[c + i * N] = rel[i];
        W.rt[c + i * N] = rt[i];
      }
      W.sf[c] = scal_f;
      W.status[c] = (uint8_t)((it << 2) | (stale ? 3 : 1));
    }
  }
  if (solve && !listed) {
    double qc[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) qc[i] = rel[i] * org[i * ST];
    stage2_assemble<NS>(P, qc, newton, newton ? S.qs[0][threadIdx.x] : 0.0,
                        newton ? S.qs[1][threadIdx.x] : 0.0, q, cellinfo, clk, j, k);
  }
}

// Whether stage 2 takes the mask's list: complete (a mask that was not
// listed, or not to its end, has n_listed below solve_cells) and less than half of
// the grid.
__device__ __forceinline__ bool mask_is_sparse_list(const uint32_t* cells, unsigned long long ncell,
                                                    const DevClock* clk) {
  return cells && clk->n_listed == clk->solve_cells && 2 * clk->solve_cells < ncell;
}

// k_stage2's form for the present mask (the same tests in k_stage2<.., true> itself
// cost it 1%: 2.129 against 2.110 ms on 2048^2 cells).  A step takes them along in
// k_dt_clip; either form solves any mask, so that a stale choice costs time only.
__device__ __forceinline__ void stage2_form(const uint32_t* cells, unsigned long long ncell,
                                            DevClock* clk) {
  clk->use_list = !mask_is_sparse_list(cells, ncell, clk) && clk->solve_cells >= LIST_MIN_CELLS;
}
__global__ void k_stage2_form(const uint32_t* cells, unsigned long long ncell, DevClock* clk) {
  stage2_form(cells, ncell, clk);
}

// Stage 2 over the grid rows [k0, k1), or over the mask's list of a sparse step; the
// kernel of the other form returns at once.  Blocks of T threads, 512
// per SM, at 128 registers (84 registers spilled 2 kB per thread and measured 2.58
// against 2.04 ms on 2048^2 cells).
// What bounds it is instruction fetch: the solve's code is larger than the
// instruction cache, and warps at different places in it evict each other's
// (1024^2 cells of the fractal workload, warps on their own: 54% hits, 7 of 15
// stall cycles without an instruction; in step 94%).  So the warps of a block take each
// phase together, and with LIST, where there is work for it, one block of 512
// fills the SM: 2.03 ms on 2048^2 cells against 2.18 ms in blocks of 128.  The other
// steps take blocks of 128, which wait for fewer slow cells: against blocks of
// 512, 0.271 to 0.296 ms on a radial current of 1024^2 cells after 300 steps (but
// 0.282 to 0.274 after 1000), 0.116 to 0.123 on a slope of 512^2, 0.169 to 0.176 on a
// layer of 512^2, 0.0170 to 0.0182 on a dam break of 200^2.  Rolled Jacobian
// columns (2.14 ms), a state machine with one place for residuals (2.34 ms) and 160
// registers less spill (2.01 ms, but 0.060 against 0.043 ms on 99x99) were no better.
// The kernels that this replaces, one pass per Newton iteration over lists in
// memory, took 3.55 ms on those 2048^2 cells, 0.264 ms on that radial current after
// 1000 steps and 0.234 on a 301x517 slope (0.088).
template <int NS, int T, bool LIST>
__global__ void __launch_bounds__(T, 512 / T)
    k_stage2(const __grid_constant__ DevParams Pp, double* __restrict__ q,
             const double* __restrict__ X, const uint8_t* __restrict__ mask,
             const uint8_t* __restrict__ cellinfo, const double* __restrict__ Bx,
             const double* __restrict__ By, const double* __restrict__ Bxx,
             const double* __restrict__ Bxy, const double* __restrict__ Byy,
             const double* __restrict__ gc, const __grid_constant__ NewtonWork W, DevClock* clk,
             int k0, int k1, bool list_form) {
  const DevParams& P = Pp;
  if (list_form && (clk->use_list != 0) != LIST) return;
  const bool dense =
      !LIST && mask_is_sparse_list(W.cells, (unsigned long long)P.nx * P.ny, clk);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  NewtonShared<NS, T>& S = *reinterpret_cast<NewtonShared<NS, T>*>(smem_raw);
  const int nx = P.nx;
  const long long ncell = (long long)nx * (k1 - k0);
  const long long n = dense ? (long long)clk->solve_cells : ncell;
  if ((long long)blockIdx.x * blockDim.x >= n) return;
  const double dt = clk->dt;
  stat_reset(S.st, threadIdx.x);
  __syncthreads();
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long base = (long long)blockIdx.x * blockDim.x; base < n; base += stride) {
    const long long g = base + threadIdx.x;
    int j, k;
    if (dense) {
      const uint32_t c = g < n ? W.cells[g] : 0;
      j = (int)(c % (unsigned)P.pitch);
      k = (int)(c / (unsigned)P.pitch);
    } else {
      j = (int)(g % nx);
      k = k0 + (int)(g / nx);
    }
    stage2_lane<NS, T, LIST>(P, S, q, X, mask, cellinfo, Bx, By, Bxx, Bxy, Byy, gc, W, clk, dt,
                             g < n, j, k);
  }
  __syncthreads();
  stat_flush(S.st, clk, threadIdx.x);
}

// The remaining iterations of entry e of the list (valid: e is inside the
// list), the sign guard and the assembly.
template <int NS>
__device__ __forceinline__ void stage2_rest_lane(const DevParams& P, double* __restrict__ q,
                                                 const uint8_t* __restrict__ cellinfo,
                                                 const double* __restrict__ Bx,
                                                 const double* __restrict__ By,
                                                 const NewtonWork& W, DevClock* clk, double dt,
                                                 bool valid, long long e, NewtonStats& st) {
  constexpr int NV = 4 + NS;
  const size_t N = (size_t)P.plane;
  int fin = 0;
  unsigned tr = 0;
  if (valid) {
    const uint32_t c = W.list[e];
    double q0[NV], Rj[NV], qj_org[NV], qj_rel[NV], rt[NV], qj[NV], scal_f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      q0[i] = q[c + i * N];
      Rj[i] = W.Rj[c + i * N];
      qj[i] = W.qsi[c + i * N];
      qj_rel[i] = W.x[c + i * N];
      rt[i] = W.rt[c + i * N];
    }
    const double qs1 = qj[1], qs2 = qj[2];
    scal_f = W.sf[c];
    const int status = W.status[c];
    bool stale = (status & 2) != 0, done;
    newton_scale<NS>(qj, qj_org);
    fin = newton_finish<NS, 1>(P, (status >> 2) + 1, false, q0, Rj, qj_org, Bx[c], By[c], dt, qj_rel,
                               rt, scal_f, tr, stale, done);
#pragma unroll
    for (int i = 0; i < NV; ++i) qj[i] = qj_rel[i] * qj_org[i];
    stage2_assemble<NS>(P, qj, true, qs1, qs2, q, cellinfo, clk, (int)(c % P.pitch),
                        (int)(c / P.pitch));
  }
  stat_add(st, false, fin, tr);
}

#ifndef IMEX_REST_MINB
#define IMEX_REST_MINB 4
#endif
template <int NS>
__global__ void __launch_bounds__(STAGE2_THREADS, IMEX_REST_MINB)
    k_stage2_rest(const __grid_constant__ DevParams Pp, double* __restrict__ q,
                  const uint8_t* __restrict__ cellinfo, const double* __restrict__ Bx,
                  const double* __restrict__ By, const __grid_constant__ NewtonWork W,
                  DevClock* clk) {
  __shared__ NewtonStats st;
  const long long n = (long long)clk->nw_count[0];
  if ((long long)blockIdx.x * blockDim.x >= n) return;
  stat_reset(st, threadIdx.x);
  __syncthreads();
  const double dt = clk->dt;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long base = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n;
       base += stride) {
    const long long e = base + (threadIdx.x & 31);
    stage2_rest_lane<NS>(Pp, q, cellinfo, Bx, By, W, clk, dt, e < n, e, st);
  }
  __syncthreads();
  stat_flush(st, clk, threadIdx.x);
}

// Stage 2 up to the Newton solve, for the learned start and the harvest: q_si and Rj to
// the NewtonWork planes, the cells to solve to a list (with the learned start the
// one that also holds the network's inputs).
#ifndef IMEX_FIRST_MINB
#define IMEX_FIRST_MINB 6
#endif
template <int NS>
__global__ void __launch_bounds__(STAGE2_THREADS, IMEX_FIRST_MINB)
    k_stage2_first(const __grid_constant__ DevParams Pp, const double* __restrict__ q,
                   const double* __restrict__ X, const uint8_t* __restrict__ mask,
                   const double* __restrict__ Bx, const double* __restrict__ By,
                   const double* __restrict__ Bxx, const double* __restrict__ Bxy,
                   const double* __restrict__ Byy, const double* __restrict__ gc,
                   const __grid_constant__ NewtonWork W, DevClock* clk) {
  const DevParams& P = Pp;
  constexpr int NV = 4 + NS;
  __shared__ NewtonStats st;
  const int nx = P.nx;
  const long long ncell = (long long)nx * P.ny;
  const size_t N = (size_t)P.plane;
  const double dt = clk->dt;
  stat_reset(st, threadIdx.x);
  __syncthreads();
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long base = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < ncell;
       base += stride) {
    const long long g = base + (threadIdx.x & 31);
    const bool valid = g < ncell;
    const size_t c = valid ? (size_t)(g / nx) * P.pitch + (size_t)(g % nx) : 0;
    bool newton = false;
    float fw[WARM_IN];
    if (valid && mask[c]) {
      double q0[NV], Xc[NV], qsi[NV], Rj[NV], bx, by;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        q0[i] = q[c + i * N];
        Xc[i] = X[c + i * N];
      }
      newton = stage2_start<NS>(P, q0, Xc, c, Bx, By, Bxx, Bxy, Byy, gc, dt, qsi, Rj, bx, by);
      W.status[c] = newton ? 1 : 0;
      if (newton) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          W.qsi[c + i * N] = qsi[i];
          W.Rj[c + i * N] = Rj[i];
        }
      }
      if (newton && W.warm) warm_features<NS>(qsi, q0, Rj, dt, bx, by, fw);
      if (!newton) {
#pragma unroll
        for (int i = 0; i < NV; ++i) W.x[c + i * N] = qsi[i];
      }
    }
    stat_add(st, newton, 0, 0);
    if (W.warm) {
      const unsigned int slot = list_append(newton, (uint32_t)c, W.wlist, &clk->nw_count[3]);
      if (newton) {
#pragma unroll
        for (int i = 0; i < WARM_IN; ++i) W.feat[(size_t)slot * WARM_IN + i] = fw[i];
      }
    } else {
      list_append(newton, (uint32_t)c, W.list, &clk->nw_count[0]);
    }
  }
  __syncthreads();
  stat_flush(st, clk, threadIdx.x);
}

// The network's momentum guesses for the cells of the warm-start list:
// 16 cells per warp through the tensor-core forward pass.
template <int NS>
__global__ void __launch_bounds__(32 * mlp::WARPS)
    k_warm_predict(const __grid_constant__ DevParams Pp, NewtonWork W, DevClock* clk,
                   const __nv_bfloat16* __restrict__ gW, const float* __restrict__ gP,
                   WarmNorm nrm) {
  const DevParams& P = Pp;
  const size_t N = (size_t)P.plane;
  extern __shared__ __align__(16) unsigned char smem[];
  __nv_bfloat16* sW = reinterpret_cast<__nv_bfloat16*>(smem);
  float* sP = reinterpret_cast<float*>(smem + mlp::NBW * sizeof(__nv_bfloat16));
  __shared__ float xin[mlp::WARPS][16 * WARM_IN];
  __shared__ float yout[mlp::WARPS][16 * WARM_OUT];
  mlp::load_net(gW, gP, sW, sP);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long n = (long long)clk->nw_count[3];
  for (long long r0 = ((long long)blockIdx.x * mlp::WARPS + warp) * 16; r0 < n;
       r0 += (long long)gridDim.x * mlp::WARPS * 16) {
    const int nv = (int)((n - r0) < 16 ? (n - r0) : 16);
    for (int e = lane; e < 16 * WARM_IN; e += 32) {
      const int r = e / WARM_IN, k = e % WARM_IN;
      xin[warp][e] = r < nv ? (W.feat[(size_t)(r0 + r) * WARM_IN + k] - nrm.x_mean[k]) / nrm.x_std[k]
                            : 0.0f;
    }
    __syncwarp();
    mlp::forward16(xin[warp], nv, sW, sP, yout[warp], WARM_OUT, nullptr);
    __syncwarp();
    if (lane < nv) {
      const uint32_t c = W.wlist[r0 + lane];
      const double m = W.qsi[c];
#pragma unroll
      for (int k = 0; k < WARM_OUT; ++k) {
        const double tk = (double)yout[warp][lane * WARM_OUT + k] * nrm.y_std[k] + nrm.y_mean[k];
        W.guess[c + k * N] = W.qsi[c + (1 + k) * N] + m * tk;
      }
    }
    __syncwarp();
  }
}

// The Newton solves of k_stage2_first's list, from the network's guess or from q_si:
// the iterations of stage2_lane, the block's warps together; results to
// W.x, failed warm starts to the fallback list.  Bound as k_stage2 is; it takes the
// place of iteration 1 in the kernel before and the others lane by lane
// over a list: 0.157 + 0.268 ms on 163 thousand cells of a 1024^2 radial current,
// 0.031 + 0.310 now, 0.261 + 0.392 on a layer of 1024^2 cells, 0.072 + 0.502 now.
template <int NS>
__global__ void __launch_bounds__(STAGE2_THREADS, 512 / STAGE2_THREADS)
    k_stage2_solve(const __grid_constant__ DevParams Pp, const double* __restrict__ q,
                   const double* __restrict__ Bx, const double* __restrict__ By,
                   const __grid_constant__ NewtonWork W, DevClock* clk) {
  const DevParams& P = Pp;
  constexpr int NV = 4 + NS, ST = STAGE2_THREADS;
  __shared__ NewtonShared<NS, ST> S;
  const long long n = (long long)clk->nw_count[W.warm ? 3 : 0];
  if ((long long)blockIdx.x * ST >= n) return;
  const uint32_t* cells = W.warm ? W.wlist : W.list;
  const size_t N = (size_t)P.plane;
  const double dt = clk->dt;
  double* q0 = &S.q0[0][threadIdx.x];
  double* Rj = &S.Rj[0][threadIdx.x];
  double* org = &S.org[0][threadIdx.x];
  stat_reset(S.st, threadIdx.x);
  __syncthreads();
  for (long long base = (long long)blockIdx.x * ST; base < n; base += (long long)gridDim.x * ST) {
    const bool valid = base + threadIdx.x < n;
    const uint32_t c = valid ? cells[base + threadIdx.x] : 0;
    double rel[NV], rt[NV], scal_f = 0.0, bx = 0.0, by = 0.0;
    bool go = false, need_rt = false, stale = false, fb = false;
    int it = 0;
    unsigned trials = 0;
    if (valid) {
      double g[NV];
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        q0[i * ST] = q[c + i * N];
        Rj[i * ST] = W.Rj[c + i * N];
        g[i] = W.qsi[c + i * N];
      }
      if (W.warm) {
        g[1] = W.guess[c];
        g[2] = W.guess[c + N];
      }
      bx = Bx[c];
      by = By[c];
      go = !newton_begin<NS, ST>(P, g, q0, Rj, bx, by, dt, org, rel, rt, scal_f, need_rt);
    }
#pragma unroll 1
    for (int m = 1; m <= NEWTON_MAX_IT; ++m) {
      if (!__syncthreads_or(go)) break;
      if (go) {
        go = !newton_step<NS, ST>(P, m == 1, need_rt, q0, Rj, org, bx, by, dt, rel, rt, scal_f,
                                  trials, stale);
        need_rt = false;
        it = m;
      }
    }
    if (valid) {
      double qj[NV];
#pragma unroll
      for (int i = 0; i < NV; ++i) qj[i] = rel[i] * org[i * ST];
      fb = W.warm && (go || !all_finite<NS>(qj));   // go: not converged in 100 iterations
      if (!fb) {
#pragma unroll
        for (int i = 0; i < NV; ++i) W.x[c + i * N] = qj[i];
      }
    }
    stat_add(S.st, false, valid ? max(it, 1) : 0, trials);
    if (W.warm) list_append(fb, c, W.flist, &clk->nw_fb);
  }
  __syncthreads();
  stat_flush(S.st, clk, threadIdx.x);
}

// Warm starts that failed, redone with the plain start (q_si).
template <int NS>
__global__ void __launch_bounds__(STAGE2_THREADS, IMEX_REST_MINB)
    k_stage2_fallback(const __grid_constant__ DevParams Pp, const double* __restrict__ q,
                      const double* __restrict__ Bx, const double* __restrict__ By,
                      const __grid_constant__ NewtonWork W, DevClock* clk) {
  const DevParams& P = Pp;
  constexpr int NV = 4 + NS;
  const size_t N = (size_t)P.plane;
  const double dt = clk->dt;
  const long long n = (long long)clk->nw_fb;
  unsigned long long it_sum = 0, trials = 0;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x) {
    const uint32_t c = W.flist[e];
    double q0[NV], Rj[NV], qj[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      q0[i] = q[c + i * N];
      Rj[i] = W.Rj[c + i * N];
    }
    it_sum += (unsigned long long)newton_plain<NS>(P, W, c, q0, Rj, Bx[c], By[c], dt, qj, trials);
#pragma unroll
    for (int i = 0; i < NV; ++i) W.x[c + i * N] = qj[i];
    atomicAdd(&clk->warm_fallback, 1ULL);
  }
  if (it_sum) atomicAdd(&clk->newton_iters, it_sum);
  if (trials) atomicAdd(&clk->lnsrch_trials, trials);
}

// Training pairs from the finished Newton solves (before the sign guard):
// the inputs of warm_features and the momentum change per unit q(1), for
// every hstride-th Newton cell (cells taken by a hash of their index and
// the step, so that successive steps sample different cells).  Only cells of the
// present mask: this step has written the planes of no others, where an earlier
// step may have left a solve, or (k_stage2's list) the middle of one.
template <int NS>
__global__ void __launch_bounds__(128)
    k_harvest(const __grid_constant__ DevParams Pp, const double* __restrict__ q,
              const uint8_t* __restrict__ mask, const double* __restrict__ Bx,
              const double* __restrict__ By, NewtonWork W, DevClock* clk) {
  const DevParams& P = Pp;
  constexpr int NV = 4 + NS;
  const int nx = P.nx;
  const long long ncell = (long long)nx * P.ny;
  const size_t N = (size_t)P.plane;
  const double dt = clk->dt;
  const unsigned long long salt = clk->steps * 0x9E3779B97F4A7C15ULL;
  for (long long base = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < ncell;
       base += (long long)gridDim.x * blockDim.x) {
    const long long g = base + (threadIdx.x & 31);
    bool take = false;
    size_t c = 0;
    float f[WARM_IN], y[WARM_OUT];
    if (g < ncell) {
      c = (size_t)(g / nx) * P.pitch + (size_t)(g % nx);
      unsigned long long h = ((unsigned long long)g + salt) * 0xBF58476D1CE4E5B9ULL;
      h ^= h >> 31;
      if (mask[c] && (W.status[c] & 1) && (h % W.hstride) == 0) {
        double q0[NV], qsi[NV], Rj[NV], x1, x2;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          q0[i] = q[c + i * N];
          qsi[i] = W.qsi[c + i * N];
          Rj[i] = W.Rj[c + i * N];
        }
        x1 = W.x[c + N];
        x2 = W.x[c + 2 * N];
        if (qsi[0] > 0.0 && isfinite(x1) && isfinite(x2)) {
          warm_features<NS>(qsi, q0, Rj, dt, Bx[c], By[c], f);
          y[0] = (float)((x1 - qsi[1]) / qsi[0]);
          y[1] = (float)((x2 - qsi[2]) / qsi[0]);
          take = true;
        }
      }
    }
    const unsigned m = __ballot_sync(0xffffffffu, take);
    if (!m) continue;
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    unsigned long long slot0 = 0;
    if (lane == leader) slot0 = atomicAdd(&clk->harvest_n, (unsigned long long)__popc(m));
    slot0 = __shfl_sync(0xffffffffu, slot0, leader);
    const unsigned long long slot = slot0 + __popc(m & ((1u << lane) - 1u));
    if (take && slot < W.hcap) {
#pragma unroll
      for (int i = 0; i < WARM_IN; ++i) W.hx[slot * WARM_IN + i] = f[i];
      W.hy[slot * WARM_OUT + 0] = y[0];
      W.hy[slot * WARM_OUT + 1] = y[1];
    }
  }
}

// Sign guard and assembly from the NewtonWork planes (learned start, harvest).
template <int NS>
__global__ void __launch_bounds__(STAGE2_THREADS)
    k_stage2_post(const __grid_constant__ DevParams Pp, double* __restrict__ q,
                  const uint8_t* __restrict__ mask, const uint8_t* __restrict__ cellinfo,
                  const __grid_constant__ NewtonWork W, DevClock* clk) {
  const DevParams& P = Pp;
  constexpr int NV = 4 + NS;
  const int nx = P.nx;
  const size_t N = (size_t)P.plane;
  const long long ncell = (long long)nx * P.ny;
  for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < ncell;
       g += (long long)gridDim.x * blockDim.x) {
    const int j = (int)(g % nx), k = (int)(g / nx);
    const size_t c = (size_t)k * P.pitch + j;
    if (!mask[c]) continue;
    double qc[NV], qs1 = 0.0, qs2 = 0.0;
#pragma unroll
    for (int i = 0; i < NV; ++i) qc[i] = W.x[c + i * N];
    const bool newton = (W.status[c] & 1) != 0;
    if (newton) {
      qs1 = W.qsi[c + N];
      qs2 = W.qsi[c + 2 * N];
    }
    stage2_assemble<NS>(P, qc, newton, qs1, qs2, q, cellinfo, clk, j, k);
  }
}

// Stand-alone erosion/deposition pass (imex_gpu_erosion_deposition).
template <int NS>
__device__ __forceinline__ void erosion_update_cell(const DevParams& P, double* __restrict__ q,
                                                    const double* __restrict__ Bx,
                                                    const double* __restrict__ By,
                                                    double* __restrict__ erodible,
                                                    double* __restrict__ deposit,
                                                    double* __restrict__ erosion,
                                                    double* __restrict__ Bcent, DevClock* clk,
                                                    double dt, int j, int k) {
  constexpr int NV = 4 + NS;
  const int nx = P.nx;
  const size_t c = (size_t)k * P.pitch + j;
  {
    double qc[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) qc[i] = q[c + (size_t)i * P.plane];
    double er[NS], de[NS], eo[NS], Bc = 0.0;
    const size_t N = (size_t)P.plane;
#pragma unroll
    for (int i = 0; i < NS; ++i) {
      er[i] = erodible[c + i * N];
      de[i] = deposit[c + i * N];
      eo[i] = erosion[c + i * N];
    }
    if (P.topo_change_flag) Bc = Bcent[c];
    bool bad = erosion_cell<NS>(P, qc, Bx[c], By[c], er, de, eo, &Bc, dt);
#pragma unroll
    for (int i = 0; i < NS; ++i) {
      erodible[c + i * N] = er[i];
      deposit[c + i * N] = de[i];
      erosion[c + i * N] = eo[i];
    }
    if (P.topo_change_flag) Bcent[c] = Bc;
    if (bad) record_error(clk, 6, (long long)k * nx + j);
#pragma unroll
    for (int i = 0; i < NV; ++i) q[c + (size_t)i * P.plane] = qc[i];
  }
}

template <int NS>
__global__ void __launch_bounds__(128, IMEX_EROSION_MINB)
    k_erosion(const __grid_constant__ DevParams Pp, double* __restrict__ q, const uint8_t* __restrict__ mask,
              const double* __restrict__ Bx, const double* __restrict__ By,
              double* __restrict__ erodible, double* __restrict__ deposit,
              double* __restrict__ erosion, double* __restrict__ Bcent, DevClock* clk) {
  const DevParams& P = Pp;
  const int nx = P.nx;
  const long long ncell = (long long)nx * P.ny;
  const double dt = clk->dt;
  for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < ncell;
       g += (long long)gridDim.x * blockDim.x) {
    int j = (int)(g % nx), k = (int)(g / nx);
    if (!mask[(size_t)k * P.pitch + j]) continue;
    erosion_update_cell<NS>(P, q, Bx, By, erodible, deposit, erosion, Bcent, clk, dt, j, k);
  }
}

// k_erosion over the grid rows [k0, k1) (imex_gpu_advance_host).
template <int NS>
__global__ void __launch_bounds__(128, IMEX_EROSION_MINB)
    k_erosion_rows(const __grid_constant__ DevParams Pp, double* __restrict__ q,
                   const uint8_t* __restrict__ mask, const double* __restrict__ Bx,
                   const double* __restrict__ By, double* __restrict__ erodible,
                   double* __restrict__ deposit, double* __restrict__ erosion,
                   double* __restrict__ Bcent, DevClock* clk, int k0, int k1) {
  const DevParams& P = Pp;
  const int nx = P.nx;
  const long long ncell = (long long)nx * (k1 - k0);
  const double dt = clk->dt;
  for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < ncell;
       g += (long long)gridDim.x * blockDim.x) {
    const int j = (int)(g % nx), k = k0 + (int)(g / nx);
    if (!mask[(size_t)k * P.pitch + j]) continue;
    erosion_update_cell<NS>(P, q, Bx, By, erodible, deposit, erosion, Bcent, clk, dt, j, k);
  }
}

// ============================================================ small kernels
// FMA-chain throughput probe: each thread runs 8 independent chains of
// `iters` dependent fused multiply-adds (the measured FP64 peak).
__global__ void k_fp64_probe(double* out, int iters, double a, double b) {
  double x0 = threadIdx.x * 1e-9, x1 = x0 + 1.0, x2 = x0 + 2.0, x3 = x0 + 3.0;
  double x4 = x0 + 4.0, x5 = x0 + 5.0, x6 = x0 + 6.0, x7 = x0 + 7.0;
  for (int i = 0; i < iters; ++i) {
    x0 = __fma_rn(x0, a, b); x1 = __fma_rn(x1, a, b); x2 = __fma_rn(x2, a, b); x3 = __fma_rn(x3, a, b);
    x4 = __fma_rn(x4, a, b); x5 = __fma_rn(x5, a, b); x6 = __fma_rn(x6, a, b); x7 = __fma_rn(x7, a, b);
  }
  double r = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
  if (r == 12345.678) out[0] = r;  // keeps the chains live
}

// Resets the per-step accumulators of the clock.  The mask pass lists its
// solve cells (n_listed below half of the grid's ncell) unless the mask before
// was listed and held half of the grid or more: a list that will not be used
// costs it 0.012 of 0.065 ms on 2048^2 cells.  (A new state's all-cells mask is
// not listed and says nothing of the next one.)  ncell 0, where no mask is listed:
// without the two loads, which one thread waits 0.6 us for.
__device__ __forceinline__ void step_begin(DevClock* clk, double max_dt, int reset_cells,
                                           unsigned long long ncell) {
  clk->dtmin_bits = (unsigned long long)__double_as_longlong(max_dt);
  if (reset_cells) {
    clk->n_listed =
        (ncell == 0 || clk->n_listed == 0 || 2 * clk->solve_cells < ncell) ? 0 : 1ULL << 62;
    clk->solve_cells = 0;
  }
  clk->newton_cells = 0;
  clk->newton_iters = 0;
  clk->lnsrch_trials = 0;
  clk->newton_maxit = 0;
  clk->warm_fallback = 0;
  for (int b = 0; b < 16; ++b) clk->hist[b] = 0;
}

__global__ void k_step_begin(DevClock* clk, double max_dt, int reset_cells,
                             unsigned long long ncell) {
  step_begin(clk, max_dt, reset_cells, ncell);
}

// Empties the stage-2 Newton lists (before each stage 2).
__device__ __forceinline__ void nw_reset(DevClock* clk) {
  for (int i = 0; i < 4; ++i) clk->nw_count[i] = 0;
  clk->nw_fb = 0;
}
__global__ void k_nw_reset(DevClock* clk) { nw_reset(clk); }

// dt from the CFL minimum with the driver's clipping (src/IMEX_SfloW2D.f90:359-381).
__device__ __forceinline__ void dt_clip(DevClock* clk, int clip) {
  double dt = __longlong_as_double((long long)clk->dtmin_bits);
  if (clip) {
    double t = clk->t;
    if (t + dt > clk->t_end) dt = clk->t_end - t;
    if (clk->t_output >= 0.0 && t + dt > clk->t_output) dt = clk->t_output - t;
    dt = fmin_f(dt, 1.1 * 0.5 * (clk->dt_old + clk->dt_old_old));
    clk->dt_old_old = clk->dt_old;
    clk->dt_old = dt;
  }
  clk->dt = dt;
}
// With ncell, on grids that can reach LIST_MIN_CELLS, also stage 2's form.
__global__ void k_dt_clip(DevClock* clk, int clip, const uint32_t* cells, unsigned long long ncell) {
  dt_clip(clk, clip);
  if (ncell) stage2_form(cells, ncell, clk);
}

__device__ __forceinline__ void step_end(DevClock* clk) {
  clk->t = clk->t + clk->dt;
  clk->steps += 1;
}
__global__ void k_step_end(DevClock* clk) { step_end(clk); }

// Fortran AoS q(n_vars,nx,ny) <-> SoA planes.
__global__ void k_aos_to_soa(const double* __restrict__ aos, double* __restrict__ soa, int nv,
                             int nx, int ny, long long pitch, long long plane) {
  long long n = (long long)nx * ny;
  for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < n * nv;
       g += (long long)gridDim.x * blockDim.x) {
    long long cell = g / nv;
    int v = (int)(g % nv);
    int j = (int)(cell % nx), k = (int)(cell / nx);
    soa[(size_t)v * plane + (size_t)k * pitch + j] = aos[g];
  }
}
__global__ void k_soa_to_aos(const double* __restrict__ soa, double* __restrict__ aos, int nv,
                             int nx, int ny, long long pitch, long long plane) {
  long long n = (long long)nx * ny;
  for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < n * nv;
       g += (long long)gridDim.x * blockDim.x) {
    long long cell = g / nv;
    int v = (int)(g % nv);
    int j = (int)(cell % nx), k = (int)(cell / nx);
    aos[g] = soa[(size_t)v * plane + (size_t)k * pitch + j];
  }
}

// qp planes for imex_gpu_get_state (driver's post-step convention).
template <int NS>
__global__ void k_qp_out(const __grid_constant__ DevParams Pp, const double* __restrict__ q, double* __restrict__ qp_aos,
                         const uint8_t* __restrict__ cellinfo) {
  const DevParams& P = Pp;
  constexpr int NV = 4 + NS, NP = 6 + NS;
  long long n = (long long)P.nx * P.ny;
  for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < n;
       g += (long long)gridDim.x * blockDim.x) {
    int j = (int)(g % P.nx), k = (int)(g / P.nx);
    size_t c = (size_t)k * P.pitch + j;
    double qc[NV], qpv[NP];
#pragma unroll
    for (int i = 0; i < NV; ++i) qc[i] = q[c + (size_t)i * P.plane];
    cell_qp<NS>(P, qc, qpv);
#pragma unroll
    for (int i = 0; i < NP; ++i) qp_aos[(size_t)g * NP + i] = qpv[i];
  }
}

// ==================================================== topography update
// topography_reconstruction after a bed change (src/geometry_2d.f90:683-860):
// the 5-point first and second derivatives of B_cent and the 25-point mixed
// one on the cells 3..n-2, copied to the 2-cell border; with slope
// correction, grav_coeff, its x derivative and its staggered values.  A cell
// in the border takes the stencil of its nearest interior cell, which is
// what the reference's copies leave there.
__global__ void __launch_bounds__(256)
    k_topo_geom(const __grid_constant__ DevParams Pp, const double* __restrict__ B,
                double* __restrict__ Bx, double* __restrict__ By, double* __restrict__ Bxx,
                double* __restrict__ Bxy, double* __restrict__ Byy) {
  const DevParams& P = Pp;
  const int nx = P.nx, ny = P.ny;
  const long long n = (long long)nx * ny;
  const double c1[5] = {-2.0, -1.0, 0.0, 1.0, 2.0};
  const double c2[5] = {2.0, -1.0, -2.0, -1.0, 2.0};
  const double n1x = 10.0 * P.dx, n1y = 10.0 * P.dy;
  const double n2x = 7.0 * (P.dx * P.dx), n2y = 7.0 * (P.dy * P.dy);
  const double nxy = (10.0 * P.dx) * (10.0 * P.dy);
  for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < n;
       g += (long long)gridDim.x * blockDim.x) {
    const int j = (int)(g % nx), k = (int)(g / nx);
    const int js = min(max(j, 2), nx - 3), ks = min(max(k, 2), ny - 3);
    auto b = [&](int jj, int kk) { return B[(size_t)kk * P.pitch + jj]; };
    double px = 0.0, sxx = 0.0, py = 0.0, syy = 0.0;
#pragma unroll
    for (int t = 0; t < 5; ++t) {
      px = px + c1[t] * b(js + t - 2, ks);
      sxx = sxx + c2[t] * b(js + t - 2, ks);
    }
#pragma unroll
    for (int t = 0; t < 5; ++t) {
      py = py + c1[t] * b(js, ks + t - 2);
      syy = syy + c2[t] * b(js, ks + t - 2);
    }
    double ws = 0.0;
    for (int u = 0; u < 5; ++u)
#pragma unroll
      for (int t = 0; t < 5; ++t) ws = ws + c1[t] * c1[u] * b(js + t - 2, ks + u - 2);
    const size_t c = (size_t)k * P.pitch + j;
    Bx[c] = px / n1x;
    By[c] = py / n1y;
    if (Bxx) {
      Bxx[c] = sxx / n2x;
      Byy[c] = syy / n2y;
      Bxy[c] = ws / nxy;
    }
  }
}

__device__ __forceinline__ double topo_gc(double bx, double by) {
  return 1.0 / (1.0 + bx * bx + by * by);
}

__global__ void __launch_bounds__(256)
    k_topo_gc(const __grid_constant__ DevParams Pp, const double* __restrict__ Bx,
              const double* __restrict__ By, const double* __restrict__ Bxx,
              const double* __restrict__ Bxy, double* __restrict__ gc, double* __restrict__ dgc,
              double* __restrict__ gcsx, double* __restrict__ gcsy) {
  const DevParams& P = Pp;
  const int nx = P.nx, ny = P.ny;
  const long long ncell = (long long)nx * ny, nsx = (long long)(nx + 1) * ny,
                  nsy = (long long)nx * (ny + 1);
  auto gcat = [&](int j, int k) {
    const size_t c = (size_t)k * P.pitch + j;
    return topo_gc(Bx[c], By[c]);
  };
  for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < ncell + nsx + nsy;
       g += (long long)gridDim.x * blockDim.x) {
    if (g < ncell) {
      const int j = (int)(g % nx), k = (int)(g / nx);
      const size_t c = (size_t)k * P.pitch + j;
      const double bx = Bx[c], by = By[c], gcv = topo_gc(bx, by);
      gc[c] = gcv;
      dgc[c] = -(2.0 * (gcv * gcv) * (bx * Bxx[c] + by * Bxy[c]));
    } else if (g < ncell + nsx) {
      const long long h = g - ncell;           // grav_coeff_stag_x(nx+1, ny)
      const int j = (int)(h % (nx + 1)), k = (int)(h / (nx + 1));
      double v;
      if (j == 0) v = gcat(0, k);
      else if (j == nx) v = gcat(nx - 1, k);
      else v = 0.5 * (gcat(j - 1, k) + gcat(j, k));
      gcsx[(size_t)k * (nx + 1) + j] = v;
    } else {
      const long long h = g - ncell - nsx;     // grav_coeff_stag_y(nx, ny+1)
      const int j = (int)(h % nx), k = (int)(h / nx);
      double v;
      if (k == 0) v = gcat(j, 0);
      else if (k == ny) v = gcat(j, ny - 1);
      else v = 0.5 * (gcat(j, k - 1) + gcat(j, k));
      gcsy[(size_t)k * nx + j] = v;
    }
  }
}

// ============================================================= post step
// The driver's output sweep over the solve cells after each step
// (src/IMEX_SfloW2D.f90:391-442) and its first form after the initial
// check_solve (src/IMEX_SfloW2D.f90:253-309): qp(1) kept for the volume
// print, the running maxima hmax / pdynmax / mod_vel_max, and the
// vulnerability table vuln_table(i_table) = OR over steps of
// (h >= thickness_levels(i_thk)) .AND. (p_dyn >= dyn_pres_levels(i_pdyn)),
// i_table running over i_pdyn fastest.
constexpr int POST_MAX_LEVELS = 10;
constexpr int POST_MAX_WORDS = (POST_MAX_LEVELS * POST_MAX_LEVELS + 31) / 32;

struct PostLevels {
  int n_thk, n_pdyn, n_words, pad_;
  double thk[POST_MAX_LEVELS], pdyn[POST_MAX_LEVELS];
};

struct PostPlanes {
  double* qp_h;     // qp(1,:,:) as the sweep leaves it
  double* hmax;
  double* pdynmax;
  double* mvmax;    // mod_vel_max
  uint32_t* vuln;   // n_words planes; table entry i is bit i%32 of plane i/32
};

template <int NS>
__global__ void __launch_bounds__(128)
    k_post_sweep(const __grid_constant__ DevParams Pp, const double* __restrict__ q,
                 const uint8_t* __restrict__ mask, PostPlanes W, PostLevels L, int init) {
  const DevParams& P = Pp;
  constexpr int NV = 4 + NS, NP = 6 + NS;
  const long long ncell = (long long)P.nx * P.ny;
  const size_t N = (size_t)P.plane;
  for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < ncell;
       g += (long long)gridDim.x * blockDim.x) {
    const int j = (int)(g % P.nx), k = (int)(g / P.nx);
    const size_t c = (size_t)k * P.pitch + j;
    if (!mask[c]) continue;
    double qc[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) qc[i] = q[c + i * N];
    if (qc[0] > 0.0) {
      double qpv[NP], pd;
      qc_to_qp<NS>(P, qc, qpv, &pd);
      const double h = qpv[0];
      W.qp_h[c] = h;
      W.hmax[c] = init ? h : fmax_f(W.hmax[c], h);
      const double u = qpv[NV], v = qpv[NV + 1];
      const double mv = sqrt(u * u + v * v);
      if (h > 0.001) {
        W.pdynmax[c] = init ? pd : fmax_f(W.pdynmax[c], pd);
        W.mvmax[c] = init ? mv : fmax_f(W.mvmax[c], mv);
      }
      uint32_t bits[POST_MAX_WORDS] = {0, 0, 0, 0};
      int it = 0;
      for (int a = 0; a < L.n_thk; ++a) {
        const bool thck = h >= L.thk[a];
        for (int b = 0; b < L.n_pdyn; ++b, ++it)
          if (thck && pd >= L.pdyn[b]) bits[it >> 5] |= 1u << (it & 31);
      }
      for (int w = 0; w < L.n_words; ++w) {
        uint32_t* dst = W.vuln + (size_t)w * N + c;
        *dst = init ? bits[w] : (*dst | bits[w]);
      }
    } else {
      W.qp_h[c] = 0.0;
      if (init) {
        W.hmax[c] = 0.0;
        W.pdynmax[c] = 0.0;
      }
    }
  }
}

// The driver's per-step print (src/IMEX_SfloW2D.f90:476-484) before the
// dx*dy factor: SUM(q(1,:,:)), SUM(qp(1,:,:)), COUNT(q(1,:,:) > 1e-7) and
// SUM(q(5:4+n_solid,:,:)).  Per-block partial sums in a fixed order, then
// one block folds them in block order, so the result does not vary from
// run to run.
constexpr int DIAG_THREADS = 256;
template <int NS>
__global__ void __launch_bounds__(DIAG_THREADS)
    k_post_diag(const __grid_constant__ DevParams Pp, const double* __restrict__ q,
                const double* __restrict__ qp_h, double* __restrict__ part) {
  const DevParams& P = Pp;
  const long long ncell = (long long)P.nx * P.ny;
  const size_t N = (size_t)P.plane;
  double a[4] = {0.0, 0.0, 0.0, 0.0};
  for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < ncell;
       g += (long long)gridDim.x * blockDim.x) {
    const int j = (int)(g % P.nx), k = (int)(g / P.nx);
    const size_t c = (size_t)k * P.pitch + j;
    const double h = q[c];
    a[0] += h;
    a[1] += qp_h[c];
    a[2] += (h > 1.0e-7) ? 1.0 : 0.0;
#pragma unroll
    for (int i = 0; i < NS; ++i) a[3] += q[c + (size_t)(4 + i) * N];
  }
  __shared__ double red[4][DIAG_THREADS / 32];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    double x = a[r];
    for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
    if ((threadIdx.x & 31) == 0) red[r][threadIdx.x >> 5] = x;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double x = 0.0;
    for (int w = 0; w < DIAG_THREADS / 32; ++w) x += red[threadIdx.x][w];
    part[(size_t)blockIdx.x * 4 + threadIdx.x] = x;
  }
}

__global__ void k_post_diag_fold(const double* __restrict__ part, int nblocks,
                                 double* __restrict__ out) {
  if (threadIdx.x < 4) {
    double x = 0.0;
    for (int b = 0; b < nblocks; ++b) x += part[(size_t)b * 4 + threadIdx.x];
    out[threadIdx.x] = x;
  }
}

// solve_mask_x / solve_mask_y from solve_mask (src/solver_2d.f90:779-808).
__global__ void k_masks_xy(const __grid_constant__ DevParams Pp, const uint8_t* __restrict__ mask, int8_t* mx,
                           int8_t* my) {
  const DevParams& P = Pp;
  const int nx = P.nx, ny = P.ny;
  long long nX = (long long)(nx + 1) * ny, nY = (long long)nx * (ny + 1);
  for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < nX + nY;
       g += (long long)gridDim.x * blockDim.x) {
    if (g < nX) {
      int j = (int)(g % (nx + 1)), k = (int)(g / (nx + 1));
      bool m = (j > 0 && mask[(size_t)k * P.pitch + j - 1]) || (j < nx && mask[(size_t)k * P.pitch + j]);
      mx[g] = m ? 1 : 0;
    } else {
      long long h = g - nX;
      int j = (int)(h % nx), k = (int)(h / nx);
      bool m = (k > 0 && mask[(size_t)(k - 1) * P.pitch + j]) || (k < ny && mask[(size_t)k * P.pitch + j]);
      my[h] = m ? 1 : 0;
    }
  }
}

}  // namespace IMEX_TU_NS
}  // namespace imex

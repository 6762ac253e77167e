// Damped Boltzmann-electron Picard loop with a geometric-multigrid-preconditioned CG
// linear solver, in one cooperative (persistent) kernel.
//
// Reference: DigitalTwinSimulator.recalc_poisson / _recalc_poisson_cpu
// (Python/physics_engine.py:850-902) solves, each Picard iteration,
//     A V_new = b,  b = V_fixed on Dirichlet rows, -coeff * (rho + rho_e(V)) on free rows,
// with Neumann rows copying the inward neighbour (:556-574), by SuperLU; then
//     V <- (1 - omega) V + omega V_new   (omega = 0.2)
// and finally E = -grad V with np.gradient (:871-884).
//
// Here the Dirichlet and Neumann rows are eliminated, which leaves the SPD operator
//     (4 - n_neumann_nbrs) V_i - sum_{free nbrs} V_j = coeff*rho_total_i + sum_{Dirichlet nbrs} V_fixed_j
// on the free nodes.  It is solved by FP32 MG-PCG inside an FP64 iterative-refinement
// loop (FP64 residual f - A x, FP64 dot products).  The preconditioner is one V(1,1)
// cycle: Galerkin coarse operators (9-point stencils, P bilinear), one damped-Jacobi
// sweep from zero before restriction and one after prolongation, a dense inverse on
// the coarsest level (up to a few thousand nodes, applied by all blocks).  Both smoothing sweeps are fused into the transfers, so every
// level costs one grid-wide phase going down and one going up:
//     down:  r_{l+1} = P^T (r - A w D^-1 r)
//     up:    z = m + w D^-1 (r - A m),   m = w D^-1 r + P z_{l+1}
// With d_i = w / A_ii the diagonal terms reduce to (1 - w) r_i and (1 - w) m_i, so a
// phase reads only the off-diagonal stencil, d and r.  Every load in these phases is
// issued unconditionally (masked by d > 0, the active-node test) so that a thread's
// loads overlap instead of waiting on one another.
//
// Grid-wide phases are separated by a software grid barrier (cooperative launch
// guarantees co-residency).  Every wait is bounded: on time-out the kernel sets
// PB_EF_SPIN_TIMEOUT, stops waiting at later barriers and runs to completion.
// Reductions are deterministic: one partial per block, summed in block order; the
// partials ride on the barrier that the next phase needs anyway.
#include "pb_common.cuh"
#include "pb_poisson.cuh"

namespace pb {

constexpr int FU = 1;  // fine-level nodes per thread and pass of the vector loops (4 measured slower on 257 x 1025)
constexpr float W_KEEP = (float)(1.0 - MG_JACOBI_OMEGA);

// Block index within this instance's group of blocks (a launch may solve several
// instances, each on its own contiguous range of blocks).
__device__ __forceinline__ int gbid(const PoissonArgs& a) { return (int)blockIdx.x - a.blk0; }

// Thread index of the grid-stride loops: 32-node chunks go to the blocks in turn (warp w
// of block b takes chunk w * nblk + b), so a level with fewer nodes than threads still
// spreads over every SM instead of filling the first few.  A permutation of the
// block-major index; each warp still reads 32 consecutive nodes.
__device__ __forceinline__ int gtid(const PoissonArgs& a) {
  return (((int)threadIdx.x >> 5) * a.nblk + gbid(a)) * 32 + ((int)threadIdx.x & 31);
}

// Reductions run over a fixed set of a.nvb virtual blocks (the device's SM count), whatever
// the number of blocks the instance runs on: virtual block v owns the nodes that the
// grid-stride mapping gives block v of an nvb-block launch, its partial is summed in the same
// order by whichever block runs it, and the totals add the nvb partials in a fixed order.  So
// every dot product, and with them the solve, has the same bits on any block count: a batch
// member equals its solo run, and the field-solve block count is a pure speed knob.  Block b
// runs the virtual blocks b, b + nblk, ...; with nblk = nvb the mapping is gtid's.
__device__ __forceinline__ int vtid(const PoissonArgs& a, int v) {
  return (((int)threadIdx.x >> 5) * a.nvb + v) * 32 + ((int)threadIdx.x & 31);
}

// virtual blocks run by this block
__device__ __forceinline__ int vb_count(const PoissonArgs& a) {
  return gbid(a) < a.nvb ? (a.nvb - gbid(a) + a.nblk - 1) / a.nblk : 0;
}

// the virtual-block sums' shared memory, after the coarsest right-hand side
__device__ __forceinline__ double* vb_scratch(const PoissonArgs& a) {
  extern __shared__ float4 dyn_smem[];
  return reinterpret_cast<double*>(dyn_smem + a.vb_off);
}

// the fused phases' shared memory, after the coarsest right-hand side
__device__ __forceinline__ float* fused_smem(const PoissonArgs& a) {
  extern __shared__ float4 dyn_smem[];
  return reinterpret_cast<float*>(dyn_smem + a.vb_off);
}

// grid barrier of this instance's blocks (grid_sync: bounded, release/acquire)
__device__ __forceinline__ void grid_barrier(const PoissonArgs& a) { grid_sync(a.bar, a.errflags, a.nblk, gbid(a)); }

// phase tracing (block 0, thread 0): time since the previous mark is added to trace[k]
__device__ __forceinline__ void tmark(const PoissonArgs& a, int k) {
  if (a.trace && gbid(a) == 0 && threadIdx.x == 0) {
    unsigned long long now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    unsigned long long last = a.trace[31];
    if (last) a.trace[k] += now - last;
    a.trace[31] = now;
  }
}

// ----------------------------------------------------------------- deterministic sums
__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
  return v;
}

// Partials of the virtual blocks a block runs: after the loop of its k-th virtual block each
// warp adds its two sums to shared memory (vb_add, no block barrier); vb_flush then sums each
// virtual block's 32 warp sums in warp order (the tree of one warp_sum) and writes them to
// ring slot `slot` (read after the next barrier).  vbs holds 2 x 32 doubles per virtual
// block of the block (PoissonArgs::vb_off).
__device__ __forceinline__ void vb_add(double* vbs, int k, double v0, double v1) {
  v0 = warp_sum(v0);
  v1 = warp_sum(v1);
  if ((threadIdx.x & 31) == 0) {
    double* w = vbs + (size_t)(k * 32 + (threadIdx.x >> 5)) * 2;
    w[0] = v0;
    w[1] = v1;
  }
}

__device__ __forceinline__ void vb_flush(const PoissonArgs& a, double* vbs, int slot, int nk) {
  __syncthreads();
  const int lane = threadIdx.x & 31;
  double* part = a.partials + (size_t)(slot & 3) * 2 * a.nvb;
  for (int k = (int)(threadIdx.x >> 5); k < nk; k += (int)(blockDim.x >> 5)) {
    double s0 = vbs[(size_t)(k * 32 + lane) * 2], s1 = vbs[(size_t)(k * 32 + lane) * 2 + 1];
    s0 = warp_sum(s0);
    s1 = warp_sum(s1);
    if (lane == 0) {
      const int v = gbid(a) + k * a.nblk;
      part[v] = s0;
      part[a.nvb + v] = s1;
    }
  }
  __syncthreads();  // vbs is reused by the next reduction
}

// Grid totals of a slot, after a barrier; the same order in every block.
__device__ __forceinline__ void get_sums(const PoissonArgs& a, int slot, double& t0, double& t1) {
  __shared__ double bc[2];
  if (threadIdx.x < 32) {
    const double* part = a.partials + (size_t)(slot & 3) * 2 * a.nvb;
    double s0 = 0.0, s1 = 0.0;
    // all of a lane's loads issued before the first add (one L2 round trip for up to 256
    // virtual blocks); the adds keep the order v = lane, lane + 32, ...
    for (int base = 0; base < a.nvb; base += 256) {
      double v0[8], v1[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int b = base + q * 32 + (int)threadIdx.x;
        v0[q] = b < a.nvb ? __ldcg(part + b) : 0.0;
        v1[q] = b < a.nvb ? __ldcg(part + a.nvb + b) : 0.0;
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        s0 += v0[q];
        s1 += v1[q];
      }
    }
    s0 = warp_sum(s0);
    s1 = warp_sum(s1);
    if (threadIdx.x == 0) { bc[0] = s0; bc[1] = s1; }
  }
  __syncthreads();
  t0 = bc[0];
  t1 = bc[1];
  __syncthreads();
}

// ----------------------------------------------------------------- level-0 (5-point) operator
// neighbours W, E, S, N of node i = (y, x); -1 outside the grid
__device__ __forceinline__ void nbrs0(const PoissonArgs& a, int i, int y, int x, int j[4]) {
  j[0] = x > 0 ? i - 1 : -1;
  j[1] = x < a.nx - 1 ? i + 1 : -1;
  int ys = y - 1, yn = y + 1;
  if (a.periodic) { if (ys < 0) ys += a.ny; if (yn >= a.ny) yn -= a.ny; }
  j[2] = ys >= 0 ? ys * a.nx + x : -1;
  j[3] = yn < a.ny ? yn * a.nx + x : -1;
}

// (A v)_i at a free node, v arbitrary on non-free nodes (masked); all loads issued up front
template <class T>
__device__ __forceinline__ T apply0(const PoissonArgs& a, const T* v, int i, int y, int x) {
  int j[4];
  nbrs0(a, i, y, x, j);
  uint8_t c[4];
  T vj[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int jj = j[k] >= 0 ? j[k] : i;
    c[k] = j[k] >= 0 ? __ldg(a.cls + jj) : (uint8_t)NC_NEU;
    vj[k] = *(v + jj);
  }
  const T vi = *(v + i);
  T s = (T)0;
  int nneu = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    s += c[k] == NC_FREE ? vj[k] : (T)0;
    nneu += c[k] == NC_NEU;
  }
  return (T)(4 - nneu) * vi - s;
}

// ----------------------------------------------------------------- transfer phases
// Restricted residual at coarse node (I, J) of level 1, from the fine level F (5-point
// operator, off-diagonals -1 to every neighbour; d r is zero on non-free nodes):
//   sum_children w_f * [f active] * ((1 - w) r_f + sum_{k nbr of f} d_k r_k).
// r is the fine residual; each patch node is loaded once.  wrapC: the coarse level's
// prolongation wraps in y.
__device__ __forceinline__ float restrict0(const MgLevel& F, const float* r, int I, int J, bool wrapC) {
  const int ny = F.ny, nx = F.nx;
  int ro[5];
  bool rv[5];
#pragma unroll
  for (int t = 0; t < 5; ++t) {
    int y = 2 * I + t - 2;
    if (F.per) { if (y < 0) y += ny; else if (y >= ny) y -= ny; }
    rv[t] = y >= 0 && y < ny;
    ro[t] = y * nx;
  }
  int xo[5];
  bool cv[5];
#pragma unroll
  for (int u = 0; u < 5; ++u) {
    xo[u] = 2 * J + u - 2;
    cv[u] = xo[u] >= 0 && xo[u] < nx;
  }
  float zp[5][5], rq[5][5], dq[5][5];
#pragma unroll
  for (int t = 0; t < 5; ++t)
#pragma unroll
    for (int u = 0; u < 5; ++u) {
      if ((t == 0 || t == 4) && (u == 0 || u == 4)) { zp[t][u] = rq[t][u] = dq[t][u] = 0.0f; continue; }
      const bool ok = rv[t] && cv[u];
      const int j = ok ? ro[t] + xo[u] : 0;
      const float d = __ldg(F.dinv + j), rj = *(r + j);
      dq[t][u] = d;
      rq[t][u] = rj;
      zp[t][u] = ok ? d * rj : 0.0f;
    }
  float s = 0.0f;
#pragma unroll
  for (int da = -1; da <= 1; ++da) {
    const int t = da + 2;
    const int yf = 2 * I + da;
    const bool rowok = rv[t] && (da < 0 ? (yf >= 0 || wrapC) : (yf < ny));
#pragma unroll
    for (int db = -1; db <= 1; ++db) {
      const int u = db + 2;
      const bool ok = rowok && cv[u];
      const float res = W_KEEP * rq[t][u] + ((zp[t][u - 1] + zp[t][u + 1]) + (zp[t - 1][u] + zp[t + 1][u]));
      const float w = (da ? 0.5f : 1.0f) * (db ? 0.5f : 1.0f);
      s += (ok && dq[t][u] > 0.0f) ? w * res : 0.0f;
    }
  }
  return s;
}

// (P z_c) at fine node (y, x) of the level above C
__device__ __forceinline__ float prolong(const MgLevel& C, const float* zc, int y, int x) {
  const int I0 = y >> 1, J0 = x >> 1, ay = y & 1, bx = x & 1;
  int I1 = I0 + 1;
  bool m10 = ay != 0;
  if (I1 >= C.ny) { if (C.wrapP) I1 -= C.ny; else m10 = false; }
  const int J1 = J0 + 1;
  const bool m01 = bx != 0 && J1 < C.nx;
  const int i00 = I0 * C.nx + J0;
  const int i01 = m01 ? I0 * C.nx + J1 : i00;
  const int i10 = m10 ? I1 * C.nx + J0 : i00;
  const int i11 = (m10 && m01) ? I1 * C.nx + J1 : i00;
  const float z00 = *(zc + i00), z01 = *(zc + i01), z10 = *(zc + i10), z11 = *(zc + i11);
  const float w = (ay ? 0.5f : 1.0f) * (bx ? 0.5f : 1.0f);
  return w * (z00 + (m01 ? z01 : 0.0f) + (m10 ? z10 : 0.0f) + ((m10 && m01) ? z11 : 0.0f));
}

// Post-smoothed correction on the fine level F (5-point operator, off-diagonals -1) from
// z_c of level 1, tile by tile:
//   z_i = (1 - w) m_i + d_i (r_i + sum_{k nbr of i} m_k),  m = [active] (d r + P z_c).
// The block forms m once per node of its tile and a one-node halo in shared memory (a node's
// m is used by the five stars that contain it), then z from the tile.  The tiles are
// a.ut_y x a.ut_x nearly equal rectangles, dealt to the blocks in turn; each holds at most
// UP_TILE_MAX nodes with its halo.  up_tile0 does tile t and returns this thread's part of
// (r, z) over the tile's nodes when nu0 = 1.
__device__ double up_tile0(const PoissonArgs& a, const float* r0, int t, bool two) {
  __shared__ float mt[UP_TILE_MAX];
  float* out = two ? a.m32 : a.lev[0].z;
  const MgLevel& F = a.lev[0];
  const MgLevel& C = a.lev[1];
  const int ny = F.ny, nx = F.nx, nty = a.ut_y, ntx = a.ut_x;
  double rz = 0.0;
  {
    const int ty = t / ntx, tx = t - ty * ntx;
    const int y0 = (int)((long long)ty * ny / nty), y1 = (int)((long long)(ty + 1) * ny / nty);
    const int x0 = (int)((long long)tx * nx / ntx), x1 = (int)((long long)(tx + 1) * nx / ntx);
    const int h = y1 - y0, w = x1 - x0, w2 = w + 2, nm = (h + 2) * w2;
    for (int k = threadIdx.x; k < nm; k += blockDim.x) {
      const int ly = k / w2, lx = k - ly * w2;
      int yy = y0 + ly - 1;
      const int xx = x0 + lx - 1;
      if (F.per) { if (yy < 0) yy += ny; else if (yy >= ny) yy -= ny; }
      const bool ok = yy >= 0 && yy < ny && xx >= 0 && xx < nx;
      const int j = ok ? yy * nx + xx : 0;
      const float d = __ldg(F.dinv + j), rj = *(r0 + j);
      const float sj = two ? *(a.s32 + j) : 0.0f;
      const float pz = prolong(C, C.z, ok ? yy : 0, ok ? xx : 0);
      mt[k] = (ok && d > 0.0f) ? d * (rj + sj) + pz : 0.0f;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < h * w; k += blockDim.x) {
      const int ly = k / w, lx = k - ly * w;
      const int i = (y0 + ly) * nx + (x0 + lx);
      const float di = __ldg(F.dinv + i), ri = *(r0 + i);
      const float* mc = mt + (ly + 1) * w2 + (lx + 1);
      const float acc = ri + ((mc[-1] + mc[1]) + (mc[-w2] + mc[w2]));
      const float z = di > 0.0f ? W_KEEP * mc[0] + di * acc : 0.0f;
      __stcg(out + i, z);
      if (!two) rz += (double)ri * (double)z;
    }
    __syncthreads();
  }
  return rz;
}

// With nu0 = 2 the pre-smoothed correction is d (r + s), s = r - A d r (a.s32), and this leg
// writes the once post-smoothed m2 to a.m32; smooth0 applies the second post-sweep and the
// partial of (r, z).  With nu0 = 1 this leg leaves that partial in `slot`: the tiles are then
// laid out for nvb blocks and tile t belongs to virtual block t mod nvb.
__device__ void up_leg0_tiled(const PoissonArgs& a, const float* r0, int slot) {
  const bool two = a.nu0 == 2;
  double* vbs = vb_scratch(a);
  if (two) {
    for (int t = gbid(a); t < a.ut_y * a.ut_x; t += a.nblk) up_tile0(a, r0, t, true);
    return;
  }
  for (int v = gbid(a), kv = 0; v < a.nvb; v += a.nblk, ++kv) {
    double rz = 0.0;
    for (int t = v; t < a.ut_y * a.ut_x; t += a.nvb) rz += up_tile0(a, r0, t, false);
    vb_add(vbs, kv, rz, 0.0);
  }
  vb_flush(a, vbs, slot, vb_count(a));
}

// Second fine-level pre-sweep (nu0 = 2): s = r - A (d r) on the free nodes, i.e.
// s_i = (1 - w) r_i + sum_{k nbr of i} d_k r_k (d is zero off the free nodes).
__device__ void presmooth0(const PoissonArgs& a, const float* r, float* s_out, int tid, int nth) {
  const MgLevel& F = a.lev[0];
  const int N = F.ny * F.nx;
  for (int i0 = tid; i0 < N; i0 += FU * nth) {
    float sv[FU];
#pragma unroll
    for (int u = 0; u < FU; ++u) {
      const int i = i0 + u * nth < N ? i0 + u * nth : i0;
      const int y = i / F.nx, x = i - y * F.nx;
      int j[4];
      nbrs0(a, i, y, x, j);
      const float di = __ldg(F.dinv + i), ri = *(r + i);
      float acc = 0.0f;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int jj = j[k] >= 0 ? j[k] : i;
        const float dk = j[k] >= 0 ? __ldg(F.dinv + jj) : 0.0f;
        acc += dk * *(r + jj);
      }
      sv[u] = di > 0.0f ? W_KEEP * ri + acc : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < FU; ++u)
      if (i0 + u * nth < N) __stcg(s_out + i0 + u * nth, sv[u]);
  }
}

// Second fine-level post-sweep (nu0 = 2): z = m + d (r - A m) = (1 - w) m + d (r + sum_nbr m)
// from m = a.m32 (zero off the active nodes); leaves the partials of (r, z) in `slot`.
__device__ void smooth0(const PoissonArgs& a, const float* r, int slot) {
  const MgLevel& F = a.lev[0];
  const int N = F.ny * F.nx, nth = a.nvb * (int)blockDim.x;
  double* vbs = vb_scratch(a);
  for (int v = gbid(a), kv = 0; v < a.nvb; v += a.nblk, ++kv) {
  double rz = 0.0;
  for (int i0 = vtid(a, v); i0 < N; i0 += FU * nth) {
    float zv[FU], rv[FU];
#pragma unroll
    for (int u = 0; u < FU; ++u) {
      const int i = i0 + u * nth < N ? i0 + u * nth : i0;
      const int y = i / F.nx, x = i - y * F.nx;
      int j[4];
      nbrs0(a, i, y, x, j);
      const float di = __ldg(F.dinv + i), ri = *(r + i), mi = *(a.m32 + i);
      float sm = 0.0f;
#pragma unroll
      for (int k = 0; k < 4; ++k) sm += j[k] >= 0 ? *(a.m32 + j[k]) : 0.0f;
      zv[u] = di > 0.0f ? W_KEEP * mi + di * (ri + sm) : 0.0f;
      rv[u] = ri;
    }
#pragma unroll
    for (int u = 0; u < FU; ++u) {
      if (i0 + u * nth >= N) continue;
      __stcg(F.z + i0 + u * nth, zv[u]);
      rz += (double)rv[u] * (double)zv[u];
    }
  }
  vb_add(vbs, kv, rz, 0.0);
  }
  vb_flush(a, vbs, slot, vb_count(a));
}

// Levels >= 1: the same transfers from the host-built stencils (R on the coarse level,
// U on the fine level); out-of-grid patch entries have zero weight.
__device__ __forceinline__ float restrict_pre(const MgLevel& F, const MgLevel& C, const float* r, int I, int J,
                                              int ic) {
  const int ny = F.ny, nx = F.nx, Nc = C.ny * C.nx;
  float s = 0.0f;
#pragma unroll
  for (int t = 0; t < 5; ++t) {
    int y = 2 * I + t - 2;
    if (F.per) { if (y < 0) y += ny; else if (y >= ny) y -= ny; }
    const bool rv = y >= 0 && y < ny;
#pragma unroll
    for (int u = 0; u < 5; ++u) {
      const int x = 2 * J + u - 2;
      const bool ok = rv && x >= 0 && x < nx;
      const float w = __ldg(C.R + (size_t)(t * 5 + u) * Nc + ic);
      const float v = *(r + (ok ? y * nx + x : 0));
      s += ok ? w * v : 0.0f;
    }
  }
  return s;
}

__device__ __forceinline__ float smooth_up_pre(const MgLevel& F, const MgLevel& C, const float* r, const float* zc,
                                               int y, int x, int i) {
  const int ny = F.ny, nx = F.nx, Nf = ny * nx;
  const int I0 = y >> 1, J0 = x >> 1;
  float s = 0.0f;
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    int yy = y + t - 1;
    if (F.per) { if (yy < 0) yy += ny; else if (yy >= ny) yy -= ny; }
    const bool rv = yy >= 0 && yy < ny;
    int cy = I0 + t - 1;
    if (C.per) { if (cy < 0) cy += C.ny; else if (cy >= C.ny) cy -= C.ny; }
    const bool cvr = cy >= 0 && cy < C.ny;
#pragma unroll
    for (int u = 0; u < 3; ++u) {
      const int xx = x + u - 1;
      const bool ok = rv && xx >= 0 && xx < nx;
      const float wr = __ldg(F.U + (size_t)(t * 3 + u) * Nf + i);
      const float vr = *(r + (ok ? yy * nx + xx : i));
      s += ok ? wr * vr : 0.0f;
      const int cx = J0 + u - 1;
      const bool okc = cvr && cx >= 0 && cx < C.nx;
      const float wz = __ldg(F.U + (size_t)(9 + t * 3 + u) * Nf + i);
      const float vz = *(zc + (okc ? cy * C.nx + cx : 0));
      s += okc ? wz * vz : 0.0f;
    }
  }
  return s;
}

// restrict_pre and smooth_up_pre where the grid is not periodic: entries outside the grid have
// weight zero, so their values are read at the nearest node instead of being masked (a third
// of the instructions: 1.3 us of a leg's 3).  w, stride: the node's stencil.
__device__ __forceinline__ float restrict_leg(const MgLevel& F, const float* r, int I, int J, const float* w,
                                              size_t stride) {
  const int ny = F.ny, nx = F.nx, x0 = 2 * J;
  int xo[5];
#pragma unroll
  for (int u = 0; u < 5; ++u) xo[u] = min(max(x0 + u - 2, 0), nx - 1);
  float v[25];
#pragma unroll
  for (int t = 0; t < 5; ++t) {
    const float* const row = r + min(max(2 * I + t - 2, 0), ny - 1) * nx;
#pragma unroll
    for (int u = 0; u < 5; ++u) v[t * 5 + u] = __fmul_rn(*(w + (t * 5 + u) * stride), *(row + xo[u]));
  }
  float s = 0.0f;
#pragma unroll
  for (int k = 0; k < 25; ++k) s = __fadd_rn(s, v[k]);
  return s;
}

__device__ __forceinline__ float smooth_leg(const MgLevel& F, const MgLevel& C, const float* r, const float* zc, int y,
                                            int x, const float* w, size_t stride) {
  const int fy = F.ny, fx = F.nx, cy = C.ny, cx = C.nx, Y = y >> 1, X = x >> 1;
  const int xm = max(x - 1, 0), xp = min(x + 1, fx - 1), Xm = max(X - 1, 0), Xp = min(X + 1, cx - 1);
  float v[18];
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const float* const row = r + min(max(y + t - 1, 0), fy - 1) * fx;
    const float* const crow = zc + min(max(Y + t - 1, 0), cy - 1) * cx;
    const float* const q = w + t * 3 * stride;
    v[6 * t] = __fmul_rn(*q, *(row + xm));
    v[6 * t + 1] = __fmul_rn(*(q + 9 * stride), *(crow + Xm));
    v[6 * t + 2] = __fmul_rn(*(q + stride), *(row + x));
    v[6 * t + 3] = __fmul_rn(*(q + 10 * stride), *(crow + X));
    v[6 * t + 4] = __fmul_rn(*(q + 2 * stride), *(row + xp));
    v[6 * t + 5] = __fmul_rn(*(q + 11 * stride), *(crow + Xp));
  }
  float s = 0.0f;
#pragma unroll
  for (int k = 0; k < 18; ++k) s = __fadd_rn(s, v[k]);
  return s;
}

// grid-wide down leg: r_{l+1} from level l (all from global memory)
template <bool LV0>
__device__ void down_leg(const PoissonArgs& a, int level, int tid, int nth, const float* src0 = nullptr) {
  const MgLevel& F = a.lev[level];
  const MgLevel& C = a.lev[level + 1];
  const int Nc = C.ny * C.nx;
  for (int ic = tid; ic < Nc; ic += nth) {
    const int I = ic / C.nx, J = ic - I * C.nx;
    if (LV0) {
      // level 0 restricts (1 - w) v + sum_nbr d v of v = r (one pre-sweep) or v = s (two)
      const float s = restrict0(F, src0 ? src0 : F.r, I, J, C.wrapP != 0);
      __stcg(C.r + ic, __ldg(C.dinv + ic) > 0.0f ? s : 0.0f);
    } else {
      __stcg(C.r + ic, a.periodic ? restrict_pre(F, C, F.r, I, J, ic)
                                  : restrict_leg(F, F.r, I, J, C.R + ic, (size_t)Nc));
    }
  }
}

// grid-wide up leg of level l >= 1: z_l from r_l and z_{l+1}
__device__ void up_leg(const PoissonArgs& a, int level, int tid, int nth) {
  const MgLevel& F = a.lev[level];
  const MgLevel& C = a.lev[level + 1];
  const int N = F.ny * F.nx;
  for (int i = tid; i < N; i += nth) {
    const int y = i / F.nx, x = i - y * F.nx;
    __stcg(F.z + i, a.periodic ? smooth_up_pre(F, C, F.r, C.z, y, x, i)
                               : smooth_leg(F, C, F.r, C.z, y, x, F.U + i, (size_t)N));
  }
}

// ----------------------------------------------------------------- coarsest level
// z_c = A_c^{-1} r_c on the coarsest level, by every block of the instance: each block
// gathers r_c of the active nodes into shared memory, then one warp per row (rows dealt
// to the blocks in turn) takes the dot product with that row of the dense inverse.
// Inactive nodes of z_c are never written (zero since allocation).
__device__ void coarse_solve(const PoissonArgs& a, const float* rlev, float* zlev, float* rcs) {
  const int nc = __ldg(a.nc_dev);
  for (int k = threadIdx.x; k < nc; k += blockDim.x) rcs[k] = *(rlev + __ldg(a.cidx + k));
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int nw = a.nblk * (int)(blockDim.x >> 5);
  for (int k = (int)(threadIdx.x >> 5) * a.nblk + gbid(a); k < nc; k += nw) {
    const float* row = a.cinv + (size_t)k * nc;
    float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;
    int j = lane;
    for (; j + 96 < nc; j += 128) {
      s0 += __ldg(row + j) * rcs[j];
      s1 += __ldg(row + j + 32) * rcs[j + 32];
      s2 += __ldg(row + j + 64) * rcs[j + 64];
      s3 += __ldg(row + j + 96) * rcs[j + 96];
    }
    for (; j < nc; j += 32) s0 += __ldg(row + j) * rcs[j];
    float s = (s0 + s1) + (s2 + s3);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
    if (lane == 0) __stcg(zlev + __ldg(a.cidx + k), s);
  }
}

// z32 = M^{-1} r0 by one V(1,1) cycle, after the phase that restricted r0 to level 1
// (down_leg<true>):
// the down legs from level 1, the coarse solve, the up legs and the fine-level up leg.
// Leaves the partial of (r0, z) in `slot` and ends with a barrier.
__device__ void vcycle_below(const PoissonArgs& a, float* rcs, int slot, const float* r0) {
  const int tid = gtid(a), nth = a.nblk * blockDim.x;
  const int last = a.nlevels - 1;
  if (last == 0) {
    coarse_solve(a, r0, a.z32, rcs);
    grid_barrier(a);
    const int N = a.ny * a.nx, nv = a.nvb * (int)blockDim.x;
    double* vbs = vb_scratch(a);
    for (int v = gbid(a), kv = 0; v < a.nvb; v += a.nblk, ++kv) {
      double rz = 0.0;
      for (int i = vtid(a, v); i < N; i += nv) rz += (double)(*(r0 + i)) * (double)(*(a.z32 + i));
      vb_add(vbs, kv, rz, 0.0);
    }
    vb_flush(a, vbs, slot, vb_count(a));
    grid_barrier(a);
    return;
  }
  for (int l = 1; l < last; ++l) {
    down_leg<false>(a, l, tid, nth);
    grid_barrier(a);
    tmark(a, l < 7 ? l : 6);
  }
  coarse_solve(a, a.lev[last].r, a.lev[last].z, rcs);
  grid_barrier(a);
  tmark(a, 7);
  for (int l = last - 1; l >= 1; --l) {
    up_leg(a, l, tid, nth);
    grid_barrier(a);
    tmark(a, 8 + (l < 7 ? l : 6));
  }
  up_leg0_tiled(a, r0, slot);  // nu0 = 1: the partials of (r, z)
  if (a.nu0 == 2) {
    grid_barrier(a);
    smooth0(a, r0, slot);
  }
  grid_barrier(a);
  tmark(a, 8);
}

// E = -grad V and the solve's statistics
__device__ __forceinline__ void solve_end(const PoissonArgs& a, int tid, int nth, double n_outer, double n_inner,
                                          double last_rel, unsigned long long t_start) {
  const int N = a.ny * a.nx;
  // ---- E = -grad V (np.gradient: central inside, one-sided at the edges; periodic y fix)
  if (a.compute_field) {
    for (int i = tid; i < N; i += nth) {
      int y = i / a.nx, x = i - y * a.nx;
      const double* V = a.V;
      double ex, ey;
      if (x == 0) ex = DDIV(DSUB(-(*(V + i + 1)), -(*(V + i))), a.hx);
      else if (x == a.nx - 1) ex = DDIV(DSUB(-(*(V + i)), -(*(V + i - 1))), a.hx);
      else ex = DDIV(DSUB(-(*(V + i + 1)), -(*(V + i - 1))), a.two_hx);
      if (a.periodic && y == 0) ey = DDIV(DSUB((*(V + (size_t)(a.ny - 1) * a.nx + x)), (*(V + a.nx + x))), a.two_hy_per);
      else if (a.periodic && y == a.ny - 1) ey = DDIV(DSUB((*(V + (size_t)(a.ny - 2) * a.nx + x)), (*(V + x))), a.two_hy_per);
      else if (y == 0) ey = DDIV(DSUB(-(*(V + i + a.nx)), -(*(V + i))), a.hy);
      else if (y == a.ny - 1) ey = DDIV(DSUB(-(*(V + i)), -(*(V + i - a.nx))), a.hy);
      else ey = DDIV(DSUB(-(*(V + i + a.nx)), -(*(V + i - a.nx))), a.two_hy);
      a.Ex[i] = __double2float_rn(ex);
      a.Ey[i] = __double2float_rn(ey);
    }
  }
  tmark(a, 19);
  if (tid == 0) {
    a.stats[0] += n_outer;
    a.stats[1] += n_inner;
    a.stats[2] = last_rel;
    a.stats[3] += (double)a.iterations;
  }
  if (gbid(a) == 0 && threadIdx.x == 0) {
    unsigned long long t_end;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_end));
    a.solve_ns[0] += (t_end - t_start) * (unsigned long long)a.nblk;  // block-ns
    a.solve_ns[1] += 1;
  }
}

// V_new of node i from the solution, then the damped Picard update
__device__ __forceinline__ double picard_update(const PoissonArgs& a, int i) {
  const uint8_t c = __ldg(a.cls + i);
  double vn;
  if (c == NC_FREE) vn = (*(a.x + i));
  else if (c == NC_DIR) vn = __ldg(a.Vfixed + i);
  else {
    int y = i / a.nx, x = i - y * a.nx;
    int sy = y, sx = x;
    if (x == a.nx - 1) {
      sx = x - 1;  // right: copy (y, nx-2), which may itself be a top/bottom copy
      uint8_t cs = __ldg(a.cls + sy * a.nx + sx);
      if (cs == NC_NEU && !a.periodic) sy = (sy == 0) ? 1 : (sy == a.ny - 1 ? a.ny - 2 : sy);
    } else if (y == 0) sy = 1;
    else sy = a.ny - 2;
    int j = sy * a.nx + sx;
    uint8_t cj = __ldg(a.cls + j);
    vn = (cj == NC_DIR) ? __ldg(a.Vfixed + j) : (*(a.x + j));
  }
  if (c != NC_FREE) __stcg(a.x + i, vn);
  const double V = DADD(DMUL(a.omega_keep, (*(a.V + i))), DMUL(a.omega_new, vn));
  __stcg(a.V + i, V);
  return V;
}

// ----------------------------------------------------------------- the persistent kernel
__device__ __forceinline__ void poisson_body(const PoissonArgs& a) {
  extern __shared__ float4 dyn_smem[];
  float* rcs = reinterpret_cast<float*>(dyn_smem);  // nc floats: the coarsest r, gathered
  double* vbs = vb_scratch(a);
  const int tid = gtid(a), nth = a.nblk * blockDim.x;
  const int nv = a.nvb * (int)blockDim.x;  // stride of a virtual block's nodes (reduction loops)
  const int N = a.ny * a.nx;
  int slot = 0;
  double n_outer = 0, n_inner = 0, last_rel = 0;
  unsigned long long t_start = 0;
  if (gbid(a) == 0 && threadIdx.x == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_start));
  tmark(a, 20);

  // Dirichlet-neighbour sums (V_fixed is constant during the launch), with the mapping of
  // the right-hand-side loop that reads them: each thread reads only what it wrote, so no
  // barrier is needed between the two
  for (int v = gbid(a); v < a.nvb; v += a.nblk)
    for (int i = vtid(a, v); i < N; i += nv) {
      if (__ldg(a.cls + i) != NC_FREE) continue;
      const int y = i / a.nx, x = i - y * a.nx;
      int j[4];
      nbrs0(a, i, y, x, j);
      double s = 0.0;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (j[k] >= 0 && __ldg(a.cls + j[k]) == NC_DIR) s += __ldg(a.Vfixed + j[k]);
      a.dirsum[i] = s;
    }

  for (int pic = 0; pic < a.iterations; ++pic) {
    const double inner_at_pic = n_inner, outer_at_pic = n_outer;
    // right-hand side from the Boltzmann electron density of the current V, residual
    for (int v = gbid(a), kv = 0; v < a.nvb; v += a.nblk, ++kv) {
      const int t0 = vtid(a, v);
      double ff = 0.0, rr = 0.0;
      for (int i = t0; i < N; i += nv) {
        if (__ldg(a.cls + i) != NC_FREE) continue;
        double Vi = (*(a.V + i));
        double vm = Vi < a.V_plasma ? Vi : a.V_plasma;
        double rho_e = DMUL(a.qn0_neg, exp(DDIV(DSUB(vm, a.V_plasma), a.Te_up)));
        double rt = DADD((double)__ldg(a.rho + i), rho_e);
        double fi = DMUL(a.coeff, rt) + a.dirsum[i];
        __stcg(a.f + i, fi);
        ff += fi * fi;
      }
      for (int i = t0; i < N; i += nv) {
        if (__ldg(a.cls + i) != NC_FREE) { __stcg(a.r32 + i, 0.0f); continue; }
        const int y = i / a.nx, x = i - y * a.nx;
        double res = (*(a.f + i)) - apply0<double>(a, a.x, i, y, x);
        __stcg(a.r32 + i, (float)res);
        rr += res * res;
      }
      vb_add(vbs, kv, ff, rr);
    }
    vb_flush(a, vbs, slot, vb_count(a));
    grid_barrier(a);
    double fnorm2, rnorm2;
    get_sums(a, slot++, fnorm2, rnorm2);
    tmark(a, 17);
    const double target2 = a.tol * a.tol * fnorm2;

    for (int outer = 0; outer < a.max_outer && rnorm2 > target2 && fnorm2 > 0.0; ++outer) {
      n_outer += 1;
      // ---- FP32 MG-PCG on A e = r32 (e32 starts at zero; r32 is the current residual)
      for (int i = tid; i < N; i += nth) __stcg(a.e32 + i, 0.0f);
      double rz_old = 0.0, rr0 = rnorm2, dummy;
      for (int k = 0; k < a.max_inner; ++k) {
        n_inner += 1;
        // z32 = M r32: fine-level restriction (after a second pre-sweep when nu0 = 2),
        // then the rest of the V-cycle
        if (a.nlevels > 1 && a.nu0 == 2) {
          presmooth0(a, a.r32, a.s32, tid, nth);
          grid_barrier(a);
        }
        if (a.nlevels > 1) down_leg<true>(a, 0, tid, nth, a.nu0 == 2 ? a.s32 : nullptr);
        grid_barrier(a);
        tmark(a, 0);
        vcycle_below(a, rcs, slot, a.r32);  // (r, z) partial in slot, barrier
        double rz;
        get_sums(a, slot++, rz, dummy);
        const double beta = k == 0 ? 0.0 : rz / rz_old;
        // FU nodes per thread and pass: every load of the pass is issued before the first
        // store, so the loads of different nodes overlap (the sums keep the node order)
        for (int v = gbid(a), kv = 0; v < a.nvb; v += a.nblk, ++kv) {
          double pq_p = 0.0;
          for (int i0 = vtid(a, v); i0 < N; i0 += FU * nv) {
            float pv[FU], qv[FU];
#pragma unroll
            for (int u = 0; u < FU; ++u) {
              const int i = i0 + u * nv < N ? i0 + u * nv : i0;
              const int y = i / a.nx, x = i - y * a.nx;
              const bool fr = __ldg(a.cls + i) == NC_FREE;
              const float az = apply0<float>(a, a.z32, i, y, x);
              const float zi = *(a.z32 + i);
              pv[u] = fr ? zi + (float)beta * (k == 0 ? 0.0f : (*(a.p32 + i))) : 0.0f;
              qv[u] = fr ? az + (float)beta * (k == 0 ? 0.0f : (*(a.q32 + i))) : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < FU; ++u) {
              if (i0 + u * nv >= N) continue;
              __stcg(a.p32 + i0 + u * nv, pv[u]);
              __stcg(a.q32 + i0 + u * nv, qv[u]);
              pq_p += (double)pv[u] * (double)qv[u];
            }
          }
          vb_add(vbs, kv, pq_p, 0.0);
        }
        vb_flush(a, vbs, slot, vb_count(a));
        grid_barrier(a);
        double pq;
        get_sums(a, slot++, pq, dummy);
        const double alpha = pq != 0.0 ? rz / pq : 0.0;
        for (int v = gbid(a), kv = 0; v < a.nvb; v += a.nblk, ++kv) {
          double rr_p = 0.0;
          for (int i0 = vtid(a, v); i0 < N; i0 += FU * nv) {
            float ev[FU], rv[FU];
            bool fr[FU];
#pragma unroll
            for (int u = 0; u < FU; ++u) {
              const int i = i0 + u * nv < N ? i0 + u * nv : i0;
              fr[u] = i0 + u * nv < N && __ldg(a.cls + i) == NC_FREE;
              ev[u] = (*(a.e32 + i)) + (float)alpha * (*(a.p32 + i));
              rv[u] = (*(a.r32 + i)) - (float)alpha * (*(a.q32 + i));
            }
#pragma unroll
            for (int u = 0; u < FU; ++u) {
              if (!fr[u]) continue;
              __stcg(a.e32 + i0 + u * nv, ev[u]);
              __stcg(a.r32 + i0 + u * nv, rv[u]);
              rr_p += (double)rv[u] * (double)rv[u];
            }
          }
          vb_add(vbs, kv, rr_p, 0.0);
        }
        vb_flush(a, vbs, slot, vb_count(a));
        grid_barrier(a);
        double rrk;
        get_sums(a, slot++, rrk, dummy);
        tmark(a, 15);
        rz_old = rz;
        // stop at the pass's reduction tol_inner (default 1e-3) or at the FP64 target
        // itself: the FP32 recurrence drifts from the true residual by ~1e-7 of the start,
        // and the FP64 residual after the correction decides whether another pass runs.
        // Stopping 10x below the target instead cost 24% more iterations and saved no
        // pass; a 1e-5 cap per pass cost 6% more solve time than 1e-3.
        if (rrk <= a.tol_inner * a.tol_inner * rr0 || rrk <= target2) break;
      }
      // ---- FP64 correction and true residual
      for (int i = tid; i < N; i += nth)
        if (__ldg(a.cls + i) == NC_FREE) __stcg(a.x + i, (*(a.x + i)) + (double)(*(a.e32 + i)));
      grid_barrier(a);
      for (int v = gbid(a), kv = 0; v < a.nvb; v += a.nblk, ++kv) {
        double rr = 0.0;
        for (int i = vtid(a, v); i < N; i += nv) {
          if (__ldg(a.cls + i) != NC_FREE) { __stcg(a.r32 + i, 0.0f); continue; }
          const int y = i / a.nx, x = i - y * a.nx;
          double res = (*(a.f + i)) - apply0<double>(a, a.x, i, y, x);
          __stcg(a.r32 + i, (float)res);
          rr += res * res;
        }
        vb_add(vbs, kv, rr, 0.0);
      }
      vb_flush(a, vbs, slot, vb_count(a));
      grid_barrier(a);
      get_sums(a, slot++, rnorm2, dummy);
      tmark(a, 16);
    }
    if (!(rnorm2 <= target2) && fnorm2 > 0.0 && tid == 0) atomicOr(a.errflags, PB_EF_POISSON_NOCONV);
    if (a.trace && tid == 0 && pic < 5) {
      a.trace[21 + pic] += (unsigned long long)(n_inner - inner_at_pic);
      a.trace[26 + pic] += (unsigned long long)(n_outer - outer_at_pic);
    }
    last_rel = fnorm2 > 0.0 ? sqrt(rnorm2 / fnorm2) : 0.0;

    // ---- V_new on every node, then the damped Picard update
    for (int i = tid; i < N; i += nth) picard_update(a, i);
    grid_barrier(a);
    tmark(a, 18);
  }

  solve_end(a, tid, nth, n_outer, n_inner, last_rel, t_start);
}

// ----------------------------------------------------------------- fewer, longer phases
// The body of a solve whose phases are short (PoissonArgs::fused, fused_plan).  There a phase's
// own arithmetic is nothing; it costs a grid barrier (1.4 us), a trip to L2 for every
// dependent load and the index arithmetic before it.  So
//   - neighbouring phases are joined, their halos computed more than once from shared memory:
//     the residual update with the restrictions to levels 1 and 2 (four phases of
//     poisson_body), both fine post-sweeps with (r, z) (two), the Picard update with the next
//     right-hand side (two);
//   - what does not change during a launch (the nodes of the patches, their smoother weights,
//     transfer stencils, the block's rows of the coarse inverse) is laid out in shared memory
//     at its start: after a barrier the L1 holds none of it;
//   - a thread keeps its own nodes' z, p, q, r and e in registers, and loads that need no
//     total are issued before it.
// Each value is the same expression of the same operands as in poisson_body, with the same
// roundings (written out, so that contraction cannot differ), and each sum has its order: the
// warps of the virtual blocks are dealt to all blocks, and every block adds the 32 warp sums
// of a virtual block, then the virtual blocks, as vb_flush and get_sums do.  So the solve has
// the same bits on either path.
// A call of 5 Picard iterations, before (poisson_body) and now: 65 x 284 nodes 895 -> 582 us (235
// barriers -> 125 in 25 CG iterations), 81 x 321 640 -> 424, 129 x 568 1200 -> 893, 257 x 1025
// 672 -> 608, 257 x 1135 1560 -> 1347.  Of the 18 us that a CG iteration on 65 x 284 now takes, 6
// are its four barriers and 2.5 the three totals.
// RUNS: the fine post-sweeps run on the block's own nodes (their owners in the sums) with halos
// of two rows, five rows of m to one of nodes, so that (r, z) is summed in the same phase; else
// they run on the block's tile, with a barrier before the sum.  Runs win while they are short:
// 65 x 284 582 us against 601 on tiles, 85 x 374 800 against 819; 129 x 568 (runs of 256 nodes)
// 942 against 895.
// part: this virtual warp's place among the 32 nvb of a value
__device__ __forceinline__ void vw_put(const PoissonArgs& a, int slot, int which, int part, double v) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) a.wpart[(size_t)((slot & 3) * 2 + which) * 32 * a.nvb + part] = v;
}

// The totals of one value of a slot, or of both, in two parts: the loads, then the sums (other
// loads of a phase are issued in between).
template <int NV, int NVB>
struct VwTotal {
  static constexpr int NB = (NVB + PT / 32 - 1) / (PT / 32);
  double v[NV][NB];
  __device__ __forceinline__ VwTotal(const PoissonArgs& a, int slot) {
    const double* part = a.wpart + (size_t)(slot & 3) * 2 * 32 * a.nvb;
#pragma unroll
    for (int q = 0; q < NV; ++q)
#pragma unroll
      for (int e = 0; e < NB; ++e) {
        const int b = ((int)threadIdx.x >> 5) + e * (PT / 32);
        v[q][e] = b < a.nvb ? __ldcg(part + (q * a.nvb + b) * 32 + ((int)threadIdx.x & 31)) : 0.0;
      }
  }
  __device__ __forceinline__ void sums(const PoissonArgs& a, double (&t)[NV]) {
    __shared__ double vb_sum[NV][NVB];
    const int lane = (int)threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < NV; ++q)
#pragma unroll
      for (int e = 0; e < NB; ++e) {
        const int b = ((int)threadIdx.x >> 5) + e * (PT / 32);
        if (b >= a.nvb) break;
        const double s = warp_sum(v[q][e]);
        if (lane == 0) vb_sum[q][b] = s;
      }
    __syncthreads();  // the next total is at least one grid barrier away
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      double s = 0.0;
      for (int b = lane; b < a.nvb; b += 32) s += vb_sum[q][b];
      t[q] = __shfl_sync(0xFFFFFFFFu, warp_sum(s), 0);
    }
  }
  __device__ __forceinline__ double sum(const PoissonArgs& a) {
    double t[1];
    sums(a, t);
    return t[0];
  }
};

// Shared-memory layout of a block, and its sizes: one tile of level 2 with the patches of
// levels 1 and 0 under it, the up leg's two runs of nodes with two rows and columns around
// them, the coarser levels' nodes, rows of the coarse inverse.
struct FusedBlock {
  int h, w, W, np, W1, n1, hw;      // level-2 tile, patch of level 0 (row length, nodes) and level 1
  int *dj, *l1c, *l1i, *l2i, *l2b;  // node of level 0 (-1 outside; bit 30: the tile's own), of level 1
  float *dd, *rp, *sp, *r1, *rw;    // smoother weight, residual, s; level 1; stencils of level 2
  int w0, w1, n0, n;                // run patches: row lengths, nodes of the first and of both
  int *uj, *uf;                     // node; place in z1 << 9, segment << 7 and flags
  int zw[4];                        // row length of each segment's part of z1
  float *ud, *mt, *rt, *m2;
  float* z1;                        // level 1's correction on the coarse patches of the runs
  int *zn, nz;                      // their nodes (y << 16 | x)
  float* zu;                        // and their stencils
  int *zj, n2, W2;                  // level 2 under the tile's corrections: node (-1 outside)
  float* z2;
  float* crow;
  int crows;
};
// A level as its two legs between levels 2 and last read it: a copy in shared memory, and this
// block's nodes (y << 16 | x, -1 past the level's last chunk) in gtid's order
struct FusedLevel {
  MgLevel L;
  int* yx;
  int share;
};
enum : int { UF_Y = 1, UF_X = 2, UF_M01 = 4, UF_M10 = 8, UF_W = 16, UF_E = 32, UF_RING = 64, UF_M = 128 };
constexpr int DJ_OWN = 1 << 30;

// nodes of a level that a block takes in gtid's order, rounded up to whole chunks
__device__ __forceinline__ int level_share(const PoissonArgs& a, int l) {
  return 32 * (((a.lev[l].ny * a.lev[l].nx + 31) / 32 + a.nblk - 1) / a.nblk);
}

// FILL: the tables' contents too; else the layout only.
template <bool RUNS, bool FILL>
__device__ __forceinline__ void fused_tables(const PoissonArgs& a, int c0, int c1, FusedBlock& B, FusedLevel* lv) {
  const int tid = (int)threadIdx.x, N = a.ny * a.nx, nx = a.nx, last = a.nlevels - 1;
  const MgLevel &L1 = a.lev[1], &L2 = a.lev[2];
  int I0 = 0, J0 = 0;
  B.h = B.w = 0;
  if (gbid(a) < a.dt_y * a.dt_x) {
    const int ty = gbid(a) / a.dt_x, tx = gbid(a) - ty * a.dt_x;
    I0 = ty * L2.ny / a.dt_y;
    J0 = tx * L2.nx / a.dt_x;
    B.h = (ty + 1) * L2.ny / a.dt_y - I0;
    B.w = (tx + 1) * L2.nx / a.dt_x - J0;
  }
  B.hw = B.h * B.w;
  constexpr int halo = RUNS ? FUSED_HALO : FUSED_HALO_TILE, halo1 = RUNS ? 3 : 5;
  const int H = 4 * B.h + halo;
  B.W = 4 * B.w + halo;
  B.W1 = 2 * B.w + halo1;
  B.np = B.hw ? H * B.W : 0;
  B.n1 = B.hw ? (2 * B.h + halo1) * B.W1 : 0;
  const int nv = a.nvb * PT, b0 = 32 * c0, b1 = nv + 32 * c0;
  const int l0 = max(0, min(N, 32 * c1) - b0), l1 = max(0, min(N, nv + 32 * c1) - b1);
  B.w0 = l0 + 4;
  B.w1 = l1 + 4;
  B.n0 = l0 ? 5 * B.w0 : 0;
  B.n = RUNS ? B.n0 + (l1 ? 5 * B.w1 : 0) : 0;
  float* f = fused_smem(a);
  auto take = [&](int n) { float* const q = f; f += n; return q; };
  auto takei = [&](int n) { return reinterpret_cast<int*>(take(n)); };
  B.dj = takei(B.np); B.dd = take(B.np); B.rp = take(B.np); B.sp = take(B.np);
  B.l1c = takei(B.n1); B.l1i = takei(B.n1); B.r1 = take(B.n1);
  B.l2i = takei(B.hw); B.l2b = takei(B.hw); B.rw = take(25 * B.hw);
  B.uj = takei(B.n); B.uf = takei(B.n); B.ud = take(B.n);
  B.mt = take(RUNS ? B.n : B.np);
  B.rt = take(B.n);
  B.m2 = RUNS ? take(B.n) : B.sp;  // s is not read any more when the first post-sweep is written
  for (int l = 2; l <= last; ++l) {
    const int sh = level_share(a, l), Nl = a.lev[l].ny * a.lev[l].nx, lx = a.lev[l].nx;
    int* const t = takei(sh);
    for (int q = tid; FILL && q < sh; q += PT) {
      const int i = ((q >> 5) * a.nblk + gbid(a)) * 32 + (q & 31), y = i / lx;
      t[q] = i < Nl ? (y << 16) | (i - y * lx) : -1;
    }
    if (FILL && tid == 0) {
      lv[l].L = a.lev[l];
      lv[l].yx = t;
      lv[l].share = sh;
    }
  }
  if (FILL && tid == 0) lv[1].L = a.lev[1];
  // Level 1 under the runs: a run is one or two row segments (it may cross a row's end, and is no
  // longer than a row); the patch of a segment is the coarse nodes that its two rows and columns
  // on every side interpolate from.  seg: first run column, fine row, coarse origin, size, place
  int seg_u[4], seg_c0[4], seg_w[4], seg_at[4], nz = 0;
  B.zn = reinterpret_cast<int*>(f);
  if (!RUNS && B.hw) {
    // the coarse nodes that the tile and two rows and columns around it interpolate from, each as
    // its places in the patches of level 1 (the right-hand side) and level 2 (the correction)
    const int Ya = max(0, 2 * I0 - 1), Yb = min(L1.ny - 1, 2 * (I0 + B.h) + 1);
    const int Xa = max(0, 2 * J0 - 1), Xb = min(L1.nx - 1, 2 * (J0 + B.w) + 1), sw = Xb - Xa + 1;
    B.W2 = B.w + 4;
    B.n2 = (B.h + 4) * B.W2;
    nz = (Yb - Ya + 1) * sw;
    seg_c0[0] = Ya << 16 | Xa;
    seg_w[0] = sw;
    for (int k = tid; FILL && k < nz; k += PT) {
      const int y = Ya + k / sw, x = Xa + k % sw;
      B.zn[k] = ((y - 2 * I0 + 2) * B.W1 + x - 2 * J0 + 2) << 16 | (((y >> 1) - I0 + 2) * B.W2 + (x >> 1) - J0 + 2);
    }
  }
#pragma unroll
  for (int q = 0; q < (RUNS ? 4 : 0); ++q) {
    const int o = q >> 1, l = o ? l1 : l0, b = o ? b1 : b0;
    const int y = b / nx + (q & 1), x0 = b - (b / nx) * nx, first = nx - x0;  // columns of the run in its first row
    const int ua = q & 1 ? first : 0, ub = q & 1 ? l : min(l, first);
    seg_u[q] = ua;
    seg_at[q] = nz;
    seg_c0[q] = seg_w[q] = 0;
    if (ub <= ua) continue;
    const int xa = max(0, (q & 1 ? 0 : x0) - 2), xb = min(nx - 1, (q & 1 ? 0 : x0) + (ub - ua) - 1 + 2);
    const int Ya = max(0, y - 2) >> 1, Yb = min(L1.ny - 1, (min(a.ny - 1, y + 2) >> 1) + 1);
    const int Xa = xa >> 1, Xb = min(L1.nx - 1, (xb >> 1) + 1);
    const int sw = Xb - Xa + 1, cnt = (Yb - Ya + 1) * sw;
    seg_c0[q] = Ya << 16 | Xa;
    seg_w[q] = sw;
    for (int k = tid; FILL && k < cnt; k += PT) B.zn[nz + k] = (Ya + k / sw) << 16 | (Xa + k % sw);
    nz += cnt;
  }
  B.nz = nz;
#pragma unroll
  for (int q = 0; q < 4; ++q) B.zw[q] = RUNS || q == 0 ? seg_w[q] : 0;
  takei(nz);
  B.z1 = take(nz);
  B.zu = take(18 * nz);
  if (!RUNS) {
    if (!B.hw) B.n2 = B.W2 = 0;
    B.zj = takei(B.n2);
    B.z2 = take(B.n2);
    B.uf = takei(B.np);
    for (int k = tid; FILL && k < B.n2; k += PT) {
      const int y = I0 - 2 + k / B.W2, x = J0 - 2 + k % B.W2;
      B.zj[k] = (unsigned)y < (unsigned)L2.ny && (unsigned)x < (unsigned)L2.nx ? y * L2.nx + x : -1;
    }
  }
  B.crow = f;
  const int nc = __ldg(a.nc_dev), lane = tid & 31;
  B.crows = min((int)((size_t)a.croom / max(nc, 1)), (nc + a.nblk - 1) / a.nblk);
  if (!FILL) return;
  __syncthreads();
  for (int k = tid; k < nz; k += PT) {
    const int i = RUNS ? (B.zn[k] >> 16) * L1.nx + (B.zn[k] & 0xFFFF)
                       : ((seg_c0[0] >> 16) + k / seg_w[0]) * L1.nx + (seg_c0[0] & 0xFFFF) + k % seg_w[0];
#pragma unroll 6
    for (int e = 0; e < 18; ++e) B.zu[e * nz + k] = __ldg(L1.U + (size_t)e * (L1.ny * L1.nx) + i);
  }
  // level-0 patch of the tile: node (4 I0 - 7, 4 J0 - 7) first
  for (int k = tid; k < B.np; k += PT) {
    const int ly = k / B.W, lx = k - ly * B.W, y = 4 * I0 - 7 + ly, x = 4 * J0 - 7 + lx;
    const bool in = (unsigned)y < (unsigned)a.ny && (unsigned)x < (unsigned)nx;
    const bool own = in && ly >= 7 && ly < 7 + 4 * B.h && lx >= 7 && lx < 7 + 4 * B.w;
    B.dj[k] = in ? (y * nx + x) | (own ? DJ_OWN : 0) : -1;
    B.dd[k] = in ? __ldg(a.lev[0].dinv + y * nx + x) : 0.0f;
    if (!RUNS) {
      const int py = ly - 7, px = lx - 7, Y = y >> 1, X = x >> 1;  // distance from the tile
      int uf = 0;
      if (in && py >= -2 && py < 4 * B.h + 2 && px >= -2 && px < 4 * B.w + 2)
        uf = ((Y - (seg_c0[0] >> 16)) * seg_w[0] + X - (seg_c0[0] & 0xFFFF)) << 9 | UF_M | (y & 1 ? UF_Y : 0) |
             (x & 1 ? UF_X : 0) | ((x & 1) && X + 1 < L1.nx ? UF_M01 : 0) | ((y & 1) && Y + 1 < L1.ny ? UF_M10 : 0) |
             (py >= -1 && py < 4 * B.h + 1 && px >= -1 && px < 4 * B.w + 1 ? UF_RING : 0);
      B.uf[k] = uf;
    }
  }
  // level-1 patch: node (2 I0 - 2, 2 J0 - 2) first; its place in the level-0 patch
  for (int k = tid; k < B.n1; k += PT) {
    const int ly = k / B.W1, lx = k - ly * B.W1, I = 2 * I0 - 2 + ly, J = 2 * J0 - 2 + lx;
    const bool in = (unsigned)I < (unsigned)L1.ny && (unsigned)J < (unsigned)L1.nx;
    const bool act = in && __ldg(L1.dinv + I * L1.nx + J) > 0.0f;
    const bool own = in && ly >= 2 && ly < 2 + 2 * B.h && lx >= 2 && lx < 2 + 2 * B.w;
    B.l1c[k] = act ? (2 * ly + 3) * B.W + 2 * lx + 3 : -1;
    B.l1i[k] = own ? I * L1.nx + J : -1;
  }
  for (int k = tid; k < B.hw; k += PT) {
    const int ly = k / B.w, lx = k - ly * B.w, ic = (I0 + ly) * L2.nx + J0 + lx;
    B.l2i[k] = ic;
    B.l2b[k] = 2 * ly * B.W1 + 2 * lx;
#pragma unroll 5
    for (int e = 0; e < 25; ++e) B.rw[e * B.hw + k] = __ldg(L2.R + (size_t)e * (L2.ny * L2.nx) + ic);
  }
  for (int k = tid; k < B.n; k += PT) {
    const bool o = k >= B.n0;
    const int q = o ? k - B.n0 : k, w = o ? B.w1 : B.w0, ly = q / w, lx = q - ly * w;
    const int j = (o ? b1 : b0) + (ly - 2) * nx + lx - 2;
    int uj = -1, uf = 0;
    float d = 0.0f;
    // a column before the first segment's row or after the second's lies in another row, and
    // nothing reads it
    const int g = 2 * o + (lx - 2 >= seg_u[2 * o + 1] && seg_w[2 * o + 1] > 0);
    const int x0 = (o ? b1 : b0) - ((o ? b1 : b0) / nx) * nx, xx = g & 1 ? lx - 2 - seg_u[g] : x0 + lx - 2;
    if (j >= 0 && j < N && xx >= 0 && xx < nx) {
      const int y = j / nx, x = j - y * nx, Y = y >> 1, X = x >> 1;
      uj = j;
      d = __ldg(a.lev[0].dinv + j);
      uf = (seg_at[g] + (Y - (seg_c0[g] >> 16)) * seg_w[g] + X - (seg_c0[g] & 0xFFFF)) << 9 | (g << 7) | (y & 1 ? UF_Y : 0) | (x & 1 ? UF_X : 0) | ((x & 1) && X + 1 < L1.nx ? UF_M01 : 0) |
           ((y & 1) && Y + 1 < L1.ny ? UF_M10 : 0) | (x > 0 ? UF_W : 0) | (x < nx - 1 ? UF_E : 0) |
           (ly >= 1 && ly <= 3 && lx >= 1 && lx <= w - 2 ? UF_RING : 0);
    }
    B.uj[k] = uj;
    B.uf[k] = uf;
    B.ud[k] = d;
  }
  for (int t = tid >> 5; t < B.crows; t += PT / 32) {
    const int k = t * a.nblk + gbid(a);
    if (k >= nc) break;
    for (int j = lane; j < nc; j += 32) B.crow[(size_t)t * nc + j] = __ldg(a.cinv + (size_t)k * nc + j);
  }
}

// The rest of the restriction from the residual in rp: s = r - A D r, level 1, level 2.
template <bool RUNS>
__device__ __forceinline__ void down_tile(const PoissonArgs& a, const FusedBlock& B) {
  const int tid = (int)threadIdx.x, W = B.W;
  const float *const dp = B.dd, *const rp = B.rp;
  float* const sp = B.sp;
  __syncthreads();
  // the patch's outermost ring gets no s (nothing reads it)
  for (int i = tid + W + 1; i < B.np - W - 1; i += PT) {
    const float d = dp[i];
    float acc = fmaf(dp[i - 1], rp[i - 1], 0.0f);
    acc = fmaf(dp[i + 1], rp[i + 1], acc);
    acc = fmaf(dp[i - W], rp[i - W], acc);
    acc = fmaf(dp[i + W], rp[i + W], acc);
    const float s = d > 0.0f ? fmaf(W_KEEP, rp[i], acc) : 0.0f;
    sp[i] = s;
    const int j = RUNS ? B.dj[i] : 0;
    if (RUNS && j >= DJ_OWN) __stcg(a.s32 + (j - DJ_OWN), s);
  }
  __syncthreads();
  for (int k = tid; k < B.n1; k += PT) {
    const int c = B.l1c[k], ic = RUNS ? B.l1i[k] : -1;
    float v = 0.0f;
    if (c >= 0) {
      float zp[5][5];
#pragma unroll
      for (int u = 0; u < 5; ++u)
#pragma unroll
        for (int x = 0; x < 5; ++x) {
          if ((u == 0 || u == 4) && (x == 0 || x == 4)) { zp[u][x] = 0.0f; continue; }
          const int i = c + (u - 2) * W + x - 2;
          zp[u][x] = __fmul_rn(dp[i], sp[i]);
        }
#pragma unroll
      for (int da = -1; da <= 1; ++da)
#pragma unroll
        for (int db = -1; db <= 1; ++db) {
          const int u = da + 2, x = db + 2, i = c + da * W + db;
          const float res = fmaf(W_KEEP, sp[i], (zp[u][x - 1] + zp[u][x + 1]) + (zp[u - 1][x] + zp[u + 1][x]));
          const float w = (da ? 0.5f : 1.0f) * (db ? 0.5f : 1.0f);
          v = __fadd_rn(v, dp[i] > 0.0f ? __fmul_rn(w, res) : 0.0f);
        }
    }
    B.r1[k] = v;
    if (RUNS && ic >= 0) __stcg(a.lev[1].r + ic, v);
  }
  __syncthreads();
  for (int k = tid; k < B.hw; k += PT) {
    const float* const rc = B.r1 + B.l2b[k];
    float v = 0.0f;  // nodes outside level 1 are zero in r1
#pragma unroll
    for (int u = 0; u < 5; ++u)
#pragma unroll
      for (int x = 0; x < 5; ++x) v = __fadd_rn(v, __fmul_rn(B.rw[(u * 5 + x) * B.hw + k], rc[u * B.W1 + x]));
    __stcg(a.lev[2].r + B.l2i[k], v);
  }
}

// Level 1's correction on the coarse patches, then both post-sweeps of the fine level on this
// block's runs: m two rows and columns beyond them,
// the first sweep one beyond, the second on this thread's own nodes (z, the residual's r).
constexpr int UP_PRE = 2;  // nodes of the runs' patches whose r and s a thread loads ahead
__device__ __forceinline__ void up_runs(const PoissonArgs& a, const FusedBlock& B, const FusedLevel* lv,
                                        const bool (&in)[2], int u, float (&zo)[2]) {
  const int tid = (int)threadIdx.x;
  const MgLevel &L1 = lv[1].L, &L2 = lv[2].L;
  // r and s first: their loads run beside those of z1
  float r0[UP_PRE], s0[UP_PRE];
#pragma unroll
  for (int e = 0; e < UP_PRE; ++e) {
    const int k = tid + e * PT, j = k < B.n ? B.uj[k] : -1;
    r0[e] = j >= 0 ? *(a.r32 + j) : 0.0f;
    s0[e] = j >= 0 ? *(a.s32 + j) : 0.0f;
  }
  for (int k = tid; k < B.nz; k += PT) {
    const int y = B.zn[k] >> 16, x = B.zn[k] & 0xFFFF;
    B.z1[k] = smooth_leg(L1, L2, L1.r, L2.z, y, x, B.zu + k, B.nz);
  }
  __syncthreads();
  for (int k = tid, e = 0; k < B.n; k += PT, ++e) {
    const int j = B.uj[k], f = B.uf[k];
    float m = 0.0f, rj = 0.0f;
    if (j >= 0) {
      const bool m01 = f & UF_M01, m10 = f & UF_M10;
      const float* const z = B.z1 + (f >> 9);
      const int Lx = (f >> 7 & 3) == 0 ? B.zw[0] : (f >> 7 & 3) == 1 ? B.zw[1] : (f >> 7 & 3) == 2 ? B.zw[2] : B.zw[3];
      float sj;
      if (e == 0) { rj = r0[0]; sj = s0[0]; }
      else if (UP_PRE > 1 && e == 1) { rj = r0[UP_PRE - 1]; sj = s0[UP_PRE - 1]; }
      else { rj = *(a.r32 + j); sj = *(a.s32 + j); }
      const float z00 = *z, z01 = m01 ? *(z + 1) : 0.0f, z10 = m10 ? *(z + Lx) : 0.0f,
                  z11 = m01 && m10 ? *(z + Lx + 1) : 0.0f, d = B.ud[k];
      const float wt = (f & UF_Y ? 0.5f : 1.0f) * (f & UF_X ? 0.5f : 1.0f);
      const float pz = __fmul_rn(wt, __fadd_rn(__fadd_rn(__fadd_rn(z00, z01), z10), z11));
      m = d > 0.0f ? fmaf(d, __fadd_rn(rj, sj), pz) : 0.0f;
    }
    B.mt[k] = m;
    B.rt[k] = rj;
  }
  __syncthreads();
  for (int k = tid; k < B.n; k += PT) {
    const int f = B.uf[k];
    float z = 0.0f;
    if (f & UF_RING) {
      const float* const m = B.mt + k;
      const float d = B.ud[k];
      const int pw = k >= B.n0 ? B.w1 : B.w0;
      const float mw = f & UF_W ? m[-1] : 0.0f, me = f & UF_E ? m[1] : 0.0f;
      const float acc = __fadd_rn(B.rt[k], __fadd_rn(__fadd_rn(mw, me), __fadd_rn(m[-pw], m[pw])));
      z = d > 0.0f ? fmaf(d, acc, __fmul_rn(W_KEEP, m[0])) : 0.0f;
    }
    B.m2[k] = z;
  }
  __syncthreads();
#pragma unroll
  for (int o = 0; o < 2; ++o) {
    zo[o] = 0.0f;
    if (!in[o]) continue;
    const int pw = o ? B.w1 : B.w0, k = (o ? B.n0 : 0) + 2 * pw + u + 2, f = B.uf[k];
    const float* const m = B.m2 + k;
    const float d = B.ud[k];
    float sm = 0.0f;
    sm = __fadd_rn(sm, f & UF_W ? m[-1] : 0.0f);
    sm = __fadd_rn(sm, f & UF_E ? m[1] : 0.0f);
    sm = __fadd_rn(sm, m[-pw]);
    sm = __fadd_rn(sm, m[pw]);
    zo[o] = d > 0.0f ? fmaf(W_KEEP, m[0], __fmul_rn(d, __fadd_rn(B.rt[k], sm))) : 0.0f;
  }
}

// The same on the block's tile, for grids whose runs are too long for their patches: r, s and
// level 1's right-hand side are the restriction's own patches, so only level 2's correction is
// read; z goes to memory for the owners of the sums.
__device__ __forceinline__ void up_tile(const PoissonArgs& a, const FusedBlock& B) {
  const int tid = (int)threadIdx.x, W = B.W;
  const float* const zc = a.lev[2].z;
  for (int k = tid; k < B.n2; k += PT) B.z2[k] = B.zj[k] >= 0 ? *(zc + B.zj[k]) : 0.0f;
  __syncthreads();
  for (int k = tid; k < B.nz; k += PT) {
    const float* const r = B.r1 + (B.zn[k] >> 16) - B.W1 - 1;
    const float* const z = B.z2 + (B.zn[k] & 0xFFFF) - B.W2 - 1;
    const float* const w = B.zu + k;
    float v = 0.0f;
#pragma unroll
    for (int t = 0; t < 3; ++t)
#pragma unroll
      for (int u = 0; u < 3; ++u) {
        v = __fadd_rn(v, __fmul_rn(w[(t * 3 + u) * B.nz], r[t * B.W1 + u]));
        v = __fadd_rn(v, __fmul_rn(w[(9 + t * 3 + u) * B.nz], z[t * B.W2 + u]));
      }
    B.z1[k] = v;
  }
  __syncthreads();
  for (int k = tid; k < B.np; k += PT) {
    const int f = B.uf[k];
    float m = 0.0f;
    if (f & UF_M) {
      const bool m01 = f & UF_M01, m10 = f & UF_M10;
      const float* const z = B.z1 + (f >> 9);
      const float z00 = z[0], z01 = m01 ? z[1] : 0.0f, z10 = m10 ? z[B.zw[0]] : 0.0f,
                  z11 = m01 && m10 ? z[B.zw[0] + 1] : 0.0f, d = B.dd[k];
      const float wt = (f & UF_Y ? 0.5f : 1.0f) * (f & UF_X ? 0.5f : 1.0f);
      const float pz = __fmul_rn(wt, __fadd_rn(__fadd_rn(__fadd_rn(z00, z01), z10), z11));
      m = d > 0.0f ? fmaf(d, __fadd_rn(B.rp[k], B.sp[k]), pz) : 0.0f;
    }
    B.mt[k] = m;
  }
  __syncthreads();
  for (int k = tid; k < B.np; k += PT) {
    float z = 0.0f;
    if (B.uf[k] & UF_RING) {
      const float* const m = B.mt + k;
      const float d = B.dd[k];
      const float acc = __fadd_rn(B.rp[k], __fadd_rn(__fadd_rn(m[-1], m[1]), __fadd_rn(m[-W], m[W])));
      z = d > 0.0f ? fmaf(d, acc, __fmul_rn(W_KEEP, m[0])) : 0.0f;
    }
    B.m2[k] = z;
  }
  __syncthreads();
  for (int k = tid; k < B.np; k += PT) {
    const int j = B.dj[k];
    if (j < DJ_OWN) continue;
    const float* const m = B.m2 + k;
    const float d = B.dd[k];
    const float sm = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(0.0f, m[-1]), m[1]), m[-W]), m[W]);
    __stcg(a.z32 + (j - DJ_OWN), d > 0.0f ? fmaf(W_KEEP, m[0], __fmul_rn(d, __fadd_rn(B.rp[k], sm))) : 0.0f);
  }
}

// coarse_solve with the block's rows of the inverse in shared memory; ci: the coarse nodes
// whose right-hand side this thread gathers, zi: the node of its warp's first row
__device__ __forceinline__ void coarse_rows(const PoissonArgs& a, const FusedBlock& B, float* rcs, int nc,
                                            const int (&ci)[2], int zi) {
  const float* const r = a.lev[a.nlevels - 1].r;
  float* const z = a.lev[a.nlevels - 1].z;
  const int tid = (int)threadIdx.x, lane = tid & 31;
  float v[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) v[e] = ci[e] >= 0 ? *(r + ci[e]) : 0.0f;
#pragma unroll
  for (int e = 0; e < 2; ++e)
    if (ci[e] >= 0) rcs[tid + e * PT] = v[e];
  for (int k = tid + 2 * PT; k < nc; k += PT) rcs[k] = *(r + __ldg(a.cidx + k));
  __syncthreads();
  for (int t = tid >> 5; t * a.nblk + gbid(a) < nc; t += PT / 32) {
    const int k = t * a.nblk + gbid(a);
    float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;
    auto dot = [&](const float* row) {
      int j = lane;
#pragma unroll 4
      for (; j + 96 < nc; j += 128) {
        s0 = fmaf(row[j], rcs[j], s0);
        s1 = fmaf(row[j + 32], rcs[j + 32], s1);
        s2 = fmaf(row[j + 64], rcs[j + 64], s2);
        s3 = fmaf(row[j + 96], rcs[j + 96], s3);
      }
      for (; j < nc; j += 32) s0 = fmaf(row[j], rcs[j], s0);
    };
    if (t < B.crows) dot(B.crow + (size_t)t * nc);
    else dot(a.cinv + (size_t)k * nc);
    float s = (s0 + s1) + (s2 + s3);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
    if (lane == 0) __stcg(z + (t < PT / 32 ? zi : __ldg(a.cidx + k)), s);
  }
}

template <bool RUNS>
__device__ __forceinline__ void poisson_body_fused(const PoissonArgs& a) {
  constexpr int NVB = RUNS ? FUSED_NVB_RUNS : FUSED_NVB_MAX, PATCH = RUNS ? FUSED_PATCH : FUSED_PATCH + 1;
  extern __shared__ float4 dyn_smem[];
  float* rcs = reinterpret_cast<float*>(dyn_smem);
  const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int N = a.ny * a.nx, nx = a.nx, nv = a.nvb * PT;
  // this block's virtual warps [c0, c1), one per warp: nodes 32 c + lane, and nv further
  const int vw = a.nvb * 32, c0 = (int)((long long)gbid(a) * vw / a.nblk),
            c1 = (int)((long long)(gbid(a) + 1) * vw / a.nblk), c = c0 + warp;
  const bool act = c < c1;
  const int part = (c % a.nvb) * 32 + c / a.nvb;
  const int last = a.nlevels - 1;
  int slot = 0;
  double n_outer = 0, n_inner = 0, last_rel = 0;
  unsigned long long t_start = 0;
  if (gbid(a) == 0 && tid == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_start));
  tmark(a, 20);

  __shared__ FusedLevel lv[MG_MAX_LEVELS];
  FusedBlock B;
  fused_tables<RUNS, false>(a, c0, c1, B, lv);
  bool laid = false;  // the tables, 10 to 15 us, are filled by the first linear solve that needs an iteration
  const int nc = __ldg(a.nc_dev);
  int ci[2], zi = -1;
#pragma unroll
  for (int e = 0; e < 2; ++e) ci[e] = tid + e * PT < nc ? __ldg(a.cidx + tid + e * PT) : -1;
  if (warp * a.nblk + gbid(a) < nc) zi = __ldg(a.cidx + warp * a.nblk + gbid(a));

  // this thread's nodes: bits 0 to 3 a free neighbour (W, E, y - 1, y + 1), 4 to 6 the diagonal,
  // 7 a free node; the Dirichlet-neighbour sums, which only it reads
  bool in[2];
  int code[2];
#pragma unroll
  for (int o = 0; o < 2; ++o) {
    const int i = 32 * c + lane + o * nv;
    in[o] = act && i < N;
    code[o] = 0;
    if (!in[o]) continue;
    const int y = i / nx, x = i - y * nx;
    int j[4];
    nbrs0(a, i, y, x, j);
    double s = 0.0;
    int diag = 4;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint8_t cl = j[k] >= 0 ? __ldg(a.cls + j[k]) : (uint8_t)NC_NEU;
      if (cl == NC_FREE) code[o] |= 1 << k;
      if (cl == NC_NEU) --diag;
      if (cl == NC_DIR) s += __ldg(a.Vfixed + j[k]);
    }
    code[o] |= diag << 4;
    if (__ldg(a.cls + i) == NC_FREE) {
      code[o] |= 128;
      a.dirsum[i] = s;
    }
  }
  // (A v)_i at a free node (apply0)
  auto apply_d = [&](int o, int i) {
    const double *const v = a.x + i, vi = *v;
    const double v0 = code[o] & 1 ? *(v - 1) : 0.0, v1 = code[o] & 2 ? *(v + 1) : 0.0,
                 v2 = code[o] & 4 ? *(v - nx) : 0.0, v3 = code[o] & 8 ? *(v + nx) : 0.0;
    return fma((double)((code[o] >> 4) & 7), vi, -DADD(DADD(DADD(DADD(0.0, v0), v1), v2), v3));
  };

  for (int pic = 0; pic < a.iterations; ++pic) {
    const double inner_at_pic = n_inner, outer_at_pic = n_outer;
    // the Picard update of the solve before, the right-hand side, the residual.  The update
    // writes x off the free nodes only, which no residual reads.
    float rv[2] = {0.0f, 0.0f};  // this thread's residuals
    if (act) {
      double ff = 0.0, rr = 0.0;
#pragma unroll 1
      for (int o = 0; o < 2; ++o) {
        if (!in[o]) continue;
        const int i = 32 * c + lane + o * nv;
        const double Vi = pic > 0 ? picard_update(a, i) : (*(a.V + i));
        if (!(code[o] & 128)) { __stcg(a.r32 + i, 0.0f); continue; }
        const double vm = Vi < a.V_plasma ? Vi : a.V_plasma;
        const double rho_e = DMUL(a.qn0_neg, exp(DDIV(DSUB(vm, a.V_plasma), a.Te_up)));
        const double rt = DADD((double)__ldg(a.rho + i), rho_e);
        const double fi = DADD(DMUL(a.coeff, rt), a.dirsum[i]);
        __stcg(a.f + i, fi);
        ff = fma(fi, fi, ff);
        const double res = DSUB(fi, apply_d(o, i));
        (o ? rv[1] : rv[0]) = (float)res;
        __stcg(a.r32 + i, (float)res);
        rr = fma(res, res, rr);
      }
      vw_put(a, slot, 0, part, ff);
      vw_put(a, slot, 1, part, rr);
    }
    grid_barrier(a);
    double norm2[2];
    VwTotal<2, NVB>(a, slot++).sums(a, norm2);
    const double fnorm2 = norm2[0];
    double rnorm2 = norm2[1];
    tmark(a, 17);
    const double target2 = a.tol * a.tol * fnorm2;

    if (!laid && rnorm2 > target2 && fnorm2 > 0.0) {
      laid = true;
      FusedBlock t;
      fused_tables<RUNS, true>(a, c0, c1, t, lv);
      __syncthreads();
    }
    for (int outer = 0; outer < a.max_outer && rnorm2 > target2 && fnorm2 > 0.0; ++outer) {
      n_outer += 1;
      double rz_old = 0.0, rr0 = rnorm2;
      float ev[2] = {0.0f, 0.0f}, pv[2] = {0.0f, 0.0f}, qv[2] = {0.0f, 0.0f};
      for (int k = tid; k < B.np; k += PT) {
        const int j = B.dj[k];
        B.rp[k] = j >= 0 ? *(a.r32 + (j & ~DJ_OWN)) : 0.0f;
      }
      down_tile<RUNS>(a, B);
      grid_barrier(a);
      tmark(a, 0);
      for (int k = 0; k < a.max_inner; ++k) {
        n_inner += 1;
        // z = M r: the V-cycle below the fine level's restriction
        for (int l = 2; l < last; ++l) {
          const MgLevel &F = lv[l].L, &C = lv[l + 1].L;
          const int* const yx = lv[l + 1].yx;
          for (int q = tid; q < lv[l + 1].share; q += PT)
            if (yx[q] >= 0) {
              const int I = yx[q] >> 16, J = yx[q] & 0xFFFF, ic = I * C.nx + J;
              __stcg(C.r + ic, restrict_leg(F, F.r, I, J, C.R + ic, (size_t)C.ny * C.nx));
            }
          grid_barrier(a);
          tmark(a, l < 7 ? l : 6);
        }
        coarse_rows(a, B, rcs, nc, ci, zi);
        grid_barrier(a);
        tmark(a, 7);
        for (int l = last - 1; l >= 2; --l) {
          const MgLevel &F = lv[l].L, &C = lv[l + 1].L;
          const int* const yx = lv[l].yx;
          for (int q = tid; q < lv[l].share; q += PT)
            if (yx[q] >= 0) {
              const int y = yx[q] >> 16, x = yx[q] & 0xFFFF, i = y * F.nx + x;
              __stcg(F.z + i, smooth_leg(F, C, F.r, C.z, y, x, F.U + i, (size_t)F.ny * F.nx));
            }
          grid_barrier(a);
          tmark(a, 8 + (l < 7 ? l : 6));
        }
        float zo[2], zn[2][4];
        auto neighbours = [&]() {
#pragma unroll
          for (int o = 0; o < 2; ++o) {
            const float* const z = a.z32 + 32 * c + lane + o * nv;
            const int f = code[o];
            zn[o][0] = f & 1 ? *(z - 1) : 0.0f;
            zn[o][1] = f & 2 ? *(z + 1) : 0.0f;
            zn[o][2] = f & 4 ? *(z - nx) : 0.0f;
            zn[o][3] = f & 8 ? *(z + nx) : 0.0f;
          }
        };
        if (RUNS) {
          up_runs(a, B, lv, in, 32 * warp + lane, zo);
#pragma unroll
          for (int o = 0; o < 2; ++o)
            if (in[o]) __stcg(a.z32 + 32 * c + lane + o * nv, zo[o]);
        } else {
          up_tile(a, B);
          grid_barrier(a);
          tmark(a, 9);
#pragma unroll
          for (int o = 0; o < 2; ++o) zo[o] = in[o] ? *(a.z32 + 32 * c + lane + o * nv) : 0.0f;
          neighbours();
        }
        if (act) {
          double rz_p = 0.0;
#pragma unroll
          for (int o = 0; o < 2; ++o)
            if (in[o]) rz_p += (double)rv[o] * (double)zo[o];
          vw_put(a, slot, 0, part, rz_p);
        }
        grid_barrier(a);
        tmark(a, 8);
        // p = z + beta p, q = A p
        VwTotal<1, NVB> tz(a, slot++);
        if (RUNS) neighbours();
        const double rz = tz.sum(a);
        const float beta = (float)(k == 0 ? 0.0 : rz / rz_old);
        if (act) {
          double pq_p = 0.0;
#pragma unroll
          for (int o = 0; o < 2; ++o) {
            const bool fr = code[o] & 128;
            const float sz = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(0.0f, zn[o][0]), zn[o][1]), zn[o][2]), zn[o][3]);
            const float az = fmaf((float)((code[o] >> 4) & 7), zo[o], -sz);
            pv[o] = fr ? fmaf(beta, pv[o], zo[o]) : 0.0f;
            qv[o] = fr ? fmaf(beta, qv[o], az) : 0.0f;
            if (in[o]) __stcg(a.q32 + 32 * c + lane + o * nv, qv[o]);
            pq_p += (double)pv[o] * (double)qv[o];
          }
          vw_put(a, slot, 0, part, pq_p);
        }
        grid_barrier(a);
        tmark(a, 14);
        // e += alpha p, r -= alpha q (on the nodes and on the tile's patch), then the next
        // V-cycle's restrictions
        VwTotal<1, NVB> tq(a, slot++);
        float qp[PATCH];
#pragma unroll
        for (int e = 0; e < PATCH; ++e) {
          const int t = tid + e * PT, j = t < B.np ? B.dj[t] : -1;
          qp[e] = j >= 0 ? *(a.q32 + (j & ~DJ_OWN)) : 0.0f;
        }
        const double pq = tq.sum(a);
        const float al = (float)(pq != 0.0 ? rz / pq : 0.0);
#pragma unroll
        for (int e = 0; e < PATCH; ++e) {
          const int t = tid + e * PT;
          if (t < B.np) B.rp[t] = fmaf(-al, qp[e], B.rp[t]);
        }
        for (int t = tid + PATCH * PT; t < B.np; t += PT)
          if (B.dj[t] >= 0) B.rp[t] = fmaf(-al, *(a.q32 + (B.dj[t] & ~DJ_OWN)), B.rp[t]);
        if (act) {
          double rr_p = 0.0;
#pragma unroll
          for (int o = 0; o < 2; ++o) {
            rv[o] = fmaf(-al, qv[o], rv[o]);
            ev[o] = fmaf(al, pv[o], ev[o]);
            if (RUNS && in[o]) __stcg(a.r32 + 32 * c + lane + o * nv, rv[o]);
            rr_p += (double)rv[o] * (double)rv[o];
          }
          vw_put(a, slot, 0, part, rr_p);
        }
        down_tile<RUNS>(a, B);
        grid_barrier(a);
        const double rrk = VwTotal<1, NVB>(a, slot++).sum(a);
        tmark(a, 15);
        rz_old = rz;
        if (rrk <= a.tol_inner * a.tol_inner * rr0 || rrk <= target2) break;  // as in poisson_body
      }
      // FP64 correction and true residual
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        const int i = 32 * c + lane + o * nv;
        if (code[o] & 128) __stcg(a.x + i, (*(a.x + i)) + (double)ev[o]);
      }
      grid_barrier(a);
      if (act) {
        double rr = 0.0;
#pragma unroll
        for (int o = 0; o < 2; ++o) {
          const int i = 32 * c + lane + o * nv;
          if (!(code[o] & 128)) continue;
          const double res = DSUB((*(a.f + i)), apply_d(o, i));
          rv[o] = (float)res;
          __stcg(a.r32 + i, rv[o]);
          rr = fma(res, res, rr);
        }
        vw_put(a, slot, 0, part, rr);
      }
      grid_barrier(a);
      rnorm2 = VwTotal<1, NVB>(a, slot++).sum(a);
      tmark(a, 16);
    }
    if (!(rnorm2 <= target2) && fnorm2 > 0.0 && gbid(a) == 0 && tid == 0) atomicOr(a.errflags, PB_EF_POISSON_NOCONV);
    if (a.trace && gbid(a) == 0 && tid == 0 && pic < 5) {
      a.trace[21 + pic] += (unsigned long long)(n_inner - inner_at_pic);
      a.trace[26 + pic] += (unsigned long long)(n_outer - outer_at_pic);
    }
    last_rel = fnorm2 > 0.0 ? sqrt(rnorm2 / fnorm2) : 0.0;
  }
#pragma unroll 1
  for (int o = 0; o < 2; ++o)
    if (in[o]) picard_update(a, 32 * c + lane + o * nv);
  grid_barrier(a);
  tmark(a, 18);
  solve_end(a, gtid(a), a.nblk * PT, n_outer, n_inner, last_rel, t_start);
}

__global__ void __launch_bounds__(PT, 1) k_poisson(const __grid_constant__ PoissonArgs a) { poisson_body(a); }
__global__ void __launch_bounds__(PT, 1) k_poisson_runs(const __grid_constant__ PoissonArgs a) {
  poisson_body_fused<true>(a);
}
__global__ void __launch_bounds__(PT, 1) k_poisson_tiles(const __grid_constant__ PoissonArgs a) {
  poisson_body_fused<false>(a);
}

__global__ void __launch_bounds__(PT, 1) k_poisson_batch(const PoissonArgs* __restrict__ args,
                                                         const int* __restrict__ blk_map) {
  __shared__ PoissonArgs sa;
  const int* lst = blk_map + blk_map[blockIdx.x];
  const int cnt = lst[0];
  for (int q = 0; q < cnt; ++q) {
    const int* src = reinterpret_cast<const int*>(args + lst[1 + q]);
    int* dst = reinterpret_cast<int*>(&sa);
    for (int k = threadIdx.x; k < (int)(sizeof(PoissonArgs) / sizeof(int)); k += blockDim.x) dst[k] = src[k];
    __syncthreads();
    poisson_body(sa);
    __syncthreads();
  }
}

}  // namespace pb

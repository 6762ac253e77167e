// Remaining step kernels: injection, SEE electron spawn, exit-angle percentile, sputter
// cell break, grid thermal conduction, PPC statistics, cell-key radix sort and the
// module-level thermal_conduction (Taichi semantics).
#include "pb_kernels.cuh"
#include "pb_misc.cuh"
#include "pb_poisson.cuh"

namespace pb {

// ------------------------------------------------------------------ helpers
__device__ __forceinline__ int dep_cell(float x, float y, float dxf, float dyf, int nx, int ny) {
  int ix = cell_round32(x, dxf, 1, nx - 2);
  int iy = cell_round32(y, dyf, 1, ny - 2);
  return iy * nx + ix;
}

// Poisson(lam) by CDF inversion with one keyed uniform (oracle/philox.py: poisson_count), by a
// warp: p_k = p_{k-1} lam / k is a chain of correctly rounded operations; its divisions by k
// take reciprocals that the lanes form 32 at a time (div_int), four dependent operations a term
// instead of a multiplication and a division.  Every lane returns the count.
__device__ int poisson_inversion(double u, double lam) {
  if (!(lam > 0.0)) return 0;
  const int lane = threadIdx.x & 31;
  double p = exp(-lam);
  double F = p;
  int k = 0;
  const int kmax = (int)(lam + 40.0 * sqrt(lam) + 100.0);
  while (u > F && k < kmax) {
    const double y = __drcp_rn((double)(k + 1 + lane));
    for (int t = 0; t < 32 && u > F && k < kmax; ++t) {
      ++k;
      const double x = DMUL(p, lam), yk = __shfl_sync(0xFFFFFFFFu, y, t);
      p = x >= 0x1p-900 ? div_int(x, (double)k, yk) : DDIV(x, (double)k);
      F = DADD(F, p);
    }
  }
  return k;
}

// ------------------------------------------------------------------ injection
// inject step A (physics_engine.py:996-1099): counts, slots and ids for this step; one warp
// (of k_step_reset)
__device__ __forceinline__ void inject_counts(const InjectArgs& a) {
  const uint32_t step = a.step_dev ? *a.step_dev : a.step;
  int n_ion = 0, n_rf = 0;
  if (a.ion_on) n_ion = poisson_inversion(philox_uniform(a.seed, 0, SITE_ION_COUNT, step, 0), a.lam);
  if (a.rf_on) {
    n_rf = (int)a.rf_num_float;
    if (philox_uniform(a.seed, 0, SITE_RF_COUNT, step, 0) < DSUB(a.rf_num_float, (double)n_rf)) ++n_rf;
  }
  if ((threadIdx.x & 31) != 0) return;
  int n_neut = a.neut_n;
  int np0 = *a.num_p, ne0 = *a.num_e;
  if (np0 + n_ion > a.cap_p) { atomicOr(a.errflags, PB_EF_CAPACITY_ION); n_ion = a.cap_p - np0; if (n_ion < 0) n_ion = 0; }
  if (ne0 + n_rf + n_neut > a.cap_e) {
    atomicOr(a.errflags, PB_EF_CAPACITY_ELE);
    int room = a.cap_e - ne0; if (room < 0) room = 0;
    if (n_rf > room) n_rf = room;
    n_neut = room - n_rf < n_neut ? room - n_rf : n_neut;
  }
  uint32_t id_i = *a.next_ion_id, id_e = *a.next_e_id;
  if ((uint64_t)id_i + n_ion > 0xFFFFFFFFull || (uint64_t)id_e + n_rf + n_neut > 0xFFFFFFFFull)
    atomicOr(a.errflags, PB_EF_ID_OVERFLOW);
  a.inj[0] = n_ion; a.inj[1] = n_rf; a.inj[2] = n_neut;
  a.inj[3] = np0; a.inj[4] = ne0;
  a.inj[5] = (int)id_i; a.inj[6] = (int)id_e;
  *a.num_p = np0 + n_ion;
  *a.num_e = ne0 + n_rf + n_neut;
  *a.next_ion_id = id_i + n_ion;
  *a.next_e_id = id_e + n_rf + n_neut;
}

// inject step B: four threads per new particle (place, and one velocity component each);
// blockIdx.y selects ions / rf / neutralizer.  The few particles make it a chain of latencies:
// with three normals in sequence per thread, each of 24 float64 divisions, it held the step up
// for 13 to 23 us on 130 x 568 and 26 us on 257 x 1025; 3 to 4 us so (div_int).
__global__ void __launch_bounds__(128) k_inject_gen(const __grid_constant__ InjectArgs a) {
  pdl_enter();
  const uint32_t step = a.step_dev ? *a.step_dev : a.step;
  const int seg = blockIdx.y;
  const int n = a.inj[seg];
  const int off = seg == 2 ? a.inj[1] : 0;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < 4 * n; e += gridDim.x * blockDim.x) {
    const int j = e >> 2, comp = (e & 3) - 1;
    const uint32_t id = (uint32_t)a.inj[seg == 0 ? 5 : 6] + off + j;
    const int slot = a.inj[seg == 0 ? 3 : 4] + off + j;
    const Soa& S = seg == 0 ? a.ions : a.eles;
    if (comp >= 0) {
      const uint32_t site = seg == 0 ? SITE_ION_V : seg == 1 ? SITE_RF_V : SITE_NEUT_V;
      const double g = philox_normal(a.seed, id, site, step, (uint32_t)comp);
      double v;
      if (seg == 0) v = comp == 0 ? DADD(a.v_bohm, DMUL(g, a.v_spread)) : DMUL(g, a.v_spread);
      else if (seg == 1) v = comp == 0 ? DADD(DMUL(fabs(g), a.v_e_src), a.v_bohm) : DMUL(g, a.v_e_src);
      else v = DMUL(g, a.v_e_th);
      (comp == 0 ? S.vx : comp == 1 ? S.vy : S.vz)[slot] = __double2float_rn(v);
      continue;
    }
    float x, y;
    if (seg == 0) {
      if (a.geometry == 2) {
        double uh = philox_uniform(a.seed, id, SITE_ION_HOLE, step, 0);
        double u = philox_uniform(a.seed, id, SITE_ION_HOLE, step, 1);
        int which = (int)DMUL(uh, 2.0);
        float lo = a.span[2 * which], hi = a.span[2 * which + 1];
        y = __double2float_rn(DADD((double)lo, DMUL((double)__fsub_rn(hi, lo), u)));
      } else {
        double u = philox_uniform(a.seed, id, SITE_ION_Y, step, 0);
        y = __double2float_rn(DADD(a.ylo, DMUL(DSUB(a.yhi, a.ylo), u)));
      }
      x = a.x_inj;
      S.cex[slot] = 0;
    } else if (seg == 1) {
      double u = philox_uniform(a.seed, id, SITE_RF_Y, step, 0);
      y = __double2float_rn(DADD(a.rf_ylo, DMUL(DSUB(a.rf_yhi, a.rf_ylo), u)));
      x = 0.1f;
    } else {
      double u = philox_uniform(a.seed, id, SITE_NEUT_Y, step, 0);
      y = __double2float_rn(DADD(0.0, DMUL(DSUB(a.neut_r, 0.0), u)));
      x = a.neut_x;
    }
    S.x[slot] = x;
    S.y[slot] = y;
    S.id[slot] = id;
    atomicAdd((seg == 0 ? a.cnt_i : a.cnt_e) + dep_cell(x, y, a.dxf, a.dyf, a.nx, a.ny), 1);
  }
}

// ------------------------------------------------------------------ single-block bitonic sort
// Sorts keys[0..n) ascending in place (one block; shared memory, or global memory with room for
// the next power of two).  Each of the log^2 steps of a short list costs a barrier in shared
// memory but a round trip to L2 in global memory, so lists of up to SORT_SMEM keys are copied.
constexpr int SORT_SMEM = 2048;
template <class T>
__device__ __forceinline__ void block_sort(T* keys, int n) {
  int m = 1;
  while (m < n) m <<= 1;
  for (int i = n + threadIdx.x; i < m; i += blockDim.x) keys[i] = (T)~(T)0;
  __syncthreads();
  for (int k = 2; k <= m; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = threadIdx.x; i < m; i += blockDim.x) {
        int l = i ^ j;
        if (l > i) {
          T a = keys[i], b = keys[l];
          bool up = (i & k) == 0;
          if ((a > b) == up) { keys[i] = b; keys[l] = a; }
        }
      }
      __syncthreads();
    }
  }
}

// ------------------------------------------------------------------ SEE electrons
// Spawned electrons in parent-id order (= the reference's array order), keyed draws by
// the parent ion, purge test against the current isBound, appended after the step's
// surviving electrons (physics_engine.py:1400-1417, 1541-1561).
__global__ void __launch_bounds__(1024) k_see_finish(const __grid_constant__ SeeArgs a) {
  pdl_enter();
  const uint32_t step = a.step_dev ? *a.step_dev : a.step;
  __shared__ int sm[32];
  __shared__ int s_base, s_total;
  __shared__ uint64_t skey[SORT_SMEM];
  __shared__ float svel[3 * 1024];
  int n = *a.see_count;
  if (n > a.see_cap) n = a.see_cap;
  const bool small = n <= SORT_SMEM;
  uint64_t* const keys = small ? skey : a.see_key;
  if (small) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) skey[i] = a.see_key[i];
    __syncthreads();
    block_sort(skey, n);
  } else {
    block_sort(a.see_key, n);
  }
  const int ne0 = *a.num_e;
  const uint32_t id0 = *a.next_e_id;
  int done = 0;
  for (int c0 = 0; c0 < n; c0 += blockDim.x) {
    // the chunk's velocity components, one per thread and turn
    const int nc = min(n - c0, (int)blockDim.x);
    for (int e = threadIdx.x; e < 3 * nc; e += blockDim.x) {
      const uint32_t parent = (uint32_t)(keys[c0 + e / 3] >> 32);
      svel[e] = __double2float_rn(DMUL(philox_normal(a.seed, parent, SITE_SEE_V, step, (uint32_t)(e % 3)), a.v_see_th));
    }
    __syncthreads();
    int r = c0 + threadIdx.x;
    bool keep = false;
    float x = 0, y = 0, vx = 0, vy = 0, vz = 0;
    if (r < n) {
      const uint32_t rec = (uint32_t)keys[r];
      x = a.see_xy[2 * rec];
      y = a.see_xy[2 * rec + 1];
      vx = svel[3 * threadIdx.x]; vy = svel[3 * threadIdx.x + 1]; vz = svel[3 * threadIdx.x + 2];
      int icx = cell_round(x, a.dxf, 0, a.nx - 1), icy = cell_round(y, a.dyf, 0, a.ny - 1);
      bool dead = a.isBound[(size_t)icy * a.nx + icx] != 0;
      dead = dead || (x < 0.0f) || (x > a.Lxf) || (y < 0.0f) || (y > a.Lyf) || (x != x);
      keep = !dead;
    }
    // block scan of keep flags (chunk order = parent order)
    unsigned b = __ballot_sync(0xFFFFFFFFu, keep);
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int pre = __popc(b & ((1u << lane) - 1));
    if (lane == 0) sm[w] = __popc(b);
    __syncthreads();
    if (threadIdx.x == 0) {
      int s = 0;
      for (int q = 0; q < (int)(blockDim.x >> 5); ++q) { int t = sm[q]; sm[q] = s; s += t; }
      s_base = done;
      s_total = s;
    }
    __syncthreads();
    if (keep) {
      int slot = ne0 + s_base + sm[w] + pre;
      if (slot < a.cap_e) {
        a.eles.x[slot] = x; a.eles.y[slot] = y;
        a.eles.vx[slot] = vx; a.eles.vy[slot] = vy; a.eles.vz[slot] = vz;
        a.eles.id[slot] = id0 + r;
        atomicAdd(a.cnt_e + dep_cell(x, y, a.dxf, a.dyf, a.nx, a.ny), 1);
      } else {
        atomicOr(a.errflags, PB_EF_CAPACITY_ELE);
      }
    }
    done += s_total;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    int tot = ne0 + done;
    *a.num_e = tot < a.cap_e ? tot : a.cap_e;
    *a.next_e_id = id0 + (uint32_t)n;
    *a.see_spawned = n;
  }
}

// ------------------------------------------------------------------ exit divergence
// np.percentile(angles, 95) for float32 data: q = f32(95)/f32(100), v = f32(n-1)*q,
// linear interpolation with NumPy's two-sided lerp, all in float32.
PB_HD float percentile95_sorted(const float* s, int n) {
  float q = 95.0f / 100.0f;
  float vi = (float)(n - 1) * q;
  if (vi >= (float)(n - 1)) return s[n - 1];
  float prev = floorf(vi);
  float g = vi - prev;
  int i = (int)prev;
  float lo = s[i], hi = s[i + 1];
  float d = hi - lo;
  return g >= 0.5f ? hi - d * (1.0f - g) : lo + d * g;
}

__device__ void theta95(float* angles, const int* count, int cap, uint64_t* scratch, double* out) {
  int n = *count;
  if (n > cap) n = cap;
  if (n <= 5) {
    if (threadIdx.x == 0) *out = __longlong_as_double(0x7ff8000000000000ll);
    return;
  }
  if (n <= 2 * SORT_SMEM) {
    __shared__ uint32_t skey[2 * SORT_SMEM];
    for (int i = threadIdx.x; i < n; i += blockDim.x) skey[i] = __float_as_uint(angles[i]);
    __syncthreads();
    block_sort(skey, n);
    if (threadIdx.x == 0) *out = (double)percentile95_sorted(reinterpret_cast<const float*>(skey), n);
    return;
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) scratch[i] = (uint64_t)__float_as_uint(angles[i]);
  __syncthreads();
  block_sort(scratch, n);
  for (int i = threadIdx.x; i < n; i += blockDim.x) angles[i] = __uint_as_float((uint32_t)scratch[i]);
  __syncthreads();
  if (threadIdx.x == 0) *out = (double)percentile95_sorted(angles, n);
}

// ------------------------------------------------------------------ sputter cell break
// broken = (damage > Thresh) & isBound -> eroded_depth += dy, isBound = 0, damage = 0,
// and the node class is recomputed so the next field solve uses the new operator
// (physics_engine.py:1443-1449, 525-552).
__global__ void k_erosion_break(double* damage, uint8_t* isBound, uint8_t* cls, double* eroded, int ny, int nx,
                                int periodic, double thresh, double dy, int* broken) {
  pdl_enter();
  int N = ny * nx;
  int cntb = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
    if (isBound[i] && damage[i] > thresh) {
      eroded[i] += dy;
      isBound[i] = 0;
      damage[i] = 0.0;
      int y = i / nx, x = i - y * nx;
      uint8_t c = 0;  // NC_FREE
      if (x == nx - 1) c = 2;
      else if (!periodic && (y == 0 || y == ny - 1)) c = 2;
      cls[i] = c;
      ++cntb;
    }
  }
  if (cntb) atomicAdd(broken, cntb);
}

// After a break the fine-level smoother weights follow the new node classes, and the
// hierarchy is marked dirty: k_mg_rebuild forms the coarse levels again before the next
// field solve.  (Should it leave them to the host, the V-cycle with the old coarse levels
// stays symmetric positive definite: its smoother part is, once every free node has its
// weight, and the coarse part adds a semidefinite term.)  The weights are the host build's,
// omega / (4 - Neumann neighbours) in double rounded to float, 0 off the free nodes.
__global__ void k_refresh_dinv0(const uint8_t* cls, float* dinv, int ny, int nx, int periodic, const int* broken,
                                int* mg_dirty) {
  pdl_enter();
  if (*broken == 0) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) *mg_dirty = 1;  // the coarse levels follow before the next solve
  const int N = ny * nx;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
    float d = 0.0f;
    if (cls[i] == NC_FREE) {
      const int y = i / nx, x = i - y * nx;
      int nneu = 0;
      // left, right, down, up; outside the grid counts as a Neumann neighbour
      nneu += x == 0 || cls[i - 1] == NC_NEU;
      nneu += x == nx - 1 || cls[i + 1] == NC_NEU;
      int yd = y - 1, yu = y + 1;
      if (periodic) { if (yd < 0) yd += ny; if (yu >= ny) yu -= ny; }
      nneu += yd < 0 || cls[yd * nx + x] == NC_NEU;
      nneu += yu >= ny || cls[yu * nx + x] == NC_NEU;
      if (nneu < 4) d = (float)(MG_JACOBI_OMEGA / (double)(4 - nneu));
    }
    dinv[i] = d;
  }
}

// ------------------------------------------------------------------ thermal
// Radiative cooling of bound cells, 10 explicit FTCS sweeps over interior bound cells
// (non-bound neighbours replaced by the centre value, T_new = max(T + dT, 300)) and the
// final clamp, fused with temporal blocking: each block owns a TT x TT output tile and
// loads a halo of SWEEPS cells (physics_engine.py:1566-1615, CPU-loop semantics).  The bound
// cells' new temperatures go to Tnext (other blocks' halos are still to be read from T);
// node_stats moves them.
// A thread keeps its cells' values, neighbour tests and indexes in registers over the sweeps;
// 1024 threads (three cells each), since a small grid has few tiles (27 on 65 x 284) and a sweep
// is latency: that grid's step took 19.5 us for it with 256 threads that indexed every cell of
// every sweep, 7.1 us so.
constexpr int TT = 32;
constexpr int HALO = 10;
constexpr int TW = TT + 2 * HALO;
constexpr int THERMAL_NT = 1024;

__global__ void __launch_bounds__(THERMAL_NT) k_thermal(const float* T, float* Tnext, const uint8_t* isBound, int ny,
                                                        int nx, float cf, float T4_300, float Fo_x, float Fo_y,
                                                        int sweeps) {
  pdl_enter();
  constexpr int PER = (TW * TW + THERMAL_NT - 1) / THERMAL_NT;
  __shared__ float buf[2][TW * TW];
  __shared__ uint8_t M[TW * TW];
  const int gx0 = blockIdx.x * TT - HALO, gy0 = blockIdx.y * TT - HALO;
  float c[PER];
  // bits 0-3: the neighbour left, right, down, up is bound; 4: swept; 5: a mask cell; 6: output; 7: bound
  unsigned flags[PER];
  int found = 0;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int k = threadIdx.x + j * THERMAL_NT;
    c[j] = 0.0f;
    flags[j] = 0u;
    if (k >= TW * TW) continue;
    const int ly = k / TW, lx = k - ly * TW;
    const int gy = gy0 + ly, gx = gx0 + lx;
    const bool in = gy >= 0 && gy < ny && gx >= 0 && gx < nx;
    uint8_t m = 0;
    if (in) {
      float t = T[(size_t)gy * nx + gx];
      m = isBound[(size_t)gy * nx + gx];
      if (m) {
        // T -= cf * (T**4 - 300**4)   (x^4 rounded once from double)
        double td = (double)t;
        float t4 = __double2float_rn(DMUL(DMUL(td, td), DMUL(td, td)));
        t = __fsub_rn(t, __fmul_rn(cf, __fsub_rn(t4, T4_300)));
        found = 1;
      }
      c[j] = t;
      // a mask cell of an even value is cooled only; node_stats moves it as every mask cell
      flags[j] = (m ? 32u : 0u) | (m & 1) << 7;
      if ((m & 1) && gy >= 1 && gy <= ny - 2 && gx >= 1 && gx <= nx - 2 && ly >= 1 && ly <= TW - 2 && lx >= 1 &&
          lx <= TW - 2)
        flags[j] |= 16u;
      if (ly >= HALO && ly < HALO + TT && lx >= HALO && lx < HALO + TT) flags[j] |= 64u;
    }
    buf[0][k] = c[j];
    M[k] = m;
  }
  if (!__syncthreads_or(found)) return;
#pragma unroll
  for (int j = 0; j < PER; ++j)
    if (flags[j] & 16u) {
      const int k = threadIdx.x + j * THERMAL_NT;
      flags[j] |= (M[k - 1] & 1u) | (M[k + 1] & 1u) << 1 | (M[k - TW] & 1u) << 2 | (M[k + TW] & 1u) << 3;
    }
  for (int s = 0; s < sweeps; ++s) {
    const float* cur = buf[s & 1];
    float* nxt = buf[(s & 1) ^ 1];
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int k = threadIdx.x + j * THERMAL_NT;
      if (k >= TW * TW) continue;
      if (flags[j] & 16u) {
        const float v = c[j];
        const float tl = flags[j] & 1u ? cur[k - 1] : v;
        const float tr = flags[j] & 2u ? cur[k + 1] : v;
        const float td = flags[j] & 4u ? cur[k - TW] : v;
        const float tu = flags[j] & 8u ? cur[k + TW] : v;
        const float c2 = __fmul_rn(2.0f, v);
        const float dT = __fadd_rn(__fmul_rn(Fo_x, __fadd_rn(__fsub_rn(tl, c2), tr)),
                                   __fmul_rn(Fo_y, __fadd_rn(__fsub_rn(td, c2), tu)));
        const float nv = __fadd_rn(v, dT);
        c[j] = (nv != nv) ? nv : (nv > 300.0f ? nv : 300.0f);
      }
      nxt[k] = c[j];
    }
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    if ((flags[j] & 96u) != 96u) continue;
    const int k = threadIdx.x + j * THERMAL_NT;
    const int ly = k / TW, lx = k - ly * TW;
    const float v = c[j];
    Tnext[(size_t)(gy0 + ly) * nx + gx0 + lx] = (v != v || !(flags[j] & 128u)) ? v : (v > 300.0f ? v : 300.0f);
  }
}

// Block-wide reduction with op; the result is valid in thread 0.  Ends with a barrier, so
// it can be called again at once.  blockDim.x is a multiple of 32.
template <class T, class Op>
__device__ __forceinline__ T block_reduce(T v, Op op, T ident) {
  __shared__ T sm[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_down_sync(0xFFFFFFFFu, v, o));
  if (lane == 0) sm[warp] = v;
  __syncthreads();
  if (warp == 0) {
    v = lane < (int)(blockDim.x >> 5) ? sm[lane] : ident;
    for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_down_sync(0xFFFFFFFFu, v, o));
  }
  __syncthreads();
  return v;
}

// One pass over the nodes, block `block` of `blocks`: the bound cells' new temperatures from
// k_thermal moved into T (Tnext not null), the electrodes' sums, and the PPC statistics: accum
// += ppc; total active cells, cells with 0 < ppc < 3, min nonzero.
constexpr int STEP_END_NT = 512;

__device__ __forceinline__ void node_stats(float* T, const float* Tnext, const uint8_t* isBound,
                                           const uint16_t* gridmask, int ngrids, double* sums, const int* ppc,
                                           double* accum, unsigned long long* stats, int N, int block, int blocks) {
  double s[16];
  int c[16];
#pragma unroll
  for (int g = 0; g < 16; ++g) { s[g] = 0.0; c[g] = 0; }
  unsigned act = 0, low = 0;
  int mn = 0x7fffffff;
  for (int i = block * blockDim.x + threadIdx.x; i < N; i += blocks * blockDim.x) {
    const unsigned m = gridmask[i];
    const int v = ppc[i];
    float t = 0.0f;
    if (Tnext && isBound[i]) T[i] = t = Tnext[i];
    else if (m) t = T[i];
    if (m) {
#pragma unroll
      for (int g = 0; g < 16; ++g)
        if (g < ngrids && (m >> g & 1u)) { s[g] += (double)t; ++c[g]; }
    }
    accum[i] += (double)v;
    if (v > 0) { ++act; if (v < 3) ++low; mn = v < mn ? v : mn; }
  }
  // one pair of atomics per block and grid (per-warp atomics on the same 2 * ngrids words
  // serialised at L2)
  const auto addd = [](double a, double b) { return a + b; };
  const auto addu = [](unsigned a, unsigned b) { return a + b; };
#pragma unroll
  for (int g = 0; g < 16; ++g) {
    if (g >= ngrids) break;
    if (!__syncthreads_or(c[g])) continue;
    const double a = block_reduce(s[g], addd, 0.0);
    const unsigned b = block_reduce((unsigned)c[g], addu, 0u);
    if (threadIdx.x == 0) { atomicAdd(sums + 2 * g, a); atomicAdd(sums + 2 * g + 1, (double)b); }
  }
  act = block_reduce(act, addu, 0u);
  low = block_reduce(low, addu, 0u);
  mn = block_reduce(mn, [](int a, int b) { return a < b ? a : b; }, 0x7fffffff);
  if (threadIdx.x == 0) {
    if (act) atomicAdd(stats, (unsigned long long)act);
    if (low) atomicAdd(stats + 1, (unsigned long long)low);
    atomicMin(stats + 2, (unsigned long long)mn);
  }
}

// ------------------------------------------------------------------ Taichi-kernel thermal sweep
// thermal_conduction_taichi (physics_engine.py:147-171): every masked cell, neighbours
// inside the domain and masked, T_new = max(T + dT, 300); unmasked cells copied.
// Four cells per thread with 16-byte accesses where the three arrays start 16-byte aligned
// (VEC); only cells of the mask read their neighbours.  Ten sweeps of 513 x 2049: 5.4 us
// each with scalar accesses, 4.4 us so (12.6 MB: 2.9 TB/s, from L2).
__device__ __forceinline__ float taichi_cell(const float* __restrict__ T, const int32_t* __restrict__ mask, int i, int iy,
                                             int ix, int nx, int ny, float c, float Fo_x, float Fo_y) {
  const float tl = (ix > 0 && __ldg(mask + i - 1) == 1) ? __ldg(T + i - 1) : c;
  const float tr = (ix < nx - 1 && __ldg(mask + i + 1) == 1) ? __ldg(T + i + 1) : c;
  const float tu = (iy < ny - 1 && __ldg(mask + i + nx) == 1) ? __ldg(T + i + nx) : c;
  const float td = (iy > 0 && __ldg(mask + i - nx) == 1) ? __ldg(T + i - nx) : c;
  const float c2 = __fmul_rn(2.0f, c);
  const float dT = __fadd_rn(__fmul_rn(Fo_x, __fadd_rn(__fsub_rn(tl, c2), tr)),
                             __fmul_rn(Fo_y, __fadd_rn(__fsub_rn(td, c2), tu)));
  const float nv = __fadd_rn(c, dT);
  return nv > 300.0f ? nv : 300.0f;
}

template <bool VEC>
__global__ void __launch_bounds__(256) k_thermal_taichi(const float* __restrict__ T, float* __restrict__ Tn,
                                                        const int32_t* __restrict__ mask, int nx, int ny, float Fo_x,
                                                        float Fo_y) {
  pdl_enter();
  const int N = nx * ny, t0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  int done = 0;
  if (VEC) {
    const int n4 = N >> 2;
    done = n4 << 2;
    for (int q = t0; q < n4; q += stride) {
      const int4 m = __ldg(reinterpret_cast<const int4*>(mask) + q);
      float4 v = __ldg(reinterpret_cast<const float4*>(T) + q);
      if (m.x == 1 || m.y == 1 || m.z == 1 || m.w == 1) {
        const int i = 4 * q;
        int iy = i / nx, ix = i - iy * nx;
        auto next = [&] { if (++ix == nx) { ix = 0; ++iy; } };
        const float4 c = v;
        if (m.x == 1) v.x = taichi_cell(T, mask, i, iy, ix, nx, ny, c.x, Fo_x, Fo_y);
        next();
        if (m.y == 1) v.y = taichi_cell(T, mask, i + 1, iy, ix, nx, ny, c.y, Fo_x, Fo_y);
        next();
        if (m.z == 1) v.z = taichi_cell(T, mask, i + 2, iy, ix, nx, ny, c.z, Fo_x, Fo_y);
        next();
        if (m.w == 1) v.w = taichi_cell(T, mask, i + 3, iy, ix, nx, ny, c.w, Fo_x, Fo_y);
      }
      reinterpret_cast<float4*>(Tn)[q] = v;
    }
  }
  for (unsigned e = (unsigned)done + t0; e < (unsigned)N; e += stride) {  // may end above 2^31
    const int i = (int)e;
    const float c = T[i];
    const int iy = i / nx, ix = i - iy * nx;
    Tn[i] = __ldg(mask + i) == 1 ? taichi_cell(T, mask, i, iy, ix, nx, ny, c, Fo_x, Fo_y) : c;
  }
}

// ------------------------------------------------------------------ cell-key radix sort
// Stable LSD radix sort of (key, index) pairs, RADIX_BITS per pass; identical permutation
// to np.argsort(key, kind="stable").  Per pass: tile digit histograms, a digit-major exclusive
// scan, and a stable scatter.  A thread's elements of a tile are loaded at once and ranked by
// its warp alone (one block barrier instead of three for every 256 elements, and one exposed
// load instead of eight): a pass of 80k particles 44 -> 22 us, of 6M 95 -> 62, of 48M 820 -> 700.
__global__ void k_sort_keys(const float* x, const float* y, const int* n_dev, int nx, int ny, float dxf, float dyf,
                            uint32_t* key, uint32_t* val) {
  pdl_enter();
  int n = *n_dev;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    key[i] = (uint32_t)dep_cell(x[i], y[i], dxf, dyf, nx, ny);
    val[i] = (uint32_t)i;
  }
}

constexpr int SORT_PER = SORT_TILE / SORT_NT;  // elements per thread: warp w takes SORT_PER chunks of 32 in a row

__global__ void __launch_bounds__(SORT_NT) k_sort_hist(const uint32_t* key, const int* n_dev, int shift,
                                                       uint32_t* hist, int ntiles) {
  pdl_enter();
  __shared__ uint32_t h[RADIX];
  const int n = *n_dev, tile = blockIdx.x, lane = threadIdx.x & 31;
  const int i0 = tile * SORT_TILE + (int)(threadIdx.x >> 5) * (32 * SORT_PER) + lane;
  uint32_t k[SORT_PER];
#pragma unroll
  for (int e = 0; e < SORT_PER; ++e) k[e] = i0 + 32 * e < n ? (key[i0 + 32 * e] >> shift) & (RADIX - 1) : RADIX;
  for (int d = threadIdx.x; d < RADIX; d += blockDim.x) h[d] = 0;
  __syncthreads();
  // where neighbours agree (sorted keys, their high digits) the lanes of one digit add once:
  // 32 adds to one word take turns; scattered digits add one by one, which a match would slow
  // (143 us against 83 on 48M keys in upload order)
#pragma unroll
  for (int e = 0; e < SORT_PER; ++e) {
    const uint32_t left = __shfl_up_sync(0xFFFFFFFFu, k[e], 1);
    if (__popc(__ballot_sync(0xFFFFFFFFu, left == k[e])) >= 8) {
      const unsigned peers = __match_any_sync(0xFFFFFFFFu, k[e]);
      if (k[e] < RADIX && (peers & ((1u << lane) - 1)) == 0) atomicAdd(&h[k[e]], (uint32_t)__popc(peers));
    } else if (k[e] < RADIX) {
      atomicAdd(&h[k[e]], 1u);
    }
  }
  __syncthreads();
  for (int d = threadIdx.x; d < RADIX; d += blockDim.x) hist[(size_t)d * ntiles + tile] = h[d];
}

// Multi-block exclusive scan of a long uint32 array: per-chunk sums (only when there are several
// chunks), then each chunk scanned from the sum of those before it, which its block adds.
constexpr int SCAN_NT = 1024, SCAN_PER = 8, SCAN_CHUNK = SCAN_NT * SCAN_PER;

__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* total) {
  __shared__ uint32_t sm[SCAN_NT / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t inc = v;
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) sm[w] = inc;
  __syncthreads();
  if (w == 0) {
    uint32_t s = lane < SCAN_NT / 32 ? sm[lane] : 0u;
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t t = __shfl_up_sync(0xFFFFFFFFu, s, o);
      if (lane >= o) s += t;
    }
    sm[lane] = s;
  }
  __syncthreads();
  const uint32_t ex = (w ? sm[w - 1] : 0u) + inc - v;
  if (total) *total = sm[SCAN_NT / 32 - 1];
  __syncthreads();
  return ex;
}

// this thread's SCAN_PER values of a chunk, zero past the end
__device__ __forceinline__ void scan_load(const uint32_t* a, int total, int base, uint32_t (&v)[SCAN_PER]) {
  if (base + SCAN_PER <= total) {
#pragma unroll
    for (int k = 0; k < SCAN_PER; k += 4) {
      const uint4 q = *reinterpret_cast<const uint4*>(a + base + k);  // a from cudaMalloc, base a multiple of 8
      v[k] = q.x; v[k + 1] = q.y; v[k + 2] = q.z; v[k + 3] = q.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < SCAN_PER; ++k) v[k] = base + k < total ? a[base + k] : 0u;
  }
}

__global__ void __launch_bounds__(SCAN_NT) k_scan_partials(const uint32_t* a, int total, uint32_t* bsum) {
  pdl_enter();
  uint32_t v[SCAN_PER], s = 0u, t;
  scan_load(a, total, blockIdx.x * SCAN_CHUNK + threadIdx.x * SCAN_PER, v);
#pragma unroll
  for (int k = 0; k < SCAN_PER; ++k) s += v[k];
  block_excl_scan(s, &t);
  if (threadIdx.x == 0) bsum[blockIdx.x] = t;
}

__global__ void __launch_bounds__(SCAN_NT) k_scan_apply(uint32_t* a, int total, const uint32_t* bsum) {
  pdl_enter();
  const int base = blockIdx.x * SCAN_CHUNK + threadIdx.x * SCAN_PER;
  uint32_t v[SCAN_PER], s = 0u, before = 0u, first = 0u;
  scan_load(a, total, base, v);
  if (blockIdx.x > 0) {
    for (int b = threadIdx.x; b < (int)blockIdx.x; b += SCAN_NT) before += bsum[b];
    block_excl_scan(before, &first);
  }
#pragma unroll
  for (int k = 0; k < SCAN_PER; ++k) s += v[k];
  uint32_t ex = block_excl_scan(s, nullptr) + first;
#pragma unroll
  for (int k = 0; k < SCAN_PER; ++k) {
    if (base + k < total) a[base + k] = ex;
    ex += v[k];
  }
}

// stable scatter: each warp ranks its elements per digit in index order, then the digits'
// counts are summed over the warps before it
__global__ void __launch_bounds__(SORT_NT) k_sort_scatter(const uint32_t* key, const uint32_t* val, const int* n_dev,
                                                          int shift, const uint32_t* offs, int ntiles,
                                                          uint32_t* key_out, uint32_t* val_out) {
  pdl_enter();
  constexpr int NW = SORT_NT / 32;
  __shared__ uint32_t count[NW][RADIX];
  const int n = *n_dev, tile = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i0 = tile * SORT_TILE + w * (32 * SORT_PER) + lane;
  uint32_t k[SORT_PER], v[SORT_PER], r[SORT_PER];
#pragma unroll
  for (int e = 0; e < SORT_PER; ++e) {
    const bool in = i0 + 32 * e < n;
    k[e] = in ? key[i0 + 32 * e] : 0u;
    v[e] = in ? val[i0 + 32 * e] : 0u;
  }
  static_assert(RADIX <= SORT_NT, "one thread per digit");
  const uint32_t off = threadIdx.x < RADIX ? offs[(size_t)threadIdx.x * ntiles + tile] : 0u;
  for (int d = lane; d < RADIX; d += 32) count[w][d] = 0u;
  __syncwarp();
#pragma unroll
  for (int e = 0; e < SORT_PER; ++e) {
    const bool in = i0 + 32 * e < n;
    const uint32_t d = (k[e] >> shift) & (RADIX - 1);
    const unsigned peers = __match_any_sync(0xFFFFFFFFu, in ? d : RADIX), before = peers & ((1u << lane) - 1);
    r[e] = in ? count[w][d] + __popc(before) : 0u;
    __syncwarp();
    if (in && before == 0) count[w][d] += __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  if (threadIdx.x < RADIX) {
    uint32_t at = off;
#pragma unroll
    for (int q = 0; q < NW; ++q) {
      const uint32_t c = count[q][threadIdx.x];
      count[q][threadIdx.x] = at;
      at += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int e = 0; e < SORT_PER; ++e) {
    if (i0 + 32 * e >= n) continue;
    const uint32_t pos = count[w][(k[e] >> shift) & (RADIX - 1)] + r[e];
    key_out[pos] = k[e];
    val_out[pos] = v[e];
  }
}

// gather one species' SoA through the permutation
__global__ void k_sort_gather(Soa src, Soa dst, const uint32_t* perm, const int* n_dev) {
  pdl_enter();
  int n = *n_dev;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint32_t j = perm[i];
    dst.x[i] = src.x[j]; dst.y[i] = src.y[j];
    dst.vx[i] = src.vx[j]; dst.vy[i] = src.vy[j]; dst.vz[i] = src.vz[j];
    dst.id[i] = src.id[j];
    if (src.cex) dst.cex[i] = src.cex[j];
  }
}

// one array through the permutation (an upload's arrays arrive one by one)
template <class T>
__global__ void __launch_bounds__(256) k_gather(const T* __restrict__ src, T* __restrict__ dst,
                                                const uint32_t* __restrict__ perm, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[i] = src[perm[i]];
}

// *top = max(*top, ids): one uint32 per thread and turn, 16 bytes where the array allows
__global__ void __launch_bounds__(256) k_max_id(const uint32_t* __restrict__ id, int n, uint32_t* top) {
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  uint32_t m = 0u;
  const int n4 = (reinterpret_cast<uintptr_t>(id) & 15u) == 0 ? n >> 2 : 0;
  for (int q = t0; q < n4; q += stride) {
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(id) + q);
    m = max(max(m, max(v.x, v.y)), max(v.z, v.w));
  }
  for (int i = 4 * n4 + t0; i < n; i += stride) m = max(m, id[i]);
  m = __reduce_max_sync(0xFFFFFFFFu, m);
  if ((threadIdx.x & 31) == 0 && m) atomicMax(top, m);
}

// copy the device count to another slot (num_dst of a sort = num_src)
__global__ void k_copy_int(const int* a, int* b) { pdl_enter(); *b = *a; }

// ------------------------------------------------------------------ distance to electrodes
// Chebyshev distance (in cells, capped at BDIST_CAP) from every node to the nearest bound
// node; the ion step uses it to skip path samples that cannot reach a bound cell.  Cells
// only ever leave isBound during a run (erosion), so the map stays a lower bound.
constexpr int BDIST_CAP = 15;

__global__ void k_bdist_rows(const uint8_t* __restrict__ isBound, uint8_t* hrow, int ny, int nx) {
  pdl_enter();
  const int N = ny * nx;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
    const int y = i / nx, x = i - y * nx;
    int best = BDIST_CAP;
    for (int d = 0; d < BDIST_CAP; ++d)
      if ((x - d >= 0 && isBound[i - d]) || (x + d < nx && isBound[i + d])) { best = d; break; }
    hrow[i] = (uint8_t)best;
  }
}

__global__ void k_bdist_cols(const uint8_t* __restrict__ hrow, uint8_t* dist, int ny, int nx) {
  pdl_enter();
  const int N = ny * nx;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
    const int y = i / nx, x = i - y * nx;
    int best = BDIST_CAP;
    for (int dy = -(BDIST_CAP - 1); dy <= BDIST_CAP - 1; ++dy) {
      const int yy = y + dy;
      if (yy < 0 || yy >= ny) continue;
      const int ady = dy < 0 ? -dy : dy;
      const int v = max(ady, (int)hrow[yy * nx + x]);
      best = min(best, v);
    }
    dist[i] = (uint8_t)best;
  }
}

// ------------------------------------------------------------------ NumPy float32 sums
// np.sum of a C-contiguous float32 array is 0 + pw(a, n), where pw is NumPy's pairwise
// summation: for n < 8 a running sum from 0; for 8 <= n <= 128 eight running sums over
// a[q], a[q + 8], ... (q = 0..7, started at a[q]) while a full group of eight remains,
// combined as ((r0 + r1) + (r2 + r3)) + ((r4 + r5) + (r6 + r7)), then the remaining
// elements in order; above 128, pw(a, m) + pw(a + m, n - m) with m = n / 2 rounded down to
// a multiple of 8.  All in float32.  The host lays out that tree for n (leaf ranges, and
// the internal nodes by height); k_pw_leaves sums the leaves and k_pw_combine the internal
// nodes, so the result is NumPy's, bit for bit.  Element i is a_i^2 + b_i^2 (+ c_i^2),
// rounded as NumPy evaluates a**2 + b**2 + c**2 on float32 arrays.
struct PwSrc {
  const float* a;
  const float* b;
  const float* c;  // may be null
};

__device__ __forceinline__ float pw_elem(const PwSrc& s, long long i) {
  const float a = __ldg(s.a + i), b = __ldg(s.b + i);
  float v = __fadd_rn(__fmul_rn(a, a), __fmul_rn(b, b));
  if (s.c) {
    const float c = __ldg(s.c + i);
    v = __fadd_rn(v, __fmul_rn(c, c));
  }
  return v;
}

__global__ void k_pw_leaves(PwSrc src, const long long* __restrict__ leaf_lo, int nleaves, float* vals) {
  pdl_enter();
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nleaves; k += gridDim.x * blockDim.x) {
    const long long lo = leaf_lo[k];
    const int n = (int)(leaf_lo[k + 1] - lo);
    float res;
    if (n < 8) {
      res = 0.0f;
      for (int i = 0; i < n; ++i) res = __fadd_rn(res, pw_elem(src, lo + i));
    } else {
      float r[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) r[q] = pw_elem(src, lo + q);
      int i = 8;
      for (; i < n - (n % 8); i += 8) {
#pragma unroll
        for (int q = 0; q < 8; ++q) r[q] = __fadd_rn(r[q], pw_elem(src, lo + i + q));
      }
      res = __fadd_rn(__fadd_rn(__fadd_rn(r[0], r[1]), __fadd_rn(r[2], r[3])),
                      __fadd_rn(__fadd_rn(r[4], r[5]), __fadd_rn(r[6], r[7])));
      for (; i < n; ++i) res = __fadd_rn(res, pw_elem(src, lo + i));
    }
    vals[k] = res;
  }
}

// one block: internal node j (height order) = vals[left[j]] + vals[right[j]], stored at
// vals[nleaves + j]; then *out = 0 + the root (root < 0: no elements)
__global__ void k_pw_combine(float* vals, const int* __restrict__ left, const int* __restrict__ right,
                             const int* __restrict__ height_off, int nheights, int nleaves, int root, float* out) {
  pdl_enter();
  for (int h = 0; h < nheights; ++h) {
    for (int j = height_off[h] + (int)threadIdx.x; j < height_off[h + 1]; j += blockDim.x)
      vals[nleaves + j] = __fadd_rn(vals[left[j]], vals[right[j]]);
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = __fadd_rn(0.0f, root >= 0 ? vals[root] : 0.0f);
}

}  // namespace pb

// Particle kernels of the PIC-MCC step for sm_100a.
//
//  * boris_push_one      bilinear E (and B) gather + 2D3V Boris + drift, in the exact
//                        operation order and precision of push_particles_boris_cpu
//                        (Python/physics_engine.py:188-254): float32 cell indices,
//                        float64 weights and velocity update, float32 drift in mm.
//  * k_push_boris        one push over caller arrays (module-level function signature).
//  * k_count_cells       NGP cell counts clip(rint(x/dx), 1, n-2), warp-aggregated.
//  * k_rho_finalize      rho from counts: the exact float32 result of the reference's
//                        sequential np.add.at (ions, then electrons).
//  * k_substep_reduce,   max predicted displacement of compute_particle_substeps (:928-966), one
//    k_substep_both      species (module call) or both of a step.
//  * k_segment_hits      8-sample path absorption test (_segment_hits_grid, :1880-1901).
//  * k_ion_step          the fused ion timestep: n_sub pushes, periodic wrap, final-cell and
//                        path hits, impact heating, SEE spawn records, sputter damage, exit
//                        diagnostics, stable compaction (single pass, decoupled look-back),
//                        CEX collision, PPC and next-step deposit counts (:1166-1739).
//  * k_ele_step          the fused electron timestep: pushes, wrap, purge (:1534-1561).
#include "pb_kernels.cuh"

namespace pb {

constexpr int NT = 256;    // threads per block of the step kernels
constexpr int IPT = 4;     // particles per thread of the default tile
constexpr int TILE = NT * IPT;       // particles per block and tile (default)
constexpr int TILE_MIN = NT * 2;     // the smaller tile of the particles-per-block knob
constexpr long long SPIN_LIMIT = 1ll << 22;  // polls of a predecessor tile (~1-2 s) before giving up

// ------------------------------------------------------------------ field gather + push
__device__ __forceinline__ double gather4(const float* __restrict__ F, size_t r0, size_t r1, int ix0, int ix1,
                                          double w00, double w10, double w01, double w11) {
  double a = DMUL((double)__ldg(F + r0 + ix0), w00);
  double b = DMUL((double)__ldg(F + r0 + ix1), w10);
  double c = DMUL((double)__ldg(F + r1 + ix0), w01);
  double d = DMUL((double)__ldg(F + r1 + ix1), w11);
  return DADD(DADD(DADD(a, b), c), d);
}

// The two float4 of one cell's corners (32 bytes, 32-byte aligned) in one load.  A gather of
// particles in scattered cells is bound by the cache's tag lookups, one per lane and load
// instruction, so one 256-bit load instead of two of 128 bits halves them.
__device__ __forceinline__ void ldg_corners(const float4* __restrict__ p, float4& a, float4& b) {
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
      : "l"(p));
}

// The same from the per-cell corner array: Ec[2c] holds Ex at (iy0, ix0), (iy0, ix0 + 1),
// (iy0 + 1, ix0), (iy0 + 1, ix0 + 1) of cell c = iy0 * nx + ix0, Ec[2c + 1] the same of
// Ey: one 16-byte load per component instead of four scalar loads, same arithmetic.
__device__ __forceinline__ void gather4v(const float4 a, const float4 b, double w00, double w10, double w01,
                                         double w11, double& ex, double& ey) {
  ex = DADD(DADD(DADD(DMUL((double)a.x, w00), DMUL((double)a.y, w10)), DMUL((double)a.z, w01)),
            DMUL((double)a.w, w11));
  ey = DADD(DADD(DADD(DMUL((double)b.x, w00), DMUL((double)b.y, w10)), DMUL((double)b.z, w01)),
            DMUL((double)b.w, w11));
}
__device__ __forceinline__ void gather4c(const float4* __restrict__ Ec, size_t c, double w00, double w10,
                                         double w01, double w11, double& ex, double& ey) {
  float4 a, b;
  ldg_corners(Ec + 2 * c, a, b);
  gather4v(a, b, w00, w10, w01, w11, ex, ey);
}

// The window of the corner array staged in shared memory for a tile (PB_OPT_TMA_TILE):
// cells [bx, bx + TB_W) x [by, by + TB_H); cells outside it are read from global memory.
struct EBox {
  const float4* box;  // nullptr: no window staged
  int bx, by;
};

// Builds the corner array from Ex and Ey (cells of the last row and column are not used:
// the gather clamps the lower corner to ny - 2, nx - 2).  With ebound, also the largest
// |Ex| + |Ey| over the nodes (every node is a corner of some cell), as float bits through
// an unsigned max: a NaN (0x7FC00000) or infinity wins, which disables the bound below.
__global__ void k_e_corners(const float* __restrict__ Ex, const float* __restrict__ Ey, float4* __restrict__ Ec,
                            int ny, int nx, unsigned* ebound) {
  pdl_enter();
  const int N = ny * nx;
  unsigned m = 0u;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < N; c += gridDim.x * blockDim.x) {
    const int iy = c / nx, ix = c - iy * nx;
    if (iy >= ny - 1 || ix >= nx - 1) continue;
    const int r1 = c + nx;
    const float4 a = make_float4(__ldg(Ex + c), __ldg(Ex + c + 1), __ldg(Ex + r1), __ldg(Ex + r1 + 1));
    const float4 b = make_float4(__ldg(Ey + c), __ldg(Ey + c + 1), __ldg(Ey + r1), __ldg(Ey + r1 + 1));
    Ec[2 * c] = a;
    Ec[2 * c + 1] = b;
    m = max(m, max(max(__float_as_uint(fabsf(a.x) + fabsf(b.x)), __float_as_uint(fabsf(a.y) + fabsf(b.y))),
                   max(__float_as_uint(fabsf(a.z) + fabsf(b.z)), __float_as_uint(fabsf(a.w) + fabsf(b.w)))));
  }
  if (!ebound) return;
  __shared__ unsigned wm[32];
  m = __reduce_max_sync(0xFFFFFFFFu, m);
  if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = threadIdx.x < (blockDim.x >> 5) ? wm[threadIdx.x] : 0u;
    m = __reduce_max_sync(0xFFFFFFFFu, m);
    if (threadIdx.x == 0 && m) atomicMax(ebound, m);
  }
}

// HAS_B = false: the B arrays are all +0 (the simulator never writes them), so
// t = h * (+0) is a signed zero, t2 = +0 and 1 + t2 = 1 exactly; s = 2 t / 1 = 2 t.  The
// remaining operations are kept, so signed zeros come out as in the reference.
// floor(q) as an int and the fraction q - floor(q), exactly and without conversion
// instructions, for 0 <= q < 2^22: adding 2^23 with rounding down leaves floor(q) in the
// low mantissa bits of the sum, and q minus the floor is exact in float.  Returns whether
// q is in that range (false for NaN); fl and frac are meaningful only then, and the
// caller takes the general path otherwise.  No branch, so that the callers can test both
// coordinates with one.
__device__ __forceinline__ bool floor_frac(float q, int& fl, float& frac) {
  const float t = __fadd_rd(q, 8388608.0f);
  fl = __float_as_int(t) - 0x4B000000;
  frac = __fsub_rn(q, __fsub_rn(t, 8388608.0f));
  return (q >= 0.0f) & (q < 4194304.0f);
}

// RN(x / d) without the reciprocal instruction: q = x * inv (inv = RN(1/d)) and one
// Markstein correction q += (x - q d) inv, accepted when |x - q d| < ulp(q) |d| / 2.  The
// residual is exact (one FMA) for q within an ulp of x / d, and a quotient of two floats
// is never a midpoint, so the test holds exactly when q is the correctly rounded quotient.
// Zero, powers of two (whose lower half-ulp is smaller), tiny and non-finite q fail the
// test.  Checked on the host against IEEE division for every float |x| < 64 and ten grid
// spacings: no mismatch, the test accepts 84% of those inputs (nearly all positions in a
// grid).  div_fast returns whether q is accepted, without a branch.
__device__ __forceinline__ bool div_fast(float x, float d, float inv, float& q) {
  q = __fmul_rn(x, inv);
  q = __fmaf_rn(__fmaf_rn(-q, d, x), inv, q);
  const float r = __fmaf_rn(-q, d, x);
  const unsigned int b = __float_as_uint(q), e = b & 0x7F800000u;
  const float h = __fmul_rn(__uint_as_float((e - (24u << 23)) & 0x7F800000u), fabsf(d));
  return (e > (26u << 23)) & (e < 0x7F800000u) & ((b & 0x007FFFFFu) != 0u) & (fabsf(r) < h);
}
// RN(x / d) by bracketing, without the division instruction.  q0 = RN(x inv) (inv =
// RN(1/d)) is within 1.5 ulp of x / d, and r0 = RN(q0 d - x) (one FMA) is within a relative
// 2^-24 of the exact q0 d - x when it is a normal float.  The exact quotient is
// x / d = q0 - (q0 d - x) / d, and lo <= (1/d)(1 - 2^-24), hi >= (1/d)(1 + 2^-24) (inv moved
// two float steps down and up), so x / d lies between q0 - r0 lo and q0 - r0 hi.  Rounding
// is monotone: when qa = RN(q0 - r0 lo) and qb = RN(q0 - r0 hi) (one FMA each) are equal,
// RN(x / d) is that value.  |x| >= 2^-80 keeps r0 out of the subnormal range; NaN, infinite
// and overflowing quotients give NaN or unequal values, and NaN brackets never agree.  The
// test fails only when x / d lies within about 2^-22 ulp of a rounding midpoint.  Returns
// whether q is accepted, without a branch (k_div_check counts misses over every float x).
__device__ __forceinline__ bool div_bracket(float x, float d, float inv, float lo, float hi, float& q) {
  const float q0 = __fmul_rn(x, inv);
  const float r0 = __fmaf_rn(q0, d, -x);
  q = __fmaf_rn(-r0, lo, q0);
  const float qb = __fmaf_rn(-r0, hi, q0);
  return (q == qb) & (fabsf(x) >= 0x1p-80f);
}

// Checks div_bracket for one spacing over all 2^32 bit patterns of x: out[0] counts the
// accepted quotients that differ in any bit from __fdiv_rn(x, d); out[1] the rejected x
// among those a grid's cells can hold (x >= 2^-80, x / d < 2^22); out[2] all such x.
__global__ void k_div_check(float d, unsigned long long* out) {
  float inv, lo, hi;
  rcp_axis(d, inv, lo, hi);
  unsigned long long miss = 0, rej = 0, cand = 0;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long k = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; k < (1ull << 32);
       k += stride) {
    const float x = __uint_as_float((unsigned)k);
    const float qd = __fdiv_rn(x, d);
    float q;
    const bool ok = div_bracket(x, d, inv, lo, hi, q);
    if (ok && __float_as_uint(q) != __float_as_uint(qd)) ++miss;
    if (x >= 0x1p-80f && qd < 4194304.0f) {
      ++cand;
      if (!ok) ++rej;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    miss += __shfl_xor_sync(0xFFFFFFFFu, miss, o);
    rej += __shfl_xor_sync(0xFFFFFFFFu, rej, o);
    cand += __shfl_xor_sync(0xFFFFFFFFu, cand, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (miss) atomicAdd(out, miss);
    if (rej) atomicAdd(out + 1, rej);
    if (cand) atomicAdd(out + 2, cand);
  }
}

// The same with a branch per quotient, for callers that need one quotient at a time.
__device__ __forceinline__ float div_rn_checked(float x, float d, float inv) {
  float q = __fmul_rn(x, inv);
  q = __fmaf_rn(__fmaf_rn(-q, d, x), inv, q);
  const float r = __fmaf_rn(-q, d, x);
  const unsigned int b = __float_as_uint(q), e = b & 0x7F800000u;
  if (e > (26u << 23) && e < 0x7F800000u && (b & 0x007FFFFFu) != 0u) {
    const float h = __fmul_rn(__uint_as_float(e - (24u << 23)), fabsf(d));
    if (fabsf(r) < h) return q;
  }
  return __fdiv_rn(x, d);
}

// CORN: E is gathered from the corner array Ec (B = 0 only); otherwise from Ex, Ey.
// LIGHT: the cell position from div_fast and, inside the grid, the cell index and fraction
// from floor_frac, each pair tested with one branch: six fewer XU-pipe instructions
// (reciprocal and conversions) per substep.  The step kernels are bound by instruction
// issue and use it (measured 7% faster for the ion step, whose 64 registers it does not
// raise); the module-level push and the B != 0 path keep the plain division.
// Cell and bilinear weights of a push at (x, y): float32 quotients x / dx, y / dy, the
// clamped floor cell (ix0, iy0) and the float64 weights of the reference's gather.
template <bool LIGHT>
__device__ __forceinline__ void push_cell(float x, float y, int nx, int ny, float dxf, float dyf, const Rcp& rc,
                                          float* q_start, int& ix0, int& iy0, double& w00, double& w10,
                                          double& w01, double& w11) {
  float ixf, iyf;
  if (LIGHT) {
    const bool okq = div_bracket(x, dxf, rc.ix, rc.ix_lo, rc.ix_hi, ixf) &
                     div_bracket(y, dyf, rc.iy, rc.iy_lo, rc.iy_hi, iyf);
    if (!okq) { ixf = __fdiv_rn(x, dxf); iyf = __fdiv_rn(y, dyf); }
  } else {
    ixf = __fdiv_rn(x, dxf);
    iyf = __fdiv_rn(y, dyf);
  }
  double fx, fy;
  // inside the grid the clamp is a no-op and ixf - ix0 is the exact float fraction
  int fxi, fyi;
  float frx, fry;
  bool inside = false;
  if (LIGHT) {
    // one unsigned compare per coordinate: a floor in [0, n - 2] (n - 2 < 2^22) from the
    // rounded-down sum implies 0 <= q < n - 1, the range floor_frac needs; negative, huge,
    // infinite and NaN q give a floor outside it (tests/test_div_method.py)
    floor_frac(ixf, fxi, frx);
    floor_frac(iyf, fyi, fry);
    inside = ((unsigned)fxi <= (unsigned)(nx - 2)) & ((unsigned)fyi <= (unsigned)(ny - 2));
  }
  if (inside) {
    ix0 = fxi;
    iy0 = fyi;
    fx = (double)frx;
    fy = (double)fry;
  } else {
    ix0 = clampi(np_f2i32(floorf(ixf)), 0, nx - 2);
    iy0 = clampi(np_f2i32(floorf(iyf)), 0, ny - 2);
    fx = DSUB((double)ixf, (double)ix0);
    fy = DSUB((double)iyf, (double)iy0);
  }
  if (q_start) { q_start[0] = ixf; q_start[1] = iyf; }  // x / dx, y / dy at the start position
  const double gx = DSUB(1.0, fx), gy = DSUB(1.0, fy);
  w00 = DMUL(gx, gy); w10 = DMUL(fx, gy); w01 = DMUL(gx, fy); w11 = DMUL(fx, fy);
}

// A float as a double scaled by 2^-896, from its bits (sign, then the 8 exponent bits as the
// low bits of the 11-bit exponent, then the mantissa): exact for every finite float, zero
// and subnormals included, with integer instructions instead of the conversion unit.
// Infinities and NaN come out finite, so it is used only on values known to be finite.
__device__ __forceinline__ double f2d_scaled(float f) {
  const int b = __float_as_int(f);
  return __hiloint2double((b >> 3) & (int)0x8FFFFFFF, (int)((unsigned)b << 29));
}

// Half kick, rotation (B = 0: t = s = h * (+0)), half kick and drift from the gathered E.
// VBITS (callers know vx, vy finite): vx and vy become doubles by their bits, and
// RN(vx 2^-896 * 2^896 + h ex) in one FMA is the rounded sum of the converted value.
template <bool VBITS = false>
__device__ __forceinline__ void push_update_b0(float& x, float& y, float& vx, float& vy, float& vz, double ex,
                                               double ey, double h, float dtf) {
  const double vmx = VBITS ? __fma_rn(f2d_scaled(vx), 0x1p896, DMUL(h, ex)) : DADD((double)vx, DMUL(h, ex));
  const double vmy = VBITS ? __fma_rn(f2d_scaled(vy), 0x1p896, DMUL(h, ey)) : DADD((double)vy, DMUL(h, ey));
  if ((vmx != 0.0) & (vmy != 0.0) & (vz != 0.0f) & (fabs(vmx) < INFINITY) & (fabs(vmy) < INFINITY) &
      (fabsf(vz) < INFINITY)) {
    // every cross-product term below is a signed zero (t = s = h * (+0)), and a finite
    // nonzero value plus a zero is that value: the rotation is the identity, bit for bit
    // (vz goes to double and back unchanged, so it is left as it is)
    vx = __double2float_rn(DADD(vmx, DMUL(h, ex)));
    vy = __double2float_rn(DADD(vmy, DMUL(h, ey)));
    x = __fadd_rn(x, __fmul_rn(__fmul_rn(vx, dtf), 1000.0f));
    y = __fadd_rn(y, __fmul_rn(__fmul_rn(vy, dtf), 1000.0f));
    return;
  }
  const double vmz = (double)vz;
  const double tx = DMUL(h, 0.0), ty = tx, tz = tx;
  const double sx = DMUL(2.0, tx), sy = sx, sz = sx;
  const double vpx = DADD(vmx, DSUB(DMUL(vmy, tz), DMUL(vmz, ty)));
  const double vpy = DADD(vmy, DSUB(DMUL(vmz, tx), DMUL(vmx, tz)));
  const double vpz = DADD(vmz, DSUB(DMUL(vmx, ty), DMUL(vmy, tx)));
  const double wx = DADD(vmx, DSUB(DMUL(vpy, sz), DMUL(vpz, sy)));
  const double wy = DADD(vmy, DSUB(DMUL(vpz, sx), DMUL(vpx, sz)));
  const double wz = DADD(vmz, DSUB(DMUL(vpx, sy), DMUL(vpy, sx)));
  vx = __double2float_rn(DADD(wx, DMUL(h, ex)));
  vy = __double2float_rn(DADD(wy, DMUL(h, ey)));
  vz = __double2float_rn(wz);
  x = __fadd_rn(x, __fmul_rn(__fmul_rn(vx, dtf), 1000.0f));
  y = __fadd_rn(y, __fmul_rn(__fmul_rn(vy, dtf), 1000.0f));
}

// Half kick, rotation, half kick and drift from the gathered E and B.
__device__ __forceinline__ void push_update_b(float& x, float& y, float& vx, float& vy, float& vz, double ex, double ey,
                                              double bx, double by, double bz, double h, float dtf) {
  const double vmx = DADD((double)vx, DMUL(h, ex));
  const double vmy = DADD((double)vy, DMUL(h, ey));
  const double vmz = (double)vz;
  const double tx = DMUL(h, bx), ty = DMUL(h, by), tz = DMUL(h, bz);
  const double t2 = DADD(DADD(DMUL(tx, tx), DMUL(ty, ty)), DMUL(tz, tz));
  const double den = DADD(1.0, t2);
  const double sx = DDIV(DMUL(2.0, tx), den), sy = DDIV(DMUL(2.0, ty), den), sz = DDIV(DMUL(2.0, tz), den);
  const double vpx = DADD(vmx, DSUB(DMUL(vmy, tz), DMUL(vmz, ty)));
  const double vpy = DADD(vmy, DSUB(DMUL(vmz, tx), DMUL(vmx, tz)));
  const double vpz = DADD(vmz, DSUB(DMUL(vmx, ty), DMUL(vmy, tx)));
  const double wx = DADD(vmx, DSUB(DMUL(vpy, sz), DMUL(vpz, sy)));
  const double wy = DADD(vmy, DSUB(DMUL(vpz, sx), DMUL(vpx, sz)));
  const double wz = DADD(vmz, DSUB(DMUL(vpx, sy), DMUL(vpy, sx)));
  vx = __double2float_rn(DADD(wx, DMUL(h, ex)));
  vy = __double2float_rn(DADD(wy, DMUL(h, ey)));
  vz = __double2float_rn(wz);
  x = __fadd_rn(x, __fmul_rn(__fmul_rn(vx, dtf), 1000.0f));
  y = __fadd_rn(y, __fmul_rn(__fmul_rn(vy, dtf), 1000.0f));
}

template <bool HAS_B, bool CORN = false, bool LIGHT = false>
__device__ __forceinline__ void boris_push_one(float& x, float& y, float& vx, float& vy, float& vz,
                                               const float* __restrict__ Ex, const float* __restrict__ Ey,
                                               const float* __restrict__ Bx, const float* __restrict__ By,
                                               const float* __restrict__ Bz, int nx, int ny,
                                               float dxf, float dyf, double h, float dtf,
                                               const float4* __restrict__ Ec = nullptr, Rcp rc = Rcp{},
                                               float* q_start = nullptr,
                                               EBox eb = EBox{nullptr, 0, 0}) {
  static_assert(!(HAS_B && CORN), "the corner gather has no B field");
  int ix0, iy0;
  double w00, w10, w01, w11;
  push_cell<LIGHT>(x, y, nx, ny, dxf, dyf, rc, q_start, ix0, iy0, w00, w10, w01, w11);
  int ix1 = min(ix0 + 1, nx - 1);
  int iy1 = min(iy0 + 1, ny - 1);
  size_t r0 = (size_t)iy0 * nx, r1 = (size_t)iy1 * nx;
  double ex, ey;
  if (CORN) {
    const unsigned ox = (unsigned)(ix0 - eb.bx), oy = (unsigned)(iy0 - eb.by);
    if (eb.box && ox < (unsigned)TB_W && oy < (unsigned)TB_H) {
      const float4* q = eb.box + 2 * (oy * TB_W + ox);
      gather4v(q[0], q[1], w00, w10, w01, w11, ex, ey);
    } else {
      if (LIGHT) {  // 32-bit cell index (a grid has fewer than 2^30 cells): fewer instructions
        float4 ea, eb4;
        ldg_corners(Ec + 2 * (iy0 * nx + ix0), ea, eb4);
        gather4v(ea, eb4, w00, w10, w01, w11, ex, ey);
      } else {
        gather4c(Ec, r0 + ix0, w00, w10, w01, w11, ex, ey);
      }
    }
  } else {
    ex = gather4(Ex, r0, r1, ix0, ix1, w00, w10, w01, w11);
    ey = gather4(Ey, r0, r1, ix0, ix1, w00, w10, w01, w11);
  }
  if (!HAS_B) {
    push_update_b0(x, y, vx, vy, vz, ex, ey, h, dtf);
    return;
  }
  const double bx = gather4(Bx, r0, r1, ix0, ix1, w00, w10, w01, w11);
  const double by = gather4(By, r0, r1, ix0, ix1, w00, w10, w01, w11);
  const double bz = gather4(Bz, r0, r1, ix0, ix1, w00, w10, w01, w11);
  push_update_b(x, y, vx, vy, vz, ex, ey, bx, by, bz, h, dtf);
}

// Two electrons pushed n_sub times side by side (PB_OPT_ELE_PAIRS): both cells and both
// corner loads are issued before either particle's arithmetic, so one particle's load
// latency overlaps the other's.  Each particle's operations are those of boris_push_one.
__device__ __forceinline__ void push_pair_b0(float (&x)[2], float (&y)[2], float (&vx)[2], float (&vy)[2],
                                             float (&vz)[2], int n_sub, const float4* __restrict__ Ec, int nx,
                                             int ny, float dxf, float dyf, const Rcp& rc, double h, float dtf) {
  for (int s = 0; s < n_sub; ++s) {
    int ix0[2], iy0[2];
    double w[2][4];
    float4 A[2], B[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      push_cell<true>(x[q], y[q], nx, ny, dxf, dyf, rc, nullptr, ix0[q], iy0[q], w[q][0], w[q][1],
                      w[q][2], w[q][3]);
      const size_t c = (size_t)iy0[q] * nx + ix0[q];
      ldg_corners(Ec + 2 * c, A[q], B[q]);
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      double ex, ey;
      gather4v(A[q], B[q], w[q][0], w[q][1], w[q][2], w[q][3], ex, ey);
      push_update_b0(x[q], y[q], vx[q], vy[q], vz[q], ex, ey, h, dtf);
    }
  }
}

// n_sub from the reduced displacement: max(1, ceil(ds_max / max(ds_lim, 1e-30)))
__device__ __forceinline__ int substep_count(double ds_max, double ds_lim, uint32_t* errflags) {
  double lim = ds_lim > 1e-30 ? ds_lim : 1e-30;
  double q = ceil(DDIV(ds_max, lim));
  if (!(q == q)) { if (errflags) atomicOr(errflags, PB_EF_NAN_SUBSTEP); return 1; }
  if (q > 65536.0) { if (errflags) atomicOr(errflags, PB_EF_SUBSTEP_CAP); return 65536; }
  int n = (int)q;
  return n < 1 ? 1 : n;
}

// ------------------------------------------------------------------ standalone push
// The module kernels' indexes past the last whole vector are unsigned: a count may be close to
// 2^31, and the index that ends a loop is up to a grid's threads above it.
__global__ void k_push_boris(float* x, float* y, float* vx, float* vy, float* vz, const float* Ex,
                             const float* Ey, const float* Bx, const float* By, const float* Bz, int n,
                             int nx, int ny, float dxf, float dyf, double h, float dtf) {
  pdl_enter();
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < (unsigned)n; i += gridDim.x * blockDim.x) {
    float a = x[i], b = y[i], c = vx[i], d = vy[i], e = vz[i];
    boris_push_one<true>(a, b, c, d, e, Ex, Ey, Bx, By, Bz, nx, ny, dxf, dyf, h, dtf);
    x[i] = a; y[i] = b; vx[i] = c; vy[i] = d; vz[i] = e;
  }
}

// ------------------------------------------------------------------ standalone push, many particles
// With many particles per cell the push above is bound by the sectors of its 20 scalar
// gathers (ten 32-byte sectors a particle: L1 94% and L2 72% busy, DRAM 8%, 878 us for 16M
// ions on 513 x 2049).  Packing the corners of every cell first (as the step does) makes E one
// sector a particle and B two, for one pass over the grid.  k_push_corners packs E and leaves
// per block whether any B bit is set; with every B value +0 (the reference's step) the B = 0
// push is the same operation (boris_push_one) and no B is gathered, otherwise k_push_bcorners
// packs B too.  Both pushes are launched and the wrong one returns at once, so the host need
// not wait for the flag.  16M ions on 513 x 2049: 878 us before, 170 us packed (143 us of it
// the push, 640 MB of particle state: 4.5 TB/s); with a B field 880 and 435 us.
constexpr int PUSH_FLAGS = 1184;  // blocks of k_push_corners, one flag each

__global__ void __launch_bounds__(256) k_push_corners(const float* __restrict__ Ex, const float* __restrict__ Ey,
                                                      const float* __restrict__ Bx, const float* __restrict__ By,
                                                      const float* __restrict__ Bz, float4* __restrict__ Ec, int ny,
                                                      int nx, unsigned* __restrict__ bflags) {
  const int N = ny * nx;
  unsigned bits = 0u;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < N; c += gridDim.x * blockDim.x) {
    bits |= __float_as_uint(__ldg(Bx + c)) | __float_as_uint(__ldg(By + c)) | __float_as_uint(__ldg(Bz + c));
    const int iy = c / nx, ix = c - iy * nx;
    if (iy >= ny - 1 || ix >= nx - 1) continue;
    const int r1 = c + nx;
    Ec[2 * c] = make_float4(__ldg(Ex + c), __ldg(Ex + c + 1), __ldg(Ex + r1), __ldg(Ex + r1 + 1));
    Ec[2 * c + 1] = make_float4(__ldg(Ey + c), __ldg(Ey + c + 1), __ldg(Ey + r1), __ldg(Ey + r1 + 1));
  }
  const int any = __syncthreads_or(bits != 0u);
  if (threadIdx.x == 0) bflags[blockIdx.x] = any ? 1u : 0u;
}

// whether any block of k_push_corners saw a B bit (every thread of the block calls it)
__device__ __forceinline__ bool push_any_b(const unsigned* __restrict__ bflags, int nflags) {
  unsigned f = 0u;
  for (int k = threadIdx.x; k < nflags; k += blockDim.x) f |= __ldg(bflags + k);
  return __syncthreads_or(f != 0u) != 0;
}

// B corners of cell c: Bc[2 c], Bc[2 c + 1] are Bx, By at (iy0, ix0), (iy0, ix0 + 1), (iy0 + 1, ix0),
// (iy0 + 1, ix0 + 1), Bc[2 N + c] the same of Bz
__global__ void __launch_bounds__(256) k_push_bcorners(const float* __restrict__ Bx, const float* __restrict__ By,
                                                       const float* __restrict__ Bz, float4* __restrict__ Bc, int ny,
                                                       int nx, const unsigned* __restrict__ bflags, int nflags) {
  pdl_enter();
  if (!push_any_b(bflags, nflags)) return;
  const int N = ny * nx;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < N; c += gridDim.x * blockDim.x) {
    const int iy = c / nx, ix = c - iy * nx;
    if (iy >= ny - 1 || ix >= nx - 1) continue;
    const int r1 = c + nx;
    Bc[2 * c] = make_float4(__ldg(Bx + c), __ldg(Bx + c + 1), __ldg(Bx + r1), __ldg(Bx + r1 + 1));
    Bc[2 * c + 1] = make_float4(__ldg(By + c), __ldg(By + c + 1), __ldg(By + r1), __ldg(By + r1 + 1));
    Bc[2 * N + c] = make_float4(__ldg(Bz + c), __ldg(Bz + c + 1), __ldg(Bz + r1), __ldg(Bz + r1 + 1));
  }
}

template <bool HAS_B>
__device__ __forceinline__ void push_corner_one(float& x, float& y, float& vx, float& vy, float& vz,
                                                const float4* __restrict__ Ec, const float4* __restrict__ Bc, int nx,
                                                int ny, float dxf, float dyf, double h, float dtf, const Rcp& rc) {
  if (!HAS_B) {
    boris_push_one<false, true, true>(x, y, vx, vy, vz, nullptr, nullptr, nullptr, nullptr, nullptr, nx, ny, dxf, dyf, h,
                                      dtf, Ec, rc);
    return;
  }
  int ix0, iy0;
  double w00, w10, w01, w11;
  push_cell<true>(x, y, nx, ny, dxf, dyf, rc, nullptr, ix0, iy0, w00, w10, w01, w11);
  const int c = iy0 * nx + ix0;
  float4 ea, eb, ba, bb;
  ldg_corners(Ec + 2 * c, ea, eb);
  ldg_corners(Bc + 2 * c, ba, bb);
  const float4 bc = __ldg(Bc + 2 * nx * ny + c);
  double ex, ey, bx, by, bz, unused;
  gather4v(ea, eb, w00, w10, w01, w11, ex, ey);
  gather4v(ba, bb, w00, w10, w01, w11, bx, by);
  gather4v(bc, bc, w00, w10, w01, w11, bz, unused);
  push_update_b(x, y, vx, vy, vz, ex, ey, bx, by, bz, h, dtf);
}

// VEC: the five arrays start 16-byte aligned (four particles per thread and pass, 16-byte
// loads and stores); the last n % 4 particles, and all of them otherwise, go one by one.
// Four blocks an SM (64 registers): 152 us for the 16M ions, against 193 us at 78 registers,
// 169 us at 40 and 176 us one particle a thread at 32; a software prefetch of the next four
// particles (78 registers) 192 us.
template <bool HAS_B, bool VEC>
__global__ void __launch_bounds__(256, 4) k_push_corner(float* __restrict__ x, float* __restrict__ y,
                                                     float* __restrict__ vx, float* __restrict__ vy,
                                                     float* __restrict__ vz, const float4* __restrict__ Ec,
                                                     const float4* __restrict__ Bc, int n, int nx, int ny, float dxf,
                                                     float dyf, double h, float dtf, Rcp rc,
                                                     const unsigned* __restrict__ bflags, int nflags) {
  pdl_enter();
  if (push_any_b(bflags, nflags) != HAS_B) return;
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  int done = 0;
  if (VEC) {
    const int n4 = n >> 2;
    done = n4 << 2;
    for (int q = t0; q < n4; q += stride) {
      float4 X = reinterpret_cast<float4*>(x)[q], Y = reinterpret_cast<float4*>(y)[q];
      float4 U = reinterpret_cast<float4*>(vx)[q], V = reinterpret_cast<float4*>(vy)[q];
      float4 W = reinterpret_cast<float4*>(vz)[q];
      push_corner_one<HAS_B>(X.x, Y.x, U.x, V.x, W.x, Ec, Bc, nx, ny, dxf, dyf, h, dtf, rc);
      push_corner_one<HAS_B>(X.y, Y.y, U.y, V.y, W.y, Ec, Bc, nx, ny, dxf, dyf, h, dtf, rc);
      push_corner_one<HAS_B>(X.z, Y.z, U.z, V.z, W.z, Ec, Bc, nx, ny, dxf, dyf, h, dtf, rc);
      push_corner_one<HAS_B>(X.w, Y.w, U.w, V.w, W.w, Ec, Bc, nx, ny, dxf, dyf, h, dtf, rc);
      reinterpret_cast<float4*>(x)[q] = X;
      reinterpret_cast<float4*>(y)[q] = Y;
      reinterpret_cast<float4*>(vx)[q] = U;
      reinterpret_cast<float4*>(vy)[q] = V;
      reinterpret_cast<float4*>(vz)[q] = W;
    }
  }
  for (unsigned i = (unsigned)done + t0; i < (unsigned)n; i += stride) {
    float a = x[i], b = y[i], c = vx[i], d = vy[i], e = vz[i];
    push_corner_one<HAS_B>(a, b, c, d, e, Ec, Bc, nx, ny, dxf, dyf, h, dtf, rc);
    x[i] = a; y[i] = b; vx[i] = c; vy[i] = d; vz[i] = e;
  }
}

// ------------------------------------------------------------------ NGP counting
__device__ __forceinline__ void warp_count_add(int* cnt, int cell, bool valid) {
  unsigned act = __activemask();
  unsigned key = valid ? (unsigned)cell : 0xFFFFFFFFu;
  unsigned peers = __match_any_sync(act, key);
  int leader = __ffs(peers) - 1;
  if (valid && (int)(threadIdx.x & 31) == leader) atomicAdd(cnt + cell, __popc(peers));
}

// Shared-memory cell histograms of one tile (kernel option PB_OPT_SMEM_HIST).  The cells of
// the tile's kept particles are staged in shared memory; when they span fewer than HBINS
// consecutive cell keys (the usual case for particles re-sorted by cell), each warp adds
// its runs of equal cells to shared bins (one atomic per run: consecutive lanes of sorted
// particles share cells) and the block then adds every nonzero bin to the global counts
// once.  Wider tiles (particles that moved far since the last sort) count with warp-
// aggregated global atomics as before.  Counts are integers, so the result does not depend
// on the order of the additions.
constexpr int HBINS = 1024;

// bins[c] += length of the run of equal valid c that starts at this lane (run heads only)
__device__ __forceinline__ void warp_run_add(int* bins, int c, bool valid) {
  const int lane = threadIdx.x & 31;
  const int v = valid ? c : -1;
  const int prev = __shfl_up_sync(0xFFFFFFFFu, v, 1);
  const bool head = lane == 0 || v != prev;
  const unsigned heads = __ballot_sync(0xFFFFFFFFu, head);
  const unsigned later = lane == 31 ? 0u : heads & (0xFFFFFFFFu << (lane + 1));
  const int next = later ? __ffs(later) - 1 : 32;
  if (head && valid) atomicAdd(bins + c, next - lane);
}

template <int NTHR, int TILE_SZ>
__device__ __forceinline__ void tile_hist(const int* cell, const uint8_t* keep, int* gcnt, int* bins) {
  __shared__ int red[2 * (NTHR / 32)];
  int lo = INT_MAX, hi = INT_MIN;
  for (int k = threadIdx.x; k < TILE_SZ; k += NTHR)
    if (keep[k]) { lo = min(lo, cell[k]); hi = max(hi, cell[k]); }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, o));
    hi = max(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, o));
  }
  if ((threadIdx.x & 31) == 0) { red[threadIdx.x >> 5] = lo; red[NTHR / 32 + (threadIdx.x >> 5)] = hi; }
  __syncthreads();
  lo = INT_MAX; hi = INT_MIN;
#pragma unroll
  for (int j = 0; j < NTHR / 32; ++j) { lo = min(lo, red[j]); hi = max(hi, red[NTHR / 32 + j]); }
  if (hi >= lo && hi - lo < HBINS) {
    for (int k = threadIdx.x; k < TILE_SZ; k += NTHR) {
      const bool v = keep[k] != 0;
      warp_run_add(bins, v ? cell[k] - lo : 0, v);
    }
    __syncthreads();
    for (int b = threadIdx.x; b <= hi - lo; b += NTHR) {
      const int v = bins[b];
      if (v) { atomicAdd(gcnt + lo + b, v); bins[b] = 0; }
    }
  } else if (hi >= lo) {
    for (int k = threadIdx.x; k < TILE_SZ; k += NTHR) warp_count_add(gcnt, cell[k], keep[k] != 0);
  }
  __syncthreads();
}

__device__ __forceinline__ int deposit_cell(float x, float y, float dxf, float dyf, int nx, int ny) {
  int ix = cell_round32(x, dxf, 1, nx - 2);
  int iy = cell_round32(y, dyf, 1, ny - 2);
  return iy * nx + ix;
}

// Four particles per thread and pass where both arrays start 16-byte aligned.  A warp whose
// neighbouring lanes mostly share cells (particles sorted by cell) aggregates equal cells
// before the atomics; otherwise one atomic per particle: __match_any_sync over distinct cells
// takes one round per cell and bound the kernel (6M scattered ions on 257 x 1025: 53 us,
// match unit 79% busy, DRAM 11%; 42 us so, 160 G atomics/s).  Aggregation also pays where the
// warp's particles lie in few cells without being sorted, as atomics on few words take turns:
// warps whose tests often found a particle of another lane's in a cell of theirs (some 200 cells
// or fewer) aggregate too: 20M ions scattered over 20, 60 and 150 cells take 2117, 1204 and 942 us
// with plain atomics, 954, 917 and 890 us so; over all of 257 x 1025 144 and 142 us.
struct CountCrowd {
  int met = 0, turn = 0;
  bool on = false;
  // the warp's particles in cells c[0..N); tested every fourth turn
  template <int N>
  __device__ __forceinline__ void add(int* cnt, const int (&c)[N], bool valid) {
    if ((turn++ & 3) == 0) {
      const int left = __shfl_up_sync(0xFFFFFFFFu, c[0], 1), far = __shfl_xor_sync(0xFFFFFFFFu, c[0], 16);
      bool meets = false;
#pragma unroll
      for (int k = 0; k < N && k < 2; ++k) meets |= far == c[k];
      met += __any_sync(0xFFFFFFFFu, valid && meets) ? 16 : 0;
      on = __popc(__ballot_sync(0xFFFFFFFFu, valid && left == c[0])) >= 16 || met >= turn;  // a quarter of the tests
    }
    if (on) {
#pragma unroll
      for (int k = 0; k < N; ++k) warp_count_add(cnt, c[k], valid);
    } else if (valid) {
#pragma unroll
      for (int k = 0; k < N; ++k) atomicAdd(cnt + c[k], 1);
    }
  }
};

__global__ void __launch_bounds__(256, 8) k_count_cells(const float* __restrict__ x, const float* __restrict__ y,
                                                     const int* n_dev, int n_host, int start, int* cnt, int nx, int ny,
                                                     float dxf, float dyf) {
  pdl_enter();
  const int n = n_dev ? *n_dev : n_host;
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  int done = start;
  CountCrowd crowd;
  if (start == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15u) == 0) {
    const int n4 = n >> 2, lane = threadIdx.x & 31;
    done = n4 << 2;
    for (int qb = t0 - lane; qb < n4; qb += stride) {  // the same trip count in every lane
      const int q = qb + lane;
      const bool v = q < n4;
      float4 X = make_float4(0.0f, 0.0f, 0.0f, 0.0f), Y = X;
      if (v) {
        X = __ldg(reinterpret_cast<const float4*>(x) + q);
        Y = __ldg(reinterpret_cast<const float4*>(y) + q);
      }
      const int c[4] = {deposit_cell(X.x, Y.x, dxf, dyf, nx, ny), deposit_cell(X.y, Y.y, dxf, dyf, nx, ny),
                        deposit_cell(X.z, Y.z, dxf, dyf, nx, ny), deposit_cell(X.w, Y.w, dxf, dyf, nx, ny)};
      crowd.add(cnt, c, v);
    }
  }
  for (unsigned i0 = (unsigned)done + t0 - (threadIdx.x & 31); i0 < (unsigned)n; i0 += stride) {
    const unsigned i = i0 + (threadIdx.x & 31);
    const bool v = i < (unsigned)n;
    const int c[1] = {v ? deposit_cell(x[i], y[i], dxf, dyf, nx, ny) : -1};
    crowd.add(cnt, c, v);
  }
}

// rho = seq(seq(rho0, +c, k_ion), -c, k_ele) with the float64 addend of np.add.at;
// counts are cleared for reuse
__global__ void k_rho_finalize(float* rho, int* cnt_i, int* cnt_e, int G, double cd, int accumulate) {
  pdl_enter();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < G; i += gridDim.x * blockDim.x) {
    float s = accumulate ? rho[i] : 0.0f;
    int ki = cnt_i ? cnt_i[i] : 0;
    int ke = cnt_e ? cnt_e[i] : 0;
    if (ki) s = seq_add_f32d(s, cd, (uint32_t)ki);
    if (ke) s = seq_add_f32d(s, -cd, (uint32_t)ke);
    rho[i] = s;
    if (cnt_i) cnt_i[i] = 0;
    if (cnt_e) cnt_e[i] = 0;
  }
}

// The deposit of pb_accumulate_rho on grids whose counts fit a block's shared memory: every
// block of a cluster counts its particles in a private histogram of the whole grid, then adds
// a slice of the cells over the cluster (distributed shared memory).  One cluster rounds the
// slice into rho at once, without scratch, clear or second kernel (a call of 80k ions and one
// of 20k electrons on 65 x 284 nodes, back to back with the clear of rho: 33 us by the count
// kernels, 25 us so); more clusters add it to the global counts (6M ions and 2M electrons on
// 65 x 284, whose cells the atomics crowd: 125 us by the count kernels, 77 us so).
constexpr int DEP_C = 8;

__global__ void __cluster_dims__(DEP_C, 1, 1) __launch_bounds__(1024)
    k_deposit_cluster(const float* __restrict__ x, const float* __restrict__ y, float* rho, int* __restrict__ cnt, int n,
                      int nx, int ny, float dxf, float dyf, double cd) {
  extern __shared__ int4 dep_smem[];
  int* const hist = reinterpret_cast<int*>(dep_smem);
  const int G = nx * ny;
  uint32_t rank;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  for (int i = threadIdx.x; i < (G + 3) >> 2; i += blockDim.x) dep_smem[i] = make_int4(0, 0, 0, 0);
  __syncthreads();
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  auto add = [&](float px, float py) { atomicAdd(hist + deposit_cell(px, py, dxf, dyf, nx, ny), 1); };
  int done = 0;
  if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15u) == 0) {
    const float4* const x4 = reinterpret_cast<const float4*>(x);
    const float4* const y4 = reinterpret_cast<const float4*>(y);
    const int n4 = n >> 2;
    done = n4 << 2;
    // two groups of four particles in flight per thread
    for (int q = t0; q < n4; q += 2 * stride) {
      const int r = q + stride;
      const float4 X = __ldg(x4 + q), Y = __ldg(y4 + q);
      float4 Z = X, W = Y;
      if (r < n4) { Z = __ldg(x4 + r); W = __ldg(y4 + r); }
      add(X.x, Y.x); add(X.y, Y.y); add(X.z, Y.z); add(X.w, Y.w);
      if (r < n4) { add(Z.x, W.x); add(Z.y, W.y); add(Z.z, W.z); add(Z.w, W.w); }
    }
  }
  x += done;
  y += done;
  for (unsigned i = t0; i < (unsigned)(n - done); i += stride) add(x[i], y[i]);
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  const uint32_t base = smem_addr(hist);
  uint32_t at[DEP_C];
#pragma unroll
  for (int b = 0; b < DEP_C; ++b)
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at[b]) : "r"(base), "r"((rank + b) & (DEP_C - 1)));
  const int i0 = (int)((long long)G * rank / DEP_C), i1 = (int)((long long)G * (rank + 1) / DEP_C);
  const bool direct = gridDim.x == DEP_C;
  for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
    unsigned v[DEP_C], k = 0;
#pragma unroll
    for (int b = 0; b < DEP_C; ++b)
      asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v[b]) : "r"(at[b] + 4u * (uint32_t)i) : "memory");
    const float r0 = direct ? rho[i] : 0.0f;
#pragma unroll
    for (int b = 0; b < DEP_C; ++b) k += v[b];
    if (!k) continue;
    if (direct) rho[i] = seq_add_f32d(r0, cd, k);
    else atomicAdd(cnt + i, (int)k);
  }
  // no block leaves while another may read its histogram
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// ------------------------------------------------------------------ substep reduction
__device__ __forceinline__ double gather_sub(const float* __restrict__ F, size_t r0, size_t r1, long long ix0,
                                             long long ix1, double fx, double fy) {
  double gx = DSUB(1.0, fx), gy = DSUB(1.0, fy);
  double a = DMUL(DMUL((double)__ldg(F + r0 + ix0), gx), gy);
  double b = DMUL(DMUL((double)__ldg(F + r0 + ix1), fx), gy);
  double c = DMUL(DMUL((double)__ldg(F + r1 + ix0), gx), fy);
  double d = DMUL(DMUL((double)__ldg(F + r1 + ix1), fx), fy);
  return DADD(DADD(DADD(a, b), c), d);
}

// Ec non-null: E from the corner array (same values and arithmetic as gather_sub)
__device__ __forceinline__ double predicted_ds(float x, float y, float vx, float vy, float vz,
                                               const float* Ex, const float* Ey, const float4* Ec, int nx, int ny,
                                               float dxf, float dyf, double qm, float dtf, double dt2,
                                               float inv_dx = 0.0f, float inv_dy = 0.0f) {
  // with the corner array (the step's path): the cell as in push_cell<true>
  float ixf, iyf;
  long long ix0, iy0;
  double fx, fy;
  bool inside = false;
  int fxi = 0, fyi = 0;
  float frx = 0.0f, fry = 0.0f;
  if (Ec) {
    const bool okq = div_fast(x, dxf, inv_dx, ixf) & div_fast(y, dyf, inv_dy, iyf);
    if (!okq) { ixf = __fdiv_rn(x, dxf); iyf = __fdiv_rn(y, dyf); }
    const bool okx = floor_frac(ixf, fxi, frx), oky = floor_frac(iyf, fyi, fry);
    inside = okx & oky & (fxi <= nx - 2) & (fyi <= ny - 2);
  } else {
    ixf = __fdiv_rn(x, dxf); iyf = __fdiv_rn(y, dyf);
  }
  if (inside) {
    ix0 = fxi; iy0 = fyi; fx = (double)frx; fy = (double)fry;
  } else {
    ix0 = clampll(np_f2i64(floorf(ixf)), 0, nx - 2);
    iy0 = clampll(np_f2i64(floorf(iyf)), 0, ny - 2);
    fx = DSUB((double)ixf, (double)ix0); fy = DSUB((double)iyf, (double)iy0);
  }
  size_t r0 = (size_t)iy0 * nx, r1 = (size_t)(iy0 + 1) * nx;
  double ex, ey;
  if (Ec) {
    float4 a, b;
    ldg_corners(Ec + 2 * (r0 + ix0), a, b);
    const double gx = DSUB(1.0, fx), gy = DSUB(1.0, fy);
    ex = DADD(DADD(DADD(DMUL(DMUL((double)a.x, gx), gy), DMUL(DMUL((double)a.y, fx), gy)),
                   DMUL(DMUL((double)a.z, gx), fy)), DMUL(DMUL((double)a.w, fx), fy));
    ey = DADD(DADD(DADD(DMUL(DMUL((double)b.x, gx), gy), DMUL(DMUL((double)b.y, fx), gy)),
                   DMUL(DMUL((double)b.z, gx), fy)), DMUL(DMUL((double)b.w, fx), fy));
  } else {
    ex = gather_sub(Ex, r0, r1, ix0, ix0 + 1, fx, fy);
    ey = gather_sub(Ey, r0, r1, ix0, ix0 + 1, fx, fy);
  }
  double ax = DMUL(qm, ex), ay = DMUL(qm, ey);
  double a_mag = sqrt(DADD(DMUL(ax, ax), DMUL(ay, ay)));
  float v_mag = sqrtf(__fadd_rn(__fadd_rn(__fmul_rn(vx, vx), __fmul_rn(vy, vy)), __fmul_rn(vz, vz)));
  return DADD((double)__fmul_rn(v_mag, dtf), DMUL(DMUL(0.5, a_mag), dt2));
}

// Particles that cannot raise the maximum are passed over without the gather and the
// float64 arithmetic (ebound non-null, the corner path).  predicted_ds is monotone in the
// float32 |v|^2 it takes the root of, and for a particle inside the grid (fractions in
// [0, 1], so the bilinear E is a convex combination of corner values) its acceleration
// term is at most acc = 0.5 |qm| Emax dt^2, Emax = max over nodes of |Ex| + |Ey| (the
// bound k_e_corners leaves).  With every rounding of both terms below 1e-6 relative,
// ds <= (sqrt(v2) dtf + acc)(1 + 1e-6).  A particle is therefore skipped when
// v2 < ((M (1 - 2e-4) - acc (1 + 2e-4)) / dtf)^2 (1 - 2e-4), M an exact ds already seen:
// its ds is below M, and the maximum, hence n_sub, is that of the full loop.  Positions
// outside [0, nx - 2) x [0, ny - 2) cells, NaN and infinite values are never skipped.  The
// warp shares its running maximum after each pass that evaluated any particle, so after
// the first pass nearly every particle is skipped and the loop streams 20 B per particle.
// Block `block` of `blocks` of one species' reduction.
__device__ __forceinline__ void substep_block(const float* __restrict__ x, const float* __restrict__ y,
                                              const float* __restrict__ vx, const float* __restrict__ vy,
                                              const float* __restrict__ vz, int n, const float* Ex, const float* Ey,
                                              const float4* Ec, int nx, int ny, float dxf, float dyf, double qm,
                                              float dtf, double dt2, unsigned long long* ds_max_bits,
                                              const unsigned* ebound, int block, int blocks) {
  unsigned long long m = 0ull;
  const float inv_dx = __frcp_rn(dxf), inv_dy = __frcp_rn(dyf);
  // four particles per thread and pass (16-byte loads of each array), so that a thread
  // has four sets of loads and gathers in flight; the maximum does not depend on the
  // order.  Arrays that do not all start 16-byte aligned take the one-by-one loop.
  const bool vec = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) |
                     reinterpret_cast<uintptr_t>(vx) | reinterpret_cast<uintptr_t>(vy) |
                     reinterpret_cast<uintptr_t>(vz)) & 15u) == 0;
  const int n4 = vec ? n >> 2 : 0;
  const int t0 = block * blockDim.x + threadIdx.x, stride = blocks * blockDim.x;
  if (vec && Ec && ebound) {
    const double acc = 0.5 * fabs(qm) * (double)__uint_as_float(__ldg(ebound)) * dt2;  // NaN, inf: no skips
    const double invdt2 = 1.0 / ((double)dtf * (double)dtf);
    const float xlim = (float)(nx - 2), ylim = (float)(ny - 2);
    float thr = -1.0f;  // v2 < thr: below the running maximum (none yet)
    const int lane = threadIdx.x & 31;
    for (int qb = t0 - lane; qb < n4; qb += stride) {  // the same trip count in every lane
      const int q = qb + lane;
      bool did = false;
      if (q < n4) {
        const float4 X = __ldg(reinterpret_cast<const float4*>(x) + q);
        const float4 Y = __ldg(reinterpret_cast<const float4*>(y) + q);
        const float4 U = __ldg(reinterpret_cast<const float4*>(vx) + q);
        const float4 V = __ldg(reinterpret_cast<const float4*>(vy) + q);
        const float4 W = __ldg(reinterpret_cast<const float4*>(vz) + q);
        const float px[4] = {X.x, X.y, X.z, X.w}, py[4] = {Y.x, Y.y, Y.z, Y.w};
        const float pu[4] = {U.x, U.y, U.z, U.w}, pv[4] = {V.x, V.y, V.z, V.w}, pw[4] = {W.x, W.y, W.z, W.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float v2 = __fadd_rn(__fadd_rn(__fmul_rn(pu[j], pu[j]), __fmul_rn(pv[j], pv[j])),
                                     __fmul_rn(pw[j], pw[j]));
          const bool below = (v2 < thr) & (px[j] >= 0.0f) & (py[j] >= 0.0f) &
                             (__fmul_rn(px[j], inv_dx) < xlim) & (__fmul_rn(py[j], inv_dy) < ylim);
          if (!below) {
            const double d = predicted_ds(px[j], py[j], pu[j], pv[j], pw[j], Ex, Ey, Ec, nx, ny, dxf, dyf, qm, dtf,
                                          dt2, inv_dx, inv_dy);
            const unsigned long long b = (unsigned long long)__double_as_longlong(d);
            m = b > m ? b : m;
            did = true;
          }
        }
      }
      if (__any_sync(0xFFFFFFFFu, did)) {
        for (int o = 16; o > 0; o >>= 1) {
          const unsigned long long v = __shfl_xor_sync(0xFFFFFFFFu, m, o);
          m = v > m ? v : m;
        }
        const double M = __longlong_as_double((long long)m);
        const double R = M * (1.0 - 2e-4) - acc * (1.0 + 2e-4);
        thr = R > 0.0 ? __double2float_rd(R * R * invdt2 * (1.0 - 2e-4)) : -1.0f;
      }
    }
  } else {
    for (int q = t0; q < n4; q += stride) {
      const float4 X = __ldg(reinterpret_cast<const float4*>(x) + q);
      const float4 Y = __ldg(reinterpret_cast<const float4*>(y) + q);
      const float4 U = __ldg(reinterpret_cast<const float4*>(vx) + q);
      const float4 V = __ldg(reinterpret_cast<const float4*>(vy) + q);
      const float4 W = __ldg(reinterpret_cast<const float4*>(vz) + q);
      const double d0 = predicted_ds(X.x, Y.x, U.x, V.x, W.x, Ex, Ey, Ec, nx, ny, dxf, dyf, qm, dtf, dt2, inv_dx, inv_dy);
      const double d1 = predicted_ds(X.y, Y.y, U.y, V.y, W.y, Ex, Ey, Ec, nx, ny, dxf, dyf, qm, dtf, dt2, inv_dx, inv_dy);
      const double d2 = predicted_ds(X.z, Y.z, U.z, V.z, W.z, Ex, Ey, Ec, nx, ny, dxf, dyf, qm, dtf, dt2, inv_dx, inv_dy);
      const double d3 = predicted_ds(X.w, Y.w, U.w, V.w, W.w, Ex, Ey, Ec, nx, ny, dxf, dyf, qm, dtf, dt2, inv_dx, inv_dy);
      const unsigned long long b0 = (unsigned long long)__double_as_longlong(d0);
      const unsigned long long b1 = (unsigned long long)__double_as_longlong(d1);
      const unsigned long long b2 = (unsigned long long)__double_as_longlong(d2);
      const unsigned long long b3 = (unsigned long long)__double_as_longlong(d3);
      const unsigned long long b01 = b0 > b1 ? b0 : b1, b23 = b2 > b3 ? b2 : b3;
      const unsigned long long b = b01 > b23 ? b01 : b23;
      m = b > m ? b : m;
    }
  }
  for (unsigned i = 4u * n4 + t0; i < (unsigned)n; i += stride) {
    double ds = predicted_ds(x[i], y[i], vx[i], vy[i], vz[i], Ex, Ey, Ec, nx, ny, dxf, dyf, qm, dtf, dt2, inv_dx, inv_dy);
    unsigned long long b = (unsigned long long)__double_as_longlong(ds);
    m = b > m ? b : m;
  }
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long v = __shfl_down_sync(0xFFFFFFFFu, m, o);
    m = v > m ? v : m;
  }
  __shared__ unsigned long long sm[32];
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = threadIdx.x < (blockDim.x >> 5) ? sm[threadIdx.x] : 0ull;
    for (int o = 16; o > 0; o >>= 1) {
      unsigned long long v = __shfl_down_sync(0xFFFFFFFFu, m, o);
      m = v > m ? v : m;
    }
    if (threadIdx.x == 0 && m) atomicMax(ds_max_bits, m);
  }
}

__global__ void __launch_bounds__(256, 4) k_substep_reduce(const float* x, const float* y, const float* vx,
                                                           const float* vy, const float* vz, int n, const float* Ex,
                                                           const float* Ey, const float4* Ec, int nx, int ny, float dxf,
                                                           float dyf, double qm, float dtf, double dt2,
                                                           unsigned long long* ds_max_bits, const unsigned* ebound) {
  substep_block(x, y, vx, vy, vz, n, Ex, Ey, Ec, nx, ny, dxf, dyf, qm, dtf, dt2, ds_max_bits, ebound, (int)blockIdx.x,
                (int)gridDim.x);
}

// Both species of a step in one launch: blocks below ion_blocks reduce the ions.
__global__ void __launch_bounds__(256, 4) k_substep_both(const __grid_constant__ SubstepArgs a) {
  pdl_enter();
  const int k = (int)blockIdx.x >= a.ion_blocks;
  const Soa& S = a.sp[k];
  substep_block(S.x, S.y, S.vx, S.vy, S.vz, *a.n[k], nullptr, nullptr, a.Ec, a.nx, a.ny, a.dxf, a.dyf, a.qm[k], a.dtf,
                a.dt2, a.ds_max_bits + k, a.ebound, (int)blockIdx.x - (k ? a.ion_blocks : 0),
                k ? (int)gridDim.x - a.ion_blocks : a.ion_blocks);
}

// ------------------------------------------------------------------ path absorption
struct SegHit { bool hit; int ix, iy; };

__device__ __forceinline__ SegHit segment_hit(const uint8_t* __restrict__ isBound, int nx, int ny, float dxf,
                                              float dyf, float x0, float y0, float x1, float y1) {
  SegHit r;
  r.hit = false;
  r.ix = cell_round(x1, dxf, 0, nx - 1);
  r.iy = cell_round(y1, dyf, 0, ny - 1);
  float ddx = __fsub_rn(x1, x0), ddy = __fsub_rn(y1, y0);
#pragma unroll
  for (int i = 1; i <= 8; ++i) {
    float f = (float)i * 0.125f;
    float xi = __fadd_rn(x0, __fmul_rn(ddx, f));
    float yi = __fadd_rn(y0, __fmul_rn(ddy, f));
    int cx = cell_round(xi, dxf, 0, nx - 1);
    int cy = cell_round(yi, dyf, 0, ny - 1);
    if (!r.hit && __ldg(isBound + (size_t)cy * nx + cx)) { r.hit = true; r.ix = cx; r.iy = cy; }
  }
  return r;
}

// segment_hit with the sample cells from rint_div (same cells, fewer divisions)
__device__ __forceinline__ SegHit segment_hit_f(const uint8_t* __restrict__ isBound, int nx, int ny, float dxf,
                                                float dyf, float inv_dx, float inv_dy, float x0, float y0, float x1,
                                                float y1, int ix1, int iy1) {
  SegHit r;
  r.hit = false;
  r.ix = ix1;
  r.iy = iy1;
  float ddx = __fsub_rn(x1, x0), ddy = __fsub_rn(y1, y0);
#pragma unroll
  for (int i = 1; i <= 8; ++i) {
    float f = (float)i * 0.125f;
    float xi = __fadd_rn(x0, __fmul_rn(ddx, f));
    float yi = __fadd_rn(y0, __fmul_rn(ddy, f));
    int cx = cell_round_f(xi, dxf, inv_dx, 0, nx - 1);
    int cy = cell_round_f(yi, dyf, inv_dy, 0, ny - 1);
    if (!r.hit && __ldg(isBound + (size_t)cy * nx + cx)) { r.hit = true; r.ix = cx; r.iy = cy; }
  }
  return r;
}

__global__ void k_segment_hits(const uint8_t* isBound, int nx, int ny, float dxf, float dyf, const float* x0,
                               const float* y0, const float* x1, const float* y1, int n, uint8_t* hit,
                               int64_t* hix, int64_t* hiy) {
  pdl_enter();
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < (unsigned)n; i += gridDim.x * blockDim.x) {
    SegHit s = segment_hit(isBound, nx, ny, dxf, dyf, x0[i], y0[i], x1[i], y1[i]);
    hit[i] = s.hit;
    hix[i] = s.ix;
    hiy[i] = s.iy;
  }
}

// ------------------------------------------------------------------ cross-section splines
// de Boor evaluation of a cubic B-spline (FITPACK splev convention, knots t[0..nt-1],
// coefficients c[0..nt-5]); x is clipped into the base interval.
__device__ double spline_eval(const Spline& s, double x) {
  const int k = 3;
  int n = s.nt;
  int l = k;
  while (l < n - k - 2 && x >= s.t[l + 1]) ++l;
  double d[4];
  for (int j = 0; j <= k; ++j) d[j] = s.c[j + l - k];
  for (int r = 1; r <= k; ++r)
    for (int j = k; j >= r; --j) {
      double tl = s.t[j + l - k], tr = s.t[j + 1 + l - r];
      double alpha = (x - tl) / (tr - tl);
      d[j] = (1.0 - alpha) * d[j - 1] + alpha * d[j];
    }
  return d[k];
}

// 10 ** spline(clip(log10(max(E, 1e-30)), lo, hi))  (lookup_user_cs, physics_engine.py:475-484)
__device__ __forceinline__ double user_cs(const Spline& s, float E) {
  float le = log10f(np_maxf(E, 1e-30f));
  double l = (double)le;
  l = l < s.lo ? s.lo : (l > s.hi ? s.hi : l);
  return pow(10.0, spline_eval(s, l));
}

// ------------------------------------------------------------------ tile scan / look-back
constexpr unsigned long long FLAG_AGG = 1ull << 62, FLAG_PRE = 2ull << 62, VAL_MASK = (1ull << 62) - 1;

// Exclusive prefix of tile `tile` given its aggregate (decoupled look-back, warp-parallel).
// Called by warp 0; returns the prefix in every lane.  Waits are bounded.
__device__ long long lookback_warp(unsigned long long* status, int tile, int agg, uint32_t* errflags) {
  const int lane = threadIdx.x & 31;
  if (tile == 0) {
    if (lane == 0) atomicExch(status, FLAG_PRE | (unsigned long long)agg);
    return 0;
  }
  if (lane == 0) atomicExch(status + tile, FLAG_AGG | (unsigned long long)agg);
  long long excl = 0;
  int t = tile - 1;
  while (true) {
    int tt = t - lane;
    unsigned long long v = FLAG_PRE;  // before tile 0: an inclusive prefix of 0
    if (tt >= 0) {
      long long spin = 0;
      do {
        v = *((volatile unsigned long long*)(status + tt));
      } while ((v >> 62) == 0 && ++spin < SPIN_LIMIT);
      if ((v >> 62) == 0) { atomicOr(errflags, PB_EF_SPIN_TIMEOUT); v = FLAG_PRE; }
    }
    unsigned pre = __ballot_sync(0xFFFFFFFFu, (v >> 62) == 2);
    int stop = pre ? __ffs(pre) - 1 : 31;  // nearest lane holding an inclusive prefix
    long long val = (lane <= stop) ? (long long)(v & VAL_MASK) : 0;
    for (int o = 16; o > 0; o >>= 1) val += __shfl_down_sync(0xFFFFFFFFu, val, o);
    val = __shfl_sync(0xFFFFFFFFu, val, 0);
    excl += val;
    if (pre) break;
    t -= 32;
  }
  if (lane == 0) atomicExch(status + tile, FLAG_PRE | (unsigned long long)(excl + agg));
  return excl;
}

// Block-wide exclusive scan of keep flags staged in shared memory (index order), plus
// the global base via look-back.  Fills rank[] and returns the number kept in the tile.
template <int NTHR, int TILE_SZ>
__device__ __forceinline__ int tile_compact_ranks(const uint8_t* keep, int* rank, int tile, int t0, int n,
                                                  unsigned long long* status, int* num_dst, long long& base,
                                                  uint32_t* errflags) {
  constexpr int PER = TILE_SZ / NTHR;
  __shared__ int sm[NTHR / 32];
  __shared__ long long sbase;
  __shared__ int stotal;
  int k0 = threadIdx.x * PER;
  int c = 0;
#pragma unroll
  for (int q = 0; q < PER; ++q) c += keep[k0 + q];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int inc = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) sm[w] = inc;
  __syncthreads();
  if (w == 0) {
    int v = lane < NTHR / 32 ? sm[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int t = __shfl_up_sync(0xFFFFFFFFu, v, o);
      if (lane >= o) v += t;
    }
    if (lane < NTHR / 32) sm[lane] = v;
    int total = __shfl_sync(0xFFFFFFFFu, v, NTHR / 32 - 1);
    long long b = lookback_warp(status, tile, total, errflags);
    if (lane == 0) {
      sbase = b;
      stotal = total;
      if (t0 + TILE_SZ >= n) *num_dst = (int)(b + total);
    }
  }
  __syncthreads();
  int ex = (w ? sm[w - 1] : 0) + inc - c;
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    rank[k0 + q] = ex;
    ex += keep[k0 + q];
  }
  base = sbase;
  int tot = stotal;
  __syncthreads();
  return tot;
}

// ------------------------------------------------------------------ fused ion step
// Tile of TILE particles: item k of the tile is particle t0 + k; thread t handles
// k = t, t + NT, ... (coalesced loads), results are staged in shared memory, ranked by a
// block scan in index order and written compacted (stable) at the global offset.
template <int TL>
struct IonStage {
  float x[TL], y[TL], vx[TL], vy[TL], vz[TL];
  uint32_t id[TL];
  int rank[TL];            // deposit cells (PB_OPT_SMEM_HIST) until the compaction ranks them
  uint8_t cex[TL], keep[TL];
};

// Four resident blocks of 256 per SM (64 registers, some spilled): latency hiding gains
// more than the spills cost (12% faster than three blocks at 80 registers).
// Lower-left start cell of a tile's particles (a rough floor of x / dx and y / dy, which
// only places the staged window; every gather checks membership exactly), block-wide.
template <int TL>
__device__ __forceinline__ void tile_low_cell(const IonStepArgs& a, int t0, int n, int& xlo, int& ylo) {
  __shared__ int red[2 * (NT / 32)];
  int lx = INT_MAX, ly = INT_MAX;
  for (int k = threadIdx.x; k < TL; k += NT) {
    const int i = t0 + k;
    if (i >= n) break;
    const float qx = __fmul_rn(a.src.x[i], a.inv_dx), qy = __fmul_rn(a.src.y[i], a.inv_dy);
    const int cx = qx >= 0.0f ? (qx < (float)(a.nx - 2) ? (int)qx : a.nx - 2) : 0;
    const int cy = qy >= 0.0f ? (qy < (float)(a.ny - 2) ? (int)qy : a.ny - 2) : 0;
    lx = min(lx, cx);
    ly = min(ly, cy);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lx = min(lx, __shfl_xor_sync(0xFFFFFFFFu, lx, o));
    ly = min(ly, __shfl_xor_sync(0xFFFFFFFFu, ly, o));
  }
  if ((threadIdx.x & 31) == 0) { red[threadIdx.x >> 5] = lx; red[NT / 32 + (threadIdx.x >> 5)] = ly; }
  __syncthreads();
  xlo = ylo = INT_MAX;
#pragma unroll
  for (int j = 0; j < NT / 32; ++j) { xlo = min(xlo, red[j]); ylo = min(ylo, red[NT / 32 + j]); }
  __syncthreads();
}

constexpr long long TMA_SPIN_LIMIT = 1ll << 22;  // polls of the window's mbarrier before giving up

template <bool HAS_B, int OPT, int TL>
__global__ void __launch_bounds__(NT, 4) k_ion_step(const __grid_constant__ IonStepArgs a) {
  constexpr bool HIST = (OPT & PB_OPT_SMEM_HIST) != 0;
  constexpr bool TMA = (OPT & PB_OPT_TMA_TILE) != 0 && !HAS_B;
  pdl_enter();
  const uint32_t stepk = a.step_dev ? *a.step_dev : a.step;  // Philox step key
  __shared__ IonStage<TL> st;
  __shared__ int sm_tile;
  __shared__ int hbins[HIST ? HBINS : 1];
  __shared__ int pcell[HIST ? TL : 1];
  __shared__ __align__(128) float4 ebox[TMA ? 2 * TB_W * TB_H : 1];
  __shared__ __align__(8) uint64_t ebar;
  if (HIST)
    for (int b = threadIdx.x; b < HBINS; b += NT) hbins[b] = 0;
  if (TMA && threadIdx.x == 0) mbar_init(&ebar, 1);
  uint32_t tma_phase = 0;
  bool tma_live = TMA;   // block-uniform; false after a window copy failed to complete
  const int n = *a.num_src;
  const int n_sub = substep_count(*a.ds_max, a.ds_lim, nullptr);
  const double dt_sub = DDIV(a.dt, (double)n_sub);
  const double h = DMUL(DMUL(0.5, a.qm), dt_sub);
  const float dtf = __double2float_rn(dt_sub);
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.n_sub_out = substep_count(*a.ds_max, a.ds_lim, a.errflags);
  const float pi_f = 3.14159265358979323846f;
  // per-thread event counts (32-bit: a thread sees far fewer than 2^32 ions); the exit
  // sums, whose ions are rare, go straight to shared memory, so neither holds registers
  // across the loop
  unsigned int cnt[7] = {0, 0, 0, 0, 0, 0, 0};
  __shared__ double sums[9];
  if (threadIdx.x < 9) sums[threadIdx.x] = 0.0;
  __syncthreads();

  while (true) {
    if (threadIdx.x == 0) sm_tile = atomicAdd(a.tile_counter, 1);
    __syncthreads();
    const int tile = sm_tile;
    const int t0 = tile * TL;
    if (t0 >= n) break;
    EBox eb{nullptr, 0, 0};
    if (TMA && tma_live) {
      // stage the window of E corners around the tile's particles (one TMA copy), one
      // cell of margin below and left of the lowest start cell
      int xlo, ylo;
      tile_low_cell<TL>(a, t0, n, xlo, ylo);
      eb.bx = xlo - 1;
      eb.by = ylo - 1;
      if (threadIdx.x == 0) {
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(&ebar, TB_BYTES);
        tma_load_3d(ebox, &a.ec_map, &ebar, 0, eb.bx, eb.by);
      }
      long long spin = 0;
      bool done;
      while (!(done = mbar_try_wait(&ebar, tma_phase)) && ++spin < TMA_SPIN_LIMIT) {
      }
      tma_phase ^= 1u;
      if (__syncthreads_and(done)) {
        eb.box = ebox;
      } else {
        tma_live = false;
        if (threadIdx.x == 0) atomicOr(a.errflags, PB_EF_SPIN_TIMEOUT);
      }
    }
#pragma unroll 1
    for (int k = threadIdx.x; k < TL; k += NT) {
      const int i = t0 + k;
      uint8_t kp = 0;
      int dep_cell = 0, ppc_cell = 0;
      if (i < n) {
        float x = a.src.x[i], y = a.src.y[i], vx = a.src.vx[i], vy = a.src.vy[i], vz = a.src.vz[i];
        uint8_t cx = a.src.cex[i];
        const uint32_t pid = a.src.id[i];
        const float x0 = x, y0 = y;
        float q0[2];  // x0 / dx, y0 / dy (correctly rounded), from the first substep
        boris_push_one<HAS_B, !HAS_B, !HAS_B>(x, y, vx, vy, vz, a.Ex, a.Ey, a.Bx, a.By, a.Bz, a.nx, a.ny, a.dxf,
                                              a.dyf, h, dtf, a.Ec, a.rcp, q0, eb);
        for (int s = 1; s < n_sub; ++s)
          boris_push_one<HAS_B, !HAS_B, !HAS_B>(x, y, vx, vy, vz, a.Ex, a.Ey, a.Bx, a.By, a.Bz, a.nx, a.ny, a.dxf,
                                                a.dyf, h, dtf, a.Ec, a.rcp, nullptr, eb);
        if (a.periodic) y = np_modf_pos(y, a.Lyf);
        // the final cell, the PPC cell and the deposit cell all round or truncate the same
        // correctly rounded quotients (what rint_div and trunc_div return)
        const float qx = div_rn_checked(x, a.dxf, a.inv_dx), qy = div_rn_checked(y, a.dyf, a.inv_dy);
        // entered the optics (:1316-1324)
        if (x0 < a.x_entry && x >= a.x_entry && vx > 0.0f) cnt[0]++;
        // final-cell and path hits (:1326-1336).  The 8 path samples lie in cells at most
        // max(|di|, |dj|) + 1 (Chebyshev) from the start cell; they are examined only when
        // that reaches the distance from the start cell to the nearest bound node.
        const int icx = rint_clip(qx, 0, a.nx - 1);
        const int icy = rint_clip(qy, 0, a.ny - 1);
        const bool hit_final = __ldg(a.isBound + (size_t)icy * a.nx + icx) != 0;
        const int sx0 = rint_clip(q0[0], 0, a.nx - 1);
        const int sy0 = rint_clip(q0[1], 0, a.ny - 1);
        const int reach = max(abs(icx - sx0), abs(icy - sy0)) + 1;
        SegHit sh;
        sh.hit = false; sh.ix = icx; sh.iy = icy;
        if (reach >= (int)__ldg(a.bdist + (size_t)sy0 * a.nx + sx0))
          sh = segment_hit_f(a.isBound, a.nx, a.ny, a.dxf, a.dyf, a.inv_dx, a.inv_dy, x0, y0, x, y, icx, icy);
        bool hit = hit_final || sh.hit;
        int imx = sh.hit ? sh.ix : icx, imy = sh.hit ? sh.iy : icy;
        bool oob = (x < 0.0f) || (x > a.x_plume) || (x != x);
        if (!a.periodic) oob = oob || (y < 0.0f) || (y > a.Lyf);
        if (hit) cnt[4]++;
        if (hit && !oob) cnt[3]++;
        // heating, SEE, sputtering for hits beyond x = 0.25 mm (:1359-1449)
        if (hit && x > 0.25f) {
          float v2 = __fadd_rn(__fadd_rn(__fmul_rn(vx, vx), __fmul_rn(vy, vy)), __fmul_rn(vz, vz));
          size_t cell = (size_t)imy * a.nx + imx;
          if (a.thermal_on) {
            float Ej = __fmul_rn(__fmul_rn(a.k_half_m, v2), a.mw_f);
            float dT = __fmul_rn(__fdiv_rn(Ej, a.ccell_f), a.accel_f);
            atomicAdd(a.Tmap + cell, dT);
          }
          float E_eV = __fdiv_rn(__fmul_rn(a.k_half_m, v2), a.q_f);
          double gamma;
          if (a.see_spline.enabled) {
            double g = user_cs(a.see_spline, E_eV);
            gamma = g < 0.0 ? 0.0 : (g > 1.0 ? 1.0 : g);
          } else {
            float g = __fadd_rn(0.05f, __fmul_rn(1e-4f, E_eV));
            g = (g != g) ? g : (g < 0.0f ? 0.0f : (g > 1.0f ? 1.0f : g));
            gamma = (double)g;
          }
          double u = philox_uniform(a.seed, pid, SITE_SEE_SPAWN, stepk, 0);
          if (u < gamma) {
            int r = atomicAdd(a.see_count, 1);
            if (r < a.see_cap) {
              float off_x = __fdiv_rn(__fmul_rn(__fmul_rn(vx, a.dt_f), 1000.0f), 1.5f);
              float off_y = __fdiv_rn(__fmul_rn(__fmul_rn(vy, a.dt_f), 1000.0f), 1.5f);
              a.see_xy[2 * r] = __fsub_rn(x, off_x);
              a.see_xy[2 * r + 1] = __fsub_rn(y, off_y);
              a.see_key[r] = ((uint64_t)pid << 32) | (uint32_t)r;
            } else {
              atomicOr(a.errflags, PB_EF_SEE_OVERFLOW);
            }
          }
          if (a.erosion_on && E_eV > a.Eth_f) {
            double dmg;
            if (a.Y_exp == 1.0) {  // the reference's linear law, float32 (:1432-1433)
              dmg = (double)__fmul_rn(__fmul_rn(a.Y_f, __fsub_rn(E_eV, a.Eth_f)), a.mw_f);
            } else {               // Y_coeff (E - E_th)^p, float64 from the float32 excess
              dmg = DMUL(DMUL(a.Y_d, pow((double)__fsub_rn(E_eV, a.Eth_f), a.Y_exp)), a.mw_d);
            }
            atomicAdd(a.damage + cell, dmg);
          }
        }
        // exit plane diagnostics (:1451-1494), pre-collision velocities and flag
        bool crossed = (x0 <= a.x_exit) && (x > a.x_exit) && (vx > 0.0f);
        if ((x > a.x_exit) && (vx > 0.0f)) cnt[2]++;
        if (crossed) {
          cnt[1]++;
          float ve = sqrtf(__fadd_rn(__fadd_rn(__fmul_rn(vx, vx), __fmul_rn(vy, vy)), __fmul_rn(vz, vz)));
          float Ee = __fdiv_rn(__fmul_rn(a.k_half_m, __fmul_rn(ve, ve)), a.q_f);
          atomicAdd(&sums[0], (double)vx); atomicAdd(&sums[1], (double)ve); atomicAdd(&sums[2], (double)Ee);
          atomicAdd(&sums[7], (double)vx * vx); atomicAdd(&sums[8], (double)ve * ve);
          if (cx) { atomicAdd(&sums[5], (double)ve); atomicAdd(&sums[6], 1.0); }
          else { atomicAdd(&sums[3], (double)ve); atomicAdd(&sums[4], 1.0); }
          int r = atomicAdd(a.angle_count, 1);
          float ang = __fdiv_rn(__fmul_rn(fabsf(atan2f(vy, vx)), 180.0f), pi_f);
          if (r < a.angle_cap) a.angles[r] = ang; else atomicOr(a.errflags, PB_EF_ANGLE_OVERFLOW);
        }
        bool alive = !(hit || oob);
        kp = alive && ((x <= a.x_plume) || (vx < 0.0f));
        if (kp) {
          // CEX null-collision MCC on primaries (:1682-1739).  P = 1 - exp(-n sigma g dt)
          // <= |n0a| sigma_max g dt, so a draw u at or above that bound (plus the rounding
          // of the exact expression) neither collides nor ties, and the exact
          // probability is evaluated only below it.
          if (!cx && x >= 1.0f && x <= a.Lxf) {
            float vm = sqrtf(__fadd_rn(__fadd_rn(__fmul_rn(vx, vx), __fmul_rn(vy, vy)), __fmul_rn(vz, vz)));
            float g = np_maxf(vm, 1.0f);
            double u = philox_uniform(a.seed, pid, SITE_CEX_U, stepk, 0);
            if (!(g <= a.cex_g_max && u >= DADD(DMUL(a.cex_bound, (double)g), 1e-15))) {
              double nl;
              if (a.n_uniform) {
                nl = a.n0u;
              } else {
                float z_m = __fmul_rn(__fsub_rn(x, 1.0f), 1e-3f);
                z_m = z_m >= 0.0f ? z_m : 0.0f;
                float r_m = __fmul_rn(y, 1e-3f);
                float zr = __fadd_rn(z_m, a.rT_f);
                float R = sqrtf(__fadd_rn(__fmul_rn(r_m, r_m), __fmul_rn(zr, zr)));
                float th = atan2f(r_m, zr);
                float Rm = np_maxf(R, 1e-12f);
                float q1 = __fdiv_rn(a.rT_f, Rm);
                float geo = __fsub_rn(1.0f, __fdiv_rn(1.0f, sqrtf(__fadd_rn(1.0f, __fmul_rn(q1, q1)))));
                nl = DMUL(DMUL(a.n0a, (double)geo), (double)cosf(th));
              }
              nl = np_maxd(nl, 0.0);
              double sigma;
              if (a.cx_spline.enabled) {
                float Ec = __fdiv_rn(__fmul_rn(a.k_half_m, __fmul_rn(g, g)), a.q_f);
                sigma = user_cs(a.cx_spline, Ec);
              } else {
                float t = __fadd_rn(__fmul_rn(-0.8821f, logf(g)), 15.1262f);
                sigma = (double)__fmul_rn(__fmul_rn(t, t), 1e-20f);
              }
              double prob = DSUB(1.0, exp(DMUL(DMUL(DMUL(-nl, sigma), (double)g), a.dt)));
              if (fabs(u - prob) <= fabs(prob) * 8.9e-16 + 1e-300) cnt[6]++;
              if (u < prob) {
                cnt[5]++;
                u32x4 r0 = philox_block(a.seed, pid, SITE_CEX_FM, stepk, 0);
                u32x4 r1 = philox_block(a.seed, pid, SITE_CEX_FM, stepk, 1);
                u32x4 r2 = philox_block(a.seed, pid, SITE_CEX_FM, stepk, 2);
                u32x4 r3 = philox_block(a.seed, pid, SITE_CEX_FM, stepk, 3);
                u32x4 r4 = philox_block(a.seed, pid, SITE_CEX_FM, stepk, 4);
                double fmx = DMUL(2.0, DSUB(DADD(DADD(u53(r0.x, r0.y), u53(r0.z, r0.w)), u53(r1.x, r1.y)), 1.5));
                double fmy = DMUL(2.0, DSUB(DADD(DADD(u53(r1.z, r1.w), u53(r2.x, r2.y)), u53(r2.z, r2.w)), 1.5));
                double fmz = DMUL(2.0, DSUB(DADD(DADD(u53(r3.x, r3.y), u53(r3.z, r3.w)), u53(r4.x, r4.y)), 1.5));
                vx = __double2float_rn(DMUL(a.neut_vth, fmx));
                vy = __double2float_rn(DMUL(a.neut_vth, fmy));
                vz = __double2float_rn(DMUL(a.neut_vth, fmz));
                cx = 1;
              }
            }
          }
          // PPC map with truncated cells (:1749-1757), next-step deposit cell (rounded)
          ppc_cell = trunc_clip(qy, 0, a.ny - 1) * a.nx + trunc_clip(qx, 0, a.nx - 1);
          dep_cell = rint_clip(qy, 1, a.ny - 2) * a.nx + rint_clip(qx, 1, a.nx - 2);
        }
        st.x[k] = x; st.y[k] = y; st.vx[k] = vx; st.vy[k] = vy; st.vz[k] = vz;
        st.cex[k] = cx; st.id[k] = pid;
      }
      st.keep[k] = kp;
      if (HIST) {
        st.rank[k] = dep_cell;
        pcell[k] = ppc_cell;
      } else {
        // warp-aggregated counts (consecutive lanes, near-sorted cells)
        warp_count_add(a.ppc, ppc_cell, kp != 0);
        warp_count_add(a.cnt, dep_cell, kp != 0);
      }
    }
    __syncthreads();
    if (HIST) {
      tile_hist<NT, TL>(pcell, st.keep, a.ppc, hbins);
      tile_hist<NT, TL>(st.rank, st.keep, a.cnt, hbins);
    }
    long long base;
    tile_compact_ranks<NT, TL>(st.keep, st.rank, tile, t0, n, a.tile_status, a.num_dst, base, a.errflags);
    for (int k = threadIdx.x; k < TL; k += NT) {
      if (!st.keep[k]) continue;
      long long pos = base + st.rank[k];
      a.dst.x[pos] = st.x[k]; a.dst.y[pos] = st.y[k];
      a.dst.vx[pos] = st.vx[k]; a.dst.vy[pos] = st.vy[k]; a.dst.vz[pos] = st.vz[k];
      a.dst.cex[pos] = st.cex[k]; a.dst.id[pos] = st.id[k];
    }
    __syncthreads();
  }
  if (TMA && !tma_live && threadIdx.x == 0) {
    // a window copy did not complete in time: wait (bounded) for it before the block's
    // shared memory is released
    long long spin = 0;
    while (!mbar_try_wait(&ebar, tma_phase ^ 1u) && ++spin < TMA_SPIN_LIMIT) {
    }
  }
  // flush per-thread tallies
#pragma unroll
  for (int j = 0; j < 7; ++j) {
    unsigned long long v = cnt[j];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(a.counters + j, v);
  }
  __syncthreads();
  if (threadIdx.x < 9 && sums[threadIdx.x] != 0.0) atomicAdd(a.exit_sums + threadIdx.x, sums[threadIdx.x]);
}

// ------------------------------------------------------------------ fused electron step
template <int TL>
struct EleStage {
  float x[TL], y[TL], vx[TL], vy[TL], vz[TL];
  uint32_t id[TL];
  int rank[TL];
  uint8_t keep[TL];
};

// The end of one electron's step after its pushes: periodic wrap, purge test and the
// next step's deposit cell; the survivor is staged in shared memory at tile slot k.
template <int TL>
__device__ __forceinline__ void ele_finish(const EleStepArgs& a, EleStage<TL>& st, int k, int i, float x, float y,
                                           float vx, float vy, float vz, uint8_t& kp, int& dep_cell) {
  if (a.periodic) y = np_modf_pos(y, a.Lyf);
  int icx = cell_round_f(x, a.dxf, a.inv_dx, 0, a.nx - 1), icy = cell_round_f(y, a.dyf, a.inv_dy, 0, a.ny - 1);
  bool dead = __ldg(a.isBound + (size_t)icy * a.nx + icx) != 0;
  dead = dead || (x < 0.0f) || (x > a.Lxf) || (y < 0.0f) || (y > a.Lyf) || (x != x);
  kp = !dead;
  if (kp)
    dep_cell = cell_round32_f(y, a.dyf, a.inv_dy, 1, a.ny - 2) * a.nx + cell_round32_f(x, a.dxf, a.inv_dx, 1, a.nx - 2);
  st.x[k] = x; st.y[k] = y; st.vx[k] = vx; st.vy[k] = vy; st.vz[k] = vz;
  st.id[k] = a.src.id[i];
}

template <bool HAS_B, int OPT, int TL>
__global__ void __launch_bounds__(NT) k_ele_step(EleStepArgs a) {
  constexpr bool HIST = (OPT & PB_OPT_SMEM_HIST) != 0;
  constexpr bool PAIRS = (OPT & PB_OPT_ELE_PAIRS) != 0 && !HAS_B;
  pdl_enter();
  __shared__ EleStage<TL> st;
  __shared__ int sm_tile;
  __shared__ int hbins[HIST ? HBINS : 1];
  if (HIST)
    for (int b = threadIdx.x; b < HBINS; b += NT) hbins[b] = 0;
  const int n = *a.num_src;
  const int n_sub = substep_count(*a.ds_max, a.ds_lim, nullptr);
  const double dt_sub = DDIV(a.dt, (double)n_sub);
  const double h = DMUL(DMUL(0.5, a.qm), dt_sub);
  const float dtf = __double2float_rn(dt_sub);
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.n_sub_out = substep_count(*a.ds_max, a.ds_lim, a.errflags);
  while (true) {
    if (threadIdx.x == 0) sm_tile = atomicAdd(a.tile_counter, 1);
    __syncthreads();
    const int tile = sm_tile;
    const int t0 = tile * TL;
    if (t0 >= n) break;
    if (PAIRS) {
      // items k and k + NT of a thread pushed side by side (TL = 2 NT or 4 NT: one or two pairs)
#pragma unroll 1
      for (int k = threadIdx.x; k < TL; k += 2 * NT) {
        float x[2], y[2], vx[2], vy[2], vz[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int i = t0 + k + q * NT;
          // a slot past the end pushes a copy of an in-range particle (never stored)
          const int j = i < n ? i : t0;
          x[q] = a.src.x[j]; y[q] = a.src.y[j]; vx[q] = a.src.vx[j]; vy[q] = a.src.vy[j]; vz[q] = a.src.vz[j];
        }
        push_pair_b0(x, y, vx, vy, vz, n_sub, a.Ec, a.nx, a.ny, a.dxf, a.dyf, a.rcp, h, dtf);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int kk = k + q * NT, i = t0 + kk;
          uint8_t kp = 0;
          int dep_cell = 0;
          if (i < n) ele_finish(a, st, kk, i, x[q], y[q], vx[q], vy[q], vz[q], kp, dep_cell);
          st.keep[kk] = kp;
          if (HIST) st.rank[kk] = dep_cell;
          else warp_count_add(a.cnt, dep_cell, kp != 0);
        }
      }
    } else {
#pragma unroll 1
      for (int k = threadIdx.x; k < TL; k += NT) {
        const int i = t0 + k;
        uint8_t kp = 0;
        int dep_cell = 0;
        if (i < n) {
          float x = a.src.x[i], y = a.src.y[i], vx = a.src.vx[i], vy = a.src.vy[i], vz = a.src.vz[i];
          for (int s = 0; s < n_sub; ++s)
            boris_push_one<HAS_B, !HAS_B, !HAS_B>(x, y, vx, vy, vz, a.Ex, a.Ey, a.Bx, a.By, a.Bz, a.nx, a.ny, a.dxf,
                                                  a.dyf, h, dtf, a.Ec, a.rcp);
          ele_finish(a, st, k, i, x, y, vx, vy, vz, kp, dep_cell);
        }
        st.keep[k] = kp;
        if (HIST) st.rank[k] = dep_cell;
        else warp_count_add(a.cnt, dep_cell, kp != 0);
      }
    }
    __syncthreads();
    if (HIST) tile_hist<NT, TL>(st.rank, st.keep, a.cnt, hbins);
    long long base;
    tile_compact_ranks<NT, TL>(st.keep, st.rank, tile, t0, n, a.tile_status, a.num_dst, base, a.errflags);
    for (int k = threadIdx.x; k < TL; k += NT) {
      if (!st.keep[k]) continue;
      long long pos = base + st.rank[k];
      a.dst.x[pos] = st.x[k]; a.dst.y[pos] = st.y[k];
      a.dst.vx[pos] = st.vx[k]; a.dst.vy[pos] = st.vy[k]; a.dst.vz[pos] = st.vz[k];
      a.dst.id[pos] = st.id[k];
    }
    __syncthreads();
  }
}

// One electron sub-step of k_ele_push.  EFIN (every corner value finite, from the bound
// k_e_corners leaves): a position inside the grid has weights in [0, 1], and the Ex and Ey
// values of the cell's lower-left corner are made doubles by their bits (f2d_scaled) and
// multiplied by w00 2^896 (exact), which rounds a.x w00 exactly as the converted product
// does, with two fewer conversion-unit instructions.  Other positions take boris_push_one.
// VFIN (every electron's velocity finite at the start of the step, from the sub-step
// reduction's maximum): on that path vx and vy are finite too, since a sub-step that makes
// a velocity non-finite makes the position non-finite, which never lies inside the grid
// again; they become doubles by their bits (push_update_b0<true>).
template <bool EFIN, bool VFIN>
__device__ __forceinline__ void ele_substep(float& x, float& y, float& vx, float& vy, float& vz,
                                            const EleStepArgs& a, double h, float dtf) {
  if (!EFIN) {
    boris_push_one<false, true, true>(x, y, vx, vy, vz, a.Ex, a.Ey, nullptr, nullptr, nullptr, a.nx, a.ny, a.dxf,
                                      a.dyf, h, dtf, a.Ec, a.rcp);
    return;
  }
  float ixf, iyf;
  const bool okq = div_bracket(x, a.dxf, a.rcp.ix, a.rcp.ix_lo, a.rcp.ix_hi, ixf) &
                   div_bracket(y, a.dyf, a.rcp.iy, a.rcp.iy_lo, a.rcp.iy_hi, iyf);
  int fxi, fyi;
  float frx, fry;
  floor_frac(ixf, fxi, frx);
  floor_frac(iyf, fyi, fry);
  const bool inside = okq & ((unsigned)fxi <= (unsigned)(a.nx - 2)) & ((unsigned)fyi <= (unsigned)(a.ny - 2));
  if (!inside) {
    boris_push_one<false, true, true>(x, y, vx, vy, vz, a.Ex, a.Ey, nullptr, nullptr, nullptr, a.nx, a.ny, a.dxf,
                                      a.dyf, h, dtf, a.Ec, a.rcp);
    return;
  }
  const double fx = (double)frx, fy = (double)fry;
  const double gx = DSUB(1.0, fx), gy = DSUB(1.0, fy);
  const double w00 = DMUL(gx, gy), w10 = DMUL(fx, gy), w01 = DMUL(gx, fy), w11 = DMUL(fx, fy);
  const double w00s = DMUL(w00, 0x1p896);
  float4 A, B;
  ldg_corners(a.Ec + 2 * (fyi * a.nx + fxi), A, B);
  const double ex = DADD(DADD(DADD(DMUL(f2d_scaled(A.x), w00s), DMUL((double)A.y, w10)), DMUL((double)A.z, w01)),
                         DMUL((double)A.w, w11));
  const double ey = DADD(DADD(DADD(DMUL(f2d_scaled(B.x), w00s), DMUL((double)B.y, w10)), DMUL((double)B.z, w01)),
                         DMUL((double)B.w, w11));
  push_update_b0<VFIN>(x, y, vx, vy, vz, ex, ey, h, dtf);
}

template <bool EFIN, bool VFIN>
__device__ __forceinline__ void ele_push_range(const EleStepArgs& a, uint8_t* __restrict__ keep, int n, int n_sub,
                                               double h, float dtf) {
  const int stride = gridDim.x * blockDim.x;
  // trip count uniform across a warp (the deposit count is a warp-wide vote)
  const int n_pad = (n + 31) & ~31;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_pad; i += stride) {
    int dep_cell = 0;
    bool kp = false;
    if (i < n) {
      float x = a.src.x[i], y = a.src.y[i], vx = a.src.vx[i], vy = a.src.vy[i], vz = a.src.vz[i];
      // plain path: two sub-steps per loop pass (no spills at 32 registers, 1.3% faster)
#pragma unroll (EFIN ? 1 : 2)
      for (int s = 0; s < n_sub; ++s) ele_substep<EFIN, VFIN>(x, y, vx, vy, vz, a, h, dtf);
      if (a.periodic) y = np_modf_pos(y, a.Lyf);
      const int icx = cell_round_f(x, a.dxf, a.inv_dx, 0, a.nx - 1);
      const int icy = cell_round_f(y, a.dyf, a.inv_dy, 0, a.ny - 1);
      bool dead = __ldg(a.isBound + (size_t)icy * a.nx + icx) != 0;
      dead = dead || (x < 0.0f) || (x > a.Lxf) || (y < 0.0f) || (y > a.Lyf) || (x != x);
      kp = !dead;
      if (kp)
        dep_cell = cell_round32_f(y, a.dyf, a.inv_dy, 1, a.ny - 2) * a.nx +
                   cell_round32_f(x, a.dxf, a.inv_dx, 1, a.nx - 2);
      a.src.x[i] = x; a.src.y[i] = y; a.src.vx[i] = vx; a.src.vy[i] = vy; a.src.vz[i] = vz;
      keep[i] = kp ? 1 : 0;
    }
    warp_count_add(a.cnt, dep_cell, kp);
  }
}

// ------------------------------------------------------------------ split electron step
// PB_OPT_ELE_SPLIT: the electron step as two kernels.  k_ele_push advances every electron
// independently (no shared-memory staging, no block barriers), writes it back in place and
// records whether it survives; k_ele_compact then moves the survivors to the other buffer
// in order (the same single-pass look-back as the fused kernel).  The push is compute-bound
// at many sub-steps per electron, so the extra pass over the state costs less than the
// barriers it removes.  Same operations, same bits as k_ele_step.
__global__ void __launch_bounds__(NT, 8) k_ele_push(EleStepArgs a, uint8_t* __restrict__ keep) {
  pdl_enter();
  const int n = *a.num_src;
  const int n_sub = substep_count(*a.ds_max, a.ds_lim, nullptr);
  const double dt_sub = DDIV(a.dt, (double)n_sub);
  const double h = DMUL(DMUL(0.5, a.qm), dt_sub);
  const float dtf = __double2float_rn(dt_sub);
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.n_sub_out = substep_count(*a.ds_max, a.ds_lim, a.errflags);
  // every corner value finite (and |Ex| + |Ey| below the float range): the bound's bits
  const bool efin = a.ebound && *a.ebound < 0x7F800000u;
  // every electron's |v| finite: the sub-step reduction's maximum is finite (a NaN or
  // infinite velocity gives a NaN or infinite predicted displacement, never passed over)
  const bool vfin = *a.ds_max < INFINITY;
  if (efin && vfin) ele_push_range<true, true>(a, keep, n, n_sub, h, dtf);
  else if (efin) ele_push_range<true, false>(a, keep, n, n_sub, h, dtf);
  else ele_push_range<false, false>(a, keep, n, n_sub, h, dtf);
}

struct EleCompactStage {
  float x[TILE], y[TILE], vx[TILE], vy[TILE], vz[TILE];
  uint32_t id[TILE];
  int rank[TILE];
  uint8_t keep[TILE];
};

__global__ void __launch_bounds__(NT) k_ele_compact(EleStepArgs a, const uint8_t* __restrict__ keep) {
  pdl_enter();
  __shared__ EleCompactStage st;
  __shared__ int sm_tile;
  const int n = *a.num_src;
  while (true) {
    if (threadIdx.x == 0) sm_tile = atomicAdd(a.tile_counter, 1);
    __syncthreads();
    const int tile = sm_tile;
    const int t0 = tile * TILE;
    if (t0 >= n) break;
    for (int k = threadIdx.x; k < TILE; k += NT) {
      const int i = t0 + k;
      const uint8_t kp = i < n ? keep[i] : 0;
      st.keep[k] = kp;
      if (kp) {
        st.x[k] = a.src.x[i]; st.y[k] = a.src.y[i]; st.vx[k] = a.src.vx[i]; st.vy[k] = a.src.vy[i];
        st.vz[k] = a.src.vz[i]; st.id[k] = a.src.id[i];
      }
    }
    __syncthreads();
    long long base;
    tile_compact_ranks<NT, TILE>(st.keep, st.rank, tile, t0, n, a.tile_status, a.num_dst, base, a.errflags);
    for (int k = threadIdx.x; k < TILE; k += NT) {
      if (!st.keep[k]) continue;
      const long long pos = base + st.rank[k];
      a.dst.x[pos] = st.x[k]; a.dst.y[pos] = st.y[k];
      a.dst.vx[pos] = st.vx[k]; a.dst.vy[pos] = st.vy[k]; a.dst.vz[pos] = st.vz[k];
      a.dst.id[pos] = st.id[k];
    }
    __syncthreads();
  }
}

}  // namespace pb

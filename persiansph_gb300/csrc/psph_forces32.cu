// FP32-compensated form of the pair path (precision = PSPH_FP32C): fluids
// (CalcForce11) and soil / solids (CalcForce2233).
//
// Same algorithm as psph_forces.cu (CalcForce11, Source/Interaction.cpp:25-184,
// and the wall interpolation of PrimaryComputeAcceleration,
// Source/Domain.cpp:1029-1059/:1164-1206), with the pair arithmetic in FP32:
//  - positions enter the pair kernels as (int cell, FP32 offset from the cell
//    origin); a pair's separation is (cell_i - cell_j) * CellSize + (off_i -
//    off_j), exact in the cell part and ~1e-9 m in the offset part, and the
//    periodic minimum image falls out of the wrapped cell difference;
//  - kernel, gradient, EOS-derived terms and viscosity in FP32;
//  - the acceleration and density-rate sums are Kahan-compensated in FP32;
//  - integration, material update and the dt reduction stay in FP64
//    (psph_update.cu, dt_finalize_kernel).
#include <algorithm>
#include <cfloat>

#include "psph_copies.cuh"

namespace psph {

namespace {

constexpr int kFT32 = 128;  // block size of the copy and wall-interpolation kernels
// The pair kernels take their block size at launch (Options::pair_block, 64 to
// 256 threads, picked by psph_autotune); register caps are set per kernel.
constexpr int kMaxPairBlock = 256;

struct Kahan {
  float s = 0.f, c = 0.f;
  PSPH_D void add(float x) {
    const float y = x - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
  }
  PSPH_D double value() const { return (double)s - (double)c; }
};

// Loads issued where they stand: the neighbour's velocity, density and class
// go out together with its position, ahead of the support test, so the pair
// waits for one memory round trip instead of two (a plain load would be sunk
// below the test's branch). Read-only for the kernel's lifetime.
PSPH_D float4 ld_early(const float4* p) {
  float4 r;
  asm volatile("ld.global.nc.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "l"(p));
  return r;
}
// the same for an array the kernel itself writes elsewhere (coherent path)
PSPH_D float4 ld_early_coherent(const float4* p) {
  float4 r;
  asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "l"(p));
  return r;
}

PSPH_D float2 ld_early_coherent(const float2* p) {
  float2 r;
  asm volatile("ld.global.v2.f32 {%0,%1}, [%2];" : "=f"(r.x), "=f"(r.y) : "l"(p));
  return r;
}
PSPH_D float ld_early_coherent(const float* p) {
  float r;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(r) : "l"(p));
  return r;
}

template <int DIM, int KT>
struct KernF {
  static constexpr float cw() { return (float)Kern<DIM, KT>::cw(); }
  static PSPH_D float W(float q, float cwh) {
    if (KT == 0) {
      if (q < 1.f) return cwh * (1.f - 1.5f * q * q + 0.75f * q * q * q);
      if (q < 2.f) { const float t = 2.f - q; return cwh * (0.25f * t * t * t); }
      return 0.f;
    } else if (KT == 1) {
      if (q < 2.f) { const float t = 1.f - 0.5f * q; const float t2 = t * t; return cwh * (t2 * t2) * (2.f * q + 1.f); }
      return 0.f;
    } else {
      const float a = 3.f - q, b = 2.f - q, c = 1.f - q;
      const float a2 = a * a, b2 = b * b, c2 = c * c;
      if (q < 1.f) return cwh * (a2 * a2 * a - 6.f * b2 * b2 * b + 15.f * c2 * c2 * c);
      if (q < 2.f) return cwh * (a2 * a2 * a - 6.f * b2 * b2 * b);
      if (q < 3.f) return cwh * (a2 * a2 * a);
      return 0.f;
    }
  }
  static PSPH_D float GK(float q, float inv_q, float cwg) {
    if (KT == 0) {
      if (q < 1.f) return cwg * (-3.f + 2.25f * q);
      if (q < 2.f) { const float t = 2.f - q; return cwg * inv_q * (-0.75f * t * t); }
      return 0.f;
    } else if (KT == 1) {
      if (q < 2.f) { const float t = 1.f - 0.5f * q; return cwg * -5.f * (t * t * t); }
      return 0.f;
    } else {
      const float a = 3.f - q, b = 2.f - q, c = 1.f - q;
      const float a2 = a * a, b2 = b * b, c2 = c * c;
      if (q == 0.f) return cwg * (20.f * a2 * a - 120.f * b2 * b + 300.f * c2 * c);
      if (q < 1.f) return cwg * inv_q * (-5.f * a2 * a2 + 30.f * b2 * b2 - 75.f * c2 * c2);
      if (q < 2.f) return cwg * inv_q * (-5.f * a2 * a2 + 30.f * b2 * b2);
      if (q < 3.f) return cwg * inv_q * (-5.f * a2 * a2);
      return 0.f;
    }
  }
  static PSPH_D float D2(float q, float cwg) {
    if (KT == 0) {
      if (q < 1.f) return cwg * (-3.f + 4.5f * q);
      if (q < 2.f) return cwg * (1.5f * (2.f - q));
      return 0.f;
    } else if (KT == 1) {
      if (q < 2.f) { const float t = 1.f - 0.5f * q; return cwg * (t * t) * (10.f * q - 5.f); }
      return 0.f;
    } else {
      const float a = 3.f - q, b = 2.f - q, c = 1.f - q;
      if (q < 1.f) return cwg * (20.f * a * a * a - 120.f * b * b * b + 300.f * c * c * c);
      if (q < 2.f) return cwg * (20.f * a * a * a - 120.f * b * b * b);
      if (q < 3.f) return cwg * (20.f * a * a * a);
      return 0.f;
    }
  }
  static PSPH_D float Lap(float q, float inv_q, float cwg) {
    float first;
    if (KT == 0) {
      if (q < 1.f) first = (-3.f + 2.25f * q);
      else if (q < 2.f) { const float t = 2.f - q; first = inv_q * (-0.75f * t * t); }
      else return 0.f;
    } else if (KT == 1) {
      if (q < 2.f) { const float t = 1.f - 0.5f * q; first = -5.f * t * t * t; }
      else return 0.f;
    } else {
      const float a = 3.f - q, b = 2.f - q, c = 1.f - q;
      const float a2 = a * a, b2 = b * b, c2 = c * c;
      if (q < 1.f) first = inv_q * (-5.f * a2 * a2 + 30.f * b2 * b2 - 75.f * c2 * c2);
      else if (q < 2.f) first = inv_q * (-5.f * a2 * a2 + 30.f * b2 * b2);
      else if (q < 3.f) first = inv_q * (-5.f * a2 * a2);
      else return 0.f;
    }
    return D2(q, cwg) + cwg * (DIM - 1.f) * first;
  }
};

// ---------------------------------------------------------------------------
// Preparation (FP32 copies, partner-visible wall state) and wall interpolation
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kFT32) copies32_kernel(DevView v) {
  const StepScalars* sc = v.sc;
  if (sc->all_stop) return;
  const Persist& P = cur_persist(v);
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w < sc->n) fluid_copies32(v, P, w, P.cls[w], P.X4[w].w, P.V4[w], v.S.OFF32[w], v.o.skin > 0.f ? v.S.refcell[w] : 0);
}

// Wall interpolation, bound by the neighbours' gathers. 2D: 4 lanes to a wall,
// each a 16-byte chunk of its list at a time, over the sort's list of the fixed
// particles (920 particles 10 us where one lane takes 14, 86k 11 and 14). 3D: a lane to a particle, the free ones' idle: a warp's
// walls then gather the same neighbours at the same time (1.0M particles 82 us;
// over the list of the fixed ones, whose warps lie less close, 93, with 2 and 4
// lanes to a wall 129 and 177).
template <int DIM>
constexpr int kWallLanesLog2 = DIM == 2 ? 2 : 0;

// DensitySolid / SoundSpeed of a fluid's EOS at a wall's pressure (Source/Functions.cpp:214-264), FP32
PSPH_D void wall_state32(const PClass32& Ce, float p, float* rw, float* cw) {
  const float cs2 = Ce.cs * Ce.cs, r0 = Ce.rho0, p0 = Ce.p0;
  if (Ce.pres_eq == 0) *rw = (p - p0) / cs2 + r0;
  else if (Ce.pres_eq == 1) *rw = powf((p - p0) * (7.f / (r0 * cs2)) + 1.f, 1.f / 7.f) * r0;
  else *rw = p / cs2;
  const float ratio = *rw / r0;
  *cw = (Ce.pres_eq == 1) ? fabsf(Ce.cs * ratio * ratio * ratio) : Ce.cs;  // sqrt(cs^2 ratio^6)
}

template <int DIM, int KT>
PSPH_D void interpolate_wall32(const DevView& v, const Persist& P, int w, int sub) {
  const Options& o = v.o;
  const PClass32* __restrict__ CT = v.cls32;
  const bool wall = w >= 0;
  const PClass32& C = CT[wall ? P.cls[w] : 0];
  const GridDev& g = grid_of(v, C.inst);
  const bool noslip = wall && (C.flags & CF_NOSLIP);
  const int ow = wall ? P.orig[w] : 0, cell = wall ? v.S.cellid[w] : -1;
  const float4 oi = wall ? v.S.OFF32[w] : make_float4(0.f, 0.f, 0.f, 0.f);
  const float3 cs = cell_size_f(g);
  const float gx = o.gravity32[0], gy = o.gravity32[1], gz = o.gravity32[2];
  const bool need_orient = !o.wallp_physical && (gx != 0.f || gy != 0.f || gz != 0.f);
  const bool skin = o.skin > 0.f;
  const int rc_w = (skin && need_orient && wall) ? v.S.refcell[w] : 0;
  float sk = 0.f, p = 0.f, n0 = 0.f, n1 = 0.f, n2 = 0.f;
  const float hw = fabsf(oi.w), ihw = 1.f / hw;
  // a free neighbour's density and, with a skin, its cell in the reference's grid
  const bool spec = spec32_of(v, C.inst);
  auto density_and_cell = [&](int f) {
    return spec ? ld_early_coherent(v.S.RC32 + f)
                    : make_float2(ld_early_coherent(&v.S.D32[f].w),
                                  skin && need_orient ? __int_as_float(v.S.refcell[f]) : 0.f);
  };
  // One neighbour, loaded: free particles contribute (OFF32.w is negative for a
  // fixed one; an FP32C domain has one material).
  auto visit = [&](const int f, const int code, const float4 of, const float4 vf, const float2 rr) {
    const float rho = rr.x;
    float x0, x1, x2;
    rel_pos<DIM>(cs, oi, of, code, x0, x1, x2);  // x_wall - x_fluid
    if (need_orient) {
      // the pair's cell offset in the reference's grid (with a skin the lists'
      // cells are coarser): it decides which particle the reference lists first
      const int cd = skin ? ref_code(rc_w, __float_as_int(rr.y)) : code;
      if (!first_of_pair_code(cd, ow, P.orig[f])) {
        x0 = -x0; x1 = -x1; x2 = -x2;
      }
    }
    const float ih = o.uniform_h ? ihw : 1.f / (0.5f * (hw + of.w));
    const float q = sqrtf(x0 * x0 + x1 * x1 + x2 * x2) * ih;
    const float K = KernF<DIM, KT>::W(q, KernF<DIM, KT>::cw() * (DIM == 2 ? ih * ih : ih * ih * ih));
    if (K == 0.f) return;
    sk += K;
    p += vf.w * K + (gx * x0 + gy * x1 + gz * x2) * rho * K;
    if (noslip) { n0 += vf.x * K; n1 += vf.y * K; n2 += vf.z * K; }
  };
  const int cnt = (wall && cell >= 0) ? v.S.nl_count[w] : 0;
  if (cnt >= 0) {
    // the neighbour list, 4 entries per 16-byte load, whose 12 loads go out
    // together (this kernel writes the walls' own V32 / D32, which the test then
    // rejects, so those two take the coherent path)
    const int4* __restrict__ nl4 = reinterpret_cast<const int4*>(v.S.nl) + nl_slot(w);
    const size_t N = (size_t)v.nl_stride;
    const int nch = (cnt + 3) >> 2;
    for (int c = sub; c < nch; c += 1 << kWallLanesLog2<DIM>) {
      const int4 q = nl4[(size_t)c * N];
      const int rem = cnt - 4 * c;
      const int e[4] = {q.x, rem > 1 ? q.y : q.x, rem > 2 ? q.z : q.x, rem > 3 ? q.w : q.x};
      float4 of[4], vf[4];
      float2 rr[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int f = e[t] & kIndexMask;
        of[t] = ld_early(v.S.OFF32 + f);
        vf[t] = ld_early_coherent(v.S.V32 + f);
        rr[t] = density_and_cell(f);
      }
#pragma unroll
      for (int t = 0; t < 4; ++t)
        if (t < rem && of[t].w > 0.f) visit(e[t] & kIndexMask, entry_code(e[t]), of[t], vf[t], rr[t]);
    }
  } else if (sub == 0) {  // list overflow: scan the cells
    NbrSource<DIM> src;
    src.init(v, g, w, true, 1.0f);
    while (true) {
      int code;
      const int f = src.next(v, &code);
      if (f < 0) break;
      const float4 of = v.S.OFF32[f];
      if (of.w > 0.f) visit(f, code, of, ld_early_coherent(v.S.V32 + f), density_and_cell(f));
    }
  }
#pragma unroll
  for (int d = 1; d < 1 << kWallLanesLog2<DIM>; d <<= 1) {  // the lanes' sums together
    sk += __shfl_xor_sync(0xffffffffu, sk, d);
    p += __shfl_xor_sync(0xffffffffu, p, d);
    n0 += __shfl_xor_sync(0xffffffffu, n0, d);
    n1 += __shfl_xor_sync(0xffffffffu, n1, d);
    n2 += __shfl_xor_sync(0xffffffffu, n2, d);
  }
  if (!wall || sub != 0) return;
  if (sk != 0.f) {
    p = p / sk;
    if (noslip) { n0 /= sk; n1 /= sk; n2 /= sk; }
  } else {
    p = 0.f; n0 = n1 = n2 = 0.f;
  }
  double4_32a vw = P.V4[w];
  vw.w = (double)p;
  P.V4[w] = vw;
  v.S.sumkernel[w] = sk;
  v.S.nsv4[w] = make_double4_32a(n0, n1, n2, 0.0);
  v.S.NSV32[w] = make_float4(n0, n1, n2, 0.f);
  v.S.V32[w] = make_float4(d2f_rn(vw.x), d2f_rn(vw.y), d2f_rn(vw.z), p);
  const int eos_cls = wall_eos(v, C.inst);
  float rw = d2f_rn(P.X4[w].w), cwv = 0.f;
  if (eos_cls >= 0) wall_state32(CT[eos_cls], p, &rw, &cwv);
  const float inv = 1.f / rw;
  if (spec) {
    // a wall without a free particle in its support has none to meet, but may
    // stand in a list (their margin): its terms are zeros times finite numbers
    const bool odd = sk == 0.f && !(fabsf(inv) <= FLT_MAX);
    v.S.PX32[w] = make_float4(oi.x, oi.y, oi.z, odd ? -1.f : with_sign(inv, -1.f));
    v.S.V32LO[w].w = odd ? 0.f : with_sign(cwv, inv);
  } else {
    v.S.D32[w] = make_float4(inv, p * inv * inv, cwv, rw);
  }
}

template <int DIM, int KT>
__global__ void __launch_bounds__(kFT32) prepare32_kernel(DevView v) {
  const StepScalars* sc = v.sc;
  if (sc->all_stop) return;
  const Persist& P = cur_persist(v);
  const int t = blockIdx.x * kFT32 + threadIdx.x, sub = t & ((1 << kWallLanesLog2<DIM>) - 1);
  int w = t >> kWallLanesLog2<DIM>;
  if (DIM == 2) w = w < sc->n_walls ? v.S.walls[w] : -1;
  else if (w >= sc->n || (v.cls32[P.cls[w]].flags & CF_FREE)) w = -1;
  if (w >= 0 && v.inst[v.cls32[P.cls[w]].inst].stop) w = -1;
  if (__any_sync(0xffffffffu, w >= 0)) interpolate_wall32<DIM, KT>(v, P, w, sub);  // (a wall's lanes sum together)
}

// ---------------------------------------------------------------------------
// Fluid pair force, FP32 with compensated sums, over the neighbour lists
// ---------------------------------------------------------------------------
// FL 0: every option read at run time. FL 4: the same where some fluid has several
// EOS (Options::several_eos), a wall's state then from its partner's (86k particles in
// 2D with tensile instability 55 us; with this in FL 0 58). FL 1, 2 and 3: Morris viscosity,
// squared-density gradient, no tensile instability or XSPH, one h, one EOS, and pair
// constants (artificial viscosity, masses) the same for every class, taken from
// the launch (Options::flavours32), without (1) or with (2) the strain-rate sums
// of LES and Bingham, or with the learned closure's vorticity too (3); the
// classes' flags may differ (a slip lid over no-slip walls, LES on part of the
// fluid), where forces_spec32_kernel wants them alike and is faster.
// The list walk is a counted loop so that the next neighbour's loads can be
// issued before this one's arithmetic; each pair issues all of its neighbour
// loads before the support test (ld_early).
// Register caps measured on the 6.7M-particle dam break (64 to 112 swept): the
// strain-rate flavours run best at 96 (20 warps/SM), the plain one at 80, the
// general one at 128. A tank with a slip lid, 1.0M particles, through FL 0 and its
// flavour: 916 and 495 us without rates, 1049 and 606 with LES, 1012 and 606 with
// the closure; 86k in 2D 44 and 25.
template <int DIM, int KT, int FL>
__global__ void __maxnreg__(FL == 0 || FL == 4 ? 128 : (FL == 1 ? 80 : 96)) forces_fluid32_kernel(DevView v) {
  constexpr bool SPEC = FL >= 1 && FL <= 3;
  constexpr bool CLOSURE = FL == 3;
  __shared__ unsigned long long cred[32];
  const StepScalars* sc = v.sc;
  if (sc->all_stop) return;
  const Persist& P = cur_persist(v);
  const int n = sc->n;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const Options& o = v.o;
  const PClass32* __restrict__ CT = v.cls32;
  float dtc = FLT_MAX;
  unsigned npair2 = 0;  // 2 per pair with a free partner, 1 per wall partner (the pair is counted once)
  bool active = false;
  int cell = -1, ci_cls = 0;
  if (i < n) {
    ci_cls = P.cls[i];
    bool run = !v.inst[CT[ci_cls].inst].stop;
    if (o.mix32) run = run && !v.forms[CT[ci_cls].inst].spec32;  // (forces_spec32_kernel takes those)
    active = run && (CT[ci_cls].flags & CF_FREE);
    cell = v.S.cellid[i];
    if (run && !active) {
      v.S.A4[i] = make_double4_32a(o.gravity[0], o.gravity[1], o.gravity[2], 0.0);
      v.S.zwab[i] = 1.0;
    }
  }
  const PClass32& Ci = CT[ci_cls];
  const GridDev& g = grid_of(v, Ci.inst);
  const InstState& Is = v.inst[Ci.inst];
  const int is = active ? i : 0;
  const float4 oi = v.S.OFF32[is];
  const float4 vi = v.S.V32[is];
  const float4 vil = v.S.V32LO[is];
  const float4 di4 = v.S.D32[is];
  const float di = di4.w, inv_i = di4.x, Pi = di4.y, ci_snd = di4.z, pi = vi.w;
  const float mi = Ci.mass, hi = fabsf(oi.w);
  const float mui = o.dyn_mu ? v.S.MU32[is] : Ci.mu0;
  const int fi = Ci.flags;
  const bool shep = (fi & CF_SHEPARD) && (Is.shepard_counter == o.shepard_step);
  const bool sr_self = fi & (CF_T0 | CF_LES);
  const bool use_sr = SPEC ? (FL >= 2) : (bool)o.need_sr;
  const bool xsph_on = SPEC ? false : o.xsph != 0.0;
  const float xsph = o.xsph32;
  const float3 cs = cell_size_f(g);
  const float mu_u = o.mu_u32;
  const bool uniform_mu = o.uniform_mu, dyn_mu = o.dyn_mu;
  const int vis_eq = SPEC ? 0 : o.vis_eq, grad_type = SPEC ? 0 : o.grad_type;
  Kahan ax, ay, az, dr;
  float zw = 0.f, sd = 0.f, xs0 = 0.f, xs1 = 0.f, xs2 = 0.f;
  // strain-rate sums as sums of products a_r x_c (a = c2 vab): diagonal
  // m00 m11 m22, and the off-diagonal pairs either summed (s01 = m01 + m10 ...)
  // or, with the closure (whose vorticity needs the antisymmetric part), kept
  // apart (m01, m10, ...)
  float m00 = 0.f, m11 = 0.f, m22 = 0.f, m01 = 0.f, m02 = 0.f, m12 = 0.f, m10 = 0.f, m20 = 0.f, m21 = 0.f;
  int nnb = 0;
  const bool closure = SPEC ? (CLOSURE && (fi & CF_LES)) : (o.closure && (fi & CF_LES));
  // the closure flavour always keeps the antisymmetric sums apart
  const bool split_sr = SPEC ? CLOSURE : closure;
  const bool own_eos = FL == 4 && wall_eos(v, Ci.inst) < 0;
  const float cf2 = g.cellfac2_32;
  const bool own_h = !SPEC && v.forms;
  const bool uniform_h = own_h ? v.forms[Ci.inst].uniform_h : o.uniform_h;
  const float ih_u = own_h ? v.forms[Ci.inst].spec32c.inv_h : o.inv_h32;
  auto pair = [&](const int j, const int code) {
    const float4 oj = v.S.OFF32[j];
    const float4 vjl = ld_early(v.S.V32LO + j);
    const float4 vj = ld_early(v.S.V32 + j);
    const float4 dj4 = ld_early(v.S.D32 + j);
    const int wj = __float_as_int(vjl.w);
    const int clsj = wj & 0xffff;
    float x0, x1, x2;
    rel_pos<DIM>(cs, oi, oj, code, x0, x1, x2);
    const float hb = SPEC ? hi : 0.5f * (hi + fabsf(oj.w));  // one h: (h + h) / 2 = h exactly
    const float r2 = x0 * x0 + x1 * x1 + x2 * x2;
    // the list's own support test (exact in FP32; lists with a skin hold more)
    if (r2 > cf2 * hb * hb) return;
    const PClass32& Cj = CT[SPEC ? 0 : clsj];
    const int fjf = wj >> 16;
    const bool fj = fjf & CF_FREE;
    npair2 += fj ? 1u : 2u;
    ++nnb;
    // FP32C divisions use the hardware reciprocal (2 ulp; the form's bound is 1e-5)
    const float ih = uniform_h ? ih_u : __fdividef(1.f, hb);
    const float inv_r = (r2 > 0.f) ? rsqrtf(r2) : 0.f;
    const float q = r2 * inv_r * ih;
    const float inv_q = hb * inv_r;
    const float ih2 = ih * ih;
    const float cwh = KernF<DIM, KT>::cw() * (DIM == 2 ? ih2 : ih2 * ih);
    const float cwg = cwh * ih2;
    const float GK = KernF<DIM, KT>::GK(q, inv_q, cwg);
    const float K = KernF<DIM, KT>::W(q, cwh);
    float dj = dj4.w, inv_j = dj4.x, Pj = dj4.y, cj_snd = dj4.z;
    const float pj = vj.w;
    if (own_eos && !fj) {  // wall density from this particle's EOS (Source/Interaction.cpp:53-57)
      wall_state32(Ci, pj, &dj, &cj_snd);
      inv_j = 1.f / dj;
      Pj = pj * inv_j * inv_j;
    }
    const float mj = SPEC ? (fj ? o.m_free32 : o.fpm_wall32 * mi) : (fj ? Cj.mass : Cj.fpmassc * mi);
    const float v0 = (vi.x - vj.x) + (vil.x - vjl.x), v1 = (vi.y - vj.y) + (vil.y - vjl.y),
                v2 = (vi.z - vj.z) + (vil.z - vjl.z);
    const float vx = v0 * x0 + v1 * x1 + v2 * x2;
    float PI = 0.f;
    const float Alpha = SPEC ? o.alpha32 : 0.5f * (Ci.alpha + Cj.alpha);
    const float Beta = SPEC ? o.beta32 : 0.5f * (Ci.beta + Cj.beta);
    if ((Alpha != 0.f || Beta != 0.f) && vx < 0.f) {
      const float D = r2 + 0.01f * hb * hb;
      const float t = hb * vx;
      PI = __fdividef(t * (-Alpha * 0.5f * (ci_snd + cj_snd) * D + Beta * t), D * D * (0.5f * (di + dj)));
    }
    float TI = 0.f;
    if (!SPEC && ((fi | fjf) & CF_TI)) {
      float Ri = 0.f, Rj = 0.f;
      if ((pi + pj) < 0.f) {
        if (pi < 0.f) Ri = -pi * inv_i * inv_i;
        if (pj < 0.f) Rj = -pj * inv_j * inv_j;
      }
      const float Wd = KernF<DIM, KT>::W((Ci.tid + Cj.tid) * 0.5f * ih, cwh);
      TI = (Ci.ti * Ri + Cj.ti * Rj) * powf(K / Wd, (Ci.tin + Cj.tin) * 0.5f);
    }
    float VI0 = 0.f, VI1 = 0.f, VI2 = 0.f;
    if (((fi | fjf) & CF_NOSLIP) || fj) {
      float Mu, vab0, vab1, vab2;
      if (fj) {
        vab0 = v0; vab1 = v1; vab2 = v2;
        if (uniform_mu) Mu = mu_u;
        else {
          const float muj = dyn_mu ? v.S.MU32[j] : (SPEC ? Ci.mu0 : Cj.mu0);
          Mu = __fdividef(2.f * mui * muj, mui + muj);
        }
      } else {
        const float4 ns = v.S.NSV32[j];
        vab0 = (vi.x - (2.f * vj.x - ns.x)) + (vil.x - 2.f * vjl.x);
        vab1 = (vi.y - (2.f * vj.y - ns.y)) + (vil.y - 2.f * vjl.y);
        vab2 = (vi.z - (2.f * vj.z - ns.z)) + (vil.z - 2.f * vjl.z);
        Mu = mui;
      }
      if (vis_eq <= 2) {
        float c;
        if (vis_eq == 0) c = 2.f * Mu * inv_i * inv_j * GK;
        else if (vis_eq == 1) c = 8.f * Mu / ((di + dj) * (di + dj)) * GK;
        else c = -Mu * inv_i * inv_j * KernF<DIM, KT>::Lap(q, inv_q, cwg);
        VI0 = c * vab0; VI1 = c * vab1; VI2 = c * vab2;
      } else {
        const float L = KernF<DIM, KT>::Lap(q, inv_q, cwg);
        const float S2 = KernF<DIM, KT>::D2(q, cwg);
        const float s = -Mu * inv_i * inv_j;
        const float t = vx / r2 * (-GK + S2);
        VI0 = s * (L * vab0 + (1.f / 3.f) * (GK * v0 + t * x0));
        VI1 = s * (L * vab1 + (1.f / 3.f) * (GK * v1 + t * x1));
        VI2 = s * (L * vab2 + (1.f / 3.f) * (GK * v2 + t * x2));
      }
      if (use_sr && sr_self && (((fi | fjf) & CF_T0) || ((fi & fjf) & CF_LES))) {
        // StrainRate += (m_j / rho_j) S with S = -GK [2 v_a x_a, v_a x_b + v_b x_a, ...]
        // (Source/Interaction.cpp:114-117, no 1/2): a = c2 vab, S_rc = a_r x_c + a_c x_r
        const float c2 = -GK * (mj * inv_j);
        const float a0 = c2 * vab0, a1 = c2 * vab1, a2 = c2 * vab2;
        m00 = fmaf(a0, x0, m00);
        m11 = fmaf(a1, x1, m11);
        m22 = fmaf(a2, x2, m22);
        m01 = fmaf(a0, x1, m01);
        m02 = fmaf(a0, x2, m02);
        m12 = fmaf(a1, x2, m12);
        if (split_sr) {
          m10 = fmaf(a1, x0, m10);
          m20 = fmaf(a2, x0, m20);
          m21 = fmaf(a2, x1, m21);
        } else {
          m01 = fmaf(a1, x0, m01);
          m02 = fmaf(a2, x0, m02);
          m12 = fmaf(a2, x1, m12);
        }
      }
    }
    if (xsph_on && fj) {
      const float s = xsph * mj / (0.5f * (di + dj)) * K;
      xs0 -= s * v0; xs1 -= s * v1; xs2 -= s * v2;
    }
    float s;
    if (grad_type == 0) s = -(Pi + Pj + PI + TI) * GK;
    else s = -((pi + pj) * inv_i * inv_j + PI + TI) * GK;
    ax.add(mj * (s * x0 + VI0));
    ay.add(mj * (s * x1 + VI1));
    if (DIM == 3) az.add(mj * (s * x2 + VI2));
    dr.add(mj * di * inv_j * (GK * vx));
    zw += mj * inv_j * K;
    if (shep) sd += mj * K;
  };
  const int cnt = (active && cell >= 0) ? v.S.nl_count[i] : 0;
  if (cnt >= 0) {
    const int4* __restrict__ nl4 = reinterpret_cast<const int4*>(v.S.nl) + nl_slot(i);
    const size_t N = (size_t)v.nl_stride;
    const int nch = (cnt + 3) >> 2;
    // the strain-rate flavours load the next chunk one chunk ahead (measured:
    // it helps there and costs the plain flavour a little)
    constexpr bool kAhead = SPEC && FL >= 2;
    int4 qn = (kAhead && nch > 0) ? nl4[0] : make_int4(0, 0, 0, 0);
    for (int c = 0; c < nch; ++c) {  // one 16-byte chunk of 4 entries per load
      int4 q;
      if (kAhead) {
        q = qn;
        if (c + 1 < nch) qn = nl4[(size_t)(c + 1) * N];
      } else {
        q = nl4[(size_t)c * N];
      }
      const int rem = cnt - 4 * c;
      pair(q.x & kIndexMask, entry_code(q.x));
      if (rem > 1) pair(q.y & kIndexMask, entry_code(q.y));
      if (rem > 2) pair(q.z & kIndexMask, entry_code(q.z));
      if (rem > 3) pair(q.w & kIndexMask, entry_code(q.w));
    }
  } else {  // list overflow: scan the cells
    NbrSource<DIM> src;
    src.init(v, g, i, true, 1.0f);
    while (true) {
      int code;
      const int j = src.next(v, &code);
      if (j < 0) break;
      pair(j, code);
    }
  }
  if (active) {
    const double axd = o.gb[0] + ax.value();
    const double ayd = o.gb[1] + ay.value();
    const double azd = o.gb[2] + az.value();
    const double drd = dr.value();
    v.S.A4[i] = make_double4_32a(axd, ayd, azd, drd);
    v.S.zwab[i] = zw;
    if (o.any_shepard) v.S.sumden[i] = sd;
    if (xsph_on) v.S.vxsph4[i] = make_double4_32a(xs0, xs1, xs2, 0.0);
    if (use_sr) {
      // symmetric sums 2 m_rr and m_rc + m_cr; the antisymmetric m_rc - m_cr
      // (closure) is the vorticity's
      const float sr0 = 2.f * m00, sr4 = 2.f * m11, sr8 = 2.f * m22;
      const float sr1 = split_sr ? m01 + m10 : m01, sr2 = split_sr ? m02 + m20 : m02,
                  sr5 = split_sr ? m12 + m21 : m12;
      const float w01 = m01 - m10, w02 = m02 - m20, w12 = m12 - m21;
      // the 6 distinct sums in FP32 (the FP64 tensor is built on download)
      float2* out = reinterpret_cast<float2*>(v.S.sr32 + 6 * (size_t)i);
      out[0] = make_float2(sr0, sr1);
      out[1] = make_float2(sr2, sr4);
      out[2] = make_float2(sr5, sr8);
      // Mat1's ShearRate contraction (Source/Particle.cpp:151-153) of the
      // symmetric sums, in FP32: the update and the closure take it from here
      const float temp = sr0 * sr0 + 2.f * sr1 * sr1 + 2.f * sr2 * sr2 + sr4 * sr4 + 2.f * sr5 * sr5 + sr8 * sr8;
      v.S.cshear[i] = sqrtf(0.5f * temp);
      if (closure) {
        v.S.cvort[i] = sqrtf(w01 * w01 + w02 * w02 + w12 * w12);
        v.S.cnnb[i] = (float)nnb;
        const float det =
            sr0 * (sr4 * sr8 - sr5 * sr5) - sr1 * (sr1 * sr8 - sr5 * sr2) + sr2 * (sr1 * sr5 - sr4 * sr2);
        v.S.cr3[i] = temp > 0.f ? det / (temp * sqrtf(temp)) : 0.f;
      }
    }
    // the FP64 sums are finite exactly when their FP32 parts are (checked in FP32)
    const float fin = (ax.s - ax.s) + (ax.c - ax.c) + (ay.s - ay.s) + (ay.c - ay.c) + (az.s - az.s) +
                      (az.c - az.c) + (dr.s - dr.s) + (dr.c - dr.c);
    if (!(fin == 0.f)) atomicOr(&v.sc->status, ST_NONFINITE);
    // this particle's time-step bound sqrt_h_a sqrt(h/|a|) in FP32; the
    // minimum over particles (FP32 within a warp) and AdaptiveTimeStep stay FP64
    const float ax32 = (float)axd, ay32 = (float)ayd, az32 = (float)azd;
    const float an = sqrtf(ax32 * ax32 + ay32 * ay32 + az32 * az32);
    const float cand = o.sqrt_h_a32 * sqrtf(Ci.h / an);
    if (cand < dtc) dtc = cand;
  }
  block_dt32_and_pairs(v, Ci.inst, active, dtc, (unsigned long long)npair2, cred);
}

// ---------------------------------------------------------------------------
// The same for the usual options: Morris viscosity, squared-density gradient, no
// tensile instability or XSPH, one h, and pair constants (artificial viscosity,
// masses, flags) the same for every free and every fixed class, taken from the
// launch (Options::spec32: the dam breaks, the channel). FL 1: without strain
// rates; 2: with them (LES, Bingham); 3: with the learned closure's sums too.
//
// The kernel is bound by instruction issue and the latency of its gathers, so
//  - a neighbour is three 16-byte records instead of four (PX32: offset and the
//    magnitude of 1 / density, negative for a fixed one; V32: velocity and pressure;
//    V32LO: the velocity's low-order part and the sound speed, with the density's
//    sign), what else a pair needs following from those;
//  - a lane takes two neighbours at a time: six loads in flight, and every
//    operation that both need in packed FP32x2 arithmetic (one issue slot for
//    the two values, each rounded as the scalar operation rounds);
//  - no branch on the support: outside it kernel and gradient are exact zeros;
//  - otherwise the general kernel's expressions, rounding by rounding, except
//    the artificial viscosity (one hardware reciprocal, without the densities);
//  - the compensated sums are kept apart for the even and the odd neighbours and
//    joined at the end by an exact two-sum;
//  - 2^lg lanes share a particle's list.
// Measured per step (pair kernel alone, before -> now): 6.7M particles with the
// closure 4330 -> 2700 us, 1.0M without strain rates 485 -> 320 us, 86k in 2D
// 24.6 -> 19.5 us, the 920-particle channel 34.8 -> 14.3 us. Register caps: 3D
// 128 (136, 144: 3276; the first form of this kernel at 112: 3173, at 96: 3438).
// ---------------------------------------------------------------------------
PSPH_D float2 f2(float a, float b) { return make_float2(a, b); }
PSPH_D float2 dup(float a) { return make_float2(a, a); }
PSPH_D float2 operator+(float2 a, float2 b) { return __fadd2_rn(a, b); }
PSPH_D float2 operator-(float2 a, float2 b) { return __ffma2_rn(b, dup(-1.f), a); }
PSPH_D float2 operator*(float2 a, float2 b) { return __fmul2_rn(a, b); }
PSPH_D float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
PSPH_D float rsqrt_ftz(float x) {  // 1/sqrt of a positive normal number, 2 ulp
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
PSPH_D float rcp_ftz(float x) {  // 1/x, 1 ulp
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Two Kahan sums side by side.
struct Kahan2 {
  float2 s = make_float2(0.f, 0.f), c = make_float2(0.f, 0.f);
  PSPH_D void add(float2 x) {
    const float2 y = x - c;
    const float2 t = s + y;
    c = (t - s) - y;
    s = t;
  }
};
// s - c of two compensated sums joined: the sum of the s with its rounding error
// (Knuth's two-sum) in c.
PSPH_D void join(float& s, float& c, float s2, float c2) {
  const float t = s + s2, b = t - s;
  const float e = (s - (t - b)) + (s2 - b);
  c = (c + c2) - e;
  s = t;
}

// Kernel and gradient (1/r dW/dr) of two separations in KernF's expressions; exact
// zeros outside the support.
template <int DIM, int KT>
PSPH_D void kern2(float2 q, float2 inv_q, float cwh, float cwg, float2& K, float2& GK) {
  if (KT == 1) {
    float2 t = fma2(q, dup(-0.5f), dup(1.f));
    t.x = fmaxf(t.x, 0.f);
    t.y = fmaxf(t.y, 0.f);
    const float2 t2 = t * t;
    GK = (t2 * t) * dup(cwg * -5.f);
    K = (dup(cwh) * (t2 * t2)) * fma2(q, dup(2.f), dup(1.f));
  } else {
    K = f2(KernF<DIM, KT>::W(q.x, cwh), KernF<DIM, KT>::W(q.y, cwh));
    GK = f2(KernF<DIM, KT>::GK(q.x, inv_q.x, cwg), KernF<DIM, KT>::GK(q.y, inv_q.y, cwg));
  }
}

// On a Shepard step the filter divides SumDen by ZWab: FP32 sums whose rounding
// goes into the density and, times c^2, into the next step's pressure. They are
// then taken one neighbour after the other in the order of the cells and their
// x-slabs, a slab's particles by original index, as the general kernel's
// expressions take them, so that a filtered density depends neither on the pair
// kernel's lanes nor on the sort's free-first order. (ZWab, SumDen) of particle i.
template <int DIM, int KT, bool OWN>
__device__ __forceinline__ float2 filter_sums(const DevView& v, const int* __restrict__ orig, int i, int cnt, int inst) {
  const Options& o = v.o;
  const Spec32& c32 = OWN ? v.forms[inst].spec32c : o.spec32c;
  const GridDev& g = grid_of(v, inst);
  const float3 cs = cell_size_f(g);
  const float4 xi = v.S.PX32[i];
  const float hi = c32.h, ih = OWN ? c32.inv_h : o.inv_h32, ih2 = ih * ih;
  const float cwh = KernF<DIM, KT>::cw() * (DIM == 2 ? ih2 : ih2 * ih);
  float zw = 0.f, sd = 0.f;
  auto one = [&](const int e) {
    const float4 oj = v.S.PX32[e & kIndexMask];
    float x0, x1, x2;
    rel_pos<DIM>(cs, xi, oj, entry_code(e), x0, x1, x2);
    const float r2 = x0 * x0 + x1 * x1 + x2 * x2;
    if (r2 > g.cellfac2_32 * hi * hi) return;
    const float inv_r = (r2 > 0.f) ? rsqrtf(r2) : 0.f;
    const float q = r2 * inv_r * ih;
    const float K = KernF<DIM, KT>::W(q, cwh);
    const float mj = kind_free(oj.w) ? c32.m_free : c32.m_wall;
    const float inv_j = with_sign(oj.w, v.S.V32LO[e & kIndexMask].w);
    zw += mj * inv_j * K;
    sd += mj * K;
  };
  auto entry = [&](int k) { return v.S.nl[nl_index(v.nl_stride, i, k)]; };
  for (int k = 0; k < cnt;) {
    // the entries of one slab: its free particles, then its fixed ones, each by original index
    const int code = entry_code(entry(k)), j0 = entry(k) & kIndexMask, cell = v.S.cellid[j0];
    int slab = 0;
    while (slab + 1 < o.xsub && j0 >= v.S.sstart[sort_bin(cell, o.xsub, slab + 1)]) ++slab;
    const unsigned bin = sort_bin(cell, o.xsub, slab);
    const int fixed_at = v.S.sstart[bin + 1], slab_end = v.S.sstart[bin + 2];
    auto below = [&](int e, int at) { return e < cnt && entry_code(entry(e)) == code && (entry(e) & kIndexMask) < at; };
    int mid = k, end;
    while (below(mid, fixed_at)) ++mid;
    for (end = mid; below(end, slab_end);) ++end;
    int a = k, b = mid;
    while (a < mid || b < end) {
      const int ea = a < mid ? entry(a) : 0, eb = b < end ? entry(b) : 0;
      const bool first = b >= end || (a < mid && orig[ea & kIndexMask] < orig[eb & kIndexMask]);
      one(first ? ea : eb);
      if (first) ++a;
      else ++b;
    }
    k = end;
  }
  return make_float2(zw, sd);
}

// On a Shepard step particle i's sums in that order in place of the lanes', where the
// filter can apply (ZWab above 0.6).
template <int DIM, int KT, bool OWN>
__device__ __noinline__ void filter_particle(const DevView& v, int i) {
  const Persist& P = cur_persist(v);
  const PClass32& C = v.cls32[P.cls[i]];
  if (!(C.flags & CF_SHEPARD) || v.inst[C.inst].shepard_counter != v.o.shepard_step) return;
  if (!(v.S.zwab[i] > 0.599) || v.S.cellid[i] < 0 || v.S.nl_count[i] < 0) return;
  const float2 f = filter_sums<DIM, KT, OWN>(v, P.orig, i, v.S.nl_count[i], C.inst);
  v.S.zwab[i] = f.x;
  v.S.sumden[i] = f.y;
}

constexpr int kSumsMax = 20;  // a particle's sums on their way to its thread

// OWN: an instance's own constants (InstForm), for ensembles whose instances differ.
template <int DIM, int KT, int FL, bool OWN>
__global__ void __maxnreg__(DIM == 3 ? 128 : (FL == 1 ? 96 : 112)) forces_spec32_kernel(DevView v, int lg) {
  // in 3D the partner's mass is folded into the kernel's constants (the closure
  // flavour does not fit its registers otherwise: 3204 us against 2740)
  constexpr bool FOLD = DIM == 3;
  extern __shared__ float staged[];  // kSumsMax rows of (block size >> lg), when lg > 0
  __shared__ unsigned long long cred[32];
  const StepScalars* sc = v.sc;
  if (sc->all_stop) return;
  const Persist& P = cur_persist(v);
  const int n = sc->n;
  const int lane = threadIdx.x & 31, L = 1 << lg, sub = lane & (L - 1);
  int i = (blockIdx.x * blockDim.x + threadIdx.x) >> lg;
  const Options& o = v.o;
  const PClass32* __restrict__ CT = v.cls32;
  unsigned npair2 = 0;  // 2 per pair with a free partner, 1 per wall partner (the pair is counted once)
  bool active = false;
  int cell = -1, ci_cls = 0;
  if (i < n) {
    ci_cls = P.cls[i];
    bool run = !v.inst[CT[ci_cls].inst].stop;
    if (OWN) run = run && v.forms[CT[ci_cls].inst].spec32;
    active = run && (CT[ci_cls].flags & CF_FREE);
    cell = v.S.cellid[i];
    if (run && !active && sub == 0) {
      v.S.A4[i] = make_double4_32a(o.gravity[0], o.gravity[1], o.gravity[2], 0.0);
      v.S.zwab[i] = 1.0;
    }
  }
  const PClass32& Ci = CT[ci_cls];
  const int inst_i = Ci.inst;
  const GridDev& g = grid_of(v, inst_i);
  const InstState& Is = v.inst[inst_i];
  const int is = active ? i : 0;
  const float4 xi = v.S.PX32[is];
  const float4 vi = v.S.V32[is];
  const float4 vl = v.S.V32LO[is];
  const float inv_i = with_sign(xi.w, vl.w), Pi = vi.w * inv_i * inv_i, snd_i = fabsf(vl.w);
  const Spec32& c32 = OWN ? v.forms[inst_i].spec32c : o.spec32c;
  const float inv_h = OWN ? c32.inv_h : o.inv_h32;
  const float mui = o.dyn_mu ? v.S.MU32[is] : (OWN ? c32.mu : o.mu_u32);
  const bool shep = (Ci.flags & CF_SHEPARD) && (Is.shepard_counter == o.shepard_step);
  const float3 cs = cell_size_f(g);
  const float reach2 = g.cellfac2_32 * c32.h * c32.h;
  const float ih2 = inv_h * inv_h;
  float cwh = KernF<DIM, KT>::cw() * (DIM == 2 ? ih2 : ih2 * inv_h), cwg = cwh * ih2;
  if (FOLD) {
    cwh *= c32.m_free;
    if (FL == 1) cwg *= c32.m_free;
  }
  Kahan2 ax, ay, az, dr;
  float2 zw = dup(0.f), sd = dup(0.f);
  // strain-rate sums as sums of products a_r x_c (a = c2 vab); without the
  // closure (whose vorticity needs the antisymmetric part) the off-diagonal
  // pairs summed
  float m00 = 0.f, m11 = 0.f, m22 = 0.f, m01 = 0.f, m02 = 0.f, m12 = 0.f, m10 = 0.f, m20 = 0.f, m21 = 0.f;
  int nnb = 0;
  // two neighbours; the second one counts when both is set
  auto pairs = [&](const int ea, const int eb, const bool both) {
    const int ja = ea & kIndexMask, jb = eb & kIndexMask;
    const float4 xa = ld_early(v.S.PX32 + ja), xb = ld_early(v.S.PX32 + jb);
    const float4 va = ld_early(v.S.V32 + ja), vb = ld_early(v.S.V32 + jb);
    const float4 la = ld_early(v.S.V32LO + ja), lb = ld_early(v.S.V32LO + jb);
    const int ca = entry_code(ea), cb = entry_code(eb);
    float2 x0 = fma2(f2(code_back<0>(ca), code_back<0>(cb)), dup(cs.x), f2(xi.x - xa.x, xi.x - xb.x));
    float2 x1 = fma2(f2(code_back<1>(ca), code_back<1>(cb)), dup(cs.y), f2(xi.y - xa.y, xi.y - xb.y));
    float2 x2 = dup(0.f);
    if (DIM == 3) x2 = fma2(f2(code_back<2>(ca), code_back<2>(cb)), dup(cs.z), f2(xi.z - xa.z, xi.z - xb.z));
    float2 r2 = fma2(x1, x1, x0 * x0);
    if (DIM == 3) r2 = fma2(x2, x2, r2);
    if (!both) r2.y = c32.far2;  // beyond the support: every term of it is zero
    const bool fa = kind_free(xa.w), fb = kind_free(xb.w);
    const bool ia = r2.x <= reach2, ib = r2.y <= reach2;
    npair2 += (ia ? (fa ? 1u : 2u) : 0u) + (ib ? (fb ? 1u : 2u) : 0u);
    if (FL == 3) nnb += (ia ? 1 : 0) + (ib ? 1 : 0);
    const float2 inv_r = f2(rsqrt_ftz(fmaxf(r2.x, 1e-30f)), rsqrt_ftz(fmaxf(r2.y, 1e-30f)));
    const float2 q = r2 * inv_r * dup(inv_h);
    float2 K, GK;
    kern2<DIM, KT>(q, inv_r * dup(c32.h), cwh, cwg, K, GK);
    const float2 inv_j = f2(with_sign(xa.w, la.w), with_sign(xb.w, lb.w));
    // StrainRate += (m_j / rho_j) S with S = -GK [2 v_a x_a, v_a x_b + v_b x_a, ...]
    // (Source/Interaction.cpp:114-117, no 1/2): a = c2 vab, S_rc = a_r x_c + a_c x_r;
    // before the mass is folded in, in the general kernel's roundings: a feature
    // of the closure near the edge of its range would pick the other model
    float2 c2 = dup(0.f);
    if (FL >= 2) {
      const float ka = fa ? c32.sr_free : c32.sr_wall, kb = fb ? c32.sr_free : c32.sr_wall;  // -1, or 0 where no rate is taken
      const float2 m = f2(fa ? c32.m_free : c32.m_wall, fb ? c32.m_free : c32.m_wall);
      c2 = GK * f2(ka, kb) * ((c32.wall_scaled ? m : dup(c32.m_free)) * inv_j);
      if (FOLD) GK = GK * dup(c32.m_free);
    }
    float2 mj = dup(c32.m_free);
    if (c32.wall_scaled) {
      if (FOLD) {
        const float2 w = f2(fa ? 1.f : c32.wall_scale, fb ? 1.f : c32.wall_scale);
        K = K * w;
        GK = GK * w;
      } else {
        mj = f2(fa ? c32.m_free : c32.m_wall, fb ? c32.m_free : c32.m_wall);
      }
    }
    float2 v0 = f2(vi.x - va.x, vi.x - vb.x) + f2(vl.x - la.x, vl.x - lb.x);
    float2 v1 = f2(vi.y - va.y, vi.y - vb.y) + f2(vl.y - la.y, vl.y - lb.y);
    float2 v2 = f2(vi.z - va.z, vi.z - vb.z) + f2(vl.z - la.z, vl.z - lb.z);
    float2 vx = fma2(v1, x1, v0 * x0);
    if (DIM == 3) vx = fma2(v2, x2, vx);
    // pressure and artificial viscosity: (-a c MU + b MU^2) / rho_ij with MU = h v.x / D;
    // rho_ij = (1/inv_i + 1/inv_j) / 2
    float2 s = dup(Pi) + f2(va.w, vb.w) * inv_j * inv_j;
    if (c32.av) {
      const float2 vm = f2(fminf(vx.x, 0.f), fminf(vx.y, 0.f));
      const float2 D = r2 + dup(c32.eps2);
      const float2 ivp = dup(inv_i) * inv_j;
      const float2 c = (dup(snd_i) + f2(fabsf(la.w), fabsf(lb.w))) * ivp;
      const float2 den = D * (dup(inv_i) + inv_j);
      float2 num = vm * dup(c32.neg_alpha_h) * c;
      float2 rc = f2(rcp_ftz(den.x), rcp_ftz(den.y));
      if (c32.beta_h2 != 0.f) num = fma2(vm * vm * ivp, dup(2.f * c32.beta_h2) * f2(rcp_ftz(D.x), rcp_ftz(D.y)), num);
      s = fma2(num, rc, s);
    }
    s = s * GK * dup(-1.f);
    float2 c = dup(0.f);
    float2 w0 = v0, w1 = v1, w2 = v2;
    {
      float2 mu2 = dup(2.f * mui);
      if (o.dyn_mu) {
        // harmonic mean with a free neighbour, the own viscosity with a wall
        const float ma = v.S.MU32[ja], mb = v.S.MU32[jb];
        mu2 = f2(fa ? __fdividef(4.f * mui * ma, mui + ma) : 2.f * mui, fb ? __fdividef(4.f * mui * mb, mui + mb) : 2.f * mui);
      }
      c = mu2 * dup(inv_i) * inv_j * GK;
    }
    if (!(fa && fb)) {  // walls: their no-slip velocity, or no viscous term where both slip
      if (!fa) {
        const float4 ns = v.S.NSV32[ja];
        w0.x = (vi.x - (2.f * va.x - ns.x)) + (vl.x - 2.f * la.x);
        w1.x = (vi.y - (2.f * va.y - ns.y)) + (vl.y - 2.f * la.y);
        w2.x = (vi.z - (2.f * va.z - ns.z)) + (vl.z - 2.f * la.z);
        if (!c32.wall_visc) c.x = 0.f;
      }
      if (!fb) {
        const float4 ns = v.S.NSV32[jb];
        w0.y = (vi.x - (2.f * vb.x - ns.x)) + (vl.x - 2.f * lb.x);
        w1.y = (vi.y - (2.f * vb.y - ns.y)) + (vl.y - 2.f * lb.y);
        w2.y = (vi.z - (2.f * vb.z - ns.z)) + (vl.z - 2.f * lb.z);
        if (!c32.wall_visc) c.y = 0.f;
      }
    }
    const float2 md = FOLD ? inv_j : mj * inv_j;
    if (FL >= 2) {
      const float2 a0 = c2 * w0, a1 = c2 * w1, a2 = c2 * w2;
      auto two = [](float& m, float2 a, float2 x) { m = fmaf(a.y, x.y, fmaf(a.x, x.x, m)); };
      two(m00, a0, x0);
      two(m11, a1, x1);
      two(m01, a0, x1);
      if (DIM == 3) {
        two(m22, a2, x2);
        two(m02, a0, x2);
        two(m12, a1, x2);
      }
      two(FL == 3 ? m10 : m01, a1, x0);
      two(FL == 3 ? m20 : m02, a2, x0);
      two(FL == 3 ? m21 : m12, a2, x1);
    }
    auto times_m = [&](float2 f) { return FOLD ? f : mj * f; };
    ax.add(times_m(fma2(s, x0, c * w0)));
    ay.add(times_m(fma2(s, x1, c * w1)));
    if (DIM == 3) az.add(times_m(fma2(s, x2, c * w2)));
    dr.add(md * (GK * vx));  // times rho_i at the end
    zw = fma2(md, K, zw);
    if (shep) sd = FOLD ? sd + K : fma2(mj, K, sd);
  };
  const int cnt = (active && cell >= 0) ? v.S.nl_count[i] : 0;
  if (cnt >= 0) {
    // pair p of the list: entries 2p and 2p + 1, half a 16-byte chunk
    const int2* __restrict__ nl2 = reinterpret_cast<const int2*>(v.S.nl) + 2 * (size_t)nl_slot(i);
    const size_t N = 2 * (size_t)v.nl_stride;
    const int np = (cnt + 1) >> 1;
    int2 next = (sub < np) ? nl2[(sub >> 1) * N + (sub & 1)] : make_int2(0, 0);
    for (int p = sub; p < np; p += L) {
      const int2 e = next;
      const int q = p + L;
      if (q < np) next = nl2[(size_t)(q >> 1) * N + (q & 1)];
      const bool both = 2 * p + 1 < cnt;
      pairs(e.x, both ? e.y : e.x, both);
    }
  } else if (sub == 0) {  // list overflow: scan the cells
    NbrSource<DIM> src;
    src.init(v, g, i, true, 1.0f);
    while (true) {
      int code;
      const int j = src.next(v, &code);
      if (j < 0) break;
      const int e = (int)((unsigned)code << kCodeShift) | j;
      pairs(e, e, false);
    }
  }
  // even and odd neighbours together, then the lanes of the particle
  float out[kSumsMax];
  {
    Kahan2* const k[4] = {&ax, &ay, &az, &dr};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float ss = k[e]->s.x, cc = k[e]->c.x;
      join(ss, cc, k[e]->s.y, k[e]->c.y);
      for (int m = 1; m < L; m <<= 1) {
        const float s2 = __shfl_xor_sync(0xffffffffu, ss, m), c2 = __shfl_xor_sync(0xffffffffu, cc, m);
        // the same operands in the same order on both sides
        const bool up = sub & m;
        float a = up ? s2 : ss, b = up ? c2 : cc;
        join(a, b, up ? ss : s2, up ? cc : c2);
        ss = a;
        cc = b;
      }
      out[2 * e] = ss;
      out[2 * e + 1] = cc;
    }
    out[8] = zw.x + zw.y;
    out[9] = sd.x + sd.y;
    const float mm[9] = {m00, m11, m22, m01, m02, m12, m10, m20, m21};
#pragma unroll
    for (int e = 0; e < 9; ++e) out[10 + e] = mm[e];
    out[19] = (float)nnb;
    const int last = FL == 1 ? 10 : (FL == 2 ? 16 : 20);
#pragma unroll
    for (int e = 8; e < 20; ++e)
      if (e < last)
        for (int m = 1; m < L; m <<= 1) out[e] += __shfl_xor_sync(0xffffffffu, out[e], m);
    if (lg > 0) {  // one thread per particle from here: full warps for the FP64 conversions
      const int np = blockDim.x >> lg;
      if (sub == 0)
#pragma unroll
        for (int e = 0; e < 20; ++e)
          if (e < last) staged[e * np + (threadIdx.x >> lg)] = out[e];
      __syncthreads();
      i = blockIdx.x * np + threadIdx.x;
      active = (int)threadIdx.x < np && i < n;
      if (active) {
#pragma unroll
        for (int e = 0; e < 20; ++e)
          if (e < last) out[e] = staged[e * np + threadIdx.x];
        ci_cls = P.cls[i];
        active = !v.inst[CT[ci_cls].inst].stop && (CT[ci_cls].flags & CF_FREE);
        if (OWN) active = active && v.forms[CT[ci_cls].inst].spec32;
      }
    }
  }
  const int inst = CT[ci_cls].inst;
  float dtc = FLT_MAX;
  if (active) {
    auto value = [&](int e) { return (double)out[2 * e] - (double)out[2 * e + 1]; };
    const double axd = o.gb[0] + value(0), ayd = o.gb[1] + value(1), azd = o.gb[2] + value(2);
    const double drd = value(3) * P.X4[i].w;
    v.S.A4[i] = make_double4_32a(axd, ayd, azd, drd);
    v.S.zwab[i] = out[8];
    if (o.any_shepard) v.S.sumden[i] = out[9];
    if (FL >= 2) {
      const float* m = out + 10;
      // symmetric sums 2 m_rr and m_rc + m_cr; the antisymmetric m_rc - m_cr
      // (closure) is the vorticity's
      const float sr0 = 2.f * m[0], sr4 = 2.f * m[1], sr8 = 2.f * m[2];
      const float sr1 = FL == 3 ? m[3] + m[6] : m[3], sr2 = FL == 3 ? m[4] + m[7] : m[4],
                  sr5 = FL == 3 ? m[5] + m[8] : m[5];
      // the 6 distinct sums in FP32 (the FP64 tensor is built on download)
      float2* q = reinterpret_cast<float2*>(v.S.sr32 + 6 * (size_t)i);
      q[0] = make_float2(sr0, sr1);
      q[1] = make_float2(sr2, sr4);
      q[2] = make_float2(sr5, sr8);
      // Mat1's ShearRate contraction (Source/Particle.cpp:151-153) of the
      // symmetric sums, in FP32: the update and the closure take it from here
      const float temp = sr0 * sr0 + 2.f * sr1 * sr1 + 2.f * sr2 * sr2 + sr4 * sr4 + 2.f * sr5 * sr5 + sr8 * sr8;
      v.S.cshear[i] = sqrtf(0.5f * temp);
      if (FL == 3 && (CT[ci_cls].flags & CF_LES)) {
        const float w01 = m[3] - m[6], w02 = m[4] - m[7], w12 = m[5] - m[8];
        v.S.cvort[i] = sqrtf(w01 * w01 + w02 * w02 + w12 * w12);
        v.S.cnnb[i] = out[19];
        const float det =
            sr0 * (sr4 * sr8 - sr5 * sr5) - sr1 * (sr1 * sr8 - sr5 * sr2) + sr2 * (sr1 * sr5 - sr4 * sr2);
        v.S.cr3[i] = temp > 0.f ? det / (temp * sqrtf(temp)) : 0.f;
      }
    }
    // the FP64 sums are finite exactly when their FP32 parts are (checked in FP32)
    float fin = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) fin += out[e] - out[e];
    if (!(fin == 0.f)) atomicOr(&v.sc->status, ST_NONFINITE);
    // this particle's time-step bound sqrt_h_a sqrt(h/|a|) in FP32; the
    // minimum over particles (FP32 within a warp) and AdaptiveTimeStep stay FP64
    const float ax32 = d2f_rn(axd), ay32 = d2f_rn(ayd), az32 = d2f_rn(azd);
    const float an = sqrtf(ax32 * ax32 + ay32 * ay32 + az32 * az32);
    const float h = OWN ? CT[ci_cls].h : c32.h;  // (with lanes this thread's particle may be another instance's)
    const float cand = o.sqrt_h_a32 * sqrtf(h / an);
    if (cand < dtc) dtc = cand;
  }
  block_dt32_and_pairs(v, inst, active, dtc, (unsigned long long)npair2, cred);
  // the filter's sums last and in a call of its own, which then takes no registers from
  // the pair loop (5.6M particles with the closure, which never filter: 2,299 us, 2,331
  // with the call ahead of the reductions)
  if (active && o.any_shepard && v.inst[inst].shepard_counter == o.shepard_step) filter_particle<DIM, KT, OWN>(v, i);
}

// ---------------------------------------------------------------------------
// Soil / solid pair force (CalcForce2233, Source/Interaction.cpp:186-377) in
// FP32 with compensated sums. The FP64 preparation (prepare_wall_kernel:
// wall stress interpolation, partner-visible wall density, TIR) runs first;
// solid_copies32_kernel then takes the FP32 copies the pair loop reads.
// ---------------------------------------------------------------------------
// Symmetric 3x3 tensor (the stresses and TIR are symmetric: Jaumann rate of a
// symmetric stress, R diag R^T) as 6 floats in two float4: 00 01 02 11 | 12 22.
// An off-diagonal pair agrees to FP64 rounding (the two entries come from the
// same terms summed in another order), far below FP32's: the upper entry is
// taken. Conversions on the integer pipe (d2f_rn), no FP64 instruction.
PSPH_D void sym_store(float4* dst, size_t w, const double* m) {
  dst[2 * w] = make_float4(d2f_rn(m[0]), d2f_rn(m[1]), d2f_rn(m[2]), d2f_rn(m[4]));
  dst[2 * w + 1] = make_float4(d2f_rn(m[5]), d2f_rn(m[8]), 0.f, 0.f);
}

template <int DIM>
__global__ void __launch_bounds__(kFT32) solid_copies32_kernel(DevView v) {
  const StepScalars* sc = v.sc;
  if (sc->all_stop) return;
  const Persist& P = cur_persist(v);
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= sc->n) return;
  const PClass32& C = v.cls32[P.cls[w]];
  if (v.inst[C.inst].stop || (v.o.mix_soil && v.forms[C.inst].soil32)) return;  // (soil_records)
  const double4_32a vv = P.V4[w];
  float lx, ly, lz;
  const float vx = d2f_split(vv.x, &lx), vy = d2f_split(vv.y, &ly), vz = d2f_split(vv.z, &lz);
  // the velocity's low-order part: near-rigid motion (a column settling as one
  // body) makes v_i - v_j far smaller than v, and the pair differences take
  // (hi_i - hi_j) + (lo_i - lo_j), exact to ~2^-48 of |v|
  const double4_32a d = v.S.D4[w];
  const double* sg = P.sigma + tensor_row(P, w);
  v.S.V32[w] = make_float4(vx, vy, vz, d2f_rn(vv.w));
  v.S.V32LO[w] = make_float4(lx, ly, lz, 0.f);
  v.S.D32[w] = make_float4(d2f_rn(d.x), d2f_rn(d.y), d2f_rn(d.z), d2f_rn(d.w));
  sym_store(v.S.SIG32, (size_t)w, sg);
  if (v.o.any_ti) sym_store(v.S.TIR32, (size_t)w, P.tir + tensor_row(P, w));
  if (!(C.flags & CF_FREE)) {
    const double4_32a vb = (v.o.scheme == PSPH_MVERLET) ? P.H4[w] : P.H4b[w];
    v.S.VB32[w] = make_float4(d2f_rn(vb.x), d2f_rn(vb.y), d2f_rn(vb.z), 0.f);
    const double4_32a ns = v.S.nsv4[w];
    v.S.NSV32[w] = make_float4(d2f_rn(ns.x), d2f_rn(ns.y), d2f_rn(ns.z), 0.f);
  }
}

// The strain-rate (00 01 02 11 12 22) and rotation-rate (01 02 12) sums of a
// soil or solid particle, in FP32 as they are summed: the update widens them
// (36 bytes instead of two FP64 tensors), a download expands them.
PSPH_D void store_rates32(const DevView& v, int i, float s0, float s1, float s2, float s3, float s4, float s5,
                          float r0, float r1, float r2) {
  float4* q = v.S.rates32 + 3 * (size_t)i;
  q[0] = make_float4(s0, s1, s2, s3);
  q[1] = make_float4(s4, s5, r0, r1);
  q[2] = make_float4(r2, 0.f, 0.f, 0.f);
}

template <int DIM, int KT>
__global__ void __maxnreg__(128) forces_solid32_kernel(DevView v) {
  __shared__ double red[32];
  __shared__ unsigned long long cred[32];
  const StepScalars* sc = v.sc;
  if (sc->all_stop) return;
  const Persist& P = cur_persist(v);
  const int n = sc->n;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const Options& o = v.o;
  const PClass32* __restrict__ CT = v.cls32;
  double dtc = DBL_MAX;
  unsigned npair2 = 0;  // 2 per pair with a free partner, 1 per wall partner (the pair is counted once)
  bool active = false;
  int cell = -1, ci_cls = 0;
  if (i < n) {
    ci_cls = P.cls[i];
    bool run = !v.inst[CT[ci_cls].inst].stop;
    if (o.mix_soil) run = run && !v.forms[CT[ci_cls].inst].soil32;  // (forces_soil32_kernel takes those)
    active = run && (CT[ci_cls].flags & CF_FREE);
    cell = v.S.cellid[i];
    if (run && !active) {
      v.S.A4[i] = make_double4_32a(o.gravity[0], o.gravity[1], o.gravity[2], 0.0);
      v.S.zwab[i] = 1.0;
    }
  }
  const PClass32& Ci = CT[ci_cls];
  const GridDev& g = grid_of(v, Ci.inst);
  const InstState& Is = v.inst[Ci.inst];
  const int is = active ? i : 0;
  const float4 oi = v.S.OFF32[is];
  const float4 vi = v.S.V32[is];
  const float4 vil = v.S.V32LO[is];
  const float4 di4 = v.S.D32[is];
  const float di = di4.w, inv_i = di4.x, ci_snd = di4.z;
  const float mi = Ci.mass, hi = fabsf(oi.w);
  const bool shep = (Ci.flags & CF_SHEPARD) && (Is.shepard_counter == o.shepard_step);
  const float4 sa = v.S.SIG32[2 * (size_t)is], sb = v.S.SIG32[2 * (size_t)is + 1];
  const float Si[6] = {sa.x, sa.y, sa.z, sa.w, sb.x, sb.y};
  float Ti[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (o.any_ti) {
    const float4 ta = v.S.TIR32[2 * (size_t)is], tb = v.S.TIR32[2 * (size_t)is + 1];
    Ti[0] = ta.x; Ti[1] = ta.y; Ti[2] = ta.z; Ti[3] = ta.w; Ti[4] = tb.x; Ti[5] = tb.y;
  }
  const float I22 = (DIM == 2) ? 0.f : 1.f;  // Domain::I (Source/Domain.cpp:1665)
  const float3 cs = cell_size_f(g);
  const bool xsph_on = o.xsph != 0.0;
  const float xsph = (float)o.xsph;
  const int grad_type = o.grad_type;
  Kahan ax, ay, az, dr;
  float zw = 0.f, sd = 0.f, xs0 = 0.f, xs1 = 0.f, xs2 = 0.f;
  float sr0 = 0.f, sr1 = 0.f, sr2 = 0.f, sr3 = 0.f, sr4 = 0.f, sr5 = 0.f;  // 00 01 02 11 12 22
  float rr0 = 0.f, rr1 = 0.f, rr2 = 0.f;                                  // 01 02 12
  const float cf2 = (float)(g.cellfac * g.cellfac);
  NbrSource<DIM> src;
  src.init(v, g, i, active && cell >= 0, 1.0f);
  while (true) {
    int code;
    const int j = src.next(v, &code);
    if (j < 0) break;
    const float4 oj = v.S.OFF32[j];
    float x0, x1, x2;
    rel_pos<DIM>(cs, oi, oj, code, x0, x1, x2);
    const float hb = 0.5f * (hi + fabsf(oj.w));
    const float r2 = x0 * x0 + x1 * x1 + x2 * x2;
    if (r2 > cf2 * hb * hb) continue;  // the support test (the list holds a margin)
    const PClass32& Cj = CT[P.cls[j]];
    const int fjf = Cj.flags;
    const bool fj = fjf & CF_FREE;
    npair2 += fj ? 1ull : 2ull;
    const float ih = 1.f / hb;
    const float inv_r = (r2 > 0.f) ? rsqrtf(r2) : 0.f;
    const float q = r2 * inv_r * ih;
    const float ih2 = ih * ih;
    const float cwh = KernF<DIM, KT>::cw() * (DIM == 2 ? ih2 : ih2 * ih);
    const float cwg = cwh * ih2;
    const float GK = KernF<DIM, KT>::GK(q, hb * inv_r, cwg);
    const float K = KernF<DIM, KT>::W(q, cwh);
    const float4 vj = v.S.V32[j];
    const bool soil = (Ci.material * Cj.material == 9);
    float dj, inv_j, cj_snd = 0.f, mj;
    if (fj) {
      const float4 dj4 = v.S.D32[j];
      dj = dj4.w; inv_j = dj4.x; cj_snd = dj4.z; mj = Cj.mass;
    } else if (soil) {  // soil walls take the partner's density (Source/Interaction.cpp:201-205)
      dj = di; inv_j = inv_i; mj = Cj.fpmassc * mi;
    } else {
      if (o.uniform_eos) {
        const float4 dj4 = v.S.D32[j];
        dj = dj4.w; inv_j = dj4.x; cj_snd = dj4.z;
      } else {
        const PClass& C64 = v.cls[ci_cls];
        const double d64 = density_solid(C64.pres_eq, C64.cs, C64.p0, (double)vj.w, C64.rho0);
        dj = (float)d64;
        inv_j = 1.f / dj;
        cj_snd = (float)sound_speed(C64.pres_eq, C64.cs, d64, C64.rho0);
      }
      mj = Cj.fpmassc * mi;
    }
    const float4 vjl = v.S.V32LO[j];
    const float v0 = (vi.x - vj.x) + (vil.x - vjl.x), v1 = (vi.y - vj.y) + (vil.y - vjl.y),
                v2 = (vi.z - vj.z) + (vil.z - vjl.z);
    const float vx = v0 * x0 + v1 * x1 + v2 * x2;
    float PIs = 0.f;  // PIij = PIs I
    const float Alpha = 0.5f * (Ci.alpha + Cj.alpha), Beta = 0.5f * (Ci.beta + Cj.beta);
    if ((Alpha != 0.f || Beta != 0.f) && vx < 0.f) {
      const float Cij = soil ? 0.5f * (Ci.cs + Cj.cs) : 0.5f * (ci_snd + cj_snd);
      const float D = r2 + 0.01f * hb * hb;
      const float t = hb * vx;
      PIs = t * (Alpha * Cij * D + Beta * t) / (D * D * (0.5f * (di + dj)));
    }
    float vab0, vab1, vab2;
    if (fj) { vab0 = v0; vab1 = v1; vab2 = v2; }
    else if ((Ci.flags | fjf) & CF_NOSLIP) {
      const float4 ns = v.S.NSV32[j];
      vab0 = vi.x - (2.f * vj.x - ns.x);
      vab1 = vi.y - (2.f * vj.y - ns.y);
      vab2 = vi.z - (2.f * vj.z - ns.z);
    } else {
      const float4 vbj = v.S.VB32[j];
      vab0 = vi.x - vbj.x; vab1 = vi.y - vbj.y; vab2 = vi.z - vbj.z;
    }
    const float4 sja = v.S.SIG32[2 * (size_t)j], sjb = v.S.SIG32[2 * (size_t)j + 1];
    const float Sj[6] = {sja.x, sja.y, sja.z, sja.w, sjb.x, sjb.y};
    float M[6];
    if (grad_type == 0) {
      const float ci2 = inv_i * inv_i, cj2 = inv_j * inv_j;
#pragma unroll
      for (int e = 0; e < 6; ++e) M[e] = Si[e] * ci2 + Sj[e] * cj2;
    } else {
      const float c = inv_i * inv_j;
#pragma unroll
      for (int e = 0; e < 6; ++e) M[e] = (Si[e] + Sj[e]) * c;
    }
    M[0] += PIs; M[3] += PIs; M[5] += PIs * I22;
    if ((Ci.flags | fjf) & CF_TI) {
      const float Wd = KernF<DIM, KT>::W((Ci.tid + Cj.tid) * 0.5f * ih, cwh);
      const float TIs = powf(K / Wd, (Ci.tin + Cj.tin) * 0.5f);
      const float4 tja = v.S.TIR32[2 * (size_t)j], tjb = v.S.TIR32[2 * (size_t)j + 1];
      const float Tj[6] = {tja.x, tja.y, tja.z, tja.w, tjb.x, tjb.y};
#pragma unroll
      for (int e = 0; e < 6; ++e) M[e] += (Ti[e] + Tj[e]) * TIs;
    }
    const float g0 = GK * x0, g1 = GK * x1, g2 = GK * x2;
    // row vector (GK x_ij) times M (Mult, External/matvec.h:806)
    ax.add(mj * (g0 * M[0] + g1 * M[1] + g2 * M[2]));
    ay.add(mj * (g0 * M[1] + g1 * M[3] + g2 * M[4]));
    if (DIM == 3) az.add(mj * (g0 * M[2] + g1 * M[4] + g2 * M[5]));
    dr.add(mj * di * inv_j * (v0 * g0 + v1 * g1 + v2 * g2));
    const float md = mj * inv_j;
    zw += md * K;
    const float c2 = -0.5f * GK * md;
    sr0 += c2 * (2.f * vab0 * x0);
    sr1 += c2 * (vab0 * x1 + vab1 * x0);
    sr2 += c2 * (vab0 * x2 + vab2 * x0);
    sr3 += c2 * (2.f * vab1 * x1);
    sr4 += c2 * (vab1 * x2 + vab2 * x1);
    sr5 += c2 * (2.f * vab2 * x2);
    rr0 += c2 * (vab0 * x1 - vab1 * x0);
    rr1 += c2 * (vab0 * x2 - vab2 * x0);
    rr2 += c2 * (vab1 * x2 - vab2 * x1);
    if (xsph_on && fj) {
      const float s = xsph * mj / (0.5f * (di + dj)) * K;
      xs0 -= s * v0; xs1 -= s * v1; xs2 -= s * v2;
    }
    if (shep) sd += mj * K;
  }
  if (active) {
    const double axd = o.gravity[0] + o.body_force[0] + ax.value();
    const double ayd = o.gravity[1] + o.body_force[1] + ay.value();
    const double azd = o.gravity[2] + o.body_force[2] + az.value();
    const double drd = dr.value();
    v.S.A4[i] = make_double4_32a(axd, ayd, azd, drd);
    v.S.zwab[i] = zw;
    if (o.any_shepard) v.S.sumden[i] = sd;
    if (xsph_on) v.S.vxsph4[i] = make_double4_32a(xs0, xs1, xs2, 0.0);
    store_rates32(v, i, sr0, sr1, sr2, sr3, sr4, sr5, rr0, rr1, rr2);
    if (!(isfinite(axd) && isfinite(ayd) && isfinite(azd) && isfinite(drd))) atomicOr(&v.sc->status, ST_NONFINITE);
    // this particle's time-step bound sqrt_h_a sqrt(h/|a|) in FP32; the
    // minimum over particles and AdaptiveTimeStep stay FP64
    const float ax32 = (float)axd, ay32 = (float)ayd, az32 = (float)azd;
    const float an = sqrtf(ax32 * ax32 + ay32 * ay32 + az32 * az32);
    const double cand = (double)((float)o.sqrt_h_a * sqrtf(Ci.h / an));
    if (cand < dtc) dtc = cand;
  }
  block_dt_and_pairs<0>(v, Ci.inst, active, dtc, npair2, red, cred);
}

// The same for soil domains in 2D whose classes share their pair constants
// (Options::soil32: one h, artificial viscosity, sound speed, tensile-instability
// constants and flags; one free mass per instance): the granular columns. As in
// forces_spec32_kernel a lane takes two neighbours at a time in packed FP32x2
// arithmetic, and a neighbour is three 16-byte records
// (written by prepare_wall_kernel)
//   PX32  x, y, Sigma00, Sigma01      V32  vx, vy, Sigma11, 1/density (kFixedMark: fixed)
//   V32LO the low-order parts of vx and vy, vz, whether its TIR is non-zero
// In 2D the entries with a z index meet a zero separation in the acceleration.
// The tensile-instability power is evaluated only where one of the two carries a
// tensile stress (elsewhere it multiplies a zero).
// 1.0M particles in ten columns: 513 us before (nine loads a neighbour and the
// power for every pair), 197 us now.
// OWN: for ensembles whose instances differ (InstForm).
template <int KT, bool OWN>
__global__ void __maxnreg__(112) forces_soil32_kernel(DevView v) {
  __shared__ unsigned long long cred[32];
  const StepScalars* sc = v.sc;
  if (sc->all_stop) return;
  const Persist& P = cur_persist(v);
  const int n = sc->n;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const Options& o = v.o;
  const PClass32* __restrict__ CT = v.cls32;
  float dtc = FLT_MAX;
  unsigned npair2 = 0;  // 2 per pair with a free partner, 1 per wall partner (the pair is counted once)
  bool active = false;
  int cell = -1, ci_cls = 0;
  if (i < n) {
    ci_cls = P.cls[i];
    bool run = !v.inst[CT[ci_cls].inst].stop;
    if (OWN) run = run && v.forms[CT[ci_cls].inst].soil32;
    active = run && (CT[ci_cls].flags & CF_FREE);
    cell = v.S.cellid[i];
    if (run && !active) {
      v.S.A4[i] = make_double4_32a(o.gravity[0], o.gravity[1], o.gravity[2], 0.0);
      v.S.zwab[i] = 1.0;
    }
  }
  const PClass32& Ci = CT[ci_cls];
  const GridDev& g = grid_of(v, Ci.inst);
  const InstState& Is = v.inst[Ci.inst];
  const int is = active ? i : 0;
  const float4 xi = v.S.PX32[is], vi = v.S.V32[is], vl = v.S.V32LO[is];
  const float inv_i = vi.w, mi = Ci.mass, h = Ci.h, ih = 1.f / h, ih2 = ih * ih;
  const float cwh = KernF<2, KT>::cw() * ih2, cwg = cwh * ih2;
  const float ci2 = inv_i * inv_i;
  const float P00 = xi.z * ci2, P01 = xi.w * ci2, P11 = vi.z * ci2;  // the own stress over density squared
  const bool shep = (Ci.flags & CF_SHEPARD) && (Is.shepard_counter == o.shepard_step);
  const float fpm = OWN ? v.forms[Ci.inst].soil_fpm : o.fpm_wall32;
  const bool wall_scaled = fpm != 1.f, av = Ci.alpha != 0.f || Ci.beta != 0.f;
  const float ac = Ci.alpha * Ci.cs;
  const float3 cs = cell_size_f(g);
  const float reach2 = g.cellfac2_32 * h * h, far2 = 100.f * h * h, eps2 = 0.01f * h * h;
  const bool noslip = OWN ? v.forms[Ci.inst].soil_noslip : o.soil_noslip;
  Kahan2 ax, ay, dr;
  float2 zw = dup(0.f), sd = dup(0.f);
  float2 s00 = dup(0.f), s01 = dup(0.f), s11 = dup(0.f), r01 = dup(0.f), s02 = dup(0.f), s12 = dup(0.f);
  auto pairs = [&](const int ea, const int eb, const bool both) {
    const int ja = ea & kIndexMask, jb = eb & kIndexMask;
    const float4 xa = ld_early(v.S.PX32 + ja), xb = ld_early(v.S.PX32 + jb);
    const float4 va = ld_early(v.S.V32 + ja), vb = ld_early(v.S.V32 + jb);
    const float4 la = ld_early(v.S.V32LO + ja), lb = ld_early(v.S.V32LO + jb);
    const int ca = entry_code(ea), cb = entry_code(eb);
    const float2 x0 = fma2(f2(code_back<0>(ca), code_back<0>(cb)), dup(cs.x), f2(xi.x - xa.x, xi.x - xb.x));
    const float2 x1 = fma2(f2(code_back<1>(ca), code_back<1>(cb)), dup(cs.y), f2(xi.y - xa.y, xi.y - xb.y));
    float2 r2 = fma2(x1, x1, x0 * x0);
    if (!both) r2.y = far2;  // beyond the support: every term of it is zero
    const bool fa = soil_free(va.w), fb = soil_free(vb.w);
    const bool ia = r2.x <= reach2, ib = r2.y <= reach2;
    npair2 += (ia ? (fa ? 1u : 2u) : 0u) + (ib ? (fb ? 1u : 2u) : 0u);
    const float2 inv_r = f2(rsqrt_ftz(fmaxf(r2.x, 1e-30f)), rsqrt_ftz(fmaxf(r2.y, 1e-30f)));
    float2 K, GK;
    kern2<2, KT>(r2 * inv_r * dup(ih), inv_r * dup(h), cwh, cwg, K, GK);
    // soil walls take the partner's density (Source/Interaction.cpp:201-205)
    const float2 inv_j = f2(fa ? va.w : inv_i, fb ? vb.w : inv_i);
    float2 mj = dup(mi);
    if (wall_scaled) mj = f2(fa ? mi : fpm * mi, fb ? mi : fpm * mi);
    const float2 v0 = f2(vi.x - va.x, vi.x - vb.x) + f2(vl.x - la.x, vl.x - lb.x);
    const float2 v1 = f2(vi.y - va.y, vi.y - vb.y) + f2(vl.y - la.y, vl.y - lb.y);
    const float2 vx = fma2(v1, x1, v0 * x0);
    const float2 cj2 = inv_j * inv_j;
    float2 M00 = fma2(f2(xa.z, xb.z), cj2, dup(P00));
    const float2 M01_ = fma2(f2(xa.w, xb.w), cj2, dup(P01));
    float2 M11 = fma2(f2(va.z, vb.z), cj2, dup(P11));
    float2 M01 = M01_;
    if (av) {  // PIij = PI I, PI = (a c MU + b MU^2) / rho_ij with MU = h v.x / D
      const float2 t = f2(fminf(vx.x, 0.f), fminf(vx.y, 0.f)) * dup(h);
      const float2 D = r2 + dup(eps2);
      const float2 ivp = dup(2.f * inv_i) * inv_j;  // rho_ij = (1/inv_i + 1/inv_j) / 2
      const float2 den = D * D * (dup(inv_i) + inv_j);
      const float2 PI = t * fma2(dup(Ci.beta), t, dup(ac) * D) * ivp * f2(rcp_ftz(den.x), rcp_ftz(den.y));
      M00 = M00 + PI;
      M11 = M11 + PI;
    }
    if (vl.w + la.w + lb.w > 0.f) {  // a tensile stress on either side of one of the pairs
      const float Wd = KernF<2, KT>::W(Ci.tid * ih, cwh);
      auto add = [&](float k, int j, float tj, float& m00, float& m01, float& m11) {
        if (!(vl.w + tj > 0.f)) return;
        const float f = powf(k / Wd, Ci.tin);
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
        if (vl.w > 0.f) t = v.S.TIR32[2 * (size_t)is];
        if (tj > 0.f) {
          const float4 u = v.S.TIR32[2 * (size_t)j];
          t.x += u.x; t.y += u.y; t.w += u.w;
        }
        m00 += t.x * f;
        m01 += t.y * f;
        m11 += t.w * f;
      };
      add(K.x, ja, la.w, M00.x, M01.x, M11.x);
      add(K.y, jb, lb.w, M00.y, M01.y, M11.y);
    }
    const float2 g0 = GK * x0, g1 = GK * x1;
    // row vector (GK x_ij) times M (Mult, External/matvec.h:806)
    ax.add(mj * fma2(g1, M01, g0 * M00));
    ay.add(mj * fma2(g1, M11, g0 * M01));
    const float2 md = mj * inv_j;
    dr.add(md * fma2(v1, g1, v0 * g0));  // times rho_i at the end
    zw = fma2(md, K, zw);
    if (shep) sd = fma2(mj, K, sd);
    float2 w0 = v0, w1 = v1, w2 = f2(vl.z - la.z, vl.z - lb.z);
    if (!(fa && fb)) {
      auto wall = [&](int j, float4 vj, float4 lj, float& a0, float& a1, float& a2) {
        if (noslip) {
          const float4 ns = v.S.NSV32[j];
          a0 = vi.x - (2.f * vj.x - ns.x);
          a1 = vi.y - (2.f * vj.y - ns.y);
          a2 = vl.z - (2.f * lj.z - ns.z);
        } else {
          const float4 q = v.S.VB32[j];
          a0 = vi.x - q.x; a1 = vi.y - q.y; a2 = vl.z - q.z;
        }
      };
      if (!fa) wall(ja, va, la, w0.x, w1.x, w2.x);
      if (!fb) wall(jb, vb, lb, w0.y, w1.y, w2.y);
    }
    const float2 c2 = dup(-0.5f) * GK * md;
    const float2 p01 = w0 * x1, p10 = w1 * x0;
    s00 = fma2(c2, w0 * x0, s00);
    s11 = fma2(c2, w1 * x1, s11);
    s01 = fma2(c2, p01 + p10, s01);
    r01 = fma2(c2, p01 - p10, r01);
    s02 = fma2(c2, w2 * x0, s02);
    s12 = fma2(c2, w2 * x1, s12);
  };
  const int cnt = (active && cell >= 0) ? v.S.nl_count[i] : 0;
  if (cnt >= 0) {
    // pair p of the list: entries 2p and 2p + 1, half a 16-byte chunk
    const int2* __restrict__ nl2 = reinterpret_cast<const int2*>(v.S.nl) + 2 * (size_t)nl_slot(i);
    const size_t N = 2 * (size_t)v.nl_stride;
    const int np = (cnt + 1) >> 1;
    int2 next = np > 0 ? nl2[0] : make_int2(0, 0);
    for (int p = 0; p < np; ++p) {
      const int2 e = next;
      if (p + 1 < np) next = nl2[(size_t)((p + 1) >> 1) * N + ((p + 1) & 1)];
      const bool both = 2 * p + 1 < cnt;
      pairs(e.x, both ? e.y : e.x, both);
    }
  } else {  // list overflow: scan the cells
    NbrSource<2> src;
    src.init(v, g, i, true, 1.0f);
    while (true) {
      int code;
      const int j = src.next(v, &code);
      if (j < 0) break;
      const int e = (int)((unsigned)code << kCodeShift) | j;
      pairs(e, e, false);
    }
  }
  if (active) {
    auto value = [](Kahan2& k) {
      join(k.s.x, k.c.x, k.s.y, k.c.y);
      return (double)k.s.x - (double)k.c.x;
    };
    const double axd = o.gb[0] + value(ax), ayd = o.gb[1] + value(ay), azd = o.gb[2];
    const double drd = value(dr) * P.X4[i].w;
    v.S.A4[i] = make_double4_32a(axd, ayd, azd, drd);
    v.S.zwab[i] = zw.x + zw.y;
    if (o.any_shepard) v.S.sumden[i] = sd.x + sd.y;
    const float t02 = s02.x + s02.y, t12 = s12.x + s12.y;
    store_rates32(v, i, 2.f * (s00.x + s00.y), s01.x + s01.y, t02, 2.f * (s11.x + s11.y), t12, 0.f, r01.x + r01.y,
                  -t02, -t12);
    const float fin = (ax.s.x - ax.s.x) + (ax.c.x - ax.c.x) + (ay.s.x - ay.s.x) + (ay.c.x - ay.c.x) +
                      (dr.s.x - dr.s.x) + (dr.c.x - dr.c.x);
    if (!(fin == 0.f)) atomicOr(&v.sc->status, ST_NONFINITE);
    // this particle's time-step bound sqrt_h_a sqrt(h/|a|) in FP32; the
    // minimum over particles and AdaptiveTimeStep stay FP64
    const float ax32 = d2f_rn(axd), ay32 = d2f_rn(ayd), az32 = d2f_rn(azd);
    const float an = sqrtf(ax32 * ax32 + ay32 * ay32 + az32 * az32);
    const float cand = (float)o.sqrt_h_a * sqrtf(h / an);
    if (cand < dtc) dtc = cand;
  }
  block_dt32_and_pairs(v, Ci.inst, active, dtc, (unsigned long long)npair2, cred);
}

inline int nblk32(int n) { return n <= 0 ? 1 : (n + kFT32 - 1) / kFT32; }

template <int DIM>
void prepare32_dispatch(const DevView& v, cudaStream_t st) {
  const int nb = nblk32(v.ncap << kWallLanesLog2<DIM>);  // (how many walls there are is known on the device only)
  switch (v.o.kt) {
    case 0: prepare32_kernel<DIM, 0><<<nb, kFT32, 0, st>>>(v); break;
    case 1: prepare32_kernel<DIM, 1><<<nb, kFT32, 0, st>>>(v); break;
    default: prepare32_kernel<DIM, 2><<<nb, kFT32, 0, st>>>(v); break;
  }
}

template <int DIM, int KT>
void spec32_dispatch(const DevView& v, int bt, cudaStream_t st) {
  // lanes per particle: one, and 4 for the quintic spline, whose lists are more
  // than twice as long (the 920-particle channel: 24.6 us with one lane, 14.3
  // with 4; the 1M-particle Wendland dam break: 311 us with one, 365 with two).
  // As in the FP64 form it depends on nothing that an ensemble changes.
  constexpr int lg = KT == PSPH_QUINTIC_SPLINE ? 2 : 0;
  const int per = bt >> lg;
  const int nb = v.ncap <= 0 ? 1 : (v.ncap + per - 1) / per;
  const size_t sm = lg > 0 ? sizeof(float) * kSumsMax * per : 0;
  const Options& o = v.o;
  if (o.mix32) {
    if (!o.need_sr) forces_spec32_kernel<DIM, KT, 1, true><<<nb, bt, sm, st>>>(v, lg);
    else if (!o.closure) forces_spec32_kernel<DIM, KT, 2, true><<<nb, bt, sm, st>>>(v, lg);
    else forces_spec32_kernel<DIM, KT, 3, true><<<nb, bt, sm, st>>>(v, lg);
    return;
  }
  if (!o.need_sr) forces_spec32_kernel<DIM, KT, 1, false><<<nb, bt, sm, st>>>(v, lg);
  else if (!o.closure) forces_spec32_kernel<DIM, KT, 2, false><<<nb, bt, sm, st>>>(v, lg);
  else forces_spec32_kernel<DIM, KT, 3, false><<<nb, bt, sm, st>>>(v, lg);
}

template <int DIM, int KT>
void fluid32_dispatch(const DevView& v, int nb, int bt, cudaStream_t st) {
  const int fl = v.o.several_eos ? 4 : !v.o.flavours32 ? 0 : !v.o.need_sr ? 1 : !v.o.closure ? 2 : 3;
  switch (fl) {
    case 4: forces_fluid32_kernel<DIM, KT, 4><<<nb, bt, 0, st>>>(v); break;
    case 0: forces_fluid32_kernel<DIM, KT, 0><<<nb, bt, 0, st>>>(v); break;
    case 1: forces_fluid32_kernel<DIM, KT, 1><<<nb, bt, 0, st>>>(v); break;
    case 2: forces_fluid32_kernel<DIM, KT, 2><<<nb, bt, 0, st>>>(v); break;
    default: forces_fluid32_kernel<DIM, KT, 3><<<nb, bt, 0, st>>>(v); break;
  }
}

template <int KT>
void soil32_dispatch(const DevView& v, int nb, int bt, cudaStream_t st) {
  if (v.o.mix_soil) forces_soil32_kernel<KT, true><<<nb, bt, 0, st>>>(v);
  else forces_soil32_kernel<KT, false><<<nb, bt, 0, st>>>(v);
}

template <int DIM>
void forces32_dispatch(const DevView& v, cudaStream_t st) {
  const int bt = (v.o.pair_block >= 32 && v.o.pair_block <= kMaxPairBlock) ? v.o.pair_block : kFT32;
  const int nb = v.ncap <= 0 ? 1 : (v.ncap + bt - 1) / bt;
  if (DIM == 2 && (v.o.soil32 || (v.o.mix_soil & kMixSpec))) {
    switch (v.o.kt) {
      case 0: soil32_dispatch<0>(v, nb, bt, st); break;
      case 1: soil32_dispatch<1>(v, nb, bt, st); break;
      default: soil32_dispatch<2>(v, nb, bt, st); break;
    }
    if (!(v.o.mix_soil & kMixGeneral)) return;
  }
  if (v.o.has_solid) {
    switch (v.o.kt) {
      case 0: forces_solid32_kernel<DIM, 0><<<nb, bt, 0, st>>>(v); break;
      case 1: forces_solid32_kernel<DIM, 1><<<nb, bt, 0, st>>>(v); break;
      default: forces_solid32_kernel<DIM, 2><<<nb, bt, 0, st>>>(v); break;
    }
    return;
  }
  if (v.o.spec32 || (v.o.mix32 & kMixSpec)) {
    switch (v.o.kt) {
      case 0: spec32_dispatch<DIM, 0>(v, bt, st); break;
      case 1: spec32_dispatch<DIM, 1>(v, bt, st); break;
      default: spec32_dispatch<DIM, 2>(v, bt, st); break;
    }
    if (!(v.o.mix32 & kMixGeneral)) return;
  }
  switch (v.o.kt) {
    case 0: fluid32_dispatch<DIM, 0>(v, nb, bt, st); break;
    case 1: fluid32_dispatch<DIM, 1>(v, nb, bt, st); break;
    default: fluid32_dispatch<DIM, 2>(v, nb, bt, st); break;
  }
}

}  // namespace

void launch_copies32(const DevView& v, cudaStream_t st) {
  if (v.o.fp32 && !v.o.has_solid) copies32_kernel<<<nblk32(v.ncap), kFT32, 0, st>>>(v);
}

void launch_prepare32(const DevView& v, cudaStream_t st) {
  if (v.o.has_solid) {  // FP64 wall stress interpolation and TIR, then the FP32 copies
    launch_prepare(v, st);
    if (v.o.soil32 || v.o.mix_soil == kMixSpec) return;  // which wrote the pair kernel's records too
    const int nb = nblk32(v.ncap);
    if (v.o.dim == 2) solid_copies32_kernel<2><<<nb, kFT32, 0, st>>>(v);
    else solid_copies32_kernel<3><<<nb, kFT32, 0, st>>>(v);
    return;
  }
  if (v.o.dim == 2) prepare32_dispatch<2>(v, st);
  else prepare32_dispatch<3>(v, st);
}

namespace {
__global__ void expand_sr32_kernel(const float* __restrict__ sr32, double* __restrict__ sr, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float* a = sr32 + 6 * (size_t)i;
  double* o = sr + 9 * (size_t)i;
  o[0] = a[0]; o[1] = a[1]; o[2] = a[2];
  o[3] = a[1]; o[4] = a[3]; o[5] = a[4];
  o[6] = a[2]; o[7] = a[4]; o[8] = a[5];
}
}  // namespace

namespace {
__global__ void expand_rates32_kernel(const float4* __restrict__ r, double* __restrict__ sr, double* __restrict__ rr,
                                      int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) widen_rates(r + 3 * (size_t)i, sr + 9 * (size_t)i, rr + 9 * (size_t)i);
}
}  // namespace

void launch_expand_sr32(const DevView& v, int n, cudaStream_t st) {
  if (n > 0 && v.S.rates32)
    expand_rates32_kernel<<<(n + 255) / 256, 256, 0, st>>>(v.S.rates32, v.S.strain_rate, v.S.rotation_rate, n);
  if (n > 0 && v.S.sr32 && v.S.strain_rate)
    expand_sr32_kernel<<<(n + 255) / 256, 256, 0, st>>>(v.S.sr32, v.S.strain_rate, n);
}

void launch_forces32(const DevView& v, cudaStream_t st) {
  if (v.o.dim == 2) forces32_dispatch<2>(v, st);
  else forces32_dispatch<3>(v, st);
}

}  // namespace psph

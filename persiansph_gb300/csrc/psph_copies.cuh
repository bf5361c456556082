// FP32 copies of a fluid particle for the FP32C pair kernels, written where its
// FP64 state is at hand: by the cell sort's reorder, or with a skin by the kernel
// that takes each step's offsets (a copy kernel of its own read that state a
// second time and was one more launch: 137 us of 6.7M particles' step, 6 of 920's).
#pragma once

#include "psph_pairs.cuh"

namespace psph {

PSPH_D void fluid_copies32(const DevView& v, const Persist& P, int w, int cls, double density, const double4_32a& vv,
                           const float4& x, int refcell) {
  const PClass32& C = v.cls32[cls];
  // every conversion on the integer pipe (d2f_rn / d2f_split: the values of
  // the conversion instruction, which runs on the FP64 pipe)
  const float p = d2f_rn(vv.w);
  float lx, ly, lz;
  const float vx = d2f_split(vv.x, &lx), vy = d2f_split(vv.y, &ly), vz = d2f_split(vv.z, &lz);
  v.S.V32[w] = make_float4(vx, vy, vz, p);
  // the velocity's low-order part: in a smooth flow v_i - v_j is far smaller
  // than v, and the pair differences take (hi_i - hi_j) + (lo_i - lo_j), exact
  // to ~2^-48 of |v|; the class index and its flags ride along in .w (class |
  // flags << 16: one load per pair, and no class-table load when the pair
  // constants are uniform)
  float lw = __int_as_float(cls | (C.flags << 16));
  if (C.flags & CF_FREE) {
    const float rho = d2f_rn(density);
    const float inv = 1.f / rho;
    const float ratio = rho / C.rho0;
    const float c = (C.pres_eq == 1) ? fabsf(C.cs * ratio * ratio * ratio) : C.cs;  // sqrt(cs^2 ratio^6)
    if (spec32_of(v, C.inst)) {  // the constant-parameter pair kernel's record (the walls' comes with their pressure)
      v.S.RC32[w] = make_float2(rho, __int_as_float(refcell));
      v.S.PX32[w] = make_float4(x.x, x.y, x.z, with_sign(inv, 1.f));
      lw = with_sign(c, rho);
    } else {
      v.S.D32[w] = make_float4(inv, p * inv * inv, c, rho);
    }
  }
  v.S.V32LO[w] = make_float4(lx, ly, lz, lw);
  // FP32 copy of a per-particle viscosity: the pair loop then converts nothing
  // (a double-to-float conversion runs on the FP64 pipe, 1/64 of the FP32 rate)
  if (v.o.dyn_mu) v.S.MU32[w] = d2f_rn(P.mu[w]);
}

}  // namespace psph

// speedy_vjp_smem.cuh -- the device adjoint of one SPEEDY column: the reverse pass of speedy_vjp.h
// (which stays its host reference) arranged for the chip.
//
// One thread per column, its per-level arrays in shared memory ([array][level][thread], like the
// forward's), every level loop rolled.  The fully unrolled form this replaces kept its arrays in
// registers and local memory: a 2.1 KB stack per thread, 31.7 k thread instructions per column in
// straight-line code that did not fit the instruction caches.  What bounds this form is
// instruction issue and the latency of its serial recurrences.
//
// Nine arrays per column: T, q, qsat, the T and q adjoints and four scratch rows (36,864 bytes per
// block at 8 levels, 73,728 at 16: three blocks per SM).  Phi and the cotangents are read again
// from L2 where they are used.  What keeps the storage this small:
//  - Every radiative recurrence and its adjoint run in one direction together.  The downward
//    fluxes D and the adjoint G of the upward ones both run down the column, and both are
//    x -> tau x + (1 - tau) s, with s the level's emission for D and its cotangent d for G
//    (longwave_down).  Going back up, the upward fluxes U and the adjoint K of the downward ones
//    do the same (longwave_rev), and each level meets all four at once, so its transmissivities,
//    blackbody terms and their adjoints are formed once for both passes.
//  - Of D and G only the values entering every second level are kept (checkpoints, 32 bytes per
//    level); the level between is stepped again from registers.
//  - The shortwave's adjoint of the upward flux runs down with the fluxes; its reverse loop
//    rebuilds the upward flux as it climbs.
//  - The convection's reverse needs one kept array (the mass flux); a warp starts it at the
//    highest cloud base of its columns and skips it where no column convects.
// The values that decide branches (saturation, convection and cloud thresholds, skin temperature,
// relative humidity gradients, limited levels) are formed with the expressions of speedy_vjp.h, so
// every branch is taken as there; adjoints use fused multiply-adds and one reciprocal of psa.
#pragma once

#include <type_traits>

#include "speedy_column_smem.cuh"
#include "speedy_vjp.h"

namespace spd {

enum { V_T, V_Q, V_QS, V_TB, V_QB, V_S0, V_S1, V_S2, V_S3, kVjpArrays };

constexpr size_t vjp_arena_bytes(int kx) {
  return (size_t)kVjpArrays * kx * kNT * sizeof(float);
}

// Packed pairs without the subnormal flush of speedy_pk.cuh, and with a fused multiply-add.  No
// sum below has a product for an operand where a fused multiply-add could take its place (ptxas
// would fuse it or not as it pleases), so that every build of the column gives the same bits.
#define SPD_PV_OP(name, op)                                                              \
  __device__ __forceinline__ float2 name(float2 a, float2 b) {                           \
    float2 d;                                                                            \
    asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t" \
        op " rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"                                  \
        : "=f"(d.x), "=f"(d.y)                                                           \
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));                                       \
    return d;                                                                            \
  }
SPD_PV_OP(pv_mul, "mul.rn.f32x2")
SPD_PV_OP(pv_add, "add.rn.f32x2")
SPD_PV_OP(pv_sub, "sub.rn.f32x2")
#undef SPD_PV_OP
__device__ __forceinline__ float2 pv_fma(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "mov.b64 rc, {%6, %7};\n\tfma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float hsum(float2 a, float2 b) { return ((a.x + a.y) + b.x) + b.y; }

// One member of a batched adjoint: its fields, shape, class, level set and solar table.
struct VjpMemberDev {
  spd_inputs_t in;
  spd_cotangents_t ct;
  spd_grads_t gr;
  int C, il, kx, cls;
  uint32_t* S;
  ZonalRow* table;
};

// Where an adjoint launch takes its members from: a plan's member table and tile list, or (when
// `members` is null) the one member given by value, whose tile t covers columns t*kNT ..
struct VjpSource {
  const VjpMemberDev* members;
  const Tile* tiles;
  VjpMemberDev single;
  int nmembers;
};

// A field pointer of the block's member record (in shared memory), read where it is used: held
// from the start, the record's 28 pointers would take 56 registers through the whole column.
template <class P>
__device__ __forceinline__ P* load_field(P* const& at) {
  uint64_t v;
  asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"((uint32_t)__cvta_generic_to_shared(&at)));
  return reinterpret_cast<P*>(v);
}

// The member's fields that the column reads again and again, at this column.
struct VjpColumn {
  const float *phi, *ct_t, *ct_q;  // level k is k * C further
  size_t C;
  __device__ __forceinline__ float at(const float* p, int k) const { return __ldg(p + k * C); }
};

// ---------------------------------------------------------------------------------------------
// Longwave
// ---------------------------------------------------------------------------------------------
enum { LV_TOP, LV_SECOND, LV_MID, LV_LAST };  // levels 0, 1, 2..kx-2, kx-1

// What the longwave passes share: column scalars.
struct LwCol {
  float psa, acl1, acl2;
  int icltop;
};

// One level: transmissivities, band fractions (times 1 - epslw), blackbody terms, and what their
// adjoints need (longwave_radiation.py:42-68, :204-226, shortwave_radiation.py:174-206).
struct LwLev {
  float2 t01, t23, f01, f23;
  float s0, s1, t, dd, grad;
};

template <int KIND>
__device__ __forceinline__ void lw_absorption(const ConstsD& CD, const LwCol& w, float q, int k,
                                              float& a0, float& a2, float& a3) {
  const spd_params_t& p = CD.K.p;
  a0 = p.ablwin;
  if (KIND == LV_TOP) {
    a2 = a3 = 0.0f;
    return;
  }
  a2 = p.ablwv1 * q;
  a3 = p.ablwv2 * q;
  if (KIND == LV_MID) {
    a0 = a0 + ((k > w.icltop) ? w.acl1 : w.acl2);
    a2 = fmaxf(a2, w.acl2);
    a3 = fmaxf(a3, w.acl2);
  }
}

__device__ __forceinline__ void lw_fractions(float temp, float wlw, float2& f01, float2& f23) {
  const float j = fminf(fmaxf(temp, 200.0f), 320.0f);
  const float a1 = j - 247.0f, a2 = j - 282.0f, a3 = j - 315.0f;
  const float f1 = fmaf(-3.0e-6f * a1, a1, 0.148f);
  const float f2 = fmaf(-5.2e-6f * a2, a2, 0.356f);
  const float f3 = fmaf(1.0e-5f * a3, a3, 0.314f);
  const float f0 = 1.0f - ((f1 + f2) + f3);
  f01 = pv_mul(bc(wlw), pk(f0, f1));
  f23 = pv_mul(bc(wlw), pk(f2, f3));
}

// tm, t, tp: temperatures of levels k - 1, k, k + 1 (those that exist).
template <int KX, int KIND>
__device__ __forceinline__ void lw_level(const ConstsD& CD, const LwCol& w, int k, float tm,
                                         float t, float tp, float q, LwLev& L) {
  const spd_vgrid_t& vg = CD.K.vg;
  float a0, a2, a3;
  lw_absorption<KIND>(CD, w, q, k, a0, a2, a3);
  const float dh = vg.dhs[k];
  L.t01 = pk(expf(-a0 * w.psa * dh), expf(-CD.D.ablco2 * w.psa * dh));
  L.t23 = KIND == LV_TOP ? bc(1.0f) : pk(expf(-a2 * w.psa * dh), expf(-a3 * w.psa * dh));
  lw_fractions(t, CD.D.w_lw, L.f01, L.f23);
  L.t = t;
  L.dd = L.grad = 0.0f;
  if (KIND == LV_TOP) {
    const float th0 = t + vg.wvi[0][1] * (tp - t);
    L.t = 0.75f * t + 0.25f * th0;  // the temperature that radiates
    const float s = L.t * L.t;
    L.s0 = kSbc * (s * s);
    L.s1 = 0.0f;
  } else if (KIND == LV_SECOND) {
    const float th0 = tm + vg.wvi[0][1] * (t - tm), th1 = t + vg.wvi[1][1] * (tp - t);
    L.t = 0.50f * t + 0.25f * (th0 + th1);
    const float s = L.t * L.t;
    L.s0 = kSbc * (s * s);
    L.s1 = 0.0f;
  } else {
    const float thm = tm + vg.wvi[k - 1][1] * (t - tm);
    if (KIND == LV_MID) {
      L.dd = (t + vg.wvi[k][1] * (tp - t)) - thm;
      L.grad = 0.5f * fmaxf(L.dd, 0.0f);
    } else {
      L.dd = t - thm;
      L.grad = fmaxf(L.dd, 0.0f);
    }
    const float st3 = kSbc * (t * t * t);
    L.s0 = st3 * t;
    L.s1 = 4.0f * st3 * L.grad;
  }
}

// Fluxes and adjoints in one band pair: x -> tau x + (1 - tau) s.
__device__ __forceinline__ float2 relax(float2 tau, float2 emis, float2 x, float2 s) {
  return pv_fma(tau, x, pv_mul(emis, s));
}

// The downward fluxes D and the adjoint G of the upward fluxes through one level; d is the
// level's cotangent (of its flux divergence).
template <int KIND>
__device__ __forceinline__ void lw_down_step(const LwLev& L, float d, float2& D01, float2& D23,
                                             float2& G01, float2& G23) {
  const float2 e01 = pv_sub(bc(1.0f), L.t01), e23 = pv_sub(bc(1.0f), L.t23);
  const float2 s01 = pv_mul(L.f01, pv_fma(e01, bc(L.s1), bc(L.s0)));
  if (KIND == LV_TOP) {  // no flux from above; bands 2 and 3 start below
    D01 = pv_mul(e01, s01);
    G01 = pv_mul(e01, bc(d));
    D23 = G23 = bc(0.0f);
    return;
  }
  const float2 s23 = pv_mul(L.f23, pv_fma(e23, bc(L.s1), bc(L.s0)));
  D01 = relax(L.t01, e01, D01, s01);
  D23 = relax(L.t23, e23, D23, s23);
  G01 = relax(L.t01, e01, G01, bc(d));
  G23 = relax(L.t23, e23, G23, bc(d));
}

// Scalars of the longwave reverse.
struct LwRev {
  float2 K01, K23;       // adjoint of the downward flux leaving the level
  float2 U01, U23;       // upward flux entering the level from below
  float sU;              // sum of U over the bands
  float dps;             // sum over levels of cotangent x flux divergence
  float psa_b, acl1_b, acl2_b;
  float hi, mid, lo;     // T adjoints of levels k + 1, k, k - 1 so far
  float st0, st1, corlw; // blackbody cotangents of the stratospheric and surface corrections
};

// One level of the reverse: D01.. and G01.. enter it from above.  Adds to the q adjoint qb.
template <int KX, int KIND>
__device__ __forceinline__ void lw_rev_level(const ConstsD& CD, const LwCol& w, const LwLev& L,
                                             int k, float t, float q, float d, float2 D01,
                                             float2 D23, float2 G01, float2 G23, LwRev& r,
                                             float& qb) {
  const spd_vgrid_t& vg = CD.K.vg;
  const spd_params_t& p = CD.K.p;
  const float2 e01 = pv_sub(bc(1.0f), L.t01), e23 = pv_sub(bc(1.0f), L.t23);
  const float2 H01 = pv_sub(r.K01, bc(d)), E01 = pv_sub(G01, bc(d));
  float2 H23 = bc(0.0f), E23 = bc(0.0f);  // bands 2 and 3 do not see level 0
  if (KIND != LV_TOP) {
    H23 = pv_sub(r.K23, bc(d));
    E23 = pv_sub(G23, bc(d));
  }
  const float2 s0 = bc(L.s0), s1 = bc(L.s1);
  float2 tb01, tb23, y01, y23;
  float s0b, s1b;
  {
    const float2 P = pv_add(H01, E01), M = pv_sub(H01, E01);
    const float2 es = pv_mul(e01, s1), X = pv_fma(es, M, pv_mul(P, s0));
    const float2 ef = pv_mul(e01, L.f01);
    tb01 = pv_fma(E01, r.U01, pv_mul(H01, D01));
    tb01 = pv_fma(neg2(L.f01), pv_fma(es, M, X), tb01);
    y01 = pv_mul(e01, X);
    const float2 a = pv_mul(ef, P), b = pv_mul(pv_mul(ef, e01), M);
    s0b = a.x + a.y;
    s1b = b.x + b.y;
    const float2 src = pv_fma(neg2(e01), s1, s0);
    r.U01 = pv_fma(L.t01, r.U01, pv_mul(ef, src));
    r.K01 = relax(L.t01, e01, r.K01, bc(d));
  }
  if (KIND != LV_TOP) {
    const float2 P = pv_add(H23, E23), M = pv_sub(H23, E23);
    const float2 es = pv_mul(e23, s1), X = pv_fma(es, M, pv_mul(P, s0));
    const float2 ef = pv_mul(e23, L.f23);
    tb23 = pv_fma(E23, r.U23, pv_mul(H23, D23));
    tb23 = pv_fma(neg2(L.f23), pv_fma(es, M, X), tb23);
    y23 = pv_mul(e23, X);
    const float2 a = pv_mul(ef, P), b = pv_mul(pv_mul(ef, e23), M);
    s0b += a.x + a.y;
    s1b += b.x + b.y;
    const float2 src = pv_fma(neg2(e23), s1, s0);
    r.U23 = pv_fma(L.t23, r.U23, pv_mul(ef, src));
    r.K23 = relax(L.t23, e23, r.K23, bc(d));
  } else {
    tb23 = y23 = bc(0.0f);
  }
  const float sU = hsum(r.U01, r.U23);  // at level 0 bands 2 and 3 pass unchanged
  r.dps = fmaf(d, r.sU - sU, r.dps);
  r.sU = sU;
  if (KIND == LV_LAST) s0b = fmaf(r.corlw, CD.D.corlw_f, s0b);
  if (KIND == LV_SECOND) s0b += r.st1;
  if (KIND == LV_TOP) s0b += r.st0;
  // band fractions (radset): derivative with respect to this level's temperature
  float tk_b;
  {
    const float wj = (t > 200.0f && t < 320.0f) ? 1.0f
                     : (t == 200.0f || t == 320.0f) ? 0.5f : 0.0f;
    const float j = fminf(fmaxf(t, 200.0f), 320.0f);
    float g = (-6.0e-6f * (j - 247.0f)) * (y01.y - y01.x);
    g = fmaf(-1.04e-5f * (j - 282.0f), y23.x - y01.x, g);
    g = fmaf(2.0e-5f * (j - 315.0f), y23.y - y01.x, g);
    tk_b = (wj * CD.D.w_lw) * g;
  }
  // transmissivities
  {
    float a0, a2, a3;
    lw_absorption<KIND>(CD, w, q, k, a0, a2, a3);
    const float2 x01 = pv_mul(pv_mul(tb01, L.t01), bc(vg.dhs[k]));
    const float2 x23 = pv_mul(pv_mul(tb23, L.t23), bc(vg.dhs[k]));
    float g = fmaf(x01.y, CD.D.ablco2, x01.x * a0);
    if (KIND != LV_TOP) {
      g = fmaf(x23.x, a2, g);
      g = fmaf(x23.y, a3, g);
      const float ab2 = -w.psa * x23.x, ab3 = -w.psa * x23.y;
      if (KIND == LV_MID) {
        const float ab0 = -w.psa * x01.x;
        const float q1 = p.ablwv1 * q, q2 = p.ablwv2 * q;
        const float w2 = spdvjp::wmax(q1, w.acl2), w3 = spdvjp::wmax(q2, w.acl2);
        qb = fmaf(ab2 * w2, p.ablwv1, fmaf(ab3 * w3, p.ablwv2, qb));
        const bool below = k > w.icltop;
        r.acl1_b += below ? ab0 : 0.0f;
        r.acl2_b += below ? 0.0f : ab0;
        r.acl2_b += fmaf(ab2, 1.0f - w2, ab3 * (1.0f - w3));
      } else {
        qb = fmaf(ab2, p.ablwv1, fmaf(ab3, p.ablwv2, qb));
      }
    }
    r.psa_b -= g;
  }
  // blackbody terms; th_j = t_j + w_j (t_{j+1} - t_j)
  if (KIND == LV_TOP) {
    const float b = s0b * (4.0f * kSbc) * (L.t * L.t * L.t);
    const float v = 0.25f * b, ww = vg.wvi[0][1];
    r.mid += fmaf(0.75f, b, v - ww * v) + tk_b;
    r.hi += ww * v;
  } else if (KIND == LV_SECOND) {
    const float b = s0b * (4.0f * kSbc) * (L.t * L.t * L.t);
    const float v = 0.25f * b, w0 = vg.wvi[0][1], w1 = vg.wvi[1][1];
    r.lo += v - w0 * v;
    r.mid += fmaf(0.50f, b, w0 * v) + (v - w1 * v) + tk_b;
    r.hi += w1 * v;
  } else {
    const float t2 = kSbc * (t * t), u4 = 4.0f * t2 * t;
    tk_b += fmaf(u4, s0b, 12.0f * t2 * L.grad * s1b);
    float db = u4 * s1b * spdvjp::wmax(L.dd, 0.0f);
    const float wm = vg.wvi[k - 1][1];
    if (KIND == LV_MID) {
      db *= 0.5f;
      const float wk = vg.wvi[k][1];
      r.hi = fmaf(wk, db, r.hi);
      tk_b += db - wk * db;
    } else {
      tk_b += db;
    }
    r.mid += tk_b - wm * db;
    r.lo += wm * db - db;
  }
}

// ---------------------------------------------------------------------------------------------
// The column
// ---------------------------------------------------------------------------------------------
// The orographic humidity correction, out of line: its power and its saturation humidities cost the
// calls that do not use it registers (T425 with 16 levels and verify 1,013 against 996 us).
static __device__ __noinline__ float qcorh_of(float phis0, float fmask, float stl, float sst,
                                              float gamlat, float pexp) {
  return spdvjp::orographic_qcorh(phis0, fmask, stl, sst, gamlat, pexp);
}

// Reverse pass of column c of member m (in shared memory), clamped into the member by the caller,
// whose `valid` says whether to store; adds the 12 parameter gradients to par.  kVerify: false
// where no column of the launch fuses verify.
template <int KX, bool kVerify>
__device__ __forceinline__ void column_vjp_smem(const ConstsD& CD, float* sm,
                                                const VjpMemberDev& m, int c, int Ci,
                                                bool valid, float* par) {
  using spdvjp::fdiv;
  using spdvjp::fdiv_full;
  using spdvjp::frcp;
  using spdvjp::wmax;
  using spdvjp::wmin;
  const Consts& K = CD.K;
  const Derived& D = CD.D;
  const spd_params_t& p = K.p;
  const spd_vgrid_t& vg = K.vg;
  constexpr int B = KX - 1;
  const size_t C = (size_t)Ci;
  auto arr = [&](int a) { return Lv{sm + (size_t)a * KX * kNT + threadIdx.x}; };
  const Lv T = arr(V_T), Q = arr(V_Q), QS = arr(V_QS), TB = arr(V_TB), QB = arr(V_QB);
  const Lv S0 = arr(V_S0), S1 = arr(V_S1), S2 = arr(V_S2), S3 = arr(V_S3);
  const bool verify = kVerify && (K.flags & SPD_FUSE_VERIFY) != 0;
  const VjpColumn col{load_field(m.in.geopotential) + c, load_field(m.ct.temperature) + c,
                      load_field(m.ct.specific_humidity) + c, C};

  // The rows that are first read further on start for L2 now, one row (128 bytes) per lane: the
  // two cotangents' levels, then the surface fields.
  {
    const int lane = threadIdx.x & 31, level = lane & 15;
    const int c0 = __shfl_sync(0xffffffffu, c, 0);  // the warp's first column
    const float* row = (lane < 16 ? col.ct_t : col.ct_q) - c + c0;
    if (level < KX) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + level * C));
    if (lane < 9) {  // alb0 .. phis0
      const float* f = load_field((&m.in.alb0)[lane]);
      asm volatile("prefetch.global.L2 [%0];" ::"l"(f + c0));
    }
  }

  // ---- forward: humidity, convection, condensation, clouds ----------------------------------
  SurfaceIn s;
  s.psa = __ldg(load_field(m.in.normalized_surface_pressure) + c);
  s.fmask = __ldg(load_field(m.in.fmask) + c);
  const float psa = s.psa;
  ColScalars o;
  uint32_t neg = 0u;  // levels whose humidity verify_state clamped
  {
    float t[KX], q[KX], phi[KX], qs[KX], dt[KX], dq[KX];
    const float* t_in = load_field(m.in.temperature) + c;
    const float* q_in = load_field(m.in.specific_humidity) + c;
#pragma unroll
    for (int k = 0; k < KX; ++k) {
      t[k] = col.at(t_in, k);
      const float qk = col.at(q_in, k);
      if (verify && qk < 0.0f) neg |= 1u << k;
      q[k] = (verify && qk < 0.0f) ? 0.0f : qk;
      phi[k] = col.at(col.phi, k);
    }
    column_first<KX>(CD, t, q, phi, s, qs, dt, dq, o);
#pragma unroll
    for (int k = 0; k < KX; ++k) {
      T[k] = t[k];
      Q[k] = q[k];
      QS[k] = qs[k];
    }
    if (verify) {  // the humidity tendency so far, until the limited levels are known
#pragma unroll
      for (int k = 0; k < KX; ++k) TB[k] = dq[k];
    }
  }
  const float rpsa = frcp(psa);
  const float cloudc = o.cloudc, clstr = o.clstr;
  const int icltop = o.icltop;
  const float qcloud = Q[KX - 2];
  const float fmask = s.fmask;
  spdvjp::Col<KX, float> cc;  // what the surface term reads (its lowest levels and scalars)
  spdvjp::SurfaceIn sf_in;
  float albsfc;
  {
    const float snowc = __ldg(load_field(m.in.snowc_am) + c), alb0 = __ldg(load_field(m.in.alb0) + c);
    sf_in.sice = __ldg(load_field(m.in.sice_am) + c);
    sf_in.snowc = snowc;
    sf_in.alb0 = alb0;
    sf_in.fmask = fmask;
    cc.snowc = snowc < 1.0f ? snowc : 1.0f;
    cc.alb_l = alb0 + cc.snowc * (p.albsn - alb0);
    const float alb_s = p.albsea + sf_in.sice * (p.albice - p.albsea);
    albsfc = alb_s + fmask * (cc.alb_l - alb_s);
  }

  // The level set and the solar rows are the pre-pass's: wait for it (this launch may start while
  // it runs), then read them past L1.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const uint32_t S = __ldcg(load_field(m.S));
  ZonalRow z;
  {
    const ZonalRow* zrow = load_field(m.table) + c % m.il;
    const float4 a = __ldcg(reinterpret_cast<const float4*>(zrow));
    const float2 b = __ldcg(reinterpret_cast<const float2*>(zrow) + 2);
    z.fsol = a.x;
    z.ozupp = a.y;
    z.ozone = a.z;
    z.zenit = a.w;
    z.stratz = b.x;
    z.sqrt_coa = b.y;
  }

  // ---- forward: shortwave (rs in S0, band-1 transmissivity in S1) ----------------------------
  const bool cmask = icltop < KX;
  const bool swon = (K.model_step % 3) == 0;
  const float refl = cmask ? p.albcl * cloudc : 0.0f;
  const float psaz = psa * z.zenit;
  const float mnq = spdvjp::vmin(p.abscl1 * qcloud, p.abscl2);
  const float acloud = cloudc * mnq;
  auto refl_at = [&](int k) {
    return k == B ? p.albcls * clstr : (((S >> k) & 1u) ? refl : 0.0f);
  };
  auto sw_inner = [&](int k, float q) {
    const float cl = (k < B && k >= icltop) ? acloud : 0.0f;
    return k < B ? D.abs1[k] + p.abswv1 * q + cl : D.abs1[k] + p.abswv1 * q;
  };
  auto sw_tau0 = [&](int k, float q) {
    if (k == 0) return expf(-psaz * vg.dhs[0] * p.absdry);
    return expf(-psaz * vg.dhs[k] * sw_inner(k, q));
  };
  auto sw_tau1 = [&](int k, float q) { return expf(-psaz * vg.dhs[k] * p.abswv2 * q); };
  const float f10 = z.fsol * 0.95f, f20 = z.fsol * 0.05f;
  float rsds, fsw0, fsw1;
  {
    const float t00 = sw_tau0(0, 0.0f);
    float f1 = t00 * (f10 - z.ozupp * psa);
    const float t01 = sw_tau0(1, Q[1]);
    S1[1] = t01;
    f1 = t01 * (f1 - z.ozone * psa);
    float f2 = f20 * sw_tau1(1, Q[1]);
#pragma unroll 2
    for (int k = 2; k < KX; ++k) {
      const float q = Q[k], t0 = sw_tau0(k, q), r = refl_at(k);
      S1[k] = t0;
      S0[k] = r * f1;
      f1 = f1 * t0 * (1.0f - r);
      f2 = f2 * sw_tau1(k, q);
    }
    rsds = f1 + f2;
    float up = f1 * albsfc;
#pragma unroll 2
    for (int k = B; k >= 2; --k) up = up * S1[k] + S0[k];
    up = up * t01 + refl_at(1);
    fsw0 = t00 * up + refl_at(0);
    fsw1 = f2;
  }

  // ---- longwave down: D with G, the adjoint of the upward fluxes -----------------------------
  // dps collects sum_k d_k dfl_k over every flux divergence (d_k: cotangent of level k's).
  // The cotangents come from L2: each loop loads its next level's before it works on this one's.
  auto ctt = [&](int k) { return col.at(col.ct_t, k); };
  auto d_of = [&](float ctk, int k) { return ctk * vg.grdscp[k] * rpsa; };
  auto d_at = [&](int k) { return d_of(ctt(k), k); };
  LwCol lw{psa, cloudc * p.ablcl1, cloudc * p.ablcl2, icltop};
  LwRev r;
  const float stratc1 = D.eps1 * psa;
  float rlds, fsw0_b, fsw1_b, rlus2_b, dB, dps;
  float2 Gs01, Gs23;
  {
    float2 D01, D23, G01, G23;
    LwLev L;
    float tm = T[0], t = T[1], ct_k = ctt(2);
    const float d0 = d_at(0), d1 = d_at(1);
    lw_level<KX, LV_TOP>(CD, lw, 0, 0.0f, tm, t, 0.0f, L);
    lw_down_step<LV_TOP>(L, d0, D01, D23, G01, G23);
    float sD = hsum(D01, D23);
    const float c1 = vg.dhs[0] * stratc1 * L.s0 + z.stratz * psa;
    dps = -d0 * (sD + c1);
    float stb = -d0 * vg.dhs[0] * L.s0;
    r.st0 = -d0 * (vg.dhs[0] * stratc1);
    float tp = T[2];
    lw_level<KX, LV_SECOND>(CD, lw, 1, tm, t, tp, Q[1], L);
    lw_down_step<LV_SECOND>(L, d1, D01, D23, G01, G23);
    float sk = hsum(D01, D23);
    dps = fmaf(d1, (sD - sk) - vg.dhs[1] * stratc1 * L.s0, dps);
    stb = fmaf(-d1 * vg.dhs[1], L.s0, stb);
    r.st1 = -d1 * (vg.dhs[1] * stratc1);
    r.psa_b = stb * D.eps1 - d0 * z.stratz;
    sD = sk;
    tm = t;
    t = tp;
    auto keep = [&](int k) {  // the fluxes entering level k (even): a checkpoint
      const int at = (k / 2 - 1) * 8;
      S0[at] = D01.x;
      S0[at + 1] = D01.y;
      S0[at + 2] = D23.x;
      S0[at + 3] = D23.y;
      S0[at + 4] = G01.x;
      S0[at + 5] = G01.y;
      S0[at + 6] = G23.x;
      S0[at + 7] = G23.y;
    };
#pragma unroll 2
    for (int k = 2; k < B; ++k) {
      if ((k & 1) == 0) keep(k);
      tp = T[k + 1];
      const float d = d_of(ct_k, k);
      ct_k = ctt(k + 1);
      lw_level<KX, LV_MID>(CD, lw, k, tm, t, tp, Q[k], L);
      lw_down_step<LV_MID>(L, d, D01, D23, G01, G23);
      sk = hsum(D01, D23);
      dps = fmaf(d, sD - sk, dps);
      sD = sk;
      tm = t;
      t = tp;
    }
    if ((B & 1) == 0) keep(B);
    lw_level<KX, LV_LAST>(CD, lw, B, tm, t, 0.0f, Q[B], L);
    dB = d_of(ct_k, B);
    lw_down_step<LV_LAST>(L, dB, D01, D23, G01, G23);
    sk = hsum(D01, D23);
    const float corlw = D.corlw_f * L.s0;
    dps = fmaf(dB, (sD - sk) - corlw, dps);
    rlds = (((p.emisfc * D01.x + p.emisfc * D01.y) + p.emisfc * D23.x) + p.emisfc * D23.y) + corlw;
    Gs01 = G01;
    Gs23 = G23;
  }

  // ---- surface fluxes, the limited levels, the surface fluxes' reverse ------------------------
  uint32_t limited = 0u;  // levels where verify_tendencies replaced dq by -q / dt
  float sfc_q_b, sfc_phi_b, sfc_qs_b, u_b, v_b, rsds_b = 0.0f, rlds_b = 0.0f;
  {
    const float phiB = col.at(col.phi, B);
    sf_in.sst = __ldg(load_field(m.in.sea_surface_temperature) + c);
    sf_in.stl = __ldg(load_field(m.in.stl_am) + c);
    sf_in.soilw = __ldg(load_field(m.in.soilw_am) + c);
    sf_in.orog = __ldg(load_field(m.in.orog) + c);
    sf_in.phis0 = __ldg(load_field(m.in.phis0) + c);
    const float ctu = col.at(load_field(m.ct.u_wind) + c, B), ctv = col.at(load_field(m.ct.v_wind) + c, B);
    cc.psa = psa;
    cc.t[B] = T[B];
    cc.t[B - 1] = T[B - 1];
    cc.q[B] = Q[B];
    cc.qsat[B] = QS[B];
    cc.phi[B] = phiB;
    cc.u = col.at(load_field(m.in.u_wind) + c, B);
    cc.v = col.at(load_field(m.in.v_wind) + c, B);
    cc.rsds = rsds;
    cc.rlds = rlds;
    const spdvjp::Ctx x{&vg, &p, K.flags, K.model_step, S};
    const spdvjp::SurfaceRow zr{z.fsol, z.ozupp, z.ozone, z.zenit, z.stratz, z.sqrt_coa};
    spdvjp::Sf<float> sf;
    sf.rdth = D.rdth;
    sf.rhdrag = D.rhdrag;
    spdvjp::surface<KX, float>(x, cc, sf_in, zr, sf);
    if (verify) {
      const float q_b = Q[B], qs_b1 = QS[B - 1];
      const float se_b = kCp * T[B] + phiB, se_b1 = kCp * T[B - 1] + col.at(col.phi, B - 1);
      const float rh_b = fdiv(q_b, QS[B]), rh_b1 = fdiv(Q[B - 1], qs_b1);
      const float dmse = se_b - se_b1 + kAlhc * (q_b - qs_b1);
      const float drh = rh_b - rh_b1;
      const int icnv = KX - o.iptop - 1;
      const float fcnv = (icnv > 0 && dmse >= 0.0f) ? p.redshc : 1.0f;
      float qt1 = 0.0f, qt0 = 0.0f;  // vertical diffusion at levels kx-2, kx-1
      if (dmse >= 0.0f) {
        if (drh >= 0.0f) {
          const float fq = fcnv * D.fshcq * QS[B] * drh;
          qt1 = fq * D.rsig[B - 1];
          qt0 = -fq * D.rsig[B];
        }
      } else if (dmse < 0.0f && drh > D.drh0) {
        const float fq = D.fvdiq2 * qs_b1 * drh;
        qt1 = fq * D.rsig[B - 1];
        qt0 = -fq * D.rsig[B];
      }
      const bool oro = (K.flags & SPD_OROGRAPHIC) != 0;
      const float qcorh =
          oro ? qcorh_of(sf_in.phis0, fmask, sf_in.stl, sf_in.sst, D.gamlat, D.pexp) : 0.0f;
      const float dts = K.dt_seconds;
      const float* q_in = load_field(m.in.specific_humidity) + c;
      float pend = 0.0f, rh_k = 0.0f;
#pragma unroll 2
      for (int k = 0; k < KX; ++k) {
        float dq = TB[k];
        if (k >= 2 && k < B - 1) {
          if (k == 2) rh_k = fdiv(Q[2], QS[2]);
          const float rh_n = fdiv(Q[k + 1], QS[k + 1]);
          const float dr = rh_n - rh_k;
          const bool cond = (D.vdcond >> k) & 1u;
          const float fq = (dr >= D.drh0v[k] && cond) ? D.fvdiq2v[k] * QS[k] * dr : 0.0f;
          const float a = 0.0f + fq * D.rsig[k];
          dq = dq + (k == 2 ? a : a + pend);
          pend = -(fq * D.rsig[k + 1]);
          rh_k = rh_n;
        } else if (k == B - 1) {
          dq = dq + (qt1 + pend);
        } else if (k == B) {
          dq = (dq + (0.0f + sf.evap2 * sf.rps * vg.grdsig[B])) + qt0;
        } else {
          dq = dq + 0.0f;
        }
        if (oro) dq = dq + fdiv_full(qcorh * D.qcorv[k], dts);
        TB[k] = dq;
      }
      // the humidity as given, read again where it was clamped, all levels' loads first
      float qi[KX];
#pragma unroll
      for (int k = 0; k < KX; ++k) qi[k] = ((neg >> k) & 1u) ? col.at(q_in, k) : Q[k];
#pragma unroll
      for (int k = 0; k < KX; ++k)
        if (!(qi[k] + dts * TB[k] >= 0.0f)) limited |= 1u << k;
    }
    // the upward pass starts from the surface's fluxes
    float2 f01, f23;
    lw_fractions(cc.tsfc, D.w_lw, f01, f23);
    r.U01 = pv_fma(f01, bc(cc.rlus2), pv_mul(bc(D.refsfc), pk(fsw0, fsw1)));
    r.U23 = pv_mul(f23, bc(cc.rlus2));
    r.sU = hsum(r.U01, r.U23);
    r.dps = fmaf(dB, p.epslw * cc.rlus2, dps);
    rlus2_b = fmaf(dB, p.epslw, hsum(pv_mul(Gs01, f01), pv_mul(Gs23, f23)));
    fsw0_b = Gs01.x * D.refsfc;
    fsw1_b = Gs01.y * D.refsfc;
    spdvjp::Bar<KX, float> bs;
    bs.t[B] = bs.t[B - 1] = bs.q[B] = bs.phi[B] = bs.qsat[B] = 0.0f;
    bs.psa = bs.u = bs.v = 0.0f;
    const float dqB_b = ((limited >> B) & 1u) ? 0.0f : col.at(col.ct_q, B) * K.q_tend_scale;
    spdvjp::surface_rev<KX, float>(x, cc, sf_in, zr, sf, ctu, ctv, ctt(B), dqB_b, rlus2_b, rsds_b,
                                   rlds_b, bs);
    r.mid = bs.t[B];
    r.lo = bs.t[B - 1];
    sfc_q_b = bs.q[B];
    sfc_phi_b = bs.phi[B];
    sfc_qs_b = bs.qsat[B];
    r.psa_b += bs.psa;
    u_b = bs.u;
    v_b = bs.v;
  }

  // ---- longwave reverse: U with K, two levels per checkpoint ---------------------------------
  {
    r.K01 = r.K23 = bc(rlds_b * p.emisfc);
    r.corlw = rlds_b - dB;
    r.acl1_b = r.acl2_b = 0.0f;
    r.hi = 0.0f;
    float tp = 0.0f, t = T[B];
    auto done = [&](int k) {  // level k's reverse is complete: level k + 1's T adjoint is final
      if (k < B) TB[k + 1] = r.hi;
      r.hi = r.mid;
      r.mid = r.lo;
      r.lo = 0.0f;
    };
    auto fetch = [&](int k, float2& D01, float2& D23, float2& G01, float2& G23) {
      const int at = (k / 2 - 1) * 8;
      D01 = pk(S0[at], S0[at + 1]);
      D23 = pk(S0[at + 2], S0[at + 3]);
      G01 = pk(S0[at + 4], S0[at + 5]);
      G23 = pk(S0[at + 6], S0[at + 7]);
    };
    float2 D01, D23, G01, G23;
    LwLev La, Lb;
    int k = B;
    if (B & 1) {  // an even level count: the last checkpoint covers kx-2 and kx-1
      fetch(B - 1, D01, D23, G01, G23);
      const float ta = T[B - 1], qa = Q[B - 1], q = Q[B];
      const float tm = T[B - 2];
      lw_level<KX, LV_MID>(CD, lw, B - 1, tm, ta, t, qa, La);
      const float da = d_at(B - 1);
      float2 Db01 = D01, Db23 = D23, Gb01 = G01, Gb23 = G23;
      lw_down_step<LV_MID>(La, da, Db01, Db23, Gb01, Gb23);
      lw_level<KX, LV_LAST>(CD, lw, B, ta, t, 0.0f, q, Lb);
      float qb = sfc_q_b;
      lw_rev_level<KX, LV_LAST>(CD, lw, Lb, B, t, q, dB, Db01, Db23, Gb01, Gb23, r, qb);
      QB[B] = qb;
      done(B);
      qb = 0.0f;
      lw_rev_level<KX, LV_MID>(CD, lw, La, B - 1, ta, qa, da, D01, D23, G01, G23, r, qb);
      QB[B - 1] = qb;
      done(B - 1);
      tp = ta;
      t = tm;
      k = B - 2;
    } else {
      fetch(B, D01, D23, G01, G23);
      const float tm = T[B - 1], q = Q[B];
      lw_level<KX, LV_LAST>(CD, lw, B, tm, t, 0.0f, q, Lb);
      float qb = sfc_q_b;
      lw_rev_level<KX, LV_LAST>(CD, lw, Lb, B, t, q, dB, D01, D23, G01, G23, r, qb);
      QB[B] = qb;
      done(B);
      tp = t;
      t = tm;
      k = B - 1;
    }
    float ct_k = ctt(k), ct_m = ctt(k - 1);
#pragma unroll 1
    for (; k >= 3; k -= 2) {  // levels k (odd) and k - 1
      fetch(k - 1, D01, D23, G01, G23);
      const float d = d_of(ct_k, k), da = d_of(ct_m, k - 1);
      ct_k = ctt(k - 2);
      ct_m = ctt(k - 3);
      const float ta = T[k - 1], tm = T[k - 2], q = Q[k], qa = Q[k - 1];
      lw_level<KX, LV_MID>(CD, lw, k - 1, tm, ta, t, qa, La);
      float2 Db01 = D01, Db23 = D23, Gb01 = G01, Gb23 = G23;
      lw_down_step<LV_MID>(La, da, Db01, Db23, Gb01, Gb23);
      lw_level<KX, LV_MID>(CD, lw, k, ta, t, tp, q, Lb);
      float qb = 0.0f;
      lw_rev_level<KX, LV_MID>(CD, lw, Lb, k, t, q, d, Db01, Db23, Gb01, Gb23, r, qb);
      QB[k] = qb;
      done(k);
      qb = 0.0f;
      lw_rev_level<KX, LV_MID>(CD, lw, La, k - 1, ta, qa, da, D01, D23, G01, G23, r, qb);
      QB[k - 1] = qb;
      done(k - 1);
      tp = ta;
      t = tm;
    }
    // levels 1 and 0: nothing enters level 0
    const float ta = T[0], q = Q[1];
    lw_level<KX, LV_TOP>(CD, lw, 0, 0.0f, ta, t, 0.0f, La);
    const float d0 = d_of(ct_m, 0), d1 = d_of(ct_k, 1);
    lw_down_step<LV_TOP>(La, d0, D01, D23, G01, G23);
    lw_level<KX, LV_SECOND>(CD, lw, 1, ta, t, tp, q, Lb);
    float qb = 0.0f;
    lw_rev_level<KX, LV_SECOND>(CD, lw, Lb, 1, t, q, d1, D01, D23, G01, G23, r, qb);
    QB[1] = qb;
    done(1);
    qb = 0.0f;
    lw_rev_level<KX, LV_TOP>(CD, lw, La, 0, ta, 0.0f, d0, bc(0.0f), bc(0.0f), bc(0.0f), bc(0.0f),
                             r, qb);
    QB[0] = qb;
    TB[1] = r.hi;
    TB[0] = r.mid;
  }
  float psa_b = r.psa_b;
  dps = r.dps;
  float cloudc_b = r.acl1_b * p.ablcl1 + r.acl2_b * p.ablcl2;

  // ---- shortwave: its downward fluxes again, with the adjoint of the upward flux, then back ---
  float clstr_b = 0.0f, qcloud_b = 0.0f;
  {
    float f1, f2 = f20, upb = fsw0_b;
    auto dsw_of = [&](float ctk, int k) { return swon ? d_of(ctk, k) : 0.0f; };
    float ct_k = ctt(2);
    const float t00 = sw_tau0(0, 0.0f);
    const float d0 = dsw_of(ctt(0), 0), d1 = dsw_of(ctt(1), 1);
    const float f1a = t00 * (f10 - z.ozupp * psa);
    upb = fmaf(upb, t00, d0 * (1.0f - t00));
    const float upb1 = upb;
    const float q1 = Q[1], t01 = sw_tau0(1, q1), t11 = sw_tau1(1, q1);
    const float g1 = f1a - z.ozone * psa;
    f1 = t01 * g1;
    upb = fmaf(upb, t01, d1 * (1.0f - t01));
    f2 = f2 * t11;
#pragma unroll 2
    for (int k = 2; k < KX; ++k) {
      const float d = dsw_of(ct_k, k);
      ct_k = ctt(min(k + 1, B));
      const float q = Q[k], t0 = sw_tau0(k, q), rk = refl_at(k);
      S0[k] = f1;
      S1[k] = t0;
      S2[k] = f2;
      S3[k] = upb;
      f1 = f1 * t0 * (1.0f - rk);
      f2 = f2 * sw_tau1(k, q);
      upb = fmaf(upb, t0, d * (1.0f - t0));
    }
    float f1_b = fmaf(upb, albsfc, rsds_b), f2_b = fsw1_b + rsds_b;
    float up = f1 * albsfc;
    float psaz_b = 0.0f, acloud_b = 0.0f, refl_b = 0.0f;
#pragma unroll 2
    for (int k = B; k >= 2; --k) {
      const float d = dsw_of(ct_k, k);
      ct_k = ctt(k - 1);
      const float q = Q[k], prev = S0[k], t0 = S1[k], f2p = S2[k], ub = S3[k];
      const float rk = refl_at(k), om = 1.0f - rk, omt = 1.0f - t0;
      const float t1 = sw_tau1(k, q), om1 = 1.0f - t1;
      dps = fmaf(d, fmaf(prev * om, omt, fmaf(f2p, om1, up * omt)), dps);
      const float t1b = (f2_b - d) * f2p;
      f2_b = fmaf(f2_b, t1, d * om1);
      const float g = fmaf(f1_b, t0, d * omt);
      const float rb = prev * (ub - g);
      const float t0b = fmaf(ub - d, up, prev * om * (f1_b - d));
      up = fmaf(up, t0, rk * prev);
      f1_b = fmaf(ub, rk, om * g);
      const float dh = vg.dhs[k];
      const float e1 = t1b * t1 * (dh * p.abswv2), e0 = t0b * t0 * dh;
      psaz_b -= fmaf(e1, q, e0 * sw_inner(k, q));
      const float ib = -e0 * psaz;
      QB[k] = fmaf(ib, p.abswv1, fmaf(-e1, psaz, QB[k]));
      if (k == B) {
        par[spdvjp::P_ALBCLS] += rb * clstr;
        clstr_b = rb * p.albcls;
      } else {
        acloud_b += (k >= icltop) ? ib : 0.0f;
        refl_b += ((S >> k) & 1u) ? rb : 0.0f;
      }
    }
    {  // level 1
      const float dh = vg.dhs[1], omt = 1.0f - t01, om1 = 1.0f - t11;
      dps = fmaf(d1, (f1a - t01 * g1) + fmaf(f20, om1, up * omt), dps);
      const float t1b = (f2_b - d1) * f20;
      const float fb = f1_b - d1;
      const float t0b = fmaf(upb1 - d1, up, fb * g1);
      const float gg = fb * t01;
      psa_b -= gg * z.ozone;
      f1_b = gg + d1;
      up = fmaf(up, t01, refl_at(1));
      const float e1 = t1b * t11 * (dh * p.abswv2), e0 = t0b * t01 * dh;
      psaz_b -= fmaf(e1, q1, e0 * sw_inner(1, q1));
      const float ib = -e0 * psaz;
      QB[1] = fmaf(ib, p.abswv1, fmaf(-e1, psaz, QB[1]));
      acloud_b += (1 >= icltop) ? ib : 0.0f;
      refl_b += ((S >> 1) & 1u) ? upb1 : 0.0f;
    }
    {  // level 0
      const float fb = f1_b - d0;
      dps = fmaf(d0, (f10 - f1a) + up * (1.0f - t00), dps);
      const float t0b = fmaf(fsw0_b - d0, up, fb * (f10 - z.ozupp * psa));
      psa_b -= fb * t00 * z.ozupp;
      psaz_b -= t0b * t00 * vg.dhs[0] * p.absdry;
      refl_b += (S & 1u) ? fsw0_b : 0.0f;
    }
    cloudc_b += acloud_b * mnq;
    qcloud_b = acloud_b * cloudc * wmin(p.abscl1 * qcloud, p.abscl2) * p.abscl1;
    psa_b += psaz_b * z.zenit;
    if (cmask) {
      par[spdvjp::P_ALBCL] += refl_b * cloudc;
      cloudc_b += refl_b * p.albcl;
    }
  }

  // ---- clouds' reverse (scalars), vertical diffusion's reverse, both level by level -----------
  // From here S0 is the phi adjoint, S1 the qsat adjoint; S2 holds the relative humidity and S3
  // the running maximum of the cloud cover's candidates.
  const Lv PB = S0, XB = S1, RHs = S2, PM = S3;
  auto dq_b = [&](int k) {
    return ((limited >> k) & 1u) ? 0.0f : col.at(col.ct_q, k) * K.q_tend_scale;
  };
  float precnv_b = 0.0f, precls_b = 0.0f;
  {
    const int nl1 = KX - 2;
    const float rh_nl1 = fdiv(Q[nl1], QS[nl1]), rh_B = fdiv(Q[B], QS[B]);
    RHs[nl1] = rh_nl1;
    RHs[B] = rh_B;
    const bool m0 = rh_nl1 > p.rhcl1;
    const float cloudc0 = m0 ? rh_nl1 - p.rhcl1 : 0.0f;
    float cmax = 0.0f;
    uint32_t mk = 0u;
#pragma unroll 2
    for (int k = 2; k < KX - 2; ++k) {
      const float q = Q[k], rh = fdiv(q, QS[k]);
      RHs[k] = rh;
      const float drh = rh - p.rhcl1;
      const bool m = drh > cloudc0 && q > p.qacl;
      if (m) mk |= 1u << k;
      const float upd = m ? drh : cloudc0;
      cmax = (k == 2) ? upd : spdvjp::vmax(cmax, upd);
      PM[k] = cmax;
    }
    const float phiB = col.at(col.phi, B), phin = col.at(col.phi, nl1);
    const float seB = kCp * T[B] + phiB, sen = kCp * T[nl1] + phin;
    const float den = phin - phiB;
    const float rden = frcp(den), gse = fdiv_full(sen - seB, den);  // den may be zero
    const float rrcl = D.rrcl;
    const float pr1v = 86.4f * (o.precnv + o.precls);
    const float pr1 = spdvjp::vmin(p.pmaxcl, pr1v);
    const float cc1 = spdvjp::vmin(1.0f, cmax * rrcl);
    const float mx = spdvjp::vmax(1e-9f, pr1);
    const float sqm = sqrtf(mx);
    const float Z = p.wpcl * sqm + cc1 * cc1;
    const bool cloud_nan = isnan(spdvjp::vmin(1.0f, Z));
    const float fstab_y = D.rgse * (gse - p.gse_s0);
    const float fstab_m = spdvjp::vmax(fstab_y, 0.0f);
    const float fstab = spdvjp::vmin(fstab_m, 1.0f);
    const float Nv = p.clsmax - 1.2f * cloudc;
    const float N = spdvjp::vmax(Nv, 0.0f);
    const float clstr1 = fstab * N;
    const float clstrl_m = spdvjp::vmax(clstr1, p.clsminl);
    // bottom levels' contributions, carried in registers: se = adjoint of cp T + phi
    float rhB_b, rhn_b = 0.0f, seB_b, sen_b, phin_x, qn_b = qcloud_b, qsB_b = sfc_qs_b, qsn_b = 0.0f;
    float qB_x = 0.0f;
    {
      const float clstrl_b = fmask * clstr_b;
      float clstr1_b = clstr_b - clstrl_b;
      rhB_b = clstrl_b * clstrl_m;
      clstr1_b += clstrl_b * rh_B * wmax(clstr1, p.clsminl);
      const float N_b = clstr1_b * fstab;
      cloudc_b += -1.2f * N_b * wmax(Nv, 0.0f);
      const float y_b = clstr1_b * N * wmin(fstab_m, 1.0f) * wmax(fstab_y, 0.0f);
      const float gse_b = y_b * D.rgse;
      const float a_b = gse_b * rden;
      sen_b = a_b;
      seB_b = -a_b;
      phin_x = -a_b * gse;
    }
    float cmax_b = 0.0f, cloudc0_b = 0.0f;
    if (!cloud_nan) {
      const float Z_b = cloudc_b * wmin(Z, 1.0f);
      const float cc_b = Z_b * 2.0f * cc1;
      const float mx_b = Z_b * p.wpcl * fdiv(0.5f, sqm);
      const float v_b = mx_b * wmax(pr1, 1e-9f) * wmin(pr1v, p.pmaxcl) * 86.4f;
      precnv_b = v_b;
      precls_b = v_b;
      cmax_b = cc_b * wmin(cmax * rrcl, 1.0f) * rrcl;
    }
    // vertical diffusion, lowest two levels (shallow convection and moisture)
    const float dqB = dq_b(B), dqn = dq_b(nl1), dtB = col.at(col.ct_t, B),
                dtn = col.at(col.ct_t, nl1);
    {
      const float dmse = seB - sen + kAlhc * (Q[B] - QS[nl1]);
      const float drh = rh_B - rh_nl1;
      const int icnv = KX - o.iptop - 1;
      const float fcnv = (icnv > 0 && dmse >= 0.0f) ? p.redshc : 1.0f;
      const float fq_b = dqn * D.rsig[nl1] - dqB * D.rsig[B];
      float dmse_b = 0.0f, drh_b = 0.0f;
      if (dmse >= 0.0f) {
        const float fx_b = dtn * D.rsig[nl1] - dtB * D.rsig[B];
        dmse_b = fx_b * fcnv * D.fshcse;
        if (drh >= 0.0f) {
          const float f = fq_b * fcnv * D.fshcq;
          qsB_b = fmaf(f, drh, qsB_b);
          drh_b = f * QS[B];
        }
      } else if (dmse < 0.0f && drh > D.drh0) {
        const float f = fq_b * D.fvdiq2;
        qsn_b = f * drh;
        drh_b = f * QS[nl1];
      }
      seB_b += dmse_b;
      sen_b -= dmse_b;
      qB_x = kAlhc * dmse_b;
      qsn_b -= kAlhc * dmse_b;
      rhB_b += drh_b;
      rhn_b -= drh_b;
    }
    // levels, bottom up.  s_up: adjoint of the lapse-rate flux between k and k + 1, which adds
    // -s to level k's dry static energy and s to level k + 1's, and -segrad times that to phi;
    // r_up: adjoint of the relative humidity difference of the pair (k, k + 1).
    float acc = 0.0f, s_up = 0.0f, r_below = 0.0f;
    float se_n = seB, phi_n = phiB, t_n_b = dtB, dq_n = dqB;
    float carry_s = 0.0f;  // s of the pair (k + 1, k + 2)
    float phi_k = phin, ct_k = dtn, cq_k = col.at(col.ct_q, nl1);
    auto finish = [&](int k, float sx, float se_x, float rh_x, float q_x, float qs_x, float phi_x) {
      const float se_b = sx + se_x;
      TB[k] = fmaf(kCp, se_b, TB[k]);
      PB[k] = fmaf(-p.segrad, sx, se_b) + phi_x;
      const float rq = frcp(QS[k]);
      const float v = rh_x * rq;
      QB[k] = QB[k] + (v + q_x);
      XB[k] = qs_x - v * RHs[k];
    };
    enum { kBottom, kNext, kMid, kTop };  // k = kx-2, kx-3, 2..kx-4, 1 and 0
    auto level = [&](auto kind, int k) {
      constexpr int KIND = decltype(kind)::value;
      constexpr bool pair = KIND == kNext || KIND == kMid;  // humidity diffuses between k, k + 1
      const float phi = phi_k, dt_k = ct_k;
      const float dq_k = ((limited >> k) & 1u) ? 0.0f : cq_k * K.q_tend_scale;
      const int kn = max(k - 1, 0);
      phi_k = col.at(col.phi, kn);
      ct_k = ctt(kn);
      cq_k = col.at(col.ct_q, kn);
      const float se = kCp * T[k] + phi;
      acc -= t_n_b;
      const float fse_b = fmaf(acc, D.rsig1[k], dt_k * D.rsig[k]);
      const float se0 = se_n - p.segrad * (phi_n - phi);
      const float sk = (se < se0) ? fse_b * D.fvdise : 0.0f;
      // level k + 1 is complete with s_k
      float dr_b = 0.0f, qs_x = 0.0f;
      if (pair) {
        const float dr = RHs[k + 1] - RHs[k];
        if (dr >= D.drh0v[k] && ((D.vdcond >> k) & 1u)) {
          const float fl = (dq_k * D.rsig[k] - dq_n * D.rsig[k + 1]) * D.fvdiq2v[k];
          qs_x = fl * dr;
          dr_b = fl * QS[k];
        }
      }
      if (KIND == kBottom) {
        finish(B, sk - carry_s, seB_b, rhB_b, qB_x, qsB_b, sfc_phi_b - phin_x);
      } else if (KIND == kNext) {
        finish(nl1, sk - carry_s, sen_b, rhn_b + dr_b, qn_b, qsn_b, phin_x);
      } else if (KIND == kMid || k == 1) {
        finish(k + 1, sk - carry_s, 0.0f, r_below + dr_b, 0.0f, s_up, 0.0f);
      } else {  // levels 1 and 0 have no relative humidity terms
        const float sx = sk - carry_s;
        TB[k + 1] = fmaf(kCp, sx, TB[k + 1]);
        PB[k + 1] = fmaf(-p.segrad, sx, sx);
        XB[k + 1] = 0.0f;
      }
      carry_s = sk;
      // what level k brings to its own completion: the cloud cover's candidate and -dr_b
      float ub = 0.0f;
      if (pair) {
        const float rh = RHs[k];
        const bool m = (mk >> k) & 1u;
        const float upd = m ? rh - p.rhcl1 : cloudc0;
        ub = cmax_b;
        if (k > 2) {
          const float pm = PM[k - 1];
          ub = cmax_b * wmax(upd, pm);
          cmax_b = cmax_b * wmax(pm, upd);
        }
        if (!m) {
          cloudc0_b += ub;
          ub = 0.0f;
        }
      }
      r_below = ub - dr_b;
      s_up = qs_x;
      se_n = se;
      phi_n = phi;
      t_n_b = dt_k;
      dq_n = dq_k;
    };
    level(std::integral_constant<int, kBottom>{}, KX - 2);
    level(std::integral_constant<int, kNext>{}, KX - 3);
#pragma unroll 2
    for (int k = KX - 4; k >= 2; --k) level(std::integral_constant<int, kMid>{}, k);
    level(std::integral_constant<int, kTop>{}, 1);
    level(std::integral_constant<int, kTop>{}, 0);
    {
      const float sx = -carry_s;
      TB[0] = fmaf(kCp, sx, TB[0]);
      PB[0] = fmaf(-p.segrad, sx, sx);
      XB[0] = 0.0f;
    }
    if (m0) {
      const float v = cloudc0_b * frcp(QS[nl1]);
      QB[nl1] = QB[nl1] + v;
      XB[nl1] = XB[nl1] - v * rh_nl1;
    }
  }

  // ---- convection: diagnosis and mass flux again, then back -----------------------------------
  // e_k: cotangent of level k's humidity flux divergence, d_k its dry static energy's.
  {
    const float q_B = Q[B], q_n = Q[B - 1], qs_B = QS[B], qs_n = QS[B - 1];
    const float seB = kCp * T[B] + col.at(col.phi, B), sen = kCp * T[B - 1] + col.at(col.phi, B - 1);
    const float mse0 = seB + kAlhc * q_B;
    const float mse1 = spdvjp::vmin(mse0, sen + kAlhc * q_n);
    const float mss0 = spdvjp::vmax(mse0, seB + kAlhc * qs_B);
    int ktop1 = KX, ktop2 = KX;
    float msthr = 0.0f;
    float mk1 = (kCp * T[KX - 3] + col.at(col.phi, KX - 3)) + kAlhc * QS[KX - 3];
    float phi_k = col.at(col.phi, KX - 4);
#pragma unroll 2
    for (int k = KX - 4; k >= 2; --k) {
      const float phi = phi_k;
      phi_k = col.at(col.phi, k - 1);
      const float mk = (kCp * T[k] + phi) + kAlhc * QS[k];
      const float m2 = mk + vg.wvi[k][1] * (mk1 - mk);
      if (mss0 > m2) ktop1 = k + 1;
      if (mse1 > m2) {
        ktop2 = k + 1;
        msthr = m2;
      }
      mk1 = mk;
    }
    const float qthr0 = p.rhbl * qs_B, qthr1 = p.rhbl * qs_n;
    const bool mask_psa = psa > p.psmin;
    const bool case1 = mask_psa && ktop1 < KX && ktop2 < KX;
    const bool case2 = mask_psa && ktop1 < KX && !(ktop2 < KX) && q_B > qthr0 && q_n > qthr1;
    // without convection every adjoint below is zero: skip a warp that has none
    const bool convects = case1 || case2;
    if (__any_sync(0xffffffffu, convects)) {
      const int iptop = convects ? ktop1 : KX + 1;
      const int kmin = __reduce_min_sync(0xffffffffu, iptop);
      float qdif = 0.0f;
      const float thrA = q_B - qthr0, thrB = (mse0 - msthr) * (float)(1.0 / 2501.0);
      if (case1) qdif = spdvjp::vmax(thrA, thrB);
      if (case2) qdif = thrA;
      const float q101 = 1.01f * q_B;
      const float qmax = spdvjp::vmax(q101, qs_B);
      const float wl = vg.wvi[B - 1][1];
      const float sb = sen + wl * (seB - sen);
      const float qb3 = q_n + wl * (q_B - q_n);
      const float qb = spdvjp::vmin(qb3, q_B);
      const float mn2y = (psa - p.psmin) * D.rdps;
      const float mn2 = spdvjp::vmin(1.0f, mn2y);
      const float fpsa = psa * mn2;
      const float den = qmax - qb;
      const float rden = frcp(den), ratio = qdif * rden;
      const float mn = spdvjp::vmin(5.0f, ratio);
      const float fmass = D.fm0 * fpsa * mn;
      const float cbmf = convects ? fmass : 0.0f * fmass;
      const float fus = fmass * seB, fuq = fmass * qmax, fds = fmass * sb, fdq = fmass * qb;
      const Lv FM = S2;
      auto e_of = [&](float cqk, int k) {
        return (((limited >> k) & 1u) ? 0.0f : cqk * K.q_tend_scale) * vg.grdsig[k] * rpsa;
      };
      auto ctq = [&](int k) { return col.at(col.ct_q, k); };
      auto e_at = [&](int k) { return e_of(ctq(k), k); };
      // mass flux, level by level upwards; collects the cotangent x divergence sum (dps) and the
      // top layer's precipitation
      float X = 0.0f, qsatb = 0.0f, fm_top = 0.0f, fsq_sum = 0.0f;
      {
        float cm = 0.0f, cs = 0.0f, cq = 0.0f;
        float fm_n = 0.f, fs_n = 0.f, fq_n = 0.f, fus_n = 0.f, fuq_n = 0.f, fds_n = 0.f, fdq_n = 0.f;
        float se_k = seB, q_k = q_B;
        float phi_m = col.at(col.phi, B - 1), ct_k = ctt(B), cq_k = ctq(B);
#pragma unroll 1
        for (int k = B; k >= kmin - 1; --k) {
          const float d = d_of(ct_k, k), e = e_of(cq_k, k), phim = phi_m;
          phi_m = col.at(col.phi, k - 2);  // kmin >= 3
          ct_k = ctt(k - 1);
          cq_k = ctq(k - 1);
          const bool lm = (k <= KX - 2) && (k >= iptop);
          const float en = lm ? D.entr[k] * psa * cbmf : 0.0f;
          cm = cm + en;
          cs = cs + en * se_k;
          cq = cq + en * q_k;
          const float fm_k = fmass + cm, fus_k = fus + cs, fuq_k = fuq + cq;
          FM[k] = fm_k;
          const float se_m = kCp * T[k - 1] + phim, q_m = Q[k - 1];
          float dse, dqa, fds_k, fdq_k;
          if (k == B) {
            fds_k = fds;
            fdq_k = fdq;
            dse = fds - fus;
            dqa = fdq - fuq;
          } else {
            const float w = vg.wvi[k - 1][1];
            fds_k = fm_k * (se_m + w * (se_k - se_m));
            fdq_k = fm_k * (q_m + w * (q_k - q_m));
            dse = lm ? fs_n - (fus_k - fds_k) : 0.0f;
            dqa = lm ? fq_n - (fuq_k - fdq_k) : 0.0f;
          }
          if (lm) {
            const float d0 = p.rhil * QS[k] - q_k;
            const float fsq = (d0 > 0.0f ? p.smf : 0.0f) * cbmf * d0;
            dqa += fsq;
            fsq_sum += fsq;
          }
          if (k == iptop - 1) {
            const float qs_k = QS[k];
            qsatb = qs_k + vg.wvi[k][1] * (QS[k + 1] - qs_k);
            fm_top = fm_n;
            X = fuq_n - fm_n * qsatb;
            const float precnv = fmaxf(X, 0.0f);
            dse = fus_n - fds_n + kAlhc * precnv;
            dqa = fuq_n - fdq_n - precnv;
          }
          if (convects) dps = fmaf(d, dse, fmaf(e, dqa, dps));
          fm_n = fm_k;
          fus_n = fus_k;
          fuq_n = fuq_k;
          fds_n = fds_k;
          fdq_n = fdq_k;
          fs_n = fus_k - fds_k;
          fq_n = fuq_k - fdq_k;
          se_k = se_m;
          q_k = q_m;
        }
      }
      const float eB = e_at(B);
      if (convects) dps = fmaf(-eB, fsq_sum, dps);
      // back down.  a, qa: adjoints of the flux differences of the level above
      float CMB = 0.0f, CSB = 0.0f, CQB = 0.0f, cbmf_b = 0.0f;
      float a_m = 0.0f, q_m_b = 0.0f;   // of level k - 1, where it is in the layer or the top
      float fds_b = 0.0f, fdq_b = 0.0f;
      float ent_b = 0.0f;
      float se_m = kCp * T[kmin - 1] + col.at(col.phi, kmin - 1), q_m = Q[kmin - 1];
      // adjoints of level k - 1 that level k completes
      float seb_m = 0.0f, qbb_m = 0.0f;
      const float fsq_sum_b = -eB;
      if (iptop == kmin) {  // the top layer k = iptop - 1 feeds level iptop's fluxes
        a_m = d_at(kmin - 1);
        q_m_b = e_at(kmin - 1);
      }
      float phi_k2 = col.at(col.phi, kmin), ct_k = ctt(kmin), cq_k = ctq(kmin);
#pragma unroll 1
      for (int k = kmin; k < KX; ++k) {
        const float d = d_of(ct_k, k), e = e_of(cq_k, k);
        const float se_k = kCp * T[k] + phi_k2, q_k = Q[k];
        const int kn = min(k + 1, B);
        phi_k2 = col.at(col.phi, kn);
        ct_k = ctt(kn);
        cq_k = ctq(kn);
        const bool lm = (k <= KX - 2) && (k >= iptop);
        const bool top = k == iptop;
        const float a = lm ? d : 0.0f, qa = lm ? e : 0.0f;
        float fus_b = a_m - a, fuq_b = q_m_b - qa;
        float fdq_bk = -fuq_b, fm_b = 0.0f, xs_b = 0.0f;
        if (top) {
          const float pb = precnv_b + kAlhc * a_m - q_m_b;
          const float Xb = pb * wmax(X, 0.0f);
          fuq_b += Xb;
          fm_b = -Xb * qsatb;
          xs_b = -Xb * fm_top;
        }
        const float fds_bk = -fus_b;
        float se_b = 0.0f, qk_b = 0.0f, qs_b = 0.0f;
        const float w = vg.wvi[k - 1][1];
        float sb3_b = 0.0f, qb3_b = 0.0f;
        if (k < B) {
          const float fm_k = FM[k];
          fm_b += fds_bk * (se_m + w * (se_k - se_m)) + fdq_bk * (q_m + w * (q_k - q_m));
          sb3_b = fds_bk * fm_k;
          qb3_b = fdq_bk * fm_k;
        } else {
          fds_b = fds_bk;
          fdq_b = fdq_bk;
        }
        CMB += fm_b;
        CSB += fus_b;
        CQB += fuq_b;
        if (lm) {
          const float ep = D.entr[k] * psa, en = ep * cbmf;
          const float en_b = CMB + CSB * se_k + CQB * q_k;
          se_b = CSB * en;
          qk_b = CQB * en;
          cbmf_b = fmaf(en_b, ep, cbmf_b);
          ent_b = fmaf(en_b, D.entu[k], ent_b);
          const float qs_k = QS[k];
          const float d0 = p.rhil * qs_k - q_k;
          if (d0 > 0.0f) {
            const float fsq_b = e + fsq_sum_b;
            cbmf_b = fmaf(fsq_b * d0, p.smf, cbmf_b);
            par[spdvjp::P_SMF] += fsq_b * d0 * cbmf;
            const float d0_b = fsq_b * (p.smf * cbmf);
            par[spdvjp::P_RHIL] += d0_b * qs_k;
            qs_b = d0_b * p.rhil;
            qk_b -= d0_b;
          }
        }
        if (k == B) {  // qb = min(qb3, q[kx-1]) and sb = sb3 join the lowest interface
          const float d_B = convects ? d : 0.0f, e_B = convects ? e : 0.0f;
          fds_b += d_B;
          fdq_b += e_B;
          const float fus_t = CSB - d_B, fuq_t = CQB - e_B;
          float fmass_b = CMB + fus_t * seB + fuq_t * qmax + fds_b * sb + fdq_b * qb;
          se_b = fmaf(fus_t, fmass, se_b);
          float qmax_b = fuq_t * fmass, qb_b = fdq_b * fmass;
          if (convects) fmass_b += cbmf_b;
          // fmass = fm0 * fpsa * min(5, qdif / (qmax - qb))
          const float A_b = fmass_b * mn;
          const float mn_b = fmass_b * (D.fm0 * fpsa);
          const float ratio_b = mn_b * wmin(ratio, 5.0f);
          const float qdif_b = ratio_b * rden;
          const float den_b = -qdif_b * ratio;
          qmax_b += den_b;
          qb_b -= den_b;
          const float fpsa_b = A_b * D.fm0;
          const float y_b = fpsa_b * psa * wmin(mn2y, 1.0f);
          psa_b += fmaf(fpsa_b, mn2, y_b * D.rdps);
          par[spdvjp::P_PSMIN] +=
              y_b * (psa - p.psmin) * (0.5f * D.rdps * D.rdps) - y_b * D.rdps;
          par[spdvjp::P_TRCNV] += -(A_b * fpsa) * D.fm0_t;
          qb3_b = qb_b * wmin(qb3, q_B);
          qk_b = fmaf(qb_b, wmin(q_B, qb3), qk_b);
          sb3_b = fds_b * fmass;
          qk_b = fmaf(qmax_b * wmax(q101, qs_B), 1.01f, qk_b);
          qs_b = fmaf(qmax_b, wmax(qs_B, q101), qs_b);
          // diagnosis: qdif = max(q - rhbl qsat, (mse0 - msthr) / 2501) or its first argument
          float qthr0_b = 0.0f;
          if (case1) {
            const float Ab = qdif_b * wmax(thrA, thrB), Bb = qdif_b * wmax(thrB, thrA);
            qk_b += Ab;
            qthr0_b = -Ab;
            const float m_b = Bb * (float)(1.0 / 2501.0);
            se_b += m_b;
            qk_b = fmaf(kAlhc, m_b, qk_b);
            const int jt = ktop2 - 1;  // the threshold level, each column its own
            const float wj = vg.wvi[jt][1];
            const float m1 = -wj * m_b, m0 = -m_b - m1;
            TB[jt] = fmaf(kCp, m0, TB[jt]);
            PB[jt] = PB[jt] + m0;
            XB[jt] = fmaf(kAlhc, m0, XB[jt]);
            TB[jt + 1] = fmaf(kCp, m1, TB[jt + 1]);
            PB[jt + 1] = PB[jt + 1] + m1;
            XB[jt + 1] = fmaf(kAlhc, m1, XB[jt + 1]);
          } else if (case2) {
            qk_b += qdif_b;
            qthr0_b = -qdif_b;
          }
          par[spdvjp::P_RHBL] += qthr0_b * qs_B;
          qs_b = fmaf(qthr0_b, p.rhbl, qs_b);
        }
        // sb3 = se_{k-1} + w (se_k - se_{k-1}), qb3 alike: completes level k - 1
        const float s1 = w * sb3_b, q1 = w * qb3_b;
        const float se_x = seb_m + (sb3_b - s1), q_x = qbb_m + (qb3_b - q1);
        TB[k - 1] = fmaf(kCp, se_x, TB[k - 1]);
        PB[k - 1] = PB[k - 1] + se_x;
        QB[k - 1] = QB[k - 1] + q_x;
        if (top) {
          const float w2 = w * xs_b;
          XB[k - 1] = XB[k - 1] + (xs_b - w2);
          qs_b += w2;
        }
        if (qs_b != 0.0f) XB[k] = XB[k] + qs_b;
        seb_m = se_b + s1;
        qbb_m = qk_b + q1;
        if (k == iptop - 1) {  // this column's top layer, below the warp's highest
          a_m = d;
          q_m_b = e;
        } else {
          a_m = a;
          q_m_b = qa;
        }
        se_m = se_k;
        q_m = q_k;
      }
      TB[B] = fmaf(kCp, seb_m, TB[B]);
      PB[B] = PB[B] + seb_m;
      QB[B] = QB[B] + qbb_m;
      // the entrainment is entmax * entu: entmax may be zero
      psa_b = fmaf(ent_b * p.entmax, cbmf, psa_b);
      par[spdvjp::P_ENTMAX] += ent_b * cbmf * psa;
    }
  }

  // ---- condensation and saturation humidity, level by level; the gradients -------------------
  {
    const float tfact = (float)(2501.0 / 1004.0);
    const float psa2 = psa * psa;
    psa_b += precls_b * (o.precls * rpsa);
    const float psum_b = -precls_b * psa;
    float psa2_b = 0.0f, rtlsc_b = 0.0f, xps = 0.0f;
    const float rdt = K.dt_seconds;
    // plain loads, each level's before the level above it is stored: a gradient may share its
    // buffer with an input or a cotangent
    float *gt = load_field(m.gr.temperature) + c, *gq = load_field(m.gr.specific_humidity) + c,
          *gp = load_field(m.gr.geopotential) + c, *gu = load_field(m.gr.u_wind) + c,
          *gv = load_field(m.gr.v_wind) + c;
    float cq_n = col.ct_q[0], ct_n = col.ct_t[0];
#pragma unroll 2
    for (int k = 0; k < KX; ++k) {
      const float ctq = cq_n * K.q_tend_scale, ctt_k = ct_n;
      const size_t in1 = (k < B ? k + 1 : B) * C;
      cq_n = col.ct_q[in1];
      ct_n = col.ct_t[in1];
      const float t = T[k], q = Q[k], qs = QS[k];
      float qs_b = XB[k], q_b = QB[k];
      const bool lim = (limited >> k) & 1u;
      const float dqa = D.rhref[k] * qs - q;
      if (k >= 1 && dqa < 0.0f) {
        const float dql = dqa * D.rtlsc;
        const float sig2 = vg.fsg[k] * vg.fsg[k];
        const float Y = p.rhlsc + p.drhlsc * (sig2 - 1.0f);
        float dql_b = (lim ? 0.0f : ctq) + psum_b * D.pfact[k];
        const float m_b = ctt_k * tfact;
        const float P = D.dqmax[k] * psa2;
        dql_b -= m_b * wmin(-dql, P);
        const float P_b = m_b * wmin(P, -dql);
        psa2_b = fmaf(P_b, D.dqmax[k], psa2_b);
        const float dqa_b = dql_b * D.rtlsc;
        rtlsc_b += dql_b * dqa + P_b * psa2 * (10.0f * sig2);
        const float rh_b = dqa_b * qs;
        qs_b = fmaf(dqa_b, D.rhref[k], qs_b);
        q_b -= dqa_b;
        const float Y_b = rh_b * wmax(Y, p.rhblsc);
        par[spdvjp::P_RHBLSC] += rh_b * wmax(p.rhblsc, Y);
        par[spdvjp::P_RHLSC] += Y_b;
        par[spdvjp::P_DRHLSC] += Y_b * (sig2 - 1.0f);
      }
      // qsat = 622 e / (sig psa - 0.378 e): with x = qsat (1 + (0.378 / 622) qsat),
      // d/dT = x c (t0 - t1) / (T - t1)^2 and d/dpsa = -x / psa
      const bool warm = t >= 273.16f;
      const float den = t - (warm ? 35.86f : 7.66f);
      const float x = fmaf(qs * (float)(0.378 / 622.0), qs, qs) * qs_b;
      xps += x;
      const float a = warm ? (float)(17.269 * (273.16 - 35.86)) : (float)(21.875 * (273.16 - 7.66));
      const float tb = TB[k] + x * fdiv(a, den * den);
      if (valid) {
        const size_t i = k * C;
        const float qk = ((neg >> k) & 1u) ? 0.0f : q_b;
        __stcs(gt + i, tb);
        __stcs(gq + i, qk + (lim ? -fdiv_full(ctq, rdt) : 0.0f));
        __stcs(gp + i, PB[k]);
        if (k < B) {
          __stcs(gu + i, 0.0f);
          __stcs(gv + i, 0.0f);
        }
      }
    }
    par[spdvjp::P_TRLSC] += -rtlsc_b * D.rtlsc_t;
    psa_b = fmaf(psa2_b, 2.0f * psa, psa_b);
    psa_b -= (xps + dps) * rpsa;
    if (valid) {
      gu[B * C] = u_b;
      gv[B * C] = v_b;
      load_field(m.gr.normalized_surface_pressure)[c] = psa_b;
    }
  }
}

}  // namespace spd

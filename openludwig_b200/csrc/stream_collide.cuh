// Fused pull-stream + collision for one 8^3 block per CTA (one cell per
// thread).  Cell stages follow kernel_cumulant.jl:70-627 and
// kernel_regularized_bgk.jl:43-325 in the same order:
//   pull + domain BCs -> obstacle bounce-back -> rho, u, sponge -> wall
//   model -> store u, rho -> WALE -> collision -> Guo forcing + store.
// The block's pull windows are staged in shared memory first (stage_block),
// rare paths (domain boundaries, level interfaces) fill their slots during
// that staging, and the per-cell path has no call sites and no
// address-taken arrays; the 27-direction loops are fully unrolled so every
// lattice constant folds.
#pragma once
#include <type_traits>

#include "level_dev.cuh"

namespace ol {

// ---------------------------------------------------------------------------
// Coarse-to-fine ghost values (physics_interpolation.jl:4-127), split into
// what a ghost position shares across directions (the parent stencil and the
// blended, interpolated rho and u) and the per-direction population.
// gx, gy, gz: 1-based fine-level global source coordinates.
// ---------------------------------------------------------------------------
// Parent cell indices fit 32 bits (every launch checks that a level's cells
// do); gathers add them to per-plane base pointers.
struct ParentStencil {
  int32_t ci[8];     // parent cell of each trilinear corner, -1 when absent
  float wx, wy, wz;  // trilinear weights
};

// Trilinear weights of the fine cell (gx, gy, gz) in the parent grid and the
// parent cell of corner s (bit 0: x + 1, bit 1: y + 1, bit 2: z + 1), or -1
// when that parent cell does not exist.
template <class DEV>
__device__ __forceinline__ int32_t parent_corner(const DEV &L, int gx, int gy, int gz, int s,
                                                 float &wx, float &wy, float &wz) {
  const float pxc = ((float)gx - 0.5f) * 0.5f;
  const float pyc = ((float)gy - 0.5f) * 0.5f;
  const float pzc = ((float)gz - 0.5f) * 0.5f;
  const int px0 = (int)floorf(pxc), py0 = (int)floorf(pyc), pz0 = (int)floorf(pzc);
  wx = pxc - (float)px0;
  wy = pyc - (float)py0;
  wz = pzc - (float)pz0;
  const int pgx = (s & 1) ? px0 + 1 : max(1, px0);
  const int pgy = (s & 2) ? py0 + 1 : max(1, py0);
  const int pgz = (s & 4) ? pz0 + 1 : max(1, pz0);
  const int pbx = (pgx - 1) / BS + 1, pby = (pgy - 1) / BS + 1, pbz = (pgz - 1) / BS + 1;
  if (pbx >= 1 && pbx <= L.pdim_x && pby >= 1 && pby <= L.pdim_y && pbz >= 1 &&
      pbz <= L.pdim_z) {
    const int pb = L.pptr[(pbx - 1) + L.pdim_x * ((pby - 1) + L.pdim_y * (pbz - 1))];
    if (pb > 0)
      return (int32_t)((L.p_block_offset + pb - 1) * BCELLS) + (pgx - 1) % BS +
             BS * ((pgy - 1) % BS) + BS * BS * ((pgz - 1) % BS);
  }
  return -1;
}

template <class DEV>
__device__ __forceinline__ void parent_stencil(const DEV &L, int gx, int gy, int gz,
                                               ParentStencil &P) {
#pragma unroll
  for (int s = 0; s < 8; ++s) P.ci[s] = parent_corner(L, gx, gy, gz, s, P.wx, P.wy, P.wz);
}

// a * (1 - w) + b * w, each product and the sum rounded on its own (as the
// reference's Float32 expression; the same bits wherever it is evaluated)
__device__ __forceinline__ float lerp_rn(float a, float b, float w) {
  return __fadd_rn(__fmul_rn(a, __fsub_rn(1.0f, w)), __fmul_rn(b, w));
}

__device__ __forceinline__ float trilerp(const float (&v)[8], float wx, float wy, float wz) {
  const float c00 = lerp_rn(v[0], v[1], wx);
  const float c01 = lerp_rn(v[4], v[5], wx);
  const float c10 = lerp_rn(v[2], v[3], wx);
  const float c11 = lerp_rn(v[6], v[7], wx);
  const float c0 = lerp_rn(c00, c10, wy);
  const float c1 = lerp_rn(c01, c11, wy);
  return lerp_rn(c0, c1, wz);
}

// Temporal blend of a parent value: lerp_rn(old, new, tw), or new alone
// without temporal interpolation.  At tw = 0 (the first child sub-step of a
// parent step) (1 - 0) * old + 0 * new rounds to old for every finite new, so
// `new` is not read there: half the parent gathers of that sub-step.
template <class NEW>
__device__ __forceinline__ float blend_parent(bool temporal, float tw, float old_v, NEW new_v) {
  if (!temporal) return new_v();
  if (tw == 0.0f) return old_v;
  return lerp_rn(old_v, new_v(), tw);
}

// Blended parent moments (rho, ux, uy, uz) of the present parent cell c at
// temporal weight tw.
__device__ __forceinline__ void corner_moments(const LevelDev &L, uint32_t c, float tw,
                                               float (&m)[4]) {
  const bool temporal = L.sp.use_temporal_interp == 1 && tw < 0.99f;
  const int64_t S = L.p_dstride;
  const float *vo = L.pvel_old, *vn = L.pvel;
  if (temporal && tw == 0.0f) {
    m[0] = L.prho_old[c]; m[1] = vo[c];
    m[2] = (vo + S)[c]; m[3] = (vo + 2 * S)[c];
    return;
  }
  const float rn = L.prho[c], uxn = vn[c], uyn = (vn + S)[c], uzn = (vn + 2 * S)[c];
  if (temporal) {
    m[0] = lerp_rn(L.prho_old[c], rn, tw);
    m[1] = lerp_rn(vo[c], uxn, tw);
    m[2] = lerp_rn((vo + S)[c], uyn, tw);
    m[3] = lerp_rn((vo + 2 * S)[c], uzn, tw);
  } else {
    m[0] = rn; m[1] = uxn; m[2] = uyn; m[3] = uzn;
  }
}

// Blended parent population k of the present parent cell c at weight tw.
template <class ST>
__device__ __forceinline__ float corner_population(const LevelDev &L, uint32_t c, int k,
                                                   float tw) {
  const bool temporal = L.sp.use_temporal_interp == 1 && tw < 0.99f;
  using T = typename ST::T;
  const T *po = (const T *)L.pf_old + (size_t)k * L.p_dstride;   // plane k
  const T *pn = (const T *)L.pf + (size_t)k * L.p_dstride;
  const float fo = temporal ? ST::load(po, c, k, L.p_inv_scale) : 0.0f;
  return blend_parent(temporal, tw, fo, [&] { return ST::load(pn, c, k, L.p_inv_scale); });
}

// Parent rho, ux, uy, uz at the ghost position: each corner blended between
// the parent's old and new state, missing corners replaced by the (possibly
// missing, then rho = 1, u = 0) first corner, then trilinear.
__device__ __forceinline__ void interp_moments(const LevelDev &L, const ParentStencil &P,
                                               float tw, float (&r)[4]) {
  float v[4][8];
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    float m[4] = {1.0f, 0.0f, 0.0f, 0.0f};
    if (P.ci[s] >= 0) corner_moments(L, (uint32_t)P.ci[s], tw, m);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i][s] = m[i];
  }
#pragma unroll
  for (int s = 1; s < 8; ++s)
    if (P.ci[s] < 0)
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i][s] = v[i][0];
#pragma unroll
  for (int i = 0; i < 4; ++i) r[i] = trilerp(v[i], P.wx, P.wy, P.wz);
}

// From the 8 corner values of f_k (absent corners already replaced): the
// interpolated f_k split into equilibrium (from the interpolated moments r)
// and non-equilibrium part, the latter rescaled by (tau_f - 1/2) /
// (tau_c - 1/2) clamped to [0.01, 100].
struct GhostScale {
  float sc;  // clamp((tau_f - 1/2) / (tau_c - 1/2), 0.01, 100)
  int comp;  // O(u^4) equilibrium
};
__device__ __forceinline__ GhostScale ghost_scale(float tau_parent, float tau, int comp) {
  const float tc = tau_parent - 0.5f, tf = tau - 0.5f;
  return {tc > 1e-6f ? fminf(fmaxf(tf / tc, 0.01f), 100.0f) : 1.0f, comp};
}
__device__ __forceinline__ GhostScale ghost_scale(const LevelDev &L) {
  return ghost_scale(L.sp.tau_parent, L.sp.tau_molecular, L.sp.compressible_corr);
}
__device__ __forceinline__ float finish_population(const GhostScale &g, int k, const float (&v)[8],
                                                   float wx, float wy, float wz,
                                                   const float (&r)[4]) {
  const float fi = trilerp(v, wx, wy, wz);
  const float fe = feq_auto(r[0], r[1], r[2], r[3], w_of(k), (float)cx_of(k), (float)cy_of(k),
                            (float)cz_of(k), g.comp);
  const float fneq = fi - fe;
  return __fadd_rn(fe, __fmul_rn(fneq, g.sc));
}

// Ghost population k at a position with stencil P and moments r (weight tw).
template <class ST>
__device__ __forceinline__ float interp_population(const LevelDev &L, int k,
                                                   const ParentStencil &P, const float (&r)[4],
                                                   float tw) {
  float v[8];
#pragma unroll
  for (int s = 0; s < 8; ++s)
    v[s] = P.ci[s] >= 0 ? corner_population<ST>(L, (uint32_t)P.ci[s], k, tw) : w_of(k);
#pragma unroll
  for (int s = 1; s < 8; ++s)
    if (P.ci[s] < 0) v[s] = v[0];
  return finish_population(ghost_scale(L), k, v, P.wx, P.wy, P.wz, r);
}

// ---------------------------------------------------------------------------
// Source value of a pull whose neighbour block is absent and whose source
// lies outside the domain or on level 1 (kernel_cumulant.jl:117-159); the
// fine-level interface case (:153-155) is interp_population, filled by
// fill_missing_flow.  x, y, z are 0-based local coordinates.
// ---------------------------------------------------------------------------
template <class ST>
__device__ __noinline__ float pull_boundary(const LevelDev &L, int k, int b,
                                            int x, int y, int z) {
  const ol_step_params &sp = L.sp;
  const int cx = cx_of(k), cy = cy_of(k), cz = cz_of(k);
  const int gx = (L.map_x[b] - 1) * BS + x + 1;
  const int gy = (L.map_y[b] - 1) * BS + y + 1;
  const int gz = (L.map_z[b] - 1) * BS + z + 1;
  const int sgx = gx - cx, sgy = gy - cy, sgz = gz - cz;
  const float w = w_of(k);
  if (sgx < 1) {
    const float noise = sp.inlet_turbulence > 0.0f
                            ? gradient_noise(gy, gz, sp.time_step_seed, 1234) *
                                  sp.inlet_turbulence * sp.u_inlet
                            : 0.0f;
    return feq_auto(1.0f, sp.u_inlet + noise, 0.0f, 0.0f, w, (float)cx, (float)cy,
                    (float)cz, sp.compressible_corr);
  }
  if (sgx > sp.nx_global)
    return feq_auto(1.0f, sp.u_inlet, 0.0f, 0.0f, w, (float)cx, (float)cy,
                    (float)cz, sp.compressible_corr);
  const size_t ci = (size_t)(L.block_offset + b) * BCELLS + x + BS * y + BS * BS * z;
  if (sgy < 1 || sgy > sp.ny_global) {
    const int km = mirror_y_of(k);
    return ST::load((const typename ST::T *)L.f_in, ci + (size_t)km * L.dstride, km,
                    L.inv_scale);
  }
  if (sgz < 1 || sgz > sp.nz_global) {
    const int km = mirror_z_of(k);
    return ST::load((const typename ST::T *)L.f_in, ci + (size_t)km * L.dstride, km,
                    L.inv_scale);
  }
  return w;
}

// ---------------------------------------------------------------------------
// WALE eddy viscosity from vel_in central differences
// (kernel_cumulant.jl:264-305, physics_utils.jl:85-123).
// ---------------------------------------------------------------------------
// Cell index of a face neighbour of the cell at local index `own` (element
// offset, own block at nbbase[13]) one step along an axis: inside the block
// `own + step`; across the face, the same cell of the face neighbour `dir`
// (`own + wrap - nbbase[13] + nbbase[dir]`); with no neighbour there, the cell
// itself (the zero-gradient fallback of physics_utils.jl:85-123).
__device__ __forceinline__ int vel_neighbor(const int *nbbase, int own, bool inside, int step,
                                            int dir, int wrap) {
  if (inside) return own + step;
  const int nb = nbbase[dir];
  return nb >= 0 ? own - nbbase[13] + nb + wrap : own;
}

// The 18 neighbour velocities the WALE gradients need (E, W, N, S, T, B
// neighbour, x/y/z component each), read from vel_in.
struct WaleVel {
  float e[3], w[3], n[3], s[3], t[3], b[3];
};

__device__ __forceinline__ void wale_load(const LevelDev &L, const int *nbbase, int x, int y, int z,
                                          WaleVel &V) {
  // the three velocity components are planes dstride apart
  const float *__restrict__ v0 = L.vel_in;
  const float *__restrict__ v1 = v0 + L.dstride;
  const float *__restrict__ v2 = v1 + L.dstride;
  const int own = nbbase[13] + x + BS * y + BS * BS * z;
  // E (x+1), W (x-1), N (y+1), S (y-1), T (z+1), B (z-1)
  const int ce = vel_neighbor(nbbase, own, x < BS - 1, 1, 14, -(BS - 1));
  const int cw = vel_neighbor(nbbase, own, x > 0, -1, 12, BS - 1);
  const int cn = vel_neighbor(nbbase, own, y < BS - 1, BS, 16, -BS * (BS - 1));
  const int cs = vel_neighbor(nbbase, own, y > 0, -BS, 10, BS * (BS - 1));
  const int ct = vel_neighbor(nbbase, own, z < BS - 1, BS * BS, 22, -BS * BS * (BS - 1));
  const int cb = vel_neighbor(nbbase, own, z > 0, -BS * BS, 4, BS * BS * (BS - 1));
  V.e[0] = __ldg(v0 + ce); V.e[1] = __ldg(v1 + ce); V.e[2] = __ldg(v2 + ce);
  V.w[0] = __ldg(v0 + cw); V.w[1] = __ldg(v1 + cw); V.w[2] = __ldg(v2 + cw);
  V.n[0] = __ldg(v0 + cn); V.n[1] = __ldg(v1 + cn); V.n[2] = __ldg(v2 + cn);
  V.s[0] = __ldg(v0 + cs); V.s[1] = __ldg(v1 + cs); V.s[2] = __ldg(v2 + cs);
  V.t[0] = __ldg(v0 + ct); V.t[1] = __ldg(v1 + ct); V.t[2] = __ldg(v2 + ct);
  V.b[0] = __ldg(v0 + cb); V.b[1] = __ldg(v1 + cb); V.b[2] = __ldg(v2 + cb);
}

__device__ __forceinline__ float wale_from(const WaleVel &V, float c_wale) {
  const float exx = V.e[0], eyx = V.e[1], ezx = V.e[2];
  const float wxx = V.w[0], wyx = V.w[1], wzx = V.w[2];
  const float nxx = V.n[0], nyx = V.n[1], nzx = V.n[2];
  const float sxx = V.s[0], syx = V.s[1], szx = V.s[2];
  const float txx = V.t[0], tyx = V.t[1], tzx = V.t[2];
  const float bxx = V.b[0], byx = V.b[1], bzx = V.b[2];
  const float g11 = 0.5f * (exx - wxx), g12 = 0.5f * (nxx - sxx), g13 = 0.5f * (txx - bxx);
  const float g21 = 0.5f * (eyx - wyx), g22 = 0.5f * (nyx - syx), g23 = 0.5f * (tyx - byx);
  const float g31 = 0.5f * (ezx - wzx), g32 = 0.5f * (nzx - szx), g33 = 0.5f * (tzx - bzx);

  const float gsq11 = g11 * g11 + g12 * g21 + g13 * g31;
  const float gsq12 = g11 * g12 + g12 * g22 + g13 * g32;
  const float gsq13 = g11 * g13 + g12 * g23 + g13 * g33;
  const float gsq21 = g21 * g11 + g22 * g21 + g23 * g31;
  const float gsq22 = g21 * g12 + g22 * g22 + g23 * g32;
  const float gsq23 = g21 * g13 + g22 * g23 + g23 * g33;
  const float gsq31 = g31 * g11 + g32 * g21 + g33 * g31;
  const float gsq32 = g31 * g12 + g32 * g22 + g33 * g32;
  const float gsq33 = g31 * g13 + g32 * g23 + g33 * g33;
  const float tr_term = third_of(gsq11 + gsq22 + gsq33);
  const float Sd11 = gsq11 - tr_term, Sd22 = gsq22 - tr_term, Sd33 = gsq33 - tr_term;
  const float Sd12 = 0.5f * (gsq12 + gsq21), Sd13 = 0.5f * (gsq13 + gsq31),
              Sd23 = 0.5f * (gsq23 + gsq32);
  const float S12 = 0.5f * (g12 + g21), S13 = 0.5f * (g13 + g31), S23 = 0.5f * (g23 + g32);
  const float OP1 = Sd11 * Sd11 + Sd22 * Sd22 + Sd33 * Sd33 +
                    2.0f * (Sd12 * Sd12 + Sd13 * Sd13 + Sd23 * Sd23);
  const float OP2 = g11 * g11 + g22 * g22 + g33 * g33 +
                    2.0f * (S12 * S12 + S13 * S13 + S23 * S23);
  // evaluated unconditionally (the floor keeps the roots defined) and selected:
  // a branch here would split the cell update's instruction schedule
  const float o1 = fmaxf(OP1, 1e-12f);
  const float r1 = sqrt_nr(o1);
  const float op2_52 = OP2 * OP2 * sqrt_nr(fmaxf(OP2, 1e-12f));
  const float den = op2_52 + o1 * sqrt_nr(r1);
  const float nu = (OP1 > 1e-12f && den > 1e-12f)
                       ? quotient_nr((c_wale * c_wale) * (o1 * r1), den) : 0.0f;
  return nu;
}

__device__ __forceinline__ float wale_nu(const LevelDev &L, const int *nbbase, int x, int y,
                                         int z) {
  WaleVel V;
  wale_load(L, nbbase, x, y, z, V);
  return wale_from(V, L.sp.c_wale);
}

// ---------------------------------------------------------------------------
// Wall-model force (kernel_cumulant.jl:220-250).  dist is in the units the
// wall-distance array carries (metres in the reference, domain_generation.jl:421).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void wall_force(float dist, float rho, float ux, float uy,
                                           float uz, float tau_mol, float &Fx, float &Fy,
                                           float &Fz) {
  Fx = Fy = Fz = 0.0f;
  if (!(dist > 0.0f && dist < 10.0f)) return;
  const float umag = sqrtf(ux * ux + uy * uy + uz * uz);
  const float nu = (tau_mol - 0.5f) / 3.0f;
  if (!(umag > 1e-6f && nu > 1e-10f)) return;
  float ut = umag * powf(nu / (dist * umag + 1e-10f), 1.0f / 7.0f) *
             powf(2.0f * 8.3f, -1.0f / 7.0f);
  ut = fmaxf(ut, 1e-6f);
  const float yp = ut * dist / nu;
  if (yp > 11.81f) {
    const float uplus = (1.0f / 0.41f) * logf(yp) + 5.2f;
    if (uplus > 0.1f) {
      ut = ut * ((umag / ut) / uplus);
      ut = fmaxf(ut, 1e-6f);
    }
  }
  const float tw = rho * ut * ut;
  const float tr = rho * nu * (umag / dist);
  if (tw > tr) {
    const float fm = (tw - tr) / dist;
    Fx = -fm * ux / umag;
    Fy = -fm * uy / umag;
    Fz = -fm * uz / umag;
  }
}

// ---------------------------------------------------------------------------
// Chimera transforms (kernel_cumulant.jl:4-26) and the cumulant collision
// (kernel_cumulant.jl:330-559).  A holds populations on entry and on exit.
//
// The cell update is bound by instruction issue and by the latency of its
// dependent chains, not by memory, so it is written for few instructions and
// straight-line code:
//   * the raw x-moments are formed first, in place; rho and the momentum are
//     sums over them (26 additions instead of 78) and the first transform
//     continues from them;
//   * a triple's zeroth moment reuses its second (m0 = b + m2);
//   * reciprocals, quotients and roots are the branch-free forms below
//     instead of calls with a slow path, so the scheduler sees one block;
//   * with omega_3 = omega_4 = 1 (the reference's defaults) every third-order
//     moment and every C_211 kind is relaxed to exactly zero, so its forward
//     transform, the fifth-order products and the zero terms of the backward
//     transform are left out (collide_cumulant<true, ...>).
//
// SUMS: the order and rounding of the sums.  kSumsShort is the form above.  The
// block pool takes the order of the written formulas -- rho and the momentum
// over the 27 populations in turn, a triple's zeroth moment as (a + b) + c, a
// product that two terms share rounded on its own -- about 80 additions a cell
// more.  Its force coefficients are read from the first hundred steps on, while
// the start's pressure wave still swings the drag through zero; there another
// rounding of any one term shows at up to 1e-3 of the coefficient vector (5e-3
// with FP16 storage), so a pool's records compare between builds only where the
// update rounds alike.  kSumsPool and kSumsPoolWs (k_sc_ws) differ in one place:
// the latter forms u_z^2 rho once, rounded, for both transforms along z.  What
// is fused is written out (fmaf, __fmul_rn), so that no compiler's choice
// enters.  A pool of one cube_3lvl case, us per coarse step: 1162, with kSumsShort
// 1148 (FP16 storage 1411 and 1386; with omega_3 = 0.9, FP32 1198 and 1191).
// ---------------------------------------------------------------------------
constexpr int kSumsShort = 0, kSumsPool = 1, kSumsPoolWs = 2;
// The block pool's form (regularized BGK has one form only).
constexpr int pool_sums(int op, bool ws = false) {
  return op != OL_OP_CUMULANT ? kSumsShort : ws ? kSumsPoolWs : kSumsPool;
}
template <int SUMS>
__device__ __forceinline__ void raw_moments(float &a, float &b, float &c) {
  const float m2 = a + c, m1 = c - a;
  a = SUMS != kSumsShort ? (a + b) + c : b + m2;
  b = m1;
  c = m2;
}
// Raw moments (m0, m1, m2) of a triple -> central ones about u.
__device__ __forceinline__ void centre(float m0, float &b, float &c, float u) {
  const float m1 = b;
  b = fmaf(-u, m0, m1);
  c = fmaf(u * u, m0, fmaf(-2.0f * u, m1, c));
}
template <int SUMS>
__device__ __forceinline__ void chim_fwd(float &a, float &b, float &c, float u) {
  raw_moments<SUMS>(a, b, c);
  centre(a, b, c, u);
}
// (m2 +- m1) / 2 as fma(+-1/2, m1, m2 / 2): the same bits (halving is exact
// at these magnitudes, so both round the same exact value once), one
// instruction fewer.
__device__ __forceinline__ void chim_bwd_from(float &a, float &b, float &c, float m0, float m1,
                                              float m2) {
  const float h = 0.5f * m2;
  c = fmaf(0.5f, m1, h);
  a = fmaf(-0.5f, m1, h);
  b = __fsub_rn(m0, m2);
}
__device__ __forceinline__ void chim_bwd(float &a, float &b, float &c, float u) {
  chim_bwd_from(a, b, c, a, fmaf(u, a, b), fmaf(u * u, a, fmaf(2.0f * u, b, c)));
}
// The same with the second moment given as a factor of r ...
__device__ __forceinline__ void chim_bwd_r(float &a, float &b, float &c, float u, float r) {
  const float m2 = fmaf(u * u, a, fmaf(r, c, __fmul_rn(2.0f * u, b)));
  chim_bwd_from(a, b, c, a, fmaf(u, a, b), m2);
}
// ... for a zero first moment ...
__device__ __forceinline__ void chim_bwd_b0(float &a, float &b, float &c, float u) {
  chim_bwd_from(a, b, c, a, u * a, fmaf(u * u, a, c));
}
// ... for the line of rho with u^2 rho rounded (kSumsPoolWs; forward, its first
// moment is not used) ...
__device__ __forceinline__ void chim_fwd_rho(float &a, float &b, float &c, float u) {
  raw_moments<kSumsPoolWs>(a, b, c);
  c = __fadd_rn(fmaf(-2.0f * u, b, c), __fmul_rn(u * u, a));
}
__device__ __forceinline__ void chim_bwd_rho(float &a, float &b, float &c, float u) {
  chim_bwd_from(a, b, c, a, u * a, __fadd_rn(c, __fmul_rn(u * u, a)));
}
// ... and for a triple that holds a first moment only.
__device__ __forceinline__ void chim_bwd_b(float &a, float &b, float &c, float u) {
  const float m1 = b, h = u * b;
  c = fmaf(0.5f, m1, h);
  a = fmaf(-0.5f, m1, h);
  b = -2.0f * h;
}

struct CumulantRates {
  float omega1, omega_bulk, omega3, omega4, omega4_diag;
  int limiter;
};

// A holds raw x-moments on entry (raw_moments over the consecutive triples)
// and populations on exit.  LOW: omega3 == omega4 == 1.
template <bool LOW, int SUMS>
__device__ __forceinline__ void collide_cumulant(float (&A)[27], float ux, float uy, float uz,
                                                 const CumulantRates &r) {
  // forward: x (consecutive triples), then y (stride 3), then z (stride 9)
#pragma unroll
  for (int i = 0; i < 9; ++i) centre(A[3 * i], A[3 * i + 1], A[3 * i + 2], ux);
#pragma unroll
  for (int zz = 0; zz < 3; ++zz)
#pragma unroll
    for (int a = 0; a < 3; ++a)
      chim_fwd<SUMS>(A[a + 9 * zz], A[a + 3 + 9 * zz], A[a + 6 + 9 * zz], uy);
  if constexpr (SUMS == kSumsPoolWs) chim_fwd_rho(A[0], A[9], A[18], uz);
  else chim_fwd<SUMS>(A[0], A[9], A[18], uz);
#pragma unroll
  for (int i = 1; i < 9; ++i) chim_fwd<SUMS>(A[i], A[i + 9], A[i + 18], uz);

  const float k000 = A[0];
  const float inv_r = recip_nr(fmaxf(k000, 0.01f));
  // index of central moment (a,b,c) = a + 3b + 9c
  auto central = [&](float k) { return __fmul_rn(k, inv_r); };
  const float c200 = central(A[2]), c020 = central(A[6]), c002 = central(A[18]);
  const float c110 = central(A[4]), c101 = central(A[10]), c011 = central(A[12]);
  // cumulant C of a fourth-order moment k: k / r - p q - 2 s t
  auto cumulant = [&](float k, float p, float q, float s, float t) {
    return fmaf(-2.0f * s, t, fmaf(k, inv_r, -__fmul_rn(p, q)));
  };
  const float C220 = cumulant(A[8], c200, c020, c110, c110);
  const float C202 = cumulant(A[20], c200, c002, c101, c101);
  const float C022 = cumulant(A[24], c020, c002, c011, c011);

  const float cs2 = 0.333333333f;
  const float om1 = r.omega1, omb = r.omega_bulk;
  const float Dtr = c200 + c020 + c002;
  const float Dtr_s = fmaf(1.0f - omb, Dtr, omb * (3.0f * cs2));
  const float D1s = __fmul_rn(1.0f - om1, c200 - c020);
  const float D2s = __fmul_rn(1.0f - om1, c200 - c002);
  const float c200s = third_of(Dtr_s + D1s + D2s);
  const float c020s = third_of(Dtr_s - 2.0f * D1s + D2s);
  const float c002s = third_of(Dtr_s + D1s - 2.0f * D2s);
  float c110s = (1.0f - om1) * c110;
  float c101s = (1.0f - om1) * c101;
  float c011s = (1.0f - om1) * c011;
  if (r.limiter == OL_LIMITER_FACTORED) {
    auto root = [](float v) { return v > 1e-30f ? sqrt_nr(v) : 0.0f; };
    const float b110 = root(c200s * c020s);
    const float b101 = root(c200s * c002s);
    const float b011 = root(c020s * c002s);
    c110s = fminf(fmaxf(c110s, -b110), b110);
    c101s = fminf(fmaxf(c101s, -b101), b101);
    c011s = fminf(fmaxf(c011s, -b011), b011);
  }
  const float o4d = 1.0f - r.omega4_diag;
  const float C220s = __fmul_rn(o4d, C220), C202s = __fmul_rn(o4d, C202),
              C022s = __fmul_rn(o4d, C022);
  const float rr = k000;
  if constexpr (LOW && SUMS == kSumsShort) {
    // e = C + 2 c^2 of each pair; t = 2 c110 c101 is shared by 211 and 222
    const float e220 = fmaf(2.0f * c110s, c110s, C220s);
    const float e202 = fmaf(2.0f * c101s, c101s, C202s);
    const float e022 = fmaf(2.0f * c011s, c011s, C022s);
    const float c220s = fmaf(c200s, c020s, e220);
    const float c202s = fmaf(c200s, c002s, e202);
    const float c022s = fmaf(c020s, c002s, e022);
    const float t = 2.0f * c110s * c101s;
    const float c211s = fmaf(c200s, c011s, t);
    const float c121s = fmaf(c020s, c101s, 2.0f * c110s * c011s);
    const float c112s = fmaf(c002s, c110s, 2.0f * c101s * c011s);
    const float c222s =
        fmaf(c002s, c220s, fmaf(c200s, e022, fmaf(c020s, e202, 4.0f * t * c011s)));
    A[8] = rr * c220s; A[20] = rr * c202s; A[24] = rr * c022s;
    A[14] = rr * c211s; A[16] = rr * c121s; A[22] = rr * c112s;
    A[26] = rr * c222s;
  } else {
    const float p = __fmul_rn(c200s, c020s), x = __fmul_rn(c200s, c011s),
                y = __fmul_rn(c020s, c101s), z = __fmul_rn(c002s, c110s);
    const float c220s = fmaf(2.0f * c110s, c110s, __fadd_rn(C220s, p));
    const float c202s = fmaf(2.0f * c101s, c101s, fmaf(c200s, c002s, C202s));
    const float c022s = fmaf(2.0f * c011s, c011s, fmaf(c020s, c002s, C022s));
    float c211s = x, c121s = y, c112s = z;
    // 222: the terms in C, those in third-order moments, the rest
    float c222s = fmaf(c002s, C220s, fmaf(c020s, C202s, __fmul_rn(c200s, C022s)));
    const float q = fmaf(z, c110s, fmaf(y, c101s, __fmul_rn(x, c011s)));
    const float rest = fmaf(__fmul_rn(8.0f * c110s, c101s), c011s, fmaf(p, c002s, 2.0f * q));
    if constexpr (!LOW) {
      const float o3 = 1.0f - r.omega3, o4 = 1.0f - r.omega4;
      auto third_order = [&](float k) { return __fmul_rn(o3, central(k)); };
      const float c210s = third_order(A[5]), c120s = third_order(A[7]);
      const float c201s = third_order(A[11]), c021s = third_order(A[15]);
      const float c102s = third_order(A[19]), c012s = third_order(A[21]);
      const float c111s = third_order(A[13]);
      const float C211s = __fmul_rn(o4, cumulant(A[14], c200, c011, c110, c101));
      const float C121s = __fmul_rn(o4, cumulant(A[16], c020, c101, c110, c011));
      const float C112s = __fmul_rn(o4, cumulant(A[22], c002, c110, c101, c011));
      c211s = __fadd_rn(C211s, c211s);
      c121s = __fadd_rn(C121s, c121s);
      c112s = __fadd_rn(C112s, c112s);
      const float c221s =
          fmaf(2.0f * c011s, c210s,
               fmaf(2.0f * c101s, c120s,
                    fmaf(4.0f * c110s, c111s, fmaf(c020s, c201s, __fmul_rn(c200s, c021s)))));
      const float c212s =
          fmaf(2.0f * c011s, c201s,
               fmaf(4.0f * c101s, c111s,
                    fmaf(2.0f * c110s, c102s, fmaf(c002s, c210s, __fmul_rn(c200s, c012s)))));
      const float c122s =
          fmaf(2.0f * c101s, c021s,
               fmaf(4.0f * c011s, c111s,
                    fmaf(2.0f * c110s, c012s, fmaf(c002s, c120s, __fmul_rn(c020s, c102s)))));
      c222s = fmaf(4.0f, fmaf(c011s, C211s, fmaf(c110s, C112s, __fmul_rn(c101s, C121s))), c222s);
      const float t = fmaf(c120s, c102s, fmaf(c201s, c021s, __fmul_rn(c210s, c012s)));
      c222s = __fadd_rn(c222s, fmaf(4.0f * c111s, c111s, 2.0f * t));
      A[5] = rr * c210s; A[7] = rr * c120s; A[11] = rr * c201s; A[15] = rr * c021s;
      A[13] = rr * c111s;
      A[17] = rr * c221s;
      A[19] = c102s; A[21] = c012s; A[23] = c212s; A[25] = c122s;  // (chim_bwd_r)
    }
    c211s = fmaf(2.0f * c110s, c101s, c211s);
    c121s = fmaf(2.0f * c110s, c011s, c121s);
    c112s = fmaf(2.0f * c101s, c011s, c112s);
    c222s = __fadd_rn(c222s, rest);
    const float s = LOW ? rr : 1.0f;
    A[8] = rr * c220s; A[14] = rr * c211s; A[16] = rr * c121s;
    A[20] = s * c202s; A[22] = s * c112s; A[24] = s * c022s; A[26] = s * c222s;
  }
  A[0] = rr;
  A[2] = rr * c200s; A[6] = rr * c020s; A[18] = rr * c002s;
  A[4] = rr * c110s; A[10] = rr * c101s; A[12] = rr * c011s;
  // backward z: (a, b) lines
  if constexpr (SUMS == kSumsPoolWs) chim_bwd_rho(A[0], A[9], A[18], uz);
  else chim_bwd_b0(A[0], A[9], A[18], uz);
  if constexpr (LOW) {  // odd total order is zero
    chim_bwd_b0(A[2], A[11], A[20], uz);
    chim_bwd_b0(A[4], A[13], A[22], uz);
    chim_bwd_b0(A[6], A[15], A[24], uz);
    chim_bwd_b0(A[8], A[17], A[26], uz);
    chim_bwd_b(A[1], A[10], A[19], uz);
    chim_bwd_b(A[3], A[12], A[21], uz);
    chim_bwd_b(A[5], A[14], A[23], uz);
    chim_bwd_b(A[7], A[16], A[25], uz);
  } else {
    A[1] = 0.0f; A[3] = 0.0f;
#pragma unroll
    for (int i = 1; i < 9; ++i) chim_bwd_r(A[i], A[i + 9], A[i + 18], uz, rr);
  }
  // backward y, then x
#pragma unroll
  for (int zz = 0; zz < 3; ++zz)
#pragma unroll
    for (int a = 0; a < 3; ++a)
      chim_bwd(A[a + 9 * zz], A[a + 3 + 9 * zz], A[a + 6 + 9 * zz], uy);
#pragma unroll
  for (int i = 0; i < 9; ++i) chim_bwd(A[3 * i], A[3 * i + 1], A[3 * i + 2], ux);
}

// ---------------------------------------------------------------------------
// Regularized BGK (kernel_regularized_bgk.jl:270-300).  A holds raw x-moments
// on entry and populations on exit.  The second moments of the
// non-equilibrium are those of the populations minus the equilibrium's, which
// are polynomials in u on this lattice (c_a in {-1, 0, 1}): rho (1/3 + u_a^2)
// and rho u_a u_b for O(u^2); the O(u^4) terms add -3/4 rho u_a^4 on the
// diagonal and nothing off it.  So the 27 equilibria are needed once instead
// of twice, and each is the even part of its direction pair plus or minus the
// odd one: 13 pairs instead of 54 evaluations, and the populations are dead
// before the first is formed (the kernel fits the warp-specialised form's 96
// registers).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void bgk_regularized(float (&A)[27], float rho, float ux, float uy,
                                                float uz, float om1, int comp) {
  // sum_k f_k c_a c_b from the x-moments: rows i = (c_y + 1) + 3 (c_z + 1)
  const float Sxx = (A[2] + A[5] + A[8]) + (A[11] + A[14] + A[17]) + (A[20] + A[23] + A[26]);
  const float Syy = (A[0] + A[6]) + (A[9] + A[15]) + (A[18] + A[24]);
  const float Szz = (A[0] + A[3] + A[6]) + (A[18] + A[21] + A[24]);
  const float Sxy = (A[7] - A[1]) + (A[16] - A[10]) + (A[25] - A[19]);
  const float Szx = (A[19] + A[22] + A[25]) - (A[1] + A[4] + A[7]);
  const float Syz = (A[0] - A[6]) + (A[24] - A[18]);
  const float xx = ux * ux, yy = uy * uy, zz = uz * uz, usq = xx + yy + zz;
  const float a4 = comp ? -0.75f : 0.0f;
  const float r3 = third_of(rho);
  const float g = 4.5f * om1, g2 = 9.0f * om1;
  const float qxx = g * (Sxx - fmaf(rho, fmaf(a4 * xx, xx, xx), r3));
  const float qyy = g * (Syy - fmaf(rho, fmaf(a4 * yy, yy, yy), r3));
  const float qzz = g * (Szz - fmaf(rho, fmaf(a4 * zz, zz, zz), r3));
  const float qxy = g2 * (Sxy - rho * ux * uy);
  const float qyz = g2 * (Syz - rho * uy * uz);
  const float qzx = g2 * (Szx - rho * uz * ux);
  const float tr = third_of(qxx + qyy + qzz);
  // even part w (base + cu^2 (e2 + e4 cu^2) + q), odd part w cu (o1 + o3 cu^2)
  const float base = rho * (comp ? fmaf(usq, fmaf(1.125f, usq, -1.5f), 1.0f)
                                 : fmaf(-1.5f, usq, 1.0f)) - tr;
  const float e2 = rho * (comp ? fmaf(-6.75f, usq, 4.5f) : 4.5f), e4 = comp ? 3.375f * rho : 0.0f;
  const float o1 = rho * (comp ? fmaf(-4.5f, usq, 3.0f) : 3.0f), o3 = comp ? 4.5f * rho : 0.0f;
  A[13] = w_of(13) * base;
#pragma unroll
  for (int k = 14; k < 27; ++k) {
    const int cx = cx_of(k), cy = cy_of(k), cz = cz_of(k);
    float cu = 0.0f, q = base;
    if (cx) { cu = cx > 0 ? ux : -ux; q += qxx; }
    if (cy) { cu = cy > 0 ? cu + uy : cu - uy; q += qyy; }
    if (cz) { cu = cz > 0 ? cu + uz : cu - uz; q += qzz; }
    if (cx * cy) q = cx * cy > 0 ? q + qxy : q - qxy;
    if (cy * cz) q = cy * cz > 0 ? q + qyz : q - qyz;
    if (cz * cx) q = cz * cx > 0 ? q + qzx : q - qzx;
    const float c2 = cu * cu;
    const float even = fmaf(c2, fmaf(e4, c2, e2), q), odd = cu * fmaf(o3, c2, o1);
    A[k] = w_of(k) * (even + odd);
    A[26 - k] = w_of(k) * (even - odd);
  }
}

// Positivity limiter (kernel_cumulant.jl:564-599).
__device__ __forceinline__ void positivity_limit(float (&A)[27], float rho, float ux, float uy,
                                              float uz, int comp) {
  float alpha = 1.0f;
#pragma unroll
  for (int k = 0; k < 27; ++k) {
    const float fe = feq_auto(rho, ux, uy, uz, w_of(k), (float)cx_of(k), (float)cy_of(k),
                              (float)cz_of(k), comp);
    const float fn = A[k] - fe;
    if (fn < 0.0f && fe > 1e-15f) alpha = fminf(alpha, fe / (fe - fn + 1e-15f));
  }
  alpha = fmaxf(alpha, 0.0f);
#pragma unroll
  for (int k = 0; k < 27; ++k) {
    const float fe = feq_auto(rho, ux, uy, uz, w_of(k), (float)cx_of(k), (float)cy_of(k),
                              (float)cz_of(k), comp);
    A[k] = fe + alpha * (A[k] - fe);
  }
}

// ---------------------------------------------------------------------------
// One cell of one block.  OP = OL_OP_*; WALE = gradients evaluated (c_wale
// != 0; with c_wale == 0 the reference's nu_eddy is exactly 0).
// ---------------------------------------------------------------------------
// ---------------------------------------------------------------------------
// Shared-memory staging of a block's 27 pull windows.
//
// E holds one halo-extended 10^3 plane per direction (E[k*1000 + (x+1) +
// 10(y+1) + 100(z+1)] for x, y, z in -1..8), so the pull of cell (x, y, z)
// in direction k is a single shared load at a compile-time offset from the
// cell's base.  The own block's 27 planes are copied with 16-byte loads; the
// 3176 out-of-block sources of the block (the slab each direction needs
// from its up to 7 neighbours) come from a per-device table of packed
// (k, neighbour direction, source cell, destination slot) entries; sources
// whose neighbour block is absent get their boundary value (inlet/outlet
// equilibrium, free-slip mirror, parent interpolation) right there.
// nbbase[dir] = element offset of neighbour `dir` within a direction plane,
// or -1 when it is absent.
// ---------------------------------------------------------------------------
constexpr int EPL = 1000;                 // floats per staged direction plane
constexpr int kStageBytes = 27 * EPL * 4;  // dynamic shared memory per CTA
constexpr int kHaloEntries = 3176;

__host__ __device__ constexpr int e_index(int x, int y, int z) {
  return (x + 1) + 10 * (y + 1) + 100 * (z + 1);
}

// Boundary values of the staging slots whose neighbour block is absent.  One
// call per thread, made only by CTAs whose block has an absent neighbour, so
// the call and its register save/restore stay off the bulk path.
template <class BC>
__device__ __noinline__ void fill_missing_slots(const int *nbbase, int t, float *E,
                                                const uint32_t *__restrict__ tab, BC bc) {
  for (int i = t; i < kHaloEntries; i += BCELLS) {
    const uint32_t te = __ldg(tab + i);
    const int k = te & 31, dir = (te >> 5) & 31, dst = te >> 19;
    if (nbbase[dir] >= 0) continue;
    const int sx = dst % 10 - 1, sy = (dst / 10) % 10 - 1, sz = dst / 100 - 1;
    E[k * EPL + dst] = bc(k, sx + cx_of(k), sy + cy_of(k), sz + cz_of(k));
  }
}

// Ring positions of the staging plane (the 488 slots of the 10^3 plane
// outside the 8^3 block), listed in the staging table after its halo entries.
constexpr int kRingEntries = 1000 - 512;
// Staging table layout: kHaloEntries packed entries, the kRingEntries ring
// slots of the 10^3 plane, then per halo entry the ring index of its slot.
constexpr int kRingIndexOffset = kHaloEntries + kRingEntries;
constexpr int kHaloTableSize = kRingIndexOffset + kHaloEntries;

// Staging planes whose slot p is never read, for a ring position p with
// outward offsets (ox, oy, oz): a direction k with c_a = o_a on the first
// axis a where o_a != 0 would pull slot p into a cell at -2 or 9 on that
// axis, outside the block.  Four of these (i = 0..3) hold the interpolated
// rho, ux, uy, uz of an interface position between the two fill phases.
__device__ __forceinline__ int stash_plane(int ox, int oy, int oz, int i) {
  const int u = (i & 1) + 1, v = (i >> 1) + 1;
  if (ox != 0) return (ox + 1) + 3 * u + 9 * v;
  if (oy != 0) return u + 3 * (oy + 1) + 9 * v;
  return u + 3 * v + 9 * (oz + 1);
}

// Boundary values of the flow staging slots whose neighbour block is absent.
// Domain boundaries (inlet, outlet, free-slip mirrors) and level-1 gaps are
// evaluated per slot by pull_boundary.  A fine-level interface slot needs the
// parent's rho and u interpolated at its source position, which every
// direction pulling from that position shares: phase 1 computes them once
// per ring position (one thread each) into stash slots, phase 2 spreads the
// (direction, slot) entries over all threads and interpolates only f_k.
template <class ST>
__device__ __noinline__ void fill_missing_flow(const LevelDev &L, const int *nbbase, int b, int t,
                                               float *E) {
  const ol_step_params &sp = L.sp;
  const uint32_t *__restrict__ tab = L.halo_tab;
  const bool fine = sp.is_level_1 == 0;
  const int gx0 = (L.map_x[b] - 1) * BS + 1, gy0 = (L.map_y[b] - 1) * BS + 1,
            gz0 = (L.map_z[b] - 1) * BS + 1;
  if (fine) {
    if (t < kRingEntries) {
      const int p = (int)__ldg(tab + kHaloEntries + t);
      const int sx = p % 10 - 1, sy = (p / 10) % 10 - 1, sz = p / 100 - 1;
      const int ox = sx < 0 ? -1 : (sx > 7 ? 1 : 0);
      const int oy = sy < 0 ? -1 : (sy > 7 ? 1 : 0);
      const int oz = sz < 0 ? -1 : (sz > 7 ? 1 : 0);
      const int sgx = gx0 + sx, sgy = gy0 + sy, sgz = gz0 + sz;
      if (nbbase[(ox + 1) + 3 * (oy + 1) + 9 * (oz + 1)] < 0 && sgx >= 1 &&
          sgx <= sp.nx_global && sgy >= 1 && sgy <= sp.ny_global && sgz >= 1 &&
          sgz <= sp.nz_global) {
        ParentStencil P;
        parent_stencil(L, sgx, sgy, sgz, P);
        float r[4];
        interp_moments(L, P, sp.temporal_weight, r);
#pragma unroll
        for (int i = 0; i < 4; ++i) E[stash_plane(ox, oy, oz, i) * EPL + p] = r[i];
      }
    }
    __syncthreads();
  }
  for (int i = t; i < kHaloEntries; i += BCELLS) {
    const uint32_t te = __ldg(tab + i);
    const int k = te & 31, dir = (te >> 5) & 31, p = te >> 19;
    if (nbbase[dir] >= 0) continue;
    const int sx = p % 10 - 1, sy = (p / 10) % 10 - 1, sz = p / 100 - 1;
    const int sgx = gx0 + sx, sgy = gy0 + sy, sgz = gz0 + sz;
    float v;
    if (fine && sgx >= 1 && sgx <= sp.nx_global && sgy >= 1 && sgy <= sp.ny_global &&
        sgz >= 1 && sgz <= sp.nz_global) {
      const int ox = sx < 0 ? -1 : (sx > 7 ? 1 : 0);
      const int oy = sy < 0 ? -1 : (sy > 7 ? 1 : 0);
      const int oz = sz < 0 ? -1 : (sz > 7 ? 1 : 0);
      float r[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) r[j] = E[stash_plane(ox, oy, oz, j) * EPL + p];
      ParentStencil P;
      parent_stencil(L, sgx, sgy, sgz, P);
      v = interp_population<ST>(L, k, P, r, sp.temporal_weight);
    } else {
      v = pull_boundary<ST>(L, k, b, sx + cx_of(k), sy + cy_of(k), sz + cz_of(k));
    }
    E[k * EPL + p] = v;
  }
}

// Separate pass over the blocks of a level: the absent-neighbour pull sources
// of block b, in staging-table order, into L.ghost[b * kHaloEntries + i].
// Same values as fill_missing_flow, from fewer gathers.  Fine cells 2m+1 and
// 2m+2 of an axis interpolate between the same parent cells m and m+1, so the
// 488 ring positions of a block fall into 152 groups (up to 2 x 2 positions)
// that share their 8 parent cells.  The unit of work is one direction of one
// group -- 1016 units for the 3176 slots -- and reads the 8 parent values
// once for its up to 4 slots (and both sub-steps of a pair).  A fine block
// touches at most 2 parent blocks per axis, so its 8 parent block ids are read
// once, next to the neighbour row, and a stencil costs no table lookups.
// The pass waits on gathers: per block there are three dependent round trips
// (neighbour row, moments, populations) instead of a stencil chain per
// position, and a third of the population gathers.  Measured per coarse step:
// cube_3lvl (3 passes) 193 -> 119 us, the two passes of sphere_ddf 58 + 58 ->
// 36 + 35 us; 256 threads at 4 CTAs per SM beat 3 CTAs with 80 registers (134)
// and 128 threads at 6 CTAs (139) in spite of a few spilled words.
constexpr int kGhostThreads = 256;
constexpr int kGhostMinBlocks = 4;  // resident CTAs per SM (64 registers per thread)
constexpr int kGhostGroups = 152, kGhostUnits = 1016;
constexpr int kGhostScan = (kGhostUnits + kGhostThreads - 1) / kGhostThreads;  // 4
// Unit table: per unit one uint4 {k | group << 5 | code << 13 | direction << 21,
// slots of positions 0 and 1, slots of positions 2 and 3 (16 bits each, 0xFFFF:
// none), 0}, sorted by direction (faces, edges, corners), then per group one
// word code | direction << 8.
constexpr int kGhostNoSlot = 0xFFFF;
constexpr int kGhostTableWords = 4 * kGhostUnits + kGhostGroups;
// Group code: pair indices p (0..5 per axis, x fastest) of positions -1 |
// 0,1 | 2,3 | 4,5 | 6,7 | 8.  Position `sub` of a group: its bits pick the
// member on the axes that have two, x first.  Returns the position's
// coordinate and trilinear weight along one axis and consumes a bit of sub.
__device__ __forceinline__ int ghost_member(int p, int &sub, float &w) {
  if (p == 0) { w = 0.75f; return -1; }
  if (p == 5) { w = 0.25f; return 8; }
  const int bit = sub & 1;
  sub >>= 1;
  w = bit ? 0.75f : 0.25f;
  return 2 * p - 2 + bit;
}

// Warp-aggregated append of `value` to a shared list when `flag` is set;
// every lane of the warp makes the call.
__device__ __forceinline__ void append_if(bool flag, int value, int *count, int16_t *list) {
  const unsigned m = __ballot_sync(0xffffffffu, flag);
  if (m == 0) return;
  const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(count, __popc(m));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (flag) list[base + __popc(m & ((1u << lane) - 1u))] = (int16_t)value;
}

// Row of block b in the ghost scratch of level L (null when the block has
// no row: no scratch, or no absent neighbour under a compact index).  DEV is
// the flow (LevelDev) or thermal (ThermalDev) level.
template <class DEV>
__device__ __forceinline__ float *ghost_row_of(const DEV &L, int b) {
  if (!L.ghost) return nullptr;
  const int r = L.gidx ? L.gidx[b] : b;
  return r >= 0 ? L.ghost + (size_t)r * kHaloEntries : nullptr;
}
// The same row of ghost_next (written by the first sub-step of a pair).
template <class DEV>
__device__ __forceinline__ float *ghost_next_row_of(const DEV &L, int b) {
  if (L.ghost_mode != kGhostPairFirst || !L.ghost_next) return nullptr;
  const int r = L.gidx ? L.gidx[b] : b;
  return r >= 0 ? L.ghost_next + (size_t)r * kHaloEntries : nullptr;
}

// What the ghost pass needs to know of a flow level; the thermal DDF
// provides the same functions for its populations (thermal.cuh).
__device__ __forceinline__ const ol_step_params &ghost_params(const LevelDev &L) { return L.sp; }
// Parent planes of moment m (0: rho, 1..3: u) and of population k, new and old.
__device__ __forceinline__ const float *ghost_moment_plane(const LevelDev &L, int m, bool old) {
  if (m == 0) return old ? L.prho_old : L.prho;
  return (old ? L.pvel_old : L.pvel) + (size_t)(m - 1) * L.p_dstride;
}
__device__ __forceinline__ const void *ghost_parent(const LevelDev &L, bool old) {
  return old ? L.pf_old : L.pf;
}
__device__ __forceinline__ float ghost_finish(const LevelDev &, const GhostScale &g, int k,
                                              const float (&v)[8], float wx, float wy, float wz,
                                              const float (&r)[4]) {
  return finish_population(g, k, v, wx, wy, wz, r);
}
__device__ __forceinline__ void ghost_moments(const LevelDev &L, const ParentStencil &P, float tw,
                                              float (&r)[4]) {
  interp_moments(L, P, tw, r);
}
template <class ST>
__device__ __forceinline__ float ghost_population(const LevelDev &L, int k, const ParentStencil &P,
                                                  const float (&r)[4], float tw, ST) {
  return interp_population<ST>(L, k, P, r, tw);
}
template <class ST>
__device__ __forceinline__ float ghost_boundary(const LevelDev &L, int k, int b, int x, int y,
                                                int z, ST) {
  return pull_boundary<ST>(L, k, b, x, y, z);
}

// A slot of a block that lies partly outside the domain (sizes that are no
// multiple of 8) but is itself inside it: interpolated on its own.
template <class ST, class DEV>
__device__ __noinline__ float ghost_slot(const DEV &L, int k, int gx, int gy, int gz, float tw) {
  ParentStencil P;
  parent_stencil(L, gx, gy, gz, P);
  float r[4];
  ghost_moments(L, P, tw, r);
  return ghost_population(L, k, P, r, tw, ST{});
}

// One CTA of kGhostThreads threads evaluates block b's row G.  With
// L.ghost_mode == kGhostPairFirst it also writes into G2 the coarse-to-fine
// slots of the pair's second sub-step (the parent does not step in between),
// reading each parent value once for both; with kGhostPairSecond those slots
// of G are already set and only the domain-boundary slots are evaluated.
template <class ST, class DEV>
__device__ __forceinline__ void ghost_fill_block(const DEV &L, int b, float *G, float *G2) {
  using T = typename ST::T;
  __shared__ int8_t kind[27];      // by direction: 0 nothing to do, 1 interpolate, 2 per slot
  __shared__ int32_t pbase[8];     // first cell of the 2 x 2 x 2 parent blocks, -1 absent
  __shared__ int n_unit;
  __shared__ int16_t unit_list[kGhostUnits];
  __shared__ float rs[4][4 * kGhostGroups];   // rho, ux, uy, uz per group position
  __shared__ float rs2[4][4 * kGhostGroups];  // the same at the second sub-step's weight
  const int t = threadIdx.x;
  const auto &sp = ghost_params(L);
  const bool precomputed = L.ghost_mode == kGhostPairSecond;
  const bool fine = sp.is_level_1 == 0;
  const int mx = L.map_x[b], my = L.map_y[b], mz = L.map_z[b];
  // lowest parent cell (1-based) of the block's stencils per axis and its block
  const int lx = 4 * (mx - 1) - 1, ly = 4 * (my - 1) - 1, lz = 4 * (mz - 1) - 1;
  const int bx0 = (max(lx, 1) - 1) / BS, by0 = (max(ly, 1) - 1) / BS, bz0 = (max(lz, 1) - 1) / BS;
  int work = 0;
  if (t < 27) {
    int kd = 0;
    if (t != 13 && L.nbr[b + L.nbr_stride * t] <= 0) {
      const int nbx = mx + t % 3 - 1, nby = my + (t / 3) % 3 - 1, nbz = mz + t / 9 - 1;
      const bool inside = nbx >= 1 && nbx * BS <= sp.nx_global && nby >= 1 &&
                          nby * BS <= sp.ny_global && nbz >= 1 && nbz * BS <= sp.nz_global;
      // the second sub-step of a pair finds its coarse-to-fine values set
      kd = fine && inside ? (precomputed ? 0 : 1) : 2;
    }
    kind[t] = (int8_t)kd;
    work = kd != 0;
  } else if (fine && t >= 32 && t < 40) {
    const int s = t - 32;
    const int px = bx0 + (s & 1), py = by0 + ((s >> 1) & 1), pz = bz0 + (s >> 2);
    int pb = 0;
    if (px < L.pdim_x && py < L.pdim_y && pz < L.pdim_z)
      pb = L.pptr[px + L.pdim_x * (py + L.pdim_y * pz)];
    pbase[s] = pb > 0 ? (int32_t)((L.p_block_offset + pb - 1) * BCELLS) : -1;
  } else if (t == 64) {
    n_unit = 0;
  }
  // (the descriptor may lie in shared memory: what the stores below must not
  // make the compiler read again is copied)
  const uint32_t *__restrict__ tab = L.ghost_units;
  const GhostScale rescale = ghost_scale(L);
  const T *const par_old = (const T *)ghost_parent(L, true);
  const T *const par_new = (const T *)ghost_parent(L, false);
  const int64_t p_dstride = L.p_dstride;
  const float p_inv_scale = L.p_inv_scale;
  uint32_t head[kGhostScan];
#pragma unroll
  for (int j = 0; j < kGhostScan; ++j) {
    const int u = t + j * kGhostThreads;
    head[j] = u < kGhostUnits ? __ldg(tab + 4 * u) : 13u << 21;
  }
  if (!__syncthreads_or(work)) return;
  const bool pair = G2 != nullptr;                         // first sub-step of a pair
  const float tw = sp.temporal_weight;
  const bool temporal = sp.use_temporal_interp == 1;
  const bool use_old = temporal && tw < 0.99f;
  const bool use_new = pair || !use_old || tw != 0.0f;
  const int gx0 = (mx - 1) * BS + 1, gy0 = (my - 1) * BS + 1, gz0 = (mz - 1) * BS + 1;
  // a parent value at this sub-step's weight and at the second sub-step's
  auto blend = [&](float fn, float fo, float &v, float &v2) {
    v = !use_old ? fn : (tw == 0.0f ? fo : lerp_rn(fo, fn, tw));
    v2 = temporal ? lerp_rn(fo, fn, kSecondSubstepWeight) : fn;
  };
  // parent cell of corner s of the group with pair indices (px, py, pz), -1 absent
  auto corner = [&](int px, int py, int pz, int s) -> int32_t {
    const int cx = (s & 1) ? lx + px + 1 : max(1, lx + px);
    const int cy = (s & 2) ? ly + py + 1 : max(1, ly + py);
    const int cz = (s & 4) ? lz + pz + 1 : max(1, lz + pz);
    const int q = ((cx - 1) / BS - bx0) + 2 * ((cy - 1) / BS - by0) + 4 * ((cz - 1) / BS - bz0);
    const int32_t base = pbase[q];
    return base < 0 ? -1
                    : base + ((cx - 1) & 7) + BS * ((cy - 1) & 7) + BS * BS * ((cz - 1) & 7);
  };
#pragma unroll
  for (int j = 0; j < kGhostScan; ++j) {
    const int u = t + j * kGhostThreads;
    append_if(kind[head[j] >> 21] != 0, u, &n_unit, unit_list);
  }
  // interpolated moments of the interface groups: one (group, moment) per thread
  if (fine && !precomputed) {
    for (int j = t; j < 4 * kGhostGroups; j += kGhostThreads) {
      const int q = j >> 2, m = j & 3;
      const uint32_t gw = __ldg(tab + 4 * kGhostUnits + q);
      if (kind[gw >> 8] != 1) continue;
      const int code = gw & 255;
      const int px = code % 6, py = (code / 6) % 6, pz = code / 36;
      const float *pn = ghost_moment_plane(L, m, false);
      const float *po = ghost_moment_plane(L, m, true);
      const float none = m == 0 ? 1.0f : 0.0f;
      float v[8], v2[8];
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const int32_t c = corner(px, py, pz, s);
        v[s] = v2[s] = none;
        if (c >= 0) blend(use_new ? pn[c] : 0.0f, use_old ? po[c] : 0.0f, v[s], v2[s]);
        else if (s > 0) { v[s] = v[0]; v2[s] = v2[0]; }
      }
#pragma unroll 1
      for (int sub = 0; sub < 4; ++sub) {
        int bits = sub;
        float wx, wy, wz;
        ghost_member(px, bits, wx);
        ghost_member(py, bits, wy);
        ghost_member(pz, bits, wz);
        if (bits) break;  // the group has fewer positions
        rs[m][4 * q + sub] = trilerp(v, wx, wy, wz);
        if (pair) rs2[m][4 * q + sub] = trilerp(v2, wx, wy, wz);
      }
    }
  }
  __syncthreads();
  for (int j = t; j < n_unit; j += kGhostThreads) {
    const int u = unit_list[j];
    const uint4 raw = __ldg((const uint4 *)tab + u);
    const int k = raw.x & 31, q = (raw.x >> 5) & 255, code = (raw.x >> 13) & 255;
    const int px = code % 6, py = (code / 6) % 6, pz = code / 36;
    if (kind[raw.x >> 21] == 1) {
      const T *po = par_old + (size_t)k * p_dstride, *pn = par_new + (size_t)k * p_dstride;
      float v[8], v2[8];
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const int32_t c = corner(px, py, pz, s);
        v[s] = v2[s] = w_of(k);
        if (c >= 0)
          blend(use_new ? ST::load(pn, c, k, p_inv_scale) : 0.0f,
                use_old ? ST::load(po, c, k, p_inv_scale) : 0.0f, v[s], v2[s]);
        else if (s > 0) { v[s] = v[0]; v2[s] = v2[0]; }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {  // this sub-step's weight, then the second one's
        if (h == 1 && !pair) break;
        float *const out = h ? G2 : G;
        const float(*const rr)[4 * kGhostGroups] = h ? rs2 : rs;
#pragma unroll 1
        for (int sub = 0; sub < 4; ++sub) {
          const uint32_t slot = ((sub < 2 ? raw.y : raw.z) >> (16 * (sub & 1))) & 0xFFFFu;
          if (slot == kGhostNoSlot) continue;
          int bits = sub;
          float wx, wy, wz;
          ghost_member(px, bits, wx);
          ghost_member(py, bits, wy);
          ghost_member(pz, bits, wz);
          const int i = 4 * q + sub;
          const float r[4] = {rr[0][i], rr[1][i], rr[2][i], rr[3][i]};
          out[slot] = ghost_finish(L, rescale, k, h ? v2 : v, wx, wy, wz, r);
        }
      }
    } else {
      for (int sub = 0; sub < 4; ++sub) {
        const uint32_t slot = ((sub < 2 ? raw.y : raw.z) >> (16 * (sub & 1))) & 0xFFFFu;
        if (slot == kGhostNoSlot) continue;
        int bits = sub;
        float w;
        const int sx = ghost_member(px, bits, w), sy = ghost_member(py, bits, w),
                  sz = ghost_member(pz, bits, w);
        const int gx = gx0 + sx, gy = gy0 + sy, gz = gz0 + sz;
        if (fine && gx >= 1 && gx <= sp.nx_global && gy >= 1 && gy <= sp.ny_global && gz >= 1 &&
            gz <= sp.nz_global) {
          if (precomputed) continue;
          G[slot] = ghost_slot<ST>(L, k, gx, gy, gz, tw);
          if (pair) G2[slot] = ghost_slot<ST>(L, k, gx, gy, gz, kSecondSubstepWeight);
        } else {
          G[slot] = ghost_boundary(L, k, b, sx + cx_of(k), sy + cy_of(k), sz + cz_of(k), ST{});
        }
      }
    }
  }
}

// Drop-in: one CTA per block of the level (rows indexed by block).
template <class ST>
__global__ void __launch_bounds__(kGhostThreads, kGhostMinBlocks)
    k_ghost_fill(const __grid_constant__ LevelDev L) {
  pdl_wait();  // the parent's new state and this level's f_in
  const int b = L.gblocks ? L.gblocks[blockIdx.x] : (int)blockIdx.x;
  ghost_fill_block<ST>(L, b, ghost_row_of(L, b), ghost_next_row_of(L, b));
}

constexpr int kHaloPerThread = (kHaloEntries + BCELLS - 1) / BCELLS;  // 7

// Asks L2 for the per-cell arrays of block nb (local index) of level L: its
// 27 population planes, velocity (WALE reads it), sponge, mask and wall
// distance, one bulk prefetch per thread t < 33.  The stream-collide launch
// issues this for the block its CTA slot takes one wave later, so that
// block's staging loads find their data in L2 (no registers, no shared
// memory, nothing to wait for).  Every run is whole and 16-byte aligned:
// blocks are 512 cells and the arrays' planes are whole blocks.
template <class ST>
__device__ __forceinline__ void prefetch_block_l2(const LevelDev &L, int nb, int t) {
  if (nb >= L.n_blocks || t >= 33) return;
  using T = typename ST::T;
  const int64_t o = (L.block_offset + nb) * BCELLS;
  const void *src = nullptr;
  unsigned bytes = BCELLS * sizeof(float);
  if (t < 27) {
    src = (const T *)L.f_in + o + (int64_t)t * L.dstride;
    bytes = BCELLS * sizeof(T);
  } else if (t < 30) {
    if (L.vel_in) src = L.vel_in + o + (int64_t)(t - 27) * L.dstride;
  } else if (t == 30) {
    src = L.sponge + o;
  } else if (t == 31) {
    src = L.obstacle + o;
    bytes = BCELLS;
  } else if (L.wall_dist) {
    src = L.wall_dist + o;
  }
  if (src) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes)
                        : "memory");
}

// The own block's 27 planes, loaded into registers with 16-byte loads
// (FP32: 7 float4 per thread; FP16: 4 x 8 halves).  The loads depend only on
// the block's own offset, so a kernel can issue them before it has read the
// neighbour table.
template <class ST> struct OwnRegs;
template <> struct OwnRegs<StoreF32> { float4 v[7]; };
template <> struct OwnRegs<StoreF16S> { uint4 v[4]; };

__device__ __forceinline__ void own_load(const void *f_in_v, int64_t dstride, int64_t own, int t,
                                         OwnRegs<StoreF32> &r) {
  const float *fin = (const float *)f_in_v;
  const int c0 = (t & 127) * 4;
#pragma unroll
  for (int j = 0; j < 7; ++j) {
    const int k = (t >> 7) + 4 * j;
    if (k < 27) r.v[j] = __ldg((const float4 *)(fin + (size_t)k * dstride + own + c0));
  }
}
__device__ __forceinline__ void own_load(const void *f_in_v, int64_t dstride, int64_t own, int t,
                                         OwnRegs<StoreF16S> &r) {
  const __half *fin = (const __half *)f_in_v;
  const int c0 = (t & 63) * 8;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int k = (t >> 6) + 8 * j;
    if (k < 27) r.v[j] = __ldg((const uint4 *)(fin + (size_t)k * dstride + own + c0));
  }
}
// Odd lanes (x = 4..7 of a row) write their four cells rotated by one, so each
// store instruction of a warp touches every bank at most twice (three times
// in x order).
__device__ __forceinline__ void own_store(const OwnRegs<StoreF32> &r, float, int t, float *E) {
  const int c0 = (t & 127) * 4;
  const int dst = e_index(c0 & 7, (c0 >> 3) & 7, c0 >> 6);
  const bool odd = t & 1;
  const int o0 = odd ? 1 : 0, o1 = odd ? 2 : 1, o2 = odd ? 3 : 2, o3 = odd ? 0 : 3;
#pragma unroll
  for (int j = 0; j < 7; ++j) {
    const int k = (t >> 7) + 4 * j;
    if (k < 27) {
      float *e = E + k * EPL + dst;
      const float4 v = r.v[j];
      e[o0] = odd ? v.y : v.x;
      e[o1] = odd ? v.z : v.y;
      e[o2] = odd ? v.w : v.z;
      e[o3] = odd ? v.x : v.w;
    }
  }
}
__device__ __forceinline__ void own_store(const OwnRegs<StoreF16S> &r, float inv_scale, int t,
                                          float *E) {
  const int c0 = (t & 63) * 8;
  const int dst = e_index(0, (c0 >> 3) & 7, c0 >> 6);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int k = (t >> 6) + 8 * j;
    if (k < 27) {
      const __half2 *h = (const __half2 *)&r.v[j];
      const float w = w_of(k), sc = w * inv_scale;
      float *e = E + k * EPL + dst;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f2 = __half22float2(h[i]);
        e[2 * i] = fmaf(f2.x, sc, w);
        e[2 * i + 1] = fmaf(f2.y, sc, w);
      }
    }
  }
}

// Halo part of the staging, then the own block's registers into E.
// ghost_row: this block's precomputed absent-neighbour values in table order
// (kHaloEntries floats), or null to compute them here with `fill`.
template <class ST, class FILL>
__device__ __forceinline__ void stage_halo(const void *f_in_v, int64_t dstride, float inv_scale,
                                           const int *nbbase, int t, float *E,
                                           const uint32_t *__restrict__ tab, bool any_missing,
                                           const float *__restrict__ ghost_row,
                                           const OwnRegs<ST> &own_regs, FILL fill) {
  using T = typename ST::T;
  const T *__restrict__ fin = (const T *)f_in_v;
  // halo sources: all table entries and source values of this thread in flight at once
  uint32_t te[kHaloPerThread];
#pragma unroll
  for (int j = 0; j < kHaloPerThread; ++j) {
    const int i = t + j * BCELLS;
    te[j] = i < kHaloEntries ? __ldg(tab + i) : 0xFFFFFFFFu;
  }
  float hv[kHaloPerThread];
  int hd[kHaloPerThread];
#pragma unroll
  for (int j = 0; j < kHaloPerThread; ++j) {
    hd[j] = -1;
    hv[j] = 0.0f;
    if (te[j] != 0xFFFFFFFFu) {
      const int k = te[j] & 31, dir = (te[j] >> 5) & 31, src = (te[j] >> 10) & 511;
      const int nb = nbbase[dir];
      if (nb >= 0) {
        hd[j] = k * EPL + (int)(te[j] >> 19);
        hv[j] = ST::load(fin, (size_t)k * dstride + nb + src, k, inv_scale);
      } else if (ghost_row) {
        hd[j] = k * EPL + (int)(te[j] >> 19);
        hv[j] = ghost_row[t + j * BCELLS];
      }
    }
  }
  own_store(own_regs, inv_scale, t, E);
#pragma unroll
  for (int j = 0; j < kHaloPerThread; ++j)
    if (hd[j] >= 0) E[hd[j]] = hv[j];
  if (any_missing && !ghost_row) fill();
}

template <class ST, class FILL>
__device__ __forceinline__ void stage_block(const void *f_in_v, int64_t dstride, float inv_scale,
                                            const int *nbbase, int t, float *E,
                                            const uint32_t *__restrict__ tab, bool any_missing,
                                            const float *__restrict__ ghost_row, FILL fill) {
  OwnRegs<ST> r;
  own_load(f_in_v, dstride, nbbase[13], t, r);
  stage_halo<ST>(f_in_v, dstride, inv_scale, nbbase, t, E, tab, any_missing, ghost_row, r, fill);
}

// Neighbour-table row -> element offsets of the 27 neighbour blocks, then a
// barrier; returns whether any neighbour of the block is absent.
__device__ __forceinline__ bool load_nbbase_sync(const int32_t *nbr, int64_t nbr_stride,
                                                 int64_t block_offset, int b, int t, int *nbbase) {
  int missing = 0;
  if (t < 27) {
    const int nb = nbr[b + nbr_stride * t];
    nbbase[t] = nb > 0 ? (int)((block_offset + nb - 1) * BCELLS) : -1;
    missing = nb <= 0;
  }
  return __syncthreads_or(missing) != 0;
}

// Stage the flow populations of block b of level L.
template <class ST>
__device__ __forceinline__ void stage_flow(const LevelDev &L, const int *nbbase, int b, int t,
                                           float *E, bool any_missing) {
  const float *ghost_row = ghost_row_of(L, b);
  stage_block<ST>(L.f_in, L.dstride, L.inv_scale, nbbase, t, E, L.halo_tab, any_missing,
                  ghost_row, [&]() { fill_missing_flow<ST>(L, nbbase, b, t, E); });
}

// The same with the own block already in registers (own_load issued before
// the neighbour table was read).
template <class ST>
__device__ __forceinline__ void stage_flow(const LevelDev &L, const int *nbbase, int b, int t,
                                           float *E, bool any_missing, const OwnRegs<ST> &r) {
  const float *ghost_row = ghost_row_of(L, b);
  stage_halo<ST>(L.f_in, L.dstride, L.inv_scale, nbbase, t, E, L.halo_tab, any_missing,
                 ghost_row, r, [&]() { fill_missing_flow<ST>(L, nbbase, b, t, E); });
}

// obs / spg: this cell's obstacle flag and sponge weight, loaded by the
// caller before staging so that their latency overlaps it.
// The 27 pulls of cell t from the staged windows.
__device__ __forceinline__ void load_pulls(const float *E, int t, float (&A)[27]) {
  const int eb = e_index(t & 7, (t >> 3) & 7, t >> 6);
#pragma unroll
  for (int k = 0; k < 27; ++k)
    A[k] = E[k * EPL + eb - (cx_of(k) + 10 * cy_of(k) + 100 * cz_of(k))];
}

// Per-cell inputs a caller may have evaluated ahead of the collision (the
// warp-specialised kernel does so before its shared-memory pulls): the wall
// distance and the WALE eddy viscosity.
struct CellAux {
  float wall_dist;
  float nu_wale;
};

// collide_cell's stores: populations (and the optional post-collision copy)
// and rho, u, straight to the level's arrays.  The descriptor's fields are
// copied to locals first: in the block pool it lies in shared memory, which a
// store through a generic pointer might alias, so that each of the 27 stores
// would wait for the plane stride to be read again (8 steps of a pool of 6
// cases: FP16 storage 6715 -> 6505 us, FP32 5515 -> 5480 us).
template <class ST>
struct GlobalOut {
  const LevelDev &L;
  size_t own;
  __device__ __forceinline__ GlobalOut(const LevelDev &L_, size_t own_) : L(L_), own(own_) {}
  __device__ __forceinline__ void macro(float rho, float ux, float uy, float uz) const {
    float *const vel = L.vel_out + own, *const r = L.rho_out + own;
    const int64_t dstride = L.dstride;
    vel[0] = ux;
    vel[dstride] = uy;
    vel[2 * dstride] = uz;
    *r = rho;
  }
  // all 27 populations, A[k] (OPP = false) or the bounce-back A[opp(k)]
  template <bool OPP>
  __device__ __forceinline__ void f_all(const float (&A)[27]) const {
    typename ST::T *const fout = (typename ST::T *)L.f_out;
    float *const fpost = L.sp.store_post_collision ? L.f_post : nullptr;
    const int64_t dstride = L.dstride;
    const float scale = L.scale;
    if (fpost) {
#pragma unroll
      for (int k = 0; k < 27; ++k) {
        const float v = A[OPP ? opp_of(k) : k];
        ST::store(fout, own + (size_t)k * dstride, k, scale, v);
        fpost[own + (size_t)k * dstride] = v;
      }
    } else {
#pragma unroll
      for (int k = 0; k < 27; ++k)
        ST::store(fout, own + (size_t)k * dstride, k, scale, A[OPP ? opp_of(k) : k]);
    }
  }
};

template <int OP, class ST, bool WALE, bool LOW = false, int SUMS = kSumsShort>
__device__ __forceinline__ void collide_cell(const LevelDev &L, const int *nbbase, float (&A)[27],
                                             int b, int t, bool obs, float spg,
                                             const CellAux *aux = nullptr);

template <int OP, class ST, bool WALE, int SUMS = kSumsShort>
__device__ __forceinline__ void stream_collide_cell(const LevelDev &L, const int *nbbase,
                                                    const float *E, int b, int t, bool obs,
                                                    float spg) {
  float A[27];
  load_pulls(E, t, A);
  collide_cell<OP, ST, WALE, false, SUMS>(L, nbbase, A, b, t, obs, spg);
}

// Device watchdog of the native path: non-finite or vanishing density.
__device__ __forceinline__ void watchdog(int32_t *status, float rho) {
  if (!(fabsf(rho) < 1e30f)) atomicOr(status, 1);
  else if (rho < 0.01f) atomicOr(status, 2);
}

// Everything after the pull: bounce-back, moments, sponge, wall model,
// WALE, collision, forcing and the stores of cell t of block b.  LOW: the
// caller knows that omega_3 = omega_4 = 1.
template <int OP, class ST, bool WALE, bool LOW, int SUMS>
__device__ __forceinline__ void collide_cell(const LevelDev &L, const int *nbbase, float (&A)[27],
                                             int b, int t, bool obs, float spg,
                                             const CellAux *aux) {
  const int x = t & 7, y = (t >> 3) & 7, z = t >> 6;
  const ol_step_params &sp = L.sp;
  const size_t own = (size_t)nbbase[13] + t;
  const GlobalOut<ST> out(L, own);

  float rho, jx, jy, jz;
  if (obs) {
    if (L.status) {
      rho = 0.0f;
#pragma unroll
      for (int k = 0; k < 27; ++k) rho += A[k];
      watchdog(L.status, rho);
    }
    out.macro(1.0f, 0.0f, 0.0f, 0.0f);
    out.template f_all<true>(A);
    return;
  }
  if constexpr (SUMS != kSumsShort) {
    rho = jx = jy = jz = 0.0f;
#pragma unroll
    for (int k = 0; k < 27; ++k) {
      rho += A[k];
      if (cx_of(k) == 1) jx += A[k]; else if (cx_of(k) == -1) jx -= A[k];
      if (cy_of(k) == 1) jy += A[k]; else if (cy_of(k) == -1) jy -= A[k];
      if (cz_of(k) == 1) jz += A[k]; else if (cz_of(k) == -1) jz -= A[k];
    }
  } else {
    // A becomes the raw x-moments (m0, m1, m2) of each (y, z) triple
#pragma unroll
    for (int i = 0; i < 9; ++i) raw_moments<kSumsShort>(A[3 * i], A[3 * i + 1], A[3 * i + 2]);
    const float s0 = A[0] + A[3] + A[6], s1 = A[9] + A[12] + A[15], s2 = A[18] + A[21] + A[24];
    rho = s0 + s1 + s2;
    jx = (A[1] + A[4] + A[7]) + (A[10] + A[13] + A[16]) + (A[19] + A[22] + A[25]);
    jy = (A[6] - A[0]) + (A[15] - A[9]) + (A[24] - A[18]);
    jz = s2 - s0;
  }
  // device watchdog (native path): report, never trap
  if (L.status) watchdog(L.status, rho);
  rho = fmaxf(rho, 0.01f);  // (an infinite density is stored as such)
  const float inv_rho = recip_nr(fminf(rho, 3e38f));
  float ux = jx * inv_rho, uy = jy * inv_rho, uz = jz * inv_rho;
  if (spg > 0.0f) {
    rho = rho * (1.0f - spg) + 1.0f * spg;
    ux = ux * (1.0f - spg) + sp.u_inlet * spg;
    uy = uy * (1.0f - spg);
    uz = uz * (1.0f - spg);
    if (sp.sponge_blend_distributions == 1) {
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        float ft[3];
#pragma unroll
        for (int j = 0; j < 3; ++j)
          ft[j] = feq_auto(1.0f, sp.u_inlet, 0.0f, 0.0f, w_of(3 * i + j), (float)cx_of(3 * i + j),
                           (float)cy_of(3 * i + j), (float)cz_of(3 * i + j), sp.compressible_corr);
        if constexpr (SUMS == kSumsShort) raw_moments<kSumsShort>(ft[0], ft[1], ft[2]);
#pragma unroll
        for (int j = 0; j < 3; ++j) A[3 * i + j] = A[3 * i + j] * (1.0f - spg) + ft[j] * spg;
      }
    }
  }
  if constexpr (SUMS != kSumsShort) {
#pragma unroll
    for (int i = 0; i < 9; ++i) raw_moments<SUMS>(A[3 * i], A[3 * i + 1], A[3 * i + 2]);
  }
  float Fx = 0.0f, Fy = 0.0f, Fz = 0.0f;
  if (sp.wall_model_active == 1 && L.wall_dist)
    wall_force(aux ? aux->wall_dist : L.wall_dist[own], rho, ux, uy, uz, sp.tau_molecular, Fx,
               Fy, Fz);
  const bool forced = (Fx != 0.0f) | (Fy != 0.0f) | (Fz != 0.0f);
  const float uxe = ux + 0.5f * Fx * inv_rho;
  const float uye = uy + 0.5f * Fy * inv_rho;
  const float uze = uz + 0.5f * Fz * inv_rho;

  out.macro(rho, ux, uy, uz);

  float nu_eddy = 0.0f;
  if (WALE) nu_eddy = aux ? aux->nu_wale : wale_nu(L, nbbase, x, y, z);
  nu_eddy = fmaxf(nu_eddy, sp.nu_sgs_background);

  float omega;  // omega_1 (cumulant) or omega (BGK)
  if (OP == OL_OP_CUMULANT) {
    const float nu_mol = third_of(sp.tau_molecular - 0.5f);
    const float tau_eff = 0.5f + 3.0f * (nu_mol + nu_eddy);
    omega = recip_nr(fminf(fmaxf(tau_eff, 0.500001f), 3e38f));
    CumulantRates r;
    r.omega1 = omega;
    r.omega_bulk = sp.omega_bulk;
    r.omega3 = sp.omega_3;
    r.omega4 = sp.omega_4;
    r.omega4_diag = sp.omega_4;
    if (sp.adaptive_omega4 == 1) {
      const float om1m2 = omega - 2.0f;
      const float Av = quotient_nr(-(om1m2 * om1m2), sp.lambda_param * omega + 1e-10f);
      r.omega4_diag = fminf(fmaxf(Av, 0.01f), 2.0f);
    }
    r.limiter = sp.limiter_type;
    if (LOW || (sp.omega_3 == 1.0f && sp.omega_4 == 1.0f))
      collide_cumulant<true, SUMS>(A, uxe, uye, uze, r);
    else
      collide_cumulant<false, SUMS>(A, uxe, uye, uze, r);
    if (sp.limiter_type == OL_LIMITER_POSITIVITY) {
      float fmin = A[0];
#pragma unroll
      for (int k = 1; k < 27; ++k) fmin = fminf(fmin, A[k]);
      if (fmin < 0.0f) positivity_limit(A, rho, uxe, uye, uze, sp.compressible_corr);
    }
  } else {
    // Regularized BGK (kernel_regularized_bgk.jl:270-316); the Guo term uses
    // c.u_eq, as kernel_cumulant.jl:610 does (the reference line 302 names
    // an undefined `cu`).
    const float tau_turb = sp.tau_molecular + nu_eddy * 3.0f;
    omega = recip_nr(fminf(fmaxf(tau_turb, 0.500001f), 3e38f));
    bgk_regularized(A, rho, uxe, uye, uze, 1.0f - omega, sp.compressible_corr);
  }
  if (forced) {
    const float g = 1.0f - 0.5f * omega;
#pragma unroll
    for (int k = 0; k < 27; ++k) {
      const float cxf = (float)cx_of(k), cyf = (float)cy_of(k), czf = (float)cz_of(k);
      const float cu = cxf * uxe + cyf * uye + czf * uze;
      const float ft = w_of(k) * 3.0f *
                       ((cxf - ux + 3.0f * cu * cxf) * Fx +
                        (cyf - uy + 3.0f * cu * cyf) * Fy +
                        (czf - uz + 3.0f * cu * czf) * Fz);
      A[k] = A[k] + g * ft;
    }
  }
  out.template f_all<false>(A);
}

}  // namespace ol

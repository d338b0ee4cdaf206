// dg_step_generic.cuh — step kernels in the geometric-factor form for any shot count and for
// batches of meshes: FP64 and FP32 (plain or Kahan-compensated), one thread per lane — an element's
// shot, or its pair of shots on packed FP32x2 (ArithP2<float2>, even stored shots) — on plane-major
// state U[plane][e*S + s] (or, for half steps of a wavefront context, element-major).
//
// The arithmetic is dg_core.cuh's.  Register budget: one sweep over the faces for both velocity
// components (each neighbour value gathered once); the stress kernel takes the volume terms first
// and the face terms after; the fields being updated are loaded only at the end.
#pragma once
#include "dg_common.cuh"
#include "dg_core.cuh"

namespace dg {

// Registers of k_velocity / k_stress: 128 a thread (16 warps an SM); two shots a thread with
// compensation hold twice the values and spill there, so they get 168 (7,200 x 24 shots, us: 14.7 -> 12.7
// and 18.5 -> 16.4).
template <class A, bool KAHAN> constexpr int gen_regs = KAHAN && sizeof(typename A::V) == 8 ? 168 : 128;

// Velocity half-step: for its own element the sponge on the five fields and the source on Vz
// (OpenMP_Function.c:25-58), then V += dt L_V(T) (OpenMP_Function.c:75-185), L_V = (1/rho) h.
template <class A, bool KAHAN, class R = typename A::R>
__device__ __forceinline__ void velocity_body(const Ops<R>& ops_, const MeshDev<R>& m, int lb, long long t) {
  using V = typename A::V;
  constexpr int SV = sizeof(V) / sizeof(R);  // shots of a lane
  const int H = m.S / SV;                    // lanes of an element
  const long long g = (long long)lb * blockDim.x + threadIdx.x;
  if (g >= (long long)m.K * H) return;
  int e, s;  // element, lane
  if (H == 1) { e = (int)g; s = 0; } else { e = (int)(g / H); s = (int)(g - (long long)e * H); }
  const typename A::Ops& ops = A::ops(ops_);
  const long long P = m.PS / SV, ES = m.ES / SV, at = e * ES + s;
  V* const U = reinterpret_cast<V*>(m.U);
  V* const C = reinterpret_cast<V*>(m.C);
  V* __restrict__ Ug = U + at;

  const int4 fc = __ldg(m.face + e);
  const auto gm = ld4(m.geo + e);
  const R rx = gm.x, sx = gm.y, rz = gm.z, sz = gm.w;
  const bool own_sponge = fc.w & 1;
  const int nbs[3] = {fc.x, fc.y, fc.z};
  V sp[NP];
#pragma unroll
  for (int i = 0; i < NP; i++) sp[i] = Bcast<V>::of(own_sponge ? ldg(m.sponge + (long long)i * m.Kp + e) : R(1));

  V txz[NP], hx[NP], hz[NP];
#pragma unroll
  for (int i = 0; i < NP; i++) txz[i] = v_mul(Ug[(24 + i) * P], sp[i]);
  {
    V txx[NP], tzz[NP];
#pragma unroll
    for (int i = 0; i < NP; i++) {
      txx[i] = v_mul(Ug[(12 + i) * P], sp[i]);
      tzz[i] = v_mul(Ug[(18 + i) * P], sp[i]);
    }
    core_velocity_rhs<A>(ops, rx, sx, rz, sz, txx, tzz, txz, [&](int j, V (&pxx)[NF], V (&pzz)[NF], V (&pxz)[NF]) {
      const int nb = nbs[j];
      if (nb < 0) {
#pragma unroll
        for (int k = 0; k < NF; k++) { pxx[k] = v_const<V>(0.f); pzz[k] = pxx[k]; pxz[k] = pxx[k]; }
        return;
      }
      const V* __restrict__ Un = U + (nb * ES + s);
#pragma unroll
      for (int k = 0; k < NF; k++) {
        const int node = nb_node(fc.w, j, k);
        pxx[k] = Un[(12 + node) * P];
        pzz[k] = Un[(18 + node) * P];
        pxz[k] = Un[(24 + node) * P];
      }
      if (nb_sponge(fc.w, j)) {
#pragma unroll
        for (int k = 0; k < NF; k++) {
          const V a = Bcast<V>::of(ldg(m.sponge + (long long)nb_node(fc.w, j, k) * m.Kp + nb));
          pxx[k] = v_mul(pxx[k], a); pzz[k] = v_mul(pzz[k], a); pxz[k] = v_mul(pxz[k], a);
        }
      }
    }, hx, hz);
  }

  const R irho = __ldg(&m.mat[e].x);
  V vx[NP], vz[NP], cvx[NP], cvz[NP];
#pragma unroll
  for (int i = 0; i < NP; i++) { vx[i] = v_mul(Ug[(0 + i) * P], sp[i]); vz[i] = v_mul(Ug[(6 + i) * P], sp[i]); }
  if (KAHAN) {
#pragma unroll
    for (int i = 0; i < NP; i++) { cvx[i] = v_mul(C[(0 + i) * P + at], sp[i]); cvz[i] = v_mul(C[(6 + i) * P + at], sp[i]); }
  }
  V srcz[NP];
#pragma unroll
  for (int i = 0; i < NP; i++) srcz[i] = v_const<V>(0.f);
  bool mine[SV], any = false;
#pragma unroll
  for (int c = 0; c < SV; c++) {
    mine[c] = __ldg(m.src_elem + s * SV + c) == e;
    any = any || mine[c];
  }
  if (any) {
    const R w = (R)__ldg(m.wavelet + t);
#pragma unroll
    for (int i = 0; i < NP; i++) {
      R x[SV];
#pragma unroll
      for (int c = 0; c < SV; c++) x[c] = mine[c] ? v_mul(ldg(m.src_fun + (s * SV + c) * NP + i), w) : R(0);
      if constexpr (SV == 2) srcz[i] = make_float2(x[0], x[1]);
      else srcz[i] = x[0];
    }
  }
  const V step = Bcast<V>::of(v_mul(m.dt, irho));
#pragma unroll
  for (int i = 0; i < NP; i++) {
    if (KAHAN) {
      v_kahan(vx[i], cvx[i], v_mul(step, hx[i]));
      v_kahan(vz[i], cvz[i], v_fma(step, hz[i], srcz[i]));
    } else {
      vx[i] = v_fma(step, hx[i], vx[i]);
      vz[i] = v_fma(step, hz[i], v_add(vz[i], srcz[i]));
    }
    Ug[(0 + i) * P] = vx[i];
    Ug[(6 + i) * P] = vz[i];
  }
  if (KAHAN) {
#pragma unroll
    for (int i = 0; i < NP; i++) { C[(0 + i) * P + at] = cvx[i]; C[(6 + i) * P + at] = cvz[i]; }
  }
}

template <class A, bool KAHAN, bool MULTI, class R = typename A::R>
__global__ void __maxnreg__((gen_regs<A, KAHAN>)) k_velocity(const __grid_constant__ Ops<R> ops,
                                                     const __grid_constant__ MeshDev<R> one,
                                                     const MeshDev<R>* __restrict__ tab,
                                                     const int2* __restrict__ btab,
                                                     Counters* __restrict__ ctr) {
  pdl_enter();
  int lb;
  const MeshDev<R>& m = *pick_mesh<MULTI>(one, tab, btab, lb);
  const long long t = ctr->v;
  if (threadIdx.x == 0 && blockIdx.x == 0) ctr->s = t;
  if (t >= m.steps) return;
  velocity_body<A, KAHAN>(ops, m, lb, t);
}

// Stress half-step: T = a T + dt L_T(V) (OpenMP_Function.c:188-306),
//   Txx += dt [ (l+2m) (dxVx + sum_j S_j nx_j dVx) + l (dzVz + sum_j S_j nz_j dVz) ]
//   Tzz += dt [ l (dxVx + ...) + (l+2m) (dzVz + ...) ]
//   Txz += dt m [ dxVz + dzVx + sum_j S_j (nz_j dVx + nx_j dVz) ]
// The trailing blocks of the grid record the receivers (V is final during this kernel).
template <class A, bool KAHAN, class R = typename A::R>
__device__ __forceinline__ void stress_body(const Ops<R>& ops_, const MeshDev<R>& m, int lb, long long t) {
  using V = typename A::V;
  constexpr int SV = sizeof(V) / sizeof(R);  // shots of a lane
  const int H = m.S / SV;                    // lanes of an element
  const long long g = (long long)lb * blockDim.x + threadIdx.x;
  if (g >= (long long)m.K * H) return;
  int e, s;  // element, lane
  if (H == 1) { e = (int)g; s = 0; } else { e = (int)(g / H); s = (int)(g - (long long)e * H); }
  const typename A::Ops& ops = A::ops(ops_);
  const long long P = m.PS / SV, ES = m.ES / SV, at = e * ES + s;
  V* const U = reinterpret_cast<V*>(m.U);
  V* const C = reinterpret_cast<V*>(m.C);
  V* __restrict__ Ug = U + at;

  V vx[NP], vz[NP];
#pragma unroll
  for (int i = 0; i < NP; i++) { vx[i] = Ug[(0 + i) * P]; vz[i] = Ug[(6 + i) * P]; }
  const int4 fc = __ldg(m.face + e);
  const auto gm = ld4(m.geo + e);
  const R rx = gm.x, sx = gm.y, rz = gm.z, sz = gm.w;

  const int nbs[3] = {fc.x, fc.y, fc.z};
  V X[NP], Z[NP], W[NP];
  core_strain<A>(ops, rx, sx, rz, sz, vx, vz, [&](int j, V (&px)[NF], V (&pz)[NF]) {
    const int nb = nbs[j];
    if (nb < 0) {
#pragma unroll
      for (int k = 0; k < NF; k++) { px[k] = v_const<V>(0.f); pz[k] = px[k]; }
      return;
    }
    const V* __restrict__ Un = U + (nb * ES + s);
#pragma unroll
    for (int k = 0; k < NF; k++) {
      const int node = nb_node(fc.w, j, k);
      px[k] = Un[(0 + node) * P];
      pz[k] = Un[(6 + node) * P];
    }
  }, X, Z, W);

  const auto mt = ld4(m.mat + e);
  const R lam = mt.y, mu = mt.z, l2m = mt.w;
  V txx[NP], tzz[NP], txz[NP], cxx[NP], czz[NP], cxz[NP];
#pragma unroll
  for (int i = 0; i < NP; i++) {
    txx[i] = Ug[(12 + i) * P];
    tzz[i] = Ug[(18 + i) * P];
    txz[i] = Ug[(24 + i) * P];
  }
  if (KAHAN) {
#pragma unroll
    for (int i = 0; i < NP; i++) {
      cxx[i] = C[(12 + i) * P + at]; czz[i] = C[(18 + i) * P + at]; cxz[i] = C[(24 + i) * P + at];
    }
  }
  if (fc.w & 1) {
#pragma unroll
    for (int i = 0; i < NP; i++) {
      const V a = Bcast<V>::of(ldg(m.sponge + (long long)i * m.Kp + e));
      txx[i] = v_mul(txx[i], a); tzz[i] = v_mul(tzz[i], a); txz[i] = v_mul(txz[i], a);
      if (KAHAN) { cxx[i] = v_mul(cxx[i], a); czz[i] = v_mul(czz[i], a); cxz[i] = v_mul(cxz[i], a); }
    }
  }
  const V dl2m = Bcast<V>::of(v_mul(m.dt, l2m)), dlam = Bcast<V>::of(v_mul(m.dt, lam)), dmu = Bcast<V>::of(v_mul(m.dt, mu));
#pragma unroll
  for (int i = 0; i < NP; i++) {
    const V dxx = v_fma(dl2m, X[i], v_mul(dlam, Z[i]));
    const V dzz = v_fma(dlam, X[i], v_mul(dl2m, Z[i]));
    if (KAHAN) {
      v_kahan(txx[i], cxx[i], dxx);
      v_kahan(tzz[i], czz[i], dzz);
      v_kahan(txz[i], cxz[i], v_mul(dmu, W[i]));
    } else {
      txx[i] = v_add(txx[i], dxx);
      tzz[i] = v_add(tzz[i], dzz);
      txz[i] = v_fma(dmu, W[i], txz[i]);
    }
    Ug[(12 + i) * P] = txx[i];
    Ug[(18 + i) * P] = tzz[i];
    Ug[(24 + i) * P] = txz[i];
  }
  if (KAHAN) {
#pragma unroll
    for (int i = 0; i < NP; i++) {
      C[(12 + i) * P + at] = cxx[i]; C[(18 + i) * P + at] = czz[i]; C[(24 + i) * P + at] = cxz[i];
    }
  }
}

template <class A, bool KAHAN, bool MULTI, class R = typename A::R>
__global__ void __maxnreg__((gen_regs<A, KAHAN>)) k_stress(const __grid_constant__ Ops<R> ops,
                                                   const __grid_constant__ MeshDev<R> one,
                                                   const MeshDev<R>* __restrict__ tab,
                                                   const int2* __restrict__ btab,
                                                   Counters* __restrict__ ctr) {
  pdl_enter();
  int lb;
  const MeshDev<R>& m = *pick_mesh<MULTI>(one, tab, btab, lb);
  const long long t = ctr->s;
  if (threadIdx.x == 0 && blockIdx.x == 0) ctr->v = t + 1;
  if (t >= m.steps) return;
  if (!MULTI) lb = stress_block(m, lb);
  if (lb >= m.n_elem_blocks) { record(m, lb - m.n_elem_blocks, t); return; }
  stress_body<A, KAHAN>(ops, m, lb, t);
}

}  // namespace dg

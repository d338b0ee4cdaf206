// dg_step_generic.cuh — step kernels in the geometric-factor form for any shot count and for
// batches of meshes: FP64 and FP32 (plain or Kahan-compensated), one thread per (element, shot),
// plane-major layout U[plane][e*S + s].
//
// The arithmetic is dg_core.cuh's.  Register budget: one sweep over the faces for both velocity
// components (each neighbour value gathered once); the stress kernel takes the volume terms first
// and the face terms after; the fields being updated are loaded only at the end.
#pragma once
#include "dg_common.cuh"
#include "dg_core.cuh"

namespace dg {

// Velocity half-step: for its own element the sponge on the five fields and the source on Vz
// (OpenMP_Function.c:25-58), then V += dt L_V(T) (OpenMP_Function.c:75-185), L_V = (1/rho) h.
template <class R, bool KAHAN>
__device__ __forceinline__ void velocity_body(const Ops<R>& ops, const MeshDev<R>& m, int lb, long long t) {
  const int S = m.S;
  const long long g = (long long)lb * blockDim.x + threadIdx.x;
  if (g >= (long long)m.K * S) return;
  int e, s;
  if (S == 1) { e = (int)g; s = 0; } else { e = (int)(g / S); s = (int)(g - (long long)e * S); }
  const long long P = m.P;
  R* __restrict__ Ug = m.U + g;

  const int4 fc = __ldg(m.face + e);
  const auto gm = ld4(m.geo + e);
  const R rx = gm.x, sx = gm.y, rz = gm.z, sz = gm.w;
  const bool own_sponge = fc.w & 1;
  const int codes[3] = {fc.x, fc.y, fc.z};
  R sp[NP];
#pragma unroll
  for (int i = 0; i < NP; i++) sp[i] = own_sponge ? ldg(m.sponge + (long long)i * m.Kp + e) : R(1);

  R txz[NP], hx[NP], hz[NP];
#pragma unroll
  for (int i = 0; i < NP; i++) txz[i] = v_mul(Ug[(24 + i) * P], sp[i]);
  {
    R txx[NP], tzz[NP];
#pragma unroll
    for (int i = 0; i < NP; i++) {
      txx[i] = v_mul(Ug[(12 + i) * P], sp[i]);
      tzz[i] = v_mul(Ug[(18 + i) * P], sp[i]);
    }
    core_velocity_rhs<ArithOps<R>>(ops, rx, sx, rz, sz, txx, tzz, txz, [&](int j, R (&pxx)[NF], R (&pzz)[NF], R (&pxz)[NF]) {
      const int code = codes[j];
      if (code < 0) {
#pragma unroll
        for (int k = 0; k < NF; k++) { pxx[k] = R(0); pzz[k] = R(0); pxz[k] = R(0); }
        return;
      }
      const int nb = code >> 4, nf = (code >> 1) & 3, flip = code & 1;
      const R* __restrict__ Un = m.U + ((long long)nb * S + s);
#pragma unroll
      for (int k = 0; k < NF; k++) {
        const int node = face_node(nf, flip ? 2 - k : k);
        pxx[k] = Un[(12 + node) * P];
        pzz[k] = Un[(18 + node) * P];
        pxz[k] = Un[(24 + node) * P];
      }
      if (code & 8) {
#pragma unroll
        for (int k = 0; k < NF; k++) {
          const R a = ldg(m.sponge + (long long)face_node(nf, flip ? 2 - k : k) * m.Kp + nb);
          pxx[k] = v_mul(pxx[k], a); pzz[k] = v_mul(pzz[k], a); pxz[k] = v_mul(pxz[k], a);
        }
      }
    }, hx, hz);
  }

  const R irho = __ldg(&m.mat[e].x);
  R vx[NP], vz[NP], cvx[NP], cvz[NP];
#pragma unroll
  for (int i = 0; i < NP; i++) { vx[i] = v_mul(Ug[(0 + i) * P], sp[i]); vz[i] = v_mul(Ug[(6 + i) * P], sp[i]); }
  if (KAHAN) {
#pragma unroll
    for (int i = 0; i < NP; i++) { cvx[i] = v_mul(m.C[(0 + i) * P + g], sp[i]); cvz[i] = v_mul(m.C[(6 + i) * P + g], sp[i]); }
  }
  R srcz[NP];
#pragma unroll
  for (int i = 0; i < NP; i++) srcz[i] = R(0);
  if (__ldg(m.src_elem + s) == e) {
    const R w = (R)__ldg(m.wavelet + t);
#pragma unroll
    for (int i = 0; i < NP; i++) srcz[i] = v_mul(ldg(m.src_fun + s * NP + i), w);
  }
  const R step = v_mul(m.dt, irho);
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
    for (int i = 0; i < NP; i++) { m.C[(0 + i) * P + g] = cvx[i]; m.C[(6 + i) * P + g] = cvz[i]; }
  }
}

template <class R, bool KAHAN, bool MULTI>
__global__ void __launch_bounds__(256, 2) k_velocity(const __grid_constant__ Ops<R> ops,
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
  velocity_body<R, KAHAN>(ops, m, lb, t);
}

// Stress half-step: T = a T + dt L_T(V) (OpenMP_Function.c:188-306),
//   Txx += dt [ (l+2m) (dxVx + sum_j S_j nx_j dVx) + l (dzVz + sum_j S_j nz_j dVz) ]
//   Tzz += dt [ l (dxVx + ...) + (l+2m) (dzVz + ...) ]
//   Txz += dt m [ dxVz + dzVx + sum_j S_j (nz_j dVx + nx_j dVz) ]
// The trailing blocks of the grid record the receivers (V is final during this kernel).
template <class R, bool KAHAN>
__device__ __forceinline__ void stress_body(const Ops<R>& ops, const MeshDev<R>& m, int lb, long long t) {
  const int S = m.S;
  const long long g = (long long)lb * blockDim.x + threadIdx.x;
  if (g >= (long long)m.K * S) return;
  int e, s;
  if (S == 1) { e = (int)g; s = 0; } else { e = (int)(g / S); s = (int)(g - (long long)e * S); }
  const long long P = m.P;
  R* __restrict__ Ug = m.U + g;

  R vx[NP], vz[NP];
#pragma unroll
  for (int i = 0; i < NP; i++) { vx[i] = Ug[(0 + i) * P]; vz[i] = Ug[(6 + i) * P]; }
  const int4 fc = __ldg(m.face + e);
  const auto gm = ld4(m.geo + e);
  const R rx = gm.x, sx = gm.y, rz = gm.z, sz = gm.w;

  const int codes[3] = {fc.x, fc.y, fc.z};
  R X[NP], Z[NP], W[NP];
  core_strain<ArithOps<R>>(ops, rx, sx, rz, sz, vx, vz, [&](int j, R (&px)[NF], R (&pz)[NF]) {
    const int code = codes[j];
    if (code < 0) {
#pragma unroll
      for (int k = 0; k < NF; k++) { px[k] = R(0); pz[k] = R(0); }
      return;
    }
    const int nb = code >> 4, nf = (code >> 1) & 3, flip = code & 1;
    const R* __restrict__ Un = m.U + ((long long)nb * S + s);
#pragma unroll
    for (int k = 0; k < NF; k++) {
      const int node = face_node(nf, flip ? 2 - k : k);
      px[k] = Un[(0 + node) * P];
      pz[k] = Un[(6 + node) * P];
    }
  }, X, Z, W);

  const auto mt = ld4(m.mat + e);
  const R lam = mt.y, mu = mt.z, l2m = mt.w;
  R txx[NP], tzz[NP], txz[NP], cxx[NP], czz[NP], cxz[NP];
#pragma unroll
  for (int i = 0; i < NP; i++) {
    txx[i] = Ug[(12 + i) * P];
    tzz[i] = Ug[(18 + i) * P];
    txz[i] = Ug[(24 + i) * P];
  }
  if (KAHAN) {
#pragma unroll
    for (int i = 0; i < NP; i++) {
      cxx[i] = m.C[(12 + i) * P + g]; czz[i] = m.C[(18 + i) * P + g]; cxz[i] = m.C[(24 + i) * P + g];
    }
  }
  if (fc.w & 1) {
#pragma unroll
    for (int i = 0; i < NP; i++) {
      const R a = ldg(m.sponge + (long long)i * m.Kp + e);
      txx[i] = v_mul(txx[i], a); tzz[i] = v_mul(tzz[i], a); txz[i] = v_mul(txz[i], a);
      if (KAHAN) { cxx[i] = v_mul(cxx[i], a); czz[i] = v_mul(czz[i], a); cxz[i] = v_mul(cxz[i], a); }
    }
  }
  const R dl2m = v_mul(m.dt, l2m), dlam = v_mul(m.dt, lam), dmu = v_mul(m.dt, mu);
#pragma unroll
  for (int i = 0; i < NP; i++) {
    const R dxx = v_fma(dl2m, X[i], v_mul(dlam, Z[i]));
    const R dzz = v_fma(dlam, X[i], v_mul(dl2m, Z[i]));
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
      m.C[(12 + i) * P + g] = cxx[i]; m.C[(18 + i) * P + g] = czz[i]; m.C[(24 + i) * P + g] = cxz[i];
    }
  }
}

template <class R, bool KAHAN, bool MULTI>
__global__ void __launch_bounds__(256, 2) k_stress(const __grid_constant__ Ops<R> ops,
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
  if (lb >= m.n_elem_blocks) { record(m, lb - m.n_elem_blocks, t); return; }
  stress_body<R, KAHAN>(ops, m, lb, t);
}

}  // namespace dg

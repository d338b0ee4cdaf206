// dg_core.cuh — the arithmetic of one element's two half steps, on register arrays, with every
// operation named (fused or not), so that kernels that feed it from global memory, shared memory
// or another block's messages give the same bits.
//
// An arithmetic A has V (the value of one lane: float, float2 = two shots, or double), R (its
// scalar) and the operator products: ArithP2<V> takes the P2 operators as compile-time constants
// (zeros skipped, +-1 as an add or a subtract: FP32), ArithOps<R> from the kernel's parameter
// bank (the parsed operator files: FP64, and FP32 with other operators).
#pragma once
#include "dg_common.cuh"

namespace dg {

__device__ __forceinline__ float v_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float v_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float v_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float v_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double v_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ double v_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double v_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double v_sub(double a, double b) { return __dsub_rn(a, b); }
// A packed product that feeds a packed sum may come out fused, rounding or not (ptxas): where both
// are meant to round, a branch or a fused operation lies between them.
__device__ __forceinline__ float2 v_fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 v_mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 v_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
// a - b, exactly rounded (b * -1 is exact)
__device__ __forceinline__ float2 v_sub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
// a scalar in every lane of a value
template <class V> struct Bcast;
template <> struct Bcast<float> { static __device__ __forceinline__ float of(float a) { return a; } };
template <> struct Bcast<double> { static __device__ __forceinline__ double of(double a) { return a; } };
template <> struct Bcast<float2> {
  static __device__ __forceinline__ float2 of(float a) { return make_float2(a, a); }
  static __device__ __forceinline__ float2 of(float2 a) { return a; }
};
// one number in every lane of T (a value, or a scalar)
template <class T> __device__ __forceinline__ T v_const(float a) { return T(a); }
template <> __device__ __forceinline__ float2 v_const<float2>(float a) { return make_float2(a, a); }

// h + c x for an operator entry c known at compile time
template <class V> __device__ __forceinline__ V v_axpy_c(float c, V x, V h) {
  if (c == 0.f) return h;
  if (c == 1.f) return v_add(h, x);
  if (c == -1.f) return v_sub(h, x);
  return v_fma(Bcast<V>::of(c), x, h);
}

template <class V_> struct ArithP2 {  // FP32, the P2 operators of the reference triangle
  using V = V_;
  using R = float;
  struct Ops {};
  static __device__ __forceinline__ Ops ops(const dg::Ops<float>&) { return {}; }
  static __device__ __forceinline__ V dr(const Ops&, int i, int n, V x, V h) { return v_axpy_c(p2_dr(i * NP + n), x, h); }
  static __device__ __forceinline__ V ds(const Ops&, int i, int n, V x, V h) { return v_axpy_c(p2_ds(i * NP + n), x, h); }
  static __device__ __forceinline__ V lift(const Ops&, int j, int i, int k, V x, V h) {
    return v_axpy_c(p2_lift((j * NP + i) * NF + k), x, h);
  }
};

template <class R_> struct ArithOps {  // operators from the parameter bank
  using V = R_;
  using R = R_;
  using Ops = dg::Ops<R>;
  static __device__ __forceinline__ const Ops& ops(const Ops& o) { return o; }
  static __device__ __forceinline__ V dr(const Ops& o, int i, int n, V x, V h) { return v_fma(o.Dr[i * NP + n], x, h); }
  static __device__ __forceinline__ V ds(const Ops& o, int i, int n, V x, V h) { return v_fma(o.Ds[i * NP + n], x, h); }
  static __device__ __forceinline__ V lift(const Ops& o, int j, int i, int k, V x, V h) {
    return v_fma(o.L[(j * NP + i) * NF + k], x, h);
  }
};

// Outward normal of face j times |face| / (4 J) from the inverse Jacobian (rx, sx, rz, sz):
// (-sx,-sz)/2, (rx+sx,rz+sz)/2, (-rx,-rz)/2 — the reference's Q / A (fun_DG.c:1118-1131).  T: a
// scalar (the lanes share the element) or a value (two elements).
template <class T>
__device__ __forceinline__ void face_normal(int j, T rx, T sx, T rz, T sz, T& nx, T& nz) {
  const T h = v_const<T>(0.5f), mh = v_const<T>(-0.5f);
  if (j == 0) { nx = v_mul(mh, sx); nz = v_mul(mh, sz); }
  else if (j == 1) { nx = v_mul(h, v_add(rx, sx)); nz = v_mul(h, v_add(rz, sz)); }
  else { nx = v_mul(mh, rx); nz = v_mul(mh, rz); }
}

// The velocity right-hand side, both directions:
//   hx = Dr (rx Txx + rz Txz) + Ds (sx Txx + sz Txz) + sum_j S_j (nx_j dTxx + nz_j dTxz)
//   hz = Dr (rx Txz + rz Tzz) + Ds (sx Txz + sz Tzz) + sum_j S_j (nz_j dTzz + nx_j dTxz)
// The faces come first (face by face, so that few neighbour values are held at a time), then the
// volume; the other order costs the wavefront step 2.5 % and FP32-Kahan on one shot 6 %.
template <class A, class T>
__device__ __forceinline__ void core_velocity_volume(const typename A::Ops& ops, T rx_, T sx_, T rz_, T sz_,
                                                     const typename A::V (&txx)[NP], const typename A::V (&tzz)[NP],
                                                     const typename A::V (&txz)[NP], typename A::V (&hx)[NP],
                                                     typename A::V (&hz)[NP]) {
  using V = typename A::V;
  const V rx = Bcast<V>::of(rx_), sx = Bcast<V>::of(sx_), rz = Bcast<V>::of(rz_), sz = Bcast<V>::of(sz_);
  V a[NP], b[NP], c[NP], d[NP];
#pragma unroll
  for (int n = 0; n < NP; n++) {
    a[n] = v_fma(rx, txx[n], v_mul(rz, txz[n]));
    b[n] = v_fma(sx, txx[n], v_mul(sz, txz[n]));
    c[n] = v_fma(rx, txz[n], v_mul(rz, tzz[n]));
    d[n] = v_fma(sx, txz[n], v_mul(sz, tzz[n]));
  }
#pragma unroll
  for (int i = 0; i < NP; i++) {
#pragma unroll
    for (int n = 0; n < NP; n++) {
      hx[i] = A::dr(ops, i, n, a[n], hx[i]);
      hz[i] = A::dr(ops, i, n, c[n], hz[i]);
      hx[i] = A::ds(ops, i, n, b[n], hx[i]);
      hz[i] = A::ds(ops, i, n, d[n], hz[i]);
    }
  }
}
// The terms of face j: pxx, pzz, pxz are the neighbour's stresses at the face's nodes in this
// element's order, the neighbour's sponge factor applied (zeros across an outer face).
template <class A, class T>
__device__ __forceinline__ void core_velocity_face(const typename A::Ops& ops, int j, T rx, T sx, T rz, T sz,
                                                   const typename A::V (&txx)[NP], const typename A::V (&tzz)[NP],
                                                   const typename A::V (&txz)[NP], const typename A::V (&pxx)[NF],
                                                   const typename A::V (&pzz)[NF], const typename A::V (&pxz)[NF],
                                                   typename A::V (&hx)[NP], typename A::V (&hz)[NP]) {
  using V = typename A::V;
  T nxs, nzs;
  face_normal(j, rx, sx, rz, sz, nxs, nzs);
  const V nx = Bcast<V>::of(nxs), nz = Bcast<V>::of(nzs);
  V fx[NF], fz[NF];
#pragma unroll
  for (int k = 0; k < NF; k++) {
    const int own = face_node(j, k);
    const V dxx = v_sub(pxx[k], txx[own]), dzz = v_sub(pzz[k], tzz[own]), dxz = v_sub(pxz[k], txz[own]);
    fx[k] = v_fma(nx, dxx, v_mul(nz, dxz));
    fz[k] = v_fma(nz, dzz, v_mul(nx, dxz));
  }
#pragma unroll
  for (int i = 0; i < NP; i++)
#pragma unroll
    for (int k = 0; k < NF; k++) {
      hx[i] = A::lift(ops, j, i, k, fx[k], hx[i]);
      hz[i] = A::lift(ops, j, i, k, fz[k], hz[i]);
    }
}
// Both, gather(j, pxx, pzz, pxz) giving the neighbour's values.
template <class A, class T, class G>
__device__ __forceinline__ void core_velocity_rhs(const typename A::Ops& ops, T rx, T sx, T rz, T sz,
                                                  const typename A::V (&txx)[NP], const typename A::V (&tzz)[NP],
                                                  const typename A::V (&txz)[NP], G&& gather, typename A::V (&hx)[NP],
                                                  typename A::V (&hz)[NP]) {
#pragma unroll
  for (int i = 0; i < NP; i++) { hx[i] = v_const<typename A::V>(0.f); hz[i] = hx[i]; }
#pragma unroll
  for (int j = 0; j < NF; j++) {
    typename A::V pxx[NF], pzz[NF], pxz[NF];
    gather(j, pxx, pzz, pxz);
    core_velocity_face<A>(ops, j, rx, sx, rz, sz, txx, tzz, txz, pxx, pzz, pxz, hx, hz);
  }
  core_velocity_volume<A>(ops, rx, sx, rz, sz, txx, tzz, txz, hx, hz);
}

// The strain rates of the stress update, volume terms (which need no neighbour) and then faces:
//   X = dx Vx + sum_j S_j nx_j dVx, Z = dz Vz + sum_j S_j nz_j dVz,
//   W = dx Vz + dz Vx + sum_j S_j (nz_j dVx + nx_j dVz)
template <class A, class T>
__device__ __forceinline__ void core_strain_volume(const typename A::Ops& ops, T rx_, T sx_, T rz_, T sz_,
                                                   const typename A::V (&vx)[NP], const typename A::V (&vz)[NP],
                                                   typename A::V (&X)[NP], typename A::V (&Z)[NP],
                                                   typename A::V (&W)[NP]) {
  using V = typename A::V;
  const V rx = Bcast<V>::of(rx_), sx = Bcast<V>::of(sx_), rz = Bcast<V>::of(rz_), sz = Bcast<V>::of(sz_);
#pragma unroll
  for (int i = 0; i < NP; i++) {
    V drx = v_const<V>(0.f), dsx = drx, drz = drx, dsz = drx;
#pragma unroll
    for (int n = 0; n < NP; n++) {
      drx = A::dr(ops, i, n, vx[n], drx);
      drz = A::dr(ops, i, n, vz[n], drz);
      dsx = A::ds(ops, i, n, vx[n], dsx);
      dsz = A::ds(ops, i, n, vz[n], dsz);
    }
    X[i] = v_fma(rx, drx, v_mul(sx, dsx));
    Z[i] = v_fma(rz, drz, v_mul(sz, dsz));
    W[i] = v_fma(rx, drz, v_fma(sx, dsz, v_fma(rz, drx, v_mul(sz, dsx))));
  }
}
// The terms of face j: px, pz are the neighbour's velocities at the face's nodes in this
// element's order (zeros across an outer face).
template <class A, class T>
__device__ __forceinline__ void core_strain_face(const typename A::Ops& ops, int j, T rx, T sx, T rz, T sz,
                                                 const typename A::V (&vx)[NP], const typename A::V (&vz)[NP],
                                                 const typename A::V (&px)[NF], const typename A::V (&pz)[NF],
                                                 typename A::V (&X)[NP], typename A::V (&Z)[NP],
                                                 typename A::V (&W)[NP]) {
  using V = typename A::V;
  T nxs, nzs;
  face_normal(j, rx, sx, rz, sz, nxs, nzs);
  const V nx = Bcast<V>::of(nxs), nz = Bcast<V>::of(nzs);
  V fa[NF], fb[NF], fw[NF];
#pragma unroll
  for (int k = 0; k < NF; k++) {
    const int own = face_node(j, k);
    const V dvx = v_sub(px[k], vx[own]), dvz = v_sub(pz[k], vz[own]);
    fa[k] = v_mul(nx, dvx);
    fb[k] = v_mul(nz, dvz);
    fw[k] = v_fma(nz, dvx, v_mul(nx, dvz));
  }
#pragma unroll
  for (int i = 0; i < NP; i++)
#pragma unroll
    for (int k = 0; k < NF; k++) {
      X[i] = A::lift(ops, j, i, k, fa[k], X[i]);
      Z[i] = A::lift(ops, j, i, k, fb[k], Z[i]);
      W[i] = A::lift(ops, j, i, k, fw[k], W[i]);
    }
}
// Both, gather(j, px, pz) giving the neighbour's values.
template <class A, class T, class G>
__device__ __forceinline__ void core_strain(const typename A::Ops& ops, T rx, T sx, T rz, T sz,
                                            const typename A::V (&vx)[NP], const typename A::V (&vz)[NP], G&& gather,
                                            typename A::V (&X)[NP], typename A::V (&Z)[NP], typename A::V (&W)[NP]) {
  core_strain_volume<A>(ops, rx, sx, rz, sz, vx, vz, X, Z, W);
#pragma unroll
  for (int j = 0; j < NF; j++) {
    typename A::V px[NF], pz[NF];
    gather(j, px, pz);
    core_strain_face<A>(ops, j, rx, sx, rz, sz, vx, vz, px, pz, X, Z, W);
  }
}

// Kahan-compensated u += d with compensation c
template <class V> __device__ __forceinline__ void v_kahan(V& u, V& c, V d) {
  const V y = v_sub(d, c);
  const V t = v_add(u, y);
  c = v_sub(v_sub(t, u), y);
  u = t;
}

}  // namespace dg

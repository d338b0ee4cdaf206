// dg_step_resident.cuh — many time steps of one mesh in one launch, the wave field resident on the
// SMs: one thread per lane (an element's shot, or pair of shots), its values in registers.
//
// Each block owns a run of consecutive elements (locality order).  A copy of its fields in shared
// memory serves the neighbours inside the block; what a neighbouring block needs crosses the GPU
// as messages: for every face between two blocks the owner sends, after each half step, the
// face's three nodes' velocities or stresses as 16-byte messages of three words and a tag (the
// step they belong to), and the receiving block polls the messages themselves and lays the
// values out beside its own lanes, so the gathers of all faces are alike.  A 16-byte access is
// single-copy atomic, so a message with the right tag is whole: no fence, no flag of its own and
// no grid barrier.  One buffer per face and half is enough: a block overwrites a velocity message
// only after the barrier behind which it has received that neighbour's next stresses, which the
// neighbour sent behind the barrier after it had received the velocities (and the same the other
// way round).  A half step has one block barrier, before its gathers; the stress half's volume
// terms, which need the element's own values only, run while the messages are on their way.
//
// A small mesh's step is bound by latency, not by bandwidth: as two launches a step, a
// 20,000-element one-shot mesh takes about 10 us a step whatever its arithmetic, most of it
// launch gaps, the round trips for codes, geometry and neighbour values, and the tail.
//
// The grid is cooperative (all blocks resident), so every wait ends; each wait is bounded all the
// same: past the limit, or once another block gave up, the thread sets the error word (in host
// memory) and polls no more, so the launch ends and the host reports the error.
#pragma once
#include "dg_common.cuh"
#include "dg_core.cuh"
#include "dg_step_ref.cuh"

namespace dg {

struct Resident {
  int nls;               // plane stride in shared memory: lanes of the largest block, its message lanes,
                         // and a lane of zeros (the last)
  int nl;                // lanes of the largest block: where the message lanes begin
  int H;                 // lanes per element
  const int* e_start;    // [blocks + 1] first element of each block
  const int* s_start;    // [blocks + 1] first message slot of each block
  const int4* link;      // [K] faces: local neighbour << 4 | sponge << 3 | face << 1 | flip (elements counted
                         // from the block's first), -1 outer, -2 - (2 slot + flip) in another block (slots
                         // counted from the block's first); w: bit 0 sponge, bit 1 some face in another block
  const int4* out;       // [K] message slot at the neighbour for each such face, -1 otherwise
  uint4* pt;             // stress messages [message][slot * H + lane]
  uint4* pv;             // velocity messages
  long long ps;          // message stride: slots * H
  const int* rec_start;  // [blocks + 1] receivers of each block:
  const int* rec_list;   //   rec_list[rec_start[b] .. rec_start[b+1])
  int* error;
  unsigned* arrived;     // blocks that have read the step counter (0 between launches)
  unsigned spin_limit;
};

// 16 bytes at once, coherent at gpu scope
__device__ __forceinline__ uint4 ld_msg(const uint4* p) {
  unsigned long long a, b;
  asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
               : "=l"(a), "=l"(b) : "l"(p) : "memory");
  return make_uint4((unsigned)a, (unsigned)(a >> 32), (unsigned)b, (unsigned)(b >> 32));
}
__device__ __forceinline__ void st_msg(uint4* p, unsigned x, unsigned y, unsigned z, unsigned tag) {
  const unsigned long long a = x | (unsigned long long)y << 32, b = z | (unsigned long long)tag << 32;
  asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }"
               ::"l"(p), "l"(a), "l"(b) : "memory");
}

// values as 32-bit words
__device__ __forceinline__ void to_words(float v, unsigned* w) { w[0] = __float_as_uint(v); }
__device__ __forceinline__ void to_words(float2 v, unsigned* w) {
  w[0] = __float_as_uint(v.x);
  w[1] = __float_as_uint(v.y);
}
__device__ __forceinline__ void to_words(double v, unsigned* w) {
  w[0] = (unsigned)__double2loint(v);
  w[1] = (unsigned)__double2hiint(v);
}
__device__ __forceinline__ void of_words(float& v, const unsigned* w) { v = __uint_as_float(w[0]); }
__device__ __forceinline__ void of_words(float2& v, const unsigned* w) {
  v = make_float2(__uint_as_float(w[0]), __uint_as_float(w[1]));
}
__device__ __forceinline__ void of_words(double& v, const unsigned* w) { v = __hiloint2double((int)w[1], (int)w[0]); }

// N values (a multiple of three words) as messages at p, p + stride, ...
template <int N, class V>
__device__ __forceinline__ void send_msgs(uint4* p, long long stride, unsigned tag, const V (&v)[N]) {
  constexpr int WV = sizeof(V) / 4, W = N * WV;
  static_assert(W % 3 == 0, "whole messages");
  unsigned w[W];
#pragma unroll
  for (int i = 0; i < N; i++) to_words(v[i], w + i * WV);
#pragma unroll
  for (int i = 0; i < W / 3; i++) st_msg(p + i * stride, w[3 * i], w[3 * i + 1], w[3 * i + 2], tag);
}
template <int N, class V>
__device__ __forceinline__ void recv_msgs(const uint4* p, long long stride, unsigned tag, const Resident& w, bool& dead,
                                          V (&v)[N]) {
  constexpr int WV = sizeof(V) / 4, W = N * WV;
  uint4 m[W / 3];
  unsigned spins = 0;
  for (;;) {
    bool ok = true;
#pragma unroll
    for (int i = 0; i < W / 3; i++) m[i] = ld_msg(p + i * stride);
#pragma unroll
    for (int i = 0; i < W / 3; i++) ok &= m[i].w == tag;
    if (ok || dead) break;
    if (++spins > w.spin_limit || ((spins & 255u) == 0 && (ld_volatile_i32(w.error) != 0))) {
      *(volatile int*)w.error = 1;
      dead = true;
    }
  }
  unsigned u[W];
#pragma unroll
  for (int i = 0; i < W / 3; i++) { u[3 * i] = m[i].x; u[3 * i + 1] = m[i].y; u[3 * i + 2] = m[i].z; }
#pragma unroll
  for (int i = 0; i < N; i++) of_words(v[i], u + i * WV);
}

// Sends the velocities or stresses of the faces that lie in other blocks.
template <class V>
__device__ __forceinline__ void send_velocity(const Resident& w, const int (&slot)[NF], int q, unsigned tag,
                                              const V (&vx)[NP], const V (&vz)[NP]) {
#pragma unroll
  for (int j = 0; j < NF; j++) {
    if (slot[j] < 0) continue;
    V v[6];
#pragma unroll
    for (int k = 0; k < NF; k++) { v[2 * k] = vx[face_node(j, k)]; v[2 * k + 1] = vz[face_node(j, k)]; }
    send_msgs(w.pv + (long long)slot[j] * w.H + q, w.ps, tag, v);
  }
}
template <class V>
__device__ __forceinline__ void send_stress(const Resident& w, const int (&slot)[NF], int q, unsigned tag,
                                            const V (&txx)[NP], const V (&tzz)[NP], const V (&txz)[NP]) {
#pragma unroll
  for (int j = 0; j < NF; j++) {
    if (slot[j] < 0) continue;
    V v[9];
#pragma unroll
    for (int k = 0; k < NF; k++) {
      const int n = face_node(j, k);
      v[3 * k] = txx[n]; v[3 * k + 1] = tzz[n]; v[3 * k + 2] = txz[n];
    }
    send_msgs(w.pt + (long long)slot[j] * w.H + q, w.ps, tag, v);
  }
}

// the mesh's state as lanes of V: value (e, plane, lane q)
template <class V, class R>
__device__ __forceinline__ V* state_at(R* U, const MeshDev<R>& m, int e, int plane, int q) {
  return reinterpret_cast<V*>(U + (long long)e * m.ES + plane * m.PS) + q;
}

// The reference's own operators and operation order (DG_FP64_REF), for k_step_resident.
struct ArithRef {
  using V = double;
  using R = double;
  using Ops = dg::Ops<double>;
};
template <class A> constexpr bool is_ref = false;
template <> constexpr bool is_ref<ArithRef> = true;

// `nsteps` steps from step t0, or, COUNT (the device's counter may be ahead of the host: a caller replays
// captured steps), from the step the counter holds, as the other forms of the step take it.  There the
// blocks count themselves, and the last to have read the counter advances it.  An instance of its own:
// reading the counter costs a one-step call of 17 us 0.5 us, a run-time choice 0.3.  The stresses held between two steps carry the sponge factor of
// the coming step already (those in global memory do not), so neighbours read them as they are;
// the stress tag of step s is seq + s, the velocity tag seq + s + 1.
template <class A, bool KAHAN, int MAXT, bool COUNT>
__global__ void __launch_bounds__(MAXT, 1) k_step_resident(const __grid_constant__ typename A::Ops ops,
                                                           const __grid_constant__ MeshDev<typename A::R> m,
                                                           const __grid_constant__ Resident w,
                                                           Counters* __restrict__ ctr, long long t0, int nsteps,
                                                           unsigned seq) {
  using V = typename A::V;
  using R = typename A::R;
  constexpr int SV = sizeof(V) / sizeof(R);  // shots of a lane
  constexpr bool REF = is_ref<A>;
  if constexpr (COUNT) {
    t0 = *(volatile const long long*)&ctr->v;
    nsteps = (int)min((long long)nsteps, m.steps - t0);
    if (nsteps <= 0) return;
  }
  extern __shared__ __align__(16) unsigned char res_smem[];
  V* const sV = reinterpret_cast<V*>(res_smem);  // [12][nls] Vx, Vz
  V* const sT = sV + 12 * w.nls;                 // [18][nls] Txx, Tzz, Txz, sponge factor applied
  const int nls = w.nls, H = w.H, l = threadIdx.x;
  const int e0 = __ldg(w.e_start + blockIdx.x), NL = (__ldg(w.e_start + blockIdx.x + 1) - e0) * H;
  const int s0 = __ldg(w.s_start + blockIdx.x) * H, NG = __ldg(w.s_start + blockIdx.x + 1) * H - s0;
  const int r0 = __ldg(w.rec_start + blockIdx.x) * H, r1 = __ldg(w.rec_start + blockIdx.x + 1) * H;
  const bool mine = l < NL;
  bool dead = false;
  // the lane's element: geometry, materials, where its faces' neighbours lie, its values
  const int el = mine ? l / H : 0, q = mine ? l - el * H : 0, e = e0 + el;
  const int4 lk = __ldg(w.link + e), ot = __ldg(w.out + e);
  const int slot[NF] = {ot.x, ot.y, ot.z};
  const auto gm = ld4(m.geo + e);
  const auto mt = ld4(m.mat + e);
  const R rx = gm.x, sx = gm.y, rz = gm.z, sz = gm.w;
  const R step = v_mul(m.dt, mt.x), dl2m = v_mul(m.dt, mt.w), dlam = v_mul(m.dt, mt.y), dmu = v_mul(m.dt, mt.z);
  const bool sponge = lk.w & 1, sends = mine && (lk.w & 2);
  int src = 0;
  unsigned short at[NF][NF];  // of face j, node k: node plane and lane of the neighbour's value
  {
    const int codes[NF] = {lk.x, lk.y, lk.z};
#pragma unroll
    for (int j = 0; j < NF; j++) {
      const int c = codes[j];
#pragma unroll
      for (int k = 0; k < NF; k++) {
        int a = nls - 1;  // outer face: zeros
        if (c >= 0) a = face_node((c >> 1) & 3, (c & 1) ? 2 - k : k) * nls + (c >> 4) * H + q;
        else if (c < -1) a = (((-2 - c) & 1) ? 2 - k : k) * nls + w.nl + ((-2 - c) >> 1) * H + q;
        at[j][k] = (unsigned short)a;
      }
    }
#pragma unroll
    for (int c = 0; c < SV; c++)
      if (mine && __ldg(m.src_elem + q * SV + c) == e) src |= 1 << c;
  }
  V vx[NP], vz[NP], txx[NP], tzz[NP], txz[NP], cc[KAHAN ? 30 : 1];
#pragma unroll
  for (int i = 0; i < NP; i++) {
    vx[i] = *state_at<V>(m.U, m, e, i, q);
    vz[i] = *state_at<V>(m.U, m, e, 6 + i, q);
    txx[i] = *state_at<V>(m.U, m, e, 12 + i, q);
    tzz[i] = *state_at<V>(m.U, m, e, 18 + i, q);
    txz[i] = *state_at<V>(m.U, m, e, 24 + i, q);
    if (sponge) {
      const V a = Bcast<V>::of(ldg(m.sponge + (long long)i * m.Kp + e));
      txx[i] = v_mul(txx[i], a); tzz[i] = v_mul(tzz[i], a); txz[i] = v_mul(txz[i], a);
    }
    if (mine) { sT[i * nls + l] = txx[i]; sT[(6 + i) * nls + l] = tzz[i]; sT[(12 + i) * nls + l] = txz[i]; }
  }
  if constexpr (KAHAN) {
#pragma unroll
    for (int p = 0; p < 30; p++) cc[p] = *state_at<V>(m.C, m, e, p, q);
  }
  for (int p = threadIdx.x; p < 30; p += blockDim.x) sV[p * nls + nls - 1] = v_const<V>(0.f);
  if (sends) send_stress(w, slot, q, seq, txx, tzz, txz);
  // message units are taken from the block's last thread down: the threads past the lanes first
  const int u0 = (int)blockDim.x - 1 - l;
  for (int s = 0; s < nsteps; s++) {
    const long long t = t0 + s;
    const unsigned tag_t = seq + (unsigned)s, tag_v = tag_t + 1u;
    // ---- velocity half: sponge, source, V += dt L_V(T) ----
    {
      V hx[NP], hz[NP];
      if constexpr (REF)
        if (mine) ref_velocity_volume<false>(ops, m, e, txx, tzz, txz, hx, hz);
      for (int u = u0; u < NG; u += blockDim.x) {
        V v[9];
        recv_msgs(w.pt + s0 + u, w.ps, tag_t, w, dead, v);
        V* g = sT + w.nl + u;
#pragma unroll
        for (int k = 0; k < NF; k++)
#pragma unroll
          for (int f = 0; f < 3; f++) g[(f * NP + k) * nls] = v[3 * k + f];
      }
      __syncthreads();
      if constexpr (COUNT) {
        if (s == 0 && l == 0 && atomicAdd(w.arrived, 1u) == gridDim.x - 1) {
          *w.arrived = 0;
          ctr->v = t0 + nsteps;
          ctr->s = t0 + nsteps - 1;
        }
      }
      if (mine) {
        if constexpr (!REF) {
#pragma unroll
          for (int i = 0; i < NP; i++) { hx[i] = v_const<V>(0.f); hz[i] = hx[i]; }
        }
#pragma unroll
        for (int j = 0; j < NF; j++) {
          V pxx[NF], pzz[NF], pxz[NF];
#pragma unroll
          for (int k = 0; k < NF; k++) {
            const V* p = sT + at[j][k];
            pxx[k] = p[0];
            pzz[k] = p[6 * nls];
            pxz[k] = p[12 * nls];
          }
          if constexpr (REF) ref_velocity_face(ops, m, e, j, txx, tzz, txz, pxx, pzz, pxz, hx, hz);
          else core_velocity_face<A>(ops, j, rx, sx, rz, sz, txx, tzz, txz, pxx, pzz, pxz, hx, hz);
        }
        if constexpr (!REF) core_velocity_volume<A>(ops, rx, sx, rz, sz, txx, tzz, txz, hx, hz);
        if (sponge) {
#pragma unroll
          for (int i = 0; i < NP; i++) {
            const V a = Bcast<V>::of(ldg(m.sponge + (long long)i * m.Kp + e));
            vx[i] = v_mul(vx[i], a);
            vz[i] = v_mul(vz[i], a);
            if constexpr (KAHAN) { cc[i] = v_mul(cc[i], a); cc[6 + i] = v_mul(cc[6 + i], a); }
          }
        }
        V sv[NP];
#pragma unroll
        for (int i = 0; i < NP; i++) sv[i] = v_const<V>(0.f);
        if (src) {
          const R wt = (R)__ldg(m.wavelet + t);
#pragma unroll
          for (int i = 0; i < NP; i++) {
            R x[SV];
#pragma unroll
            for (int c = 0; c < SV; c++)
              x[c] = (src >> c) & 1 ? v_mul(ldg(m.src_fun + (q * SV + c) * NP + i), wt) : R(0);
            if constexpr (SV == 2) sv[i] = make_float2(x[0], x[1]);
            else sv[i] = x[0];
          }
        }
        const V st = Bcast<V>::of(step);
#pragma unroll
        for (int i = 0; i < NP; i++) {
          if constexpr (KAHAN) {
            v_kahan(vx[i], cc[i], v_mul(st, hx[i]));
            v_kahan(vz[i], cc[6 + i], v_fma(st, hz[i], sv[i]));
          } else if constexpr (REF) {
            if (src) vz[i] = v_add(vz[i], sv[i]);
            vx[i] = v_add(v_mul(hx[i], m.dt), vx[i]);
            vz[i] = v_add(v_mul(hz[i], m.dt), vz[i]);
          } else {
            vx[i] = v_fma(st, hx[i], vx[i]);
            vz[i] = v_fma(st, hz[i], v_add(vz[i], sv[i]));
          }
        }
        if (sends) send_velocity(w, slot, q, tag_v, vx, vz);
#pragma unroll
        for (int i = 0; i < NP; i++) { sV[i * nls + l] = vx[i]; sV[(6 + i) * nls + l] = vz[i]; }
      }
    }
    // ---- stress half: T = a T + dt L_T(V) ----
    {
      V X[NP], Z[NP], W[NP];
      if (mine) {
        if constexpr (REF) ref_stress_volume<false>(ops, m, e, vx, vz, X, Z, W);
        else core_strain_volume<A>(ops, rx, sx, rz, sz, vx, vz, X, Z, W);
      }
      for (int u = u0; u < NG; u += blockDim.x) {
        V v[6];
        recv_msgs(w.pv + s0 + u, w.ps, tag_v, w, dead, v);
        V* g = sV + w.nl + u;
#pragma unroll
        for (int k = 0; k < NF; k++)
#pragma unroll
          for (int f = 0; f < 2; f++) g[(f * NP + k) * nls] = v[2 * k + f];
      }
      __syncthreads();
      if (mine) {
#pragma unroll
        for (int j = 0; j < NF; j++) {
          V px[NF], pz[NF];
#pragma unroll
          for (int k = 0; k < NF; k++) {
            const V* p = sV + at[j][k];
            px[k] = p[0];
            pz[k] = p[6 * nls];
          }
          if constexpr (REF) ref_stress_face(ops, m, e, j, vx, vz, px, pz, X, Z, W);
          else core_strain_face<A>(ops, j, rx, sx, rz, sz, vx, vz, px, pz, X, Z, W);
        }
        const V a2 = Bcast<V>::of(dl2m), al = Bcast<V>::of(dlam), am = Bcast<V>::of(dmu);
        const bool last = s == nsteps - 1;
#pragma unroll
        for (int i = 0; i < NP; i++) {
          const V dxx = v_fma(a2, X[i], v_mul(al, Z[i]));
          const V dzz = v_fma(al, X[i], v_mul(a2, Z[i]));
          V a{};
          if (sponge) a = Bcast<V>::of(ldg(m.sponge + (long long)i * m.Kp + e));
          if constexpr (KAHAN) {
            if (sponge) { cc[12 + i] = v_mul(cc[12 + i], a); cc[18 + i] = v_mul(cc[18 + i], a); cc[24 + i] = v_mul(cc[24 + i], a); }
            v_kahan(txx[i], cc[12 + i], dxx);
            v_kahan(tzz[i], cc[18 + i], dzz);
            v_kahan(txz[i], cc[24 + i], v_mul(am, W[i]));
          } else if constexpr (REF) {  // X, Z, W are the three stresses' rates
            txx[i] = v_add(v_mul(X[i], m.dt), txx[i]);
            tzz[i] = v_add(v_mul(Z[i], m.dt), tzz[i]);
            txz[i] = v_add(v_mul(W[i], m.dt), txz[i]);
          } else {
            txx[i] = v_add(txx[i], dxx);
            tzz[i] = v_add(tzz[i], dzz);
            txz[i] = v_fma(am, W[i], txz[i]);
          }
          if (sponge && !last) { txx[i] = v_mul(txx[i], a); tzz[i] = v_mul(tzz[i], a); txz[i] = v_mul(txz[i], a); }
        }
        if (!last) {
          if (sends) send_stress(w, slot, q, tag_v, txx, tzz, txz);
#pragma unroll
          for (int i = 0; i < NP; i++) {
            sT[i * nls + l] = txx[i]; sT[(6 + i) * nls + l] = tzz[i]; sT[(12 + i) * nls + l] = txz[i];
          }
        }
      }
      // receivers: sV holds this step's velocities until the next velocity half's barrier
      for (int k = r0 + l; k < r1; k += blockDim.x) {
        const int rq = k % H, r = __ldg(w.rec_list + k / H);
        const V* p = sV + __ldg(m.rec_node + r) * nls + (__ldg(m.rec_elem + r) - e0) * H + rq;
        R* tr = m.trace + ((t * 2) * (long long)m.n_rec + r) * m.S;
        reinterpret_cast<V*>(tr)[rq] = p[0];
        reinterpret_cast<V*>(tr + (long long)m.n_rec * m.S)[rq] = p[6 * nls];
      }
    }
  }
  if (mine) {
#pragma unroll
    for (int i = 0; i < NP; i++) {
      *state_at<V>(m.U, m, e, i, q) = vx[i];
      *state_at<V>(m.U, m, e, 6 + i, q) = vz[i];
      *state_at<V>(m.U, m, e, 12 + i, q) = txx[i];
      *state_at<V>(m.U, m, e, 18 + i, q) = tzz[i];
      *state_at<V>(m.U, m, e, 24 + i, q) = txz[i];
    }
    if constexpr (KAHAN) {
#pragma unroll
      for (int p = 0; p < 30; p++) *state_at<V>(m.C, m, e, p, q) = cc[p];
    }
  }
  if (!COUNT && blockIdx.x == 0 && threadIdx.x == 0) {
    ctr->v = t0 + nsteps;
    ctr->s = t0 + nsteps - 1;
  }
}

}  // namespace dg

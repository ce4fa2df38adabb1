// sweep_common.cuh -- pieces shared by the pair sweeps (pair_kernels.cu,
// sweep32.cu): the Oldroyd-B and colloid arrays handed to the sweeps, the
// boundary particles' rigid velocity, the per-particle pair records written
// after the density sum, the block-shared stencil-slot offsets, and the
// force epilogue (body force, store, second half kick, Oldroyd-B update).
#pragma once
#include "mcfg_internal.cuh"
#include "pair_common.cuh"
#include "sph.cuh"

namespace mcfg {

// Oldroyd-B arrays handed to the sweeps (all null for a Newtonian run).
struct NN {
  const double* ct;  // conformation tensor [d*d][n]
  double* act;       // d(ct)/dt [d*d][n]
  double* vgt;       // velocity gradient [d*d][n]
  void* qq;          // 1/n and G*ct/n^2, [1+d*d][n] in the path's type
};

// colloid arrays handed to the sweeps
struct CollArgs {
  double4_32a* v;      // state velocity (boundary particles get the rigid one)
  double4_32a* rxc;    // FP64 path: boundary particle - colloid image centre
  float4* rxcf;        // FP32 path: same
};

// particles_set_colloid_velocity.F90:73-95 with colloid_particle_velocity.F90:
// the boundary particle moves with its colloid, V + Omega x rx.  Also keeps
// rx for the no-slip pair term.  Returns the new velocity.
template <int D>
__device__ __forceinline__ double4_32a colloid_particle_update(const Consts& k, int i, int si,
                                                               const double4_32a& xi4,
                                                               const CollArgs& ca) {
  const double x[3] = {xi4.x, xi4.y, xi4.z};
  double rx[3] = {0.0, 0.0, 0.0};
  colloid_rx<D>(k, x, si - 1, rx);
  if (ca.rxc) ca.rxc[i] = make_double4_32a(rx[0], rx[1], rx[2], 0.0);
  if (ca.rxcf) ca.rxcf[i] = make_float4((float)rx[0], (float)rx[1], (float)rx[2], 0.f);
  double vn[3] = {0.0, 0.0, 0.0};
  if (k.coll_translate || k.coll_rotate) {
    const double* cd = k.coll + (size_t)(si - 1) * 12;
    vn[0] = cd[3];
    vn[1] = cd[4];
    vn[2] = D == 3 ? cd[5] : 0.0;
    if (k.coll_rotate) {
      const double r3[3] = {rx[0], rx[1], D == 3 ? rx[2] : 0.0};
      const double om[3] = {cd[6], cd[7], cd[8]};
      double w[3];
      cross3t<double>(om, r3, w);
#pragma unroll
      for (int a = 0; a < D; ++a) vn[a] += w[a];
    }
  }
  const double4_32a out = make_double4_32a(vn[0], vn[1], D == 3 ? vn[2] : 0.0, 0.0);
  ca.v[i] = out;
  return out;
}

// Per-particle prologue of the force sweep: pressure from the equation of
// state and the pair coefficients (fused into the density sweeps or run as
// k_pressure).  The FP32 path forms them in FP32.
template <bool FP64>
__device__ __forceinline__ void write_particle_records(const Consts& k, int i, double rho, double m,
                                                       int pid, const double4_32a& v,
                                                       double* __restrict__ pr,
                                                       double4_32a* __restrict__ pc,
                                                       float4* __restrict__ pcf,
                                                       float4* __restrict__ vf, const NN& nn) {
  if (!k.newtonian) {
    // Oldroyd-B: pressure tensor (p + G) I - G c
    // (particles_compute_pressure_tensor.F90:88-133) as A = (p + G)/n^2 and
    // Q = G c / n^2, with 1/n for the velocity gradient
    const double r_eos = (k.rhs_density_type == 1) ? rho : rho * m;
    const double p = eos_pressure(k, r_eos);
    pr[i] = p;
    const double inv = 1.0 / rho;
    const double inv2 = inv * inv;
    const int n = k.n, d2 = k.d * k.d;
    if (FP64) {
      pc[i] = make_double4_32a((p + k.G) * inv2, inv2, 1.0 / m, p);
      double* q = (double*)nn.qq;
      q[i] = inv;
      for (int cc = 0; cc < d2; ++cc) q[(size_t)(1 + cc) * n + i] = k.G * nn.ct[(size_t)cc * n + i] * inv2;
    } else {
      pcf[2 * i] = make_float4((float)((p + k.G) * inv2), (float)inv2, (float)(1.0 / m), (float)p);
      vf[2 * i] = make_float4((float)v.x, (float)v.y, (float)v.z, __int_as_float(pid));
      float* q = (float*)nn.qq;
      q[i] = (float)inv;
      for (int cc = 0; cc < d2; ++cc)
        q[(size_t)(1 + cc) * n + i] = (float)(k.G * nn.ct[(size_t)cc * n + i] * inv2);
    }
    return;
  }
  if (FP64) {
    const double r_eos = (k.rhs_density_type == 1) ? rho : rho * m;
    const double p = eos_pressure(k, r_eos);
    pr[i] = p;
    pc[i] = pair_coeffs(k, rho, p, m);
  } else {
    // conversions on the integer pipe (narrow, widen: the same roundings)
    const float rf = narrow(rho), mf = narrow(m);
    const float r_eos = (k.rhs_density_type == 1) ? rf : rf * mf;
    float p;
    if (k.eos_type == 1) {
      const float rg = (k.gammaf == 1.0f) ? r_eos : powf(r_eos, k.gammaf);
      p = k.c2f * (rg - k.rho_reff);
    } else {
      const float q = r_eos / k.rho_reff;
      const float qg = (k.gammaf == 1.0f) ? q : powf(q, k.gammaf);
      p = k.p0f * (qg - 1.0f);
    }
    pr[i] = widen(p);
    const float inv = 1.0f / rf;
    float4 cc;
    switch (k.rhs_force_type) {
      case 1: cc = make_float4(p * inv * inv, inv, mf, p); break;
      case 2: cc = make_float4(p * inv * inv, inv, 1.0f / mf, p); break;
      case 3: cc = make_float4(p * inv * inv, inv * inv, 1.0f / mf, p); break;
      default: cc = make_float4(p, inv * inv, 1.0f / mf, p); break;
    }
    pcf[2 * i] = cc;
    vf[2 * i] = make_float4(narrow(v.x), narrow(v.y), narrow(v.z), __int_as_float(pid));
  }
}

// A pair with a boundary particle, FP32 path: the wall or colloid particle
// takes the no-slip velocity and the fluid partner's pressure (pp_interaction_
// fw/wf/fc/cf.inc), in the Oldroyd-B model also its density and pressure
// tensor.  Wall distances come from the FP64-rounded per-particle values (one
// wall axis) or from the FP64 positions (several).  ci_w, cj_w: the two
// pressures; qi is particle i's polymer record, qie / qj those of the pair.
template <int D, bool NNW>
__device__ __forceinline__ void boundary_pair32(const Consts& k, int i, int j, int si, int sj,
                                                const float* r, float2 wdi,
                                                const float2* __restrict__ wd,
                                                const double4_32a* __restrict__ x,
                                                const CollArgs& ca, float ci_w, float cj_w,
                                                float* vi, float* vj, float& Ai, float& Aj,
                                                float& Bi, float& Bj, const float* qi, float* qie,
                                                float* qj) {
  constexpr int D2 = D * D;
  const bool other_j = (si < 0 || sj < 0) ? sj < 0 : sj > 0;  // the boundary particle is j
  float vw[3];
  bool noslip = true;
  if (si < 0 || sj < 0) {
    const int sw = (sj < 0) ? sj : si;
    const int face = -sw;
    const bool lower = (face & 1) != 0;
    float df, dw;
    if (k.wall_axis >= 0) {
      const float2 wj = wd[j];
      const float di = lower ? wdi.x : wdi.y, dj = lower ? wj.x : wj.y;
      df = (sj < 0) ? di : dj;
      dw = (sj < 0) ? dj : di;
    } else {
      const int axis = (face - 1) >> 1;
      const double x_sur = axis == 0 ? (lower ? k.min_phys[0] : k.max_phys[0])
                           : axis == 1 ? (lower ? k.min_phys[1] : k.max_phys[1])
                                       : (lower ? k.min_phys[2] : k.max_phys[2]);
      const double4_32a a4 = x[i], b4 = x[j];
      const double xa = axis == 0 ? a4.x : axis == 1 ? a4.y : a4.z;
      const double xb = axis == 0 ? b4.x : axis == 1 ? b4.y : b4.z;
      df = (float)(((sj < 0) ? xa : xb) - x_sur);
      dw = (float)(((sj < 0) ? xb : xa) - x_sur);
    }
    if (other_j)
      wall_noslip_dist<float, D>(k, df, dw, vi, sj, vw);
    else
      wall_noslip_dist<float, D>(k, df, dw, vj, si, vw);
  } else if (k.coll_noslip == 2) {
    const float4 rc4 = ca.rxcf[other_j ? j : i];
    const float rxc_[3] = {rc4.x, rc4.y, rc4.z};
    if (other_j) {
      colloid_noslip<float, D>(k, sj - 1, rxc_, r, vi, vw);
    } else {
      const float rfc[3] = {-r[0], -r[1], -r[2]};
      colloid_noslip<float, D>(k, si - 1, rxc_, rfc, vj, vw);
    }
  } else {
    noslip = false;  // frozen: the boundary particle's own (rigid) velocity
  }
  if (other_j) {
    if (noslip)
#pragma unroll
      for (int a = 0; a < D; ++a) vj[a] = vw[a];
    if (NNW) {
      Aj = Ai;
      Bj = Bi;
#pragma unroll
      for (int cc = 0; cc <= D2; ++cc) qj[cc] = qi[cc];
    } else {
      Aj = boundary_A<float>(k.rhs_force_type, ci_w, Bj);
    }
  } else {
    if (noslip)
#pragma unroll
      for (int a = 0; a < D; ++a) vi[a] = vw[a];
    if (NNW) {
      Ai = Aj;
      Bi = Bj;
#pragma unroll
      for (int cc = 0; cc <= D2; ++cc) qie[cc] = qj[cc];
    } else {
      Ai = boundary_A<float>(k.rhs_force_type, cj_w, Bi);
    }
  }
}

constexpr int kReuseTPB = 128;
// below this many particles the scalar FP32 force sweep and the FP64 density
// run 4 lanes per particle
constexpr int64_t kSplitBelow = 50000;
// and below this many the FP64 density sweep runs 8
constexpr int64_t kSplit8Below = 12000;
// Lanes per particle of the packed FP32 sweeps: a lane takes whole octets of a
// list, and a 2D particle has about four octets of pairs, a 3D one fourteen or
// more.  Measured, us a step (lanes 16 / 4 / 1): 3D rc = 3 dx 6k particles 60 /
// 73 / 160, 18k 97 / 80 / 145, 41k 170 / 132 / 161, 71k 272 / 185 / 183, 91k 327 /
// 203 / 168; 3D rc = 4 dx 8k 73 / 69 / 174, 33k 185 / 146 / 168, 91k 483 / 314 / 308;
// 2D 10k 40 / 30 / 39, 23k 50 / 39 / 40, 63k 87 / 69 / 47.
constexpr int64_t kLanes16Below = 12000, kLanes4Below = 75000, kLanes4Below2D = 20000;
inline int lanes32(int64_t n, int dim) {
  if (dim == 2) return n < kLanes4Below2D ? 4 : 1;
  return n < kLanes16Below ? 16 : n < kLanes4Below ? 4 : 1;
}

// How a sweep with S > 1 lanes per particle ends: the lanes leave their sums in
// shared memory (over the finished cell tables) and the block's first kFinish<S>
// threads run the epilogue, a particle each.  Run by one lane in S, its ~80 FP64
// instructions (64 cycles of a scheduler each, however few lanes take part) cost
// S times as much: 16,384 2D Oldroyd-B particles, four lanes, FP64 pipe 40% busy
// with it, force 25.7 us; so 20.0 us, density 18.5 -> 15.2.
template <int S>
constexpr int kFinish = kReuseTPB / S;

// FP32 offset of each stencil slot (the neighbour cell's origin minus the
// home cell's, w = Lees-Edwards velocity jump), build_table's t.o, in a
// block-shared table of kSlotTable entries: slot s of a home cell in
// Lees-Edwards state st at st * kMaxStencil + s.  The block's first threads
// fill it, then __syncthreads.
constexpr int kSlotTable = 3 * kMaxStencil;
static_assert(kSlotTable <= kReuseTPB, "one thread per slot-table entry");
template <int D>
__device__ __forceinline__ void fill_slot_offsets(const Consts& k, float4* s_slot) {
  const int e = threadIdx.x;
  if (e < kSlotTable) s_slot[e] = slot_offset<D>(k, e % kMaxStencil, e / kMaxStencil);
}

// One partner's FP32 records: offset to its cell's origin (w = species id),
// velocity (w = pid bits) and pair coefficients (A, B, C, p), and its slot.
struct JData {
  float4 o, v, c;
  int sl, j;
};

// the velocity and coefficient records lie side by side (one 32-byte load)
__device__ __forceinline__ void load_vc(const float4* __restrict__ vf, int j, float4& v,
                                        float4& c) {
  const double4_32a t = *(reinterpret_cast<const double4_32a*>(vf) + j);
  v = make_float4(__int_as_float(__double2loint(t.x)), __int_as_float(__double2hiint(t.x)),
                  __int_as_float(__double2loint(t.y)), __int_as_float(__double2hiint(t.y)));
  c = make_float4(__int_as_float(__double2loint(t.z)), __int_as_float(__double2hiint(t.z)),
                  __int_as_float(__double2loint(t.w)), __int_as_float(__double2hiint(t.w)));
}

__device__ __forceinline__ JData load_j(const int* __restrict__ s_start, int ent,
                                        const float4* __restrict__ off,
                                        const float4* __restrict__ vf) {
  JData d;
  d.sl = ent >> kLocalBits;
  d.j = s_start[d.sl * kReuseTPB + threadIdx.x] + (ent & (kMaxCellCount - 1));
  d.o = off[d.j];
  load_vc(vf, d.j, d.v, d.c);
  return d;
}

// slot offsets of the Lees-Edwards row state of the home cell
__device__ __forceinline__ const float4* slot_table(const Consts& k, const float4* s_slot,
                                                   int cell) {
  if (!k.le || cell >= k.ncell) return s_slot;
  return s_slot + le_state(k, (cell / k.nm[0]) % k.nm[1]) * kMaxStencil;
}

// ---------------------------------------------------------------------------
// Epilogue shared by both force sweeps: body force, store, second half kick.
// ---------------------------------------------------------------------------
template <int D>
__device__ __forceinline__ void force_epilogue(const Consts& k, int i, int si, const double* xi,
                                               double ax, double ay, double az,
                                               int fuse_mode, double dt,
                                               const double4_32a* __restrict__ v,
                                               double4_32a* __restrict__ f,
                                               double4_32a* __restrict__ v_out,
                                               unsigned* __restrict__ err) {
  if (!isfinite(ax) || !isfinite(ay) || !isfinite(az)) atomicOr(err, kErrNonFinite);
  if (fuse_mode >= kForceBody && si == 0) {
    // particles_apply_body_force.F90:96-353
    const double g[3] = {k.body_force[0], k.body_force[1], k.body_force[2]};
    if (k.body_force_type == 1) {
      if (k.body_on & 1) ax += g[0];
      if (k.body_on & 2) ay += g[1];
      if (D == 3 && (k.body_on & 4)) az += g[2];
    } else if (k.body_force_type == 2) {
      if (k.body_on & 1) {
        const double half = k.max_phys[D - 1] * 0.5;
        double xl = xi[D - 1];
        // positions may sit past a periodic face between list rebuilds
        if (k.periodic[D - 1]) {
          if (xl < k.min_phys[D - 1]) xl = __dadd_rn(xl, k.len[D - 1]);
          if (xl >= k.max_phys[D - 1]) xl = __dsub_rn(xl, k.len[D - 1]);
        }
        if (xl < half)
          ax += g[0];
        else if (xl > half)
          ax -= g[0];
      }
    } else if (k.body_force_type == 3) {
      if (k.body_on & 1) {
        const double kw = 2.0 * kPi / (k.max_phys[1] - k.min_phys[1]);
        ax += g[0] * sin(kw * xi[1]);
      }
    }
  }
  f[i] = make_double4_32a(ax, ay, az, 0.0);
  if (fuse_mode == kForceBodyKick) {
    // second half kick, particles_integrate_velocity.F90:84-94
    double4_32a vv = v[i];
    if (si == 0) {
      // rounded like k_integrate and the CPU restatement: v + (0.5 a) dt, no FMA
      const double hdt = halved(dt);
      vv.x = __dadd_rn(vv.x, __dmul_rn(ax, hdt));
      vv.y = __dadd_rn(vv.y, __dmul_rn(ay, hdt));
      if (D == 3) vv.z = __dadd_rn(vv.z, __dmul_rn(az, hdt));
    } else if (si < 0 && k.walls) {
      // end of the step: the face's shear velocity (moving walls)
      double vs[3] = {vv.x, vv.y, vv.z};
      wall_end_velocity<D>(k, si, vs);
      vv.x = vs[0];
      vv.y = vs[1];
      if (D == 3) vv.z = vs[2];
    }
    v_out[i] = vv;
  }
}

// Oldroyd-B per-particle update after the pair sweep: store the velocity
// gradient L, act = c L^T + L c - (c - I)/tau (particles_compute_act.F90:
// 112-156) and, inside a VV step, the second half step ct += act dt/2
// (particles_integrate_ct.F90:66-68), all in FP64.
template <int D>
__device__ __forceinline__ void nn_epilogue(const Consts& k, const NN& nn, int i, const double* L,
                                            int fuse_mode, double dt) {
  const int n = k.n;
#pragma unroll
  for (int cc = 0; cc < D * D; ++cc) nn.vgt[(size_t)cc * n + i] = L[cc];
  if (fuse_mode < kForceBody) return;
  double cm[D * D];
#pragma unroll
  for (int cc = 0; cc < D * D; ++cc) cm[cc] = nn.ct[(size_t)cc * n + i];
#pragma unroll
  for (int b = 0; b < D; ++b)
#pragma unroll
    for (int a = 0; a < D; ++a) {
      double t = 0.0;
#pragma unroll
      for (int q = 0; q < D; ++q) t = t + cm[a + D * q] * L[b + D * q] + L[a + D * q] * cm[q + D * b];
      const double act = t - (cm[a + D * b] - (a == b ? 1.0 : 0.0)) * k.inv_tau;
      nn.act[(size_t)(a + D * b) * n + i] = act;
      if (fuse_mode == kForceBodyKick)
        ((double*)nn.ct)[(size_t)(a + D * b) * n + i] =
            __dadd_rn(cm[a + D * b], __dmul_rn(__dmul_rn(act, dt), 0.5));
    }
}


}  // namespace mcfg

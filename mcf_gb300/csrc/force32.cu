// force32.cu -- FP32-mixed force sweep of the common pair forms (Newtonian
// Hu-Adams and Hu-Adams angular, no per-particle stress), two pairs an
// instruction.
//
// Bound: instruction issue, once the list arrives in time.  A pair takes ~120
// FP32 operations, ~45 integer ones for its Philox draw and ~10 special
// functions, and its partners' records come from L1.  So
//   - two entries are taken at a time with packed FP32 arithmetic (packed.cuh):
//     the two pairs are the halves of every operand, each half rounds as a pair
//     of its own, and an issue slot serves both;
//   - a thread's list comes by asynchronous 16-byte copies into a ring of its
//     own in shared memory, three octets ahead: with the list behind plain
//     loads the sweep waited on them for a third of its time, whatever its
//     other instructions;
//   - the next two partners' records are gathered during the current pairs.
// The fluid-fluid entries come first; entries with a boundary particle take
// the same loop, their velocities and coefficients replaced before packing.
// 261,568 particles, 113 pairs each: 234 us, 340 warp instructions two pairs,
// against 302 us and 265 a pair of the scalar sweep (k_force32).
//
// Reference: particles_compute_interaction.F90:609-900, rhs_force_ff_Newtonian_
// HuAdams.F90:124-239, rhs_force_ff_Newtonian_HuAdams_angular.F90.
#include <algorithm>

#include "mcfg_internal.cuh"
#include "packed.cuh"
#include "pair_common.cuh"
#include "sph.cuh"
#include "sweep_common.cuh"

namespace mcfg {

namespace {

constexpr int kHuAdams = 3, kAngular = 4;

// dW/dr of kernel_gradw (sph.cuh) for two distances
__device__ __forceinline__ F2 gradw2(const Consts& k, F2 d) {
  const F2 s = mul2(d, splat2(k.inv_hf));
  if (k.kernel_type == 1) {
    const F2 t3 = base2(3.0f, s), t2 = base2(2.0f, s), t1 = base2(1.0f, s);
    const F2 a3 = mul2(t3, t3), a2 = mul2(t2, t2), a1 = mul2(t1, t1);
    F2 g = fma2(splat2(-6.0f), mul2(a2, a2), mul2(a3, a3));
    g = fma2(splat2(15.0f), mul2(a1, a1), g);
    return mul2(splat2(5.0f * k.coef_gradf), g);
  }
  // (s om first: zero outside the support, however large s is)
  const F2 om = base2(1.0f, s);
  return mul2(splat2(12.0f * k.coef_gradf), mul2(mul2(s, om), om));
}

// sqrt of a non-negative pair
__device__ __forceinline__ F2 sqrt2(F2 a) {
  float lo, hi;
  unpack2(a, lo, hi);
  return pack2(sqrtf(lo), sqrtf(hi));
}

// u01 of two words (mcfg_internal.cuh): 1 + (r >> 9) 2^-23 from one funnel
// shift, less 1 - 2^-24 (exact)
__device__ __forceinline__ F2 u01_2(uint32_t ra, uint32_t rb) {
  return add2(pack2(__uint_as_float(__funnelshift_r(ra, 0x7fu, 9)),
                    __uint_as_float(__funnelshift_r(rb, 0x7fu, 9))),
              splat2(-0.99999994039535522461f));
}

// Box-Muller radii of two pairs, sqrt(-2 ln u): neg2log's branch away from 1
__device__ __forceinline__ F2 radius2(F2 u) {
  float a, b;
  unpack2(u, a, b);
  return sqrt2(mul2(splat2(-1.3862943611198906f), pack2(__log2f(a), __log2f(b))));
}
// both branches
__device__ __forceinline__ F2 radius2_near1(F2 u) {
  float a, b;
  unpack2(u, a, b);
  return pack2(sqrtf(neg2log(a)), sqrtf(neg2log(b)));
}

// the angle in [-pi, pi] of box_muller
__device__ __forceinline__ F2 angle2(F2 u) {
  return fma2(splat2(6.2831853071795865f), u, splat2(-3.1415926535897932f));
}

// The normals of pair_draw for two pairs (Hu-Adams: D of them, angular: one):
// the same words, radii and angles.
template <int D, int FT>
__device__ __forceinline__ void draw2(const uint32_t* rk, uint32_t step, int pidi, int pa, int pb,
                                      F2* z) {
  const uint4 a = philox4x32_10(
      make_uint4((uint32_t)min(pidi, pa), (uint32_t)max(pidi, pa), step, 0u), rk);
  const uint4 b = philox4x32_10(
      make_uint4((uint32_t)min(pidi, pb), (uint32_t)max(pidi, pb), step, 0u), rk);
  // u > 1 - 2^-10 takes the series of neg2log: the words' ten top bits are ones
  constexpr uint32_t kNear1 = 0xffc00000u;
  const F2 u1 = u01_2(a.x, b.x), u2 = u01_2(a.y, b.y);
  float s0, s1;
  if (FT == kHuAdams && D == 3) {
    const F2 u3 = u01_2(a.z, b.z), u4 = u01_2(a.w, b.w);
    F2 r1 = radius2(u1), r2 = radius2(u3);
    if (max(max(a.x, b.x), max(a.z, b.z)) >= kNear1) {
      r1 = radius2_near1(u1);
      r2 = radius2_near1(u3);
    }
    unpack2(angle2(u2), s0, s1);
    z[0] = mul2(r1, pack2(__cosf(s0), __cosf(s1)));
    z[1] = mul2(r1, pack2(__sinf(s0), __sinf(s1)));
    unpack2(angle2(u4), s0, s1);
    z[2] = mul2(r2, pack2(__cosf(s0), __cosf(s1)));
  } else {
    F2 r1 = radius2(u1);
    if (max(a.x, b.x) >= kNear1) r1 = radius2_near1(u1);
    unpack2(angle2(u2), s0, s1);
    z[0] = mul2(r1, pack2(__cosf(s0), __cosf(s1)));
    if (FT == kHuAdams) z[1] = mul2(r1, pack2(__sinf(s0), __sinf(s1)));
  }
}

// One partner in flight.
struct Partner {
  float4 o, v, c;
  int sl, j;
};

template <int S>
__device__ __forceinline__ Partner fetch(const int* __restrict__ s_start, unsigned ent,
                                         const float4* __restrict__ off,
                                         const float4* __restrict__ vf) {
  Partner p;
  p.sl = (int)(ent >> kLocalBits);
  p.j = s_start[p.sl * (kReuseTPB / S) + threadIdx.x / S] + (int)(ent & (kMaxCellCount - 1));
  p.o = off[p.j];
  load_vc(vf, p.j, p.v, p.c);
  return p;
}

// one half of the operands: separation, velocity difference, A_i + A_j, B_i + B_j
struct Half {
  float r[3], vij[3], SA, SB;
};

constexpr int kRing = 4;  // octets of a thread's list in shared memory

__device__ __forceinline__ void copy_octet(uint4* dst, const uint4* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

// S lanes per particle: lane l takes octets l, l + S, ... of each of the list's
// two segments.
template <int D, int FT, bool NOISE, int S>
__global__ void __launch_bounds__(kReuseTPB, 4)
    k_force32_packed(Consts k, const int* __restrict__ cell_start,
                     const int* __restrict__ cell_of, const uint16_t* __restrict__ nl,
                     const int* __restrict__ ncount, int cap, const float4* __restrict__ off,
                     const double4_32a* __restrict__ x, const double4_32a* __restrict__ v,
                     const float4* __restrict__ vf, const float2* __restrict__ wd,
                     double4_32a* __restrict__ f, int fuse_mode, double dt,
                     double4_32a* __restrict__ v_out, uint32_t step_arg,
                     const int64_t* __restrict__ step_ptr, float inv_sqdt,
                     unsigned* __restrict__ err, CollArgs ca) {
  const uint32_t step = step_ptr ? (uint32_t)*step_ptr : step_arg;
  __shared__ int s_start[kMaxStencil * kReuseTPB / S];
  __shared__ float4 s_slot[kSlotTable];
  __shared__ uint4 s_ring[kRing * kReuseTPB];
  const int n = k.n, tid = threadIdx.x;
  if (n == 0) return;
  fill_slot_offsets<D>(k, s_slot);
  __syncthreads();
  const int gt = blockIdx.x * kReuseTPB + tid;
  const int lane_s = gt % S;
  if (S == 1 && gt >= n) return;
  // lanes past the last particle stay for the block's end, with an empty list
  const int i = S == 1 ? gt : min(gt / S, n - 1);
  const int nc = S == 1 || gt / S < n ? ncount[i] : 0;
  const int nff = first_count(nc), no = second_count(nc);
  // the lane's octets: n0 of the first segment, then those of the second
  const int n0 = max(0, (nff + 7) / 8 - lane_s + S - 1) / S;
  const int nk = n0 + max(0, (no + 7) / 8 - lane_s + S - 1) / S;
  auto stage = [&](int kk) {
    if (kk < nk) {
      const int o = lane_s + S * (kk < n0 ? kk : kk - n0);
      const unsigned row = (unsigned)(kk < n0 ? o : list_octets(cap) - 1 - o);
      copy_octet(&s_ring[(kk % kRing) * kReuseTPB + tid],
                 reinterpret_cast<const uint4*>(nl) + (unsigned long long)row * (unsigned)n + i);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  stage(0);
  stage(1);
  stage(2);
  const int celli = cell_of[i];
  const unsigned gmask = group_mask<S>();
  if (S == 1)
    build_lane_table<D, kReuseTPB, false>(k, celli, cell_start, s_start, nullptr);
  else
    build_group_table<D, kReuseTPB, S>(k, celli, cell_start, s_start, gmask);
  const float4* slot_tab = slot_table(k, s_slot, celli);
  const float4 oi = off[i];
  const int si = __float_as_int(oi.w);
  float4 vi4, ci;
  load_vc(vf, i, vi4, ci);
  const int pidi = __float_as_int(vi4.w);
  const float2 wdi = (no > 0 && k.wall_axis >= 0) ? wd[i] : make_float2(0.f, 0.f);

  F2 acc[3], cmp[3];  // Kahan sums of the two halves
#pragma unroll
  for (int a = 0; a < 3; ++a) acc[a] = cmp[a] = splat2(0.0f);

  // fetch state: octet fk, its entries left fm, its words not yet used
  int fk = -1, fm = 0;
  uint4 q = make_uint4(0, 0, 0, 0);
  Partner pa, pb;
  bool f_both = false, f_plain = true;
  auto fetch_next = [&]() -> bool {
    if (fm <= 0) {
      if (++fk >= nk) return false;
      // octet fk has arrived when at most two younger groups are in flight
      asm volatile("cp.async.wait_group 2;" ::: "memory");
      q = s_ring[(fk % kRing) * kReuseTPB + tid];
      stage(fk + 3);
      f_plain = fk < n0;
      fm = min(8, f_plain ? nff - 8 * (lane_s + S * fk) : no - 8 * (lane_s + S * (fk - n0)));
    }
    f_both = fm > 1;
    pa = fetch<S>(s_start, q.x & 0xffffu, off, vf);
    pb = fetch<S>(s_start, f_both ? q.x >> 16 : q.x & 0xffffu, off, vf);
    q.x = q.y;
    q.y = q.z;
    q.z = q.w;
    fm -= 2;
    return true;
  };
  bool more = fetch_next();
  while (more) {
    // the operands of the two pairs, before the next partners' records take
    // the registers of these
    Half ha, hb;
    auto half = [&](const Partner& j, Half& h) {
      const float4 so = slot_tab[j.sl];
      h.r[0] = (oi.x - j.o.x) - so.x;
      h.r[1] = (oi.y - j.o.y) - so.y;
      h.r[2] = (D == 3) ? (oi.z - j.o.z) - so.z : 0.0f;
      h.vij[0] = vi4.x - (j.v.x + so.w);
      h.vij[1] = vi4.y - j.v.y;
      h.vij[2] = (D == 3) ? vi4.z - j.v.z : 0.0f;
      h.SA = ci.x + j.c.x;
      h.SB = ci.y + j.c.y;
    };
    half(pa, ha);
    half(pb, hb);
    if (!f_plain) {
      // pairs with a boundary particle
      auto boundary = [&](const Partner& j, Half& h) {
        const int sj = __float_as_int(j.o.w);
        if (si >= 0 && sj >= 0 && (si > 0) == (sj > 0)) return;  // two colloids
        float vi[3] = {vi4.x, vi4.y, vi4.z};
        float vj[3] = {j.v.x + slot_tab[j.sl].w, j.v.y, j.v.z};
        float Ai = ci.x, Aj = j.c.x, Bi = ci.y, Bj = j.c.y;
        boundary_pair32<D, false>(k, i, j.j, si, sj, h.r, wdi, wd, x, ca, ci.w, j.c.w, vi, vj, Ai,
                                  Aj, Bi, Bj, nullptr, nullptr, nullptr);
#pragma unroll
        for (int a = 0; a < D; ++a) h.vij[a] = vi[a] - vj[a];
        h.SA = Ai + Aj;
      };
      boundary(pa, ha);
      boundary(pb, hb);
    }
    const int pid_a = __float_as_int(pa.v.w), pid_b = __float_as_int(pb.v.w);
    const bool both = f_both;
    more = fetch_next();
    // never taken (offsets hold no such NaN; one that did would end the run as
    // a non-finite acceleration does): the branch ends the basic block, so
    // that the gathers are issued here and not, as the compiler otherwise
    // orders them, behind this pair's arithmetic (258 instead of 234 us)
    if (__float_as_int(oi.x) == 0x7fabcdef) {
      atomicOr(err, kErrNonFinite);
      break;
    }
    // a lone last pair: its twin is put out of the support, where every term
    // is an exact zero
    if (!both) hb.r[0] = kBeyond;
    F2 r[3], vij[3];
#pragma unroll
    for (int a = 0; a < D; ++a) {
      r[a] = pack2(ha.r[a], hb.r[a]);
      vij[a] = pack2(ha.vij[a], hb.vij[a]);
    }
    const F2 SA = pack2(ha.SA, hb.SA), SB = pack2(ha.SB, hb.SB);
    F2 d2 = fma2(r[1], r[1], mul2(r[0], r[0]));
    if (D == 3) d2 = fma2(r[2], r[2], d2);
    float dlo, dhi;
    unpack2(d2, dlo, dhi);
    const F2 u = pack2(rsqrtf(dlo), rsqrtf(dhi));
    const F2 gw = gradw2(k, mul2(d2, u));
    F2 z[3], g[3];
    if (NOISE) draw2<D, FT>(k.rk, step, pidi, pid_a, pid_b, z);
    if (FT == kHuAdams) {
      // the force along r (pair_force takes e = r/d)
      const F2 gwu = mul2(gw, u);
      const F2 f_d = mul2(splat2(k.etaf), mul2(SB, gwu));
      F2 along = mul2(SA, gwu);  // of -r
      if (NOISE) {
        // We = s (ca (e.z) e + cb (z - (e.z) e)), amplitude f_r (pair_force)
        const float cb = 0.70710678118654752440f;
        const float cr = 0.81649658092772603273f / cb - 1.0f;  // ca/cb - 1 in 3D
        const float amp = inv_sqdt * cb;
        const F2 ft =
            mul2(sqrt2(mul2(splat2(-4.0f * k.ktf), f_d)),
                 pack2(pidi < pid_a ? amp : -amp, pidi < pid_b ? amp : -amp));
        if (D == 3) {
          const F2 rz = fma2(r[2], z[2], fma2(r[1], z[1], mul2(r[0], z[0])));
          along = fma2(mul2(ft, splat2(-cr)), mul2(mul2(rz, u), u), along);
        }
#pragma unroll
        for (int a = 0; a < D; ++a)
          g[a] = fma2(ft, z[a], sub2(mul2(f_d, vij[a]), mul2(along, r[a])));
      } else {
#pragma unroll
        for (int a = 0; a < D; ++a) g[a] = sub2(mul2(f_d, vij[a]), mul2(along, r[a]));
      }
    } else {
      F2 ev = mul2(r[0], vij[0]);
#pragma unroll
      for (int a = 1; a < D; ++a) ev = fma2(r[a], vij[a], ev);
      ev = mul2(ev, u);
      const F2 Aij = mul2(SB, gw);
      const F2 f_c = mul2(Aij, mul2(SA, splat2(0.5f)));
      F2 fe = sub2(mul2(mul2(mul2(splat2(k.eta_coeff * k.etaf), Aij), ev), u), f_c);
      if (NOISE) {
        const F2 amp = mul2(splat2(sqrtf(2.0f * k.ktf * k.etaf) * inv_sqdt),
                            sqrt2(mul2(mul2(splat2(-k.eta_coeff), Aij), u)));
        fe = fma2(z[0], amp, fe);
      }
      fe = mul2(fe, u);
#pragma unroll
      for (int a = 0; a < D; ++a) g[a] = mul2(fe, r[a]);
    }
#pragma unroll
    for (int a = 0; a < D; ++a) {
      const F2 y = sub2(g[a], cmp[a]);
      const F2 t = add2(acc[a], y);
      cmp[a] = sub2(sub2(t, acc[a]), y);
      acc[a] = t;
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  // the halves' and lanes' sums (in lane order) with their corrections, then
  // both forms' factor 1/m_i; widened at the end: the FP64 pipe takes 64
  // cycles a warp and operation
  float hi[3], lo[3];
#pragma unroll
  for (int a = 0; a < D; ++a) join_sums<S>(acc[a], cmp[a], gmask, hi[a], lo[a]);
  int fi = i, fsi = si;  // the particle this thread finishes
  float im = ci.z;
  if (S > 1) {
    constexpr int P = kFinish<S>;
    float* s_sum = reinterpret_cast<float*>(s_start);
    __syncthreads();
    if (lane_s == 0) {
#pragma unroll
      for (int a = 0; a < D; ++a) {
        s_sum[(2 * a) * P + tid / S] = hi[a];
        s_sum[(2 * a + 1) * P + tid / S] = lo[a];
      }
    }
    __syncthreads();
    fi = blockIdx.x * P + tid;
    if (tid >= P || fi >= n) return;
#pragma unroll
    for (int a = 0; a < D; ++a) {
      hi[a] = s_sum[(2 * a) * P + tid];
      lo[a] = s_sum[(2 * a + 1) * P + tid];
    }
    fsi = __float_as_int(off[fi].w);
    float4 vi_, c_;
    load_vc(vf, fi, vi_, c_);
    im = c_.z;
  }
  double tot[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int a = 0; a < D; ++a) {
    const float p = hi[a] * im;
    tot[a] = widen(p) + widen(fmaf(hi[a], im, -p) + lo[a] * im);
  }
  const double4_32a xi4 = x[fi];
  const double xi[3] = {xi4.x, xi4.y, xi4.z};
  force_epilogue<D>(k, fi, fsi, xi, tot[0], tot[1], D == 3 ? tot[2] : 0.0, fuse_mode, dt, v, f,
                    v_out, err);
}

}  // namespace

bool force32_packed(Handle* h, uint32_t step, const int64_t* step_ptr, float inv_sqdt,
                    int fuse_mode, double dt) {
  const Consts& k = h->k;
  const int ft = k.rhs_force_type;
  if (!k.newtonian || k.stress || (ft != kHuAdams && ft != kAngular)) return false;
  const int S = lanes32(h->n, k.d);
  const int64_t threads = h->n * S;
  const int g = std::max(1, (int)((threads + kReuseTPB - 1) / kReuseTPB));
#define LAUNCH(DD, FT, NO, SS)                                                                  \
  k_force32_packed<DD, FT, NO, SS><<<g, kReuseTPB, 0, h->stream>>>(                             \
      k, h->cell_start, h->cell_of, h->nl, h->ncount, h->neigh_cap, h->off, h->x, h->v, h->vf,  \
      h->wd, h->f, fuse_mode, dt, h->v2, step, step_ptr, inv_sqdt, h->d_err,                    \
      CollArgs{h->v, h->rxc, h->rxcf})
#define PICK_S(DD, FT, NO)       \
  do {                           \
    if (DD == 3 && S == 16)      \
      LAUNCH(3, FT, NO, 16);     \
    else if (S == 4)             \
      LAUNCH(DD, FT, NO, 4);     \
    else                         \
      LAUNCH(DD, FT, NO, 1);     \
  } while (0)
#define PICK(DD)                                      \
  do {                                                \
    if (ft == kHuAdams) {                             \
      if (k.noise) PICK_S(DD, kHuAdams, true);        \
      else PICK_S(DD, kHuAdams, false);               \
    } else {                                          \
      if (k.noise) PICK_S(DD, kAngular, true);        \
      else PICK_S(DD, kAngular, false);               \
    }                                                 \
  } while (0)
  if (k.d == 3) PICK(3); else PICK(2);
#undef PICK
#undef PICK_S
#undef LAUNCH
  return true;
}

}  // namespace mcfg

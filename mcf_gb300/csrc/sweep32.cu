// sweep32.cu -- FP32-mixed density sweep over a candidate list.
//
// The candidates (k_scan, pair_kernels.cu) -- with neighbour-list reuse those
// within rc + skin at the last rebuild, otherwise the step's own -- are
// partitioned by species: the fluid partners of a fluid particle in the list's
// first segment; every other pair (wall, colloid, or a boundary particle's own
// pairs) in the second.  vcount packs both counts (fluid-fluid | other << 16).
//
// Each step the density sweep re-tests every candidate exactly (FP32), sums
// the number density, and writes the step's pairs as a compact list in the
// same two segments (ncount likewise).  A step's own candidates are compacted
// in place (vl == nl).  The force sweeps (force32.cu, k_force32) walk that
// list, the fluid-fluid pairs first.
//
// Reference: particles_compute_density.F90:578-867.
#include "mcfg_internal.cuh"
#include "packed.cuh"
#include "pair_common.cuh"
#include "sph.cuh"
#include "sweep_common.cuh"

namespace mcfg {

namespace {

// Does a force act between species si and sj, one of them a boundary particle?
// w-w and c-w never, c-c only between different colloids with pp_interact_cc
// (pp_interaction.inc:63-223)
__device__ __forceinline__ bool interacts(const Consts& k, int si, int sj) {
  return si == 0 || sj == 0 || (si > 0 && sj > 0 && si != sj && k.pp_cc);
}

// The kernel sum's term for two distances, W / coef (kernel_w, sph.cuh)
__device__ __forceinline__ F2 raw_w2(const Consts& k, F2 d) {
  const F2 s = mul2(d, splat2(k.inv_hf));
  if (k.kernel_type == 1) {
    const F2 t3 = base2(3.0f, s), t2 = base2(2.0f, s), t1 = base2(1.0f, s);
    const F2 q3 = mul2(t3, t3), q2 = mul2(t2, t2), q1 = mul2(t1, t1);
    const F2 w = fma2(splat2(-6.0f), mul2(mul2(q2, q2), t2), mul2(mul2(q3, q3), t3));
    return fma2(splat2(15.0f), mul2(mul2(q1, q1), t1), w);
  }
  const F2 om = base2(1.0f, s);
  return mul2(fma2(splat2(3.0f), s, splat2(1.0f)), mul2(mul2(om, om), om));
}

// Density over the candidate list, S lanes per particle.
//
// A lane takes its candidates an octet (one 16-byte load ahead) at a time,
// gathers their offsets in fours, and tests and sums them two an instruction
// (packed.cuh).  One lane a particle appends the kept entries four a store;
// several lanes (small systems, lane l octets l, l + S, ...) place theirs by a
// prefix sum, in candidate order.  Bound: issue and the latency of the gathers.
// 261,568 particles, 113 candidates each: 99 us (80 registers and 6 blocks a SM
// 116, 64 and 8 102; gathering a group ahead 112 or more) against 148 us one
// candidate and 2-byte list load at a time.  Four lanes need 104 registers
// unless held to 5 blocks a SM, whose grid then ends in a nearly empty wave (41k
// particles 58 us; 48 us with 88 registers).
template <int D, int S>
__global__ void __launch_bounds__(kReuseTPB, S == 1 ? 7 : 5)
    k_density_list(Consts k, const int* __restrict__ cell_start, const int* __restrict__ cell_of,
                   const float4* __restrict__ off, const double4_32a* __restrict__ x,
                   const double4_32a* __restrict__ v, const double* __restrict__ m,
                   const int* __restrict__ pid, const uint16_t* vl, const int* vcount, int vcap,
                   uint16_t* nl, int* ncount, int cap, double* __restrict__ rho,
                   double* __restrict__ pr, float4* __restrict__ pcf, float4* __restrict__ vf,
                   int with_pressure, unsigned* __restrict__ err, int* __restrict__ stats,
                   unsigned long long* __restrict__ pairs, NN nn, CollArgs ca) {
  __shared__ int s_start[kMaxStencil * kReuseTPB / S];
  __shared__ float4 s_slot[kSlotTable];
  __shared__ uint4 s_keep[16];
  const int n = k.n, tid = threadIdx.x;
  const int gt = blockIdx.x * kReuseTPB + tid;
  const int i = gt / S, lane_s = gt % S;
  fill_slot_offsets<D>(k, s_slot);
  if (S == 1 && tid >= kReuseTPB - 16) s_keep[tid - (kReuseTPB - 16)] = keep_entry(tid & 15);
  __syncthreads();
  int kff = 0, ko = 0, si = 0;
  int idle = 0;  // pairs within the cut-off that no force acts in
  bool acc_i = false;
  float hi = 0.0f, lo = 0.0f;  // the sum over pairs and its remainder
  if (i < n) {
    const unsigned gmask = group_mask<S>();
    const int celli = cell_of[i];
    if (S == 1)
      build_lane_table<D, kReuseTPB, false>(k, celli, cell_start, s_start, nullptr);
    else
      build_group_table<D, kReuseTPB, S>(k, celli, cell_start, s_start, gmask);
    const float4* slot_tab = slot_table(k, s_slot, celli);
    const float4 oi = off[i];
    si = __float_as_int(oi.w);
    acc_i = dyn_rho(k, si);  // else the density is constant and the sum unused
    const bool mass = k.rhs_density_type == 1;
    const int vc = vcount[i];
    const int nff = first_count(vc), ntot = nff + second_count(vc);
    const int voct = list_octets(vcap), noct = list_octets(cap);
    const bool in_place = nl == vl;
    const uint4* list4 = reinterpret_cast<const uint4*>(vl);
    F2 acc = splat2(0.0f), cmp = splat2(0.0f);
#pragma unroll 1
    for (int seg = 0; seg < 2; ++seg) {
      const bool up = seg == 0;
      const int m_ = up ? nff : ntot - nff;  // candidates of the segment
      auto octet = [&](int o) {
        return list4[(unsigned long long)(unsigned)(up ? o : voct - 1 - o) * (unsigned)n + i];
      };
      // candidates p .. p + 3 (p at least is one): their terms are added, the
      // hits that go to the force sweep returned as bits
      auto four = [&](int p, const unsigned* e) -> unsigned {
        int j[4];
        float4 o[4];
        float rx[4], ry[4], rz[4];
        unsigned ent[4], hits = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          ent[u] = u == 0 || p + u < m_ ? e[u] : e[0];
          j[u] = s_start[(ent[u] >> kLocalBits) * (kReuseTPB / S) + tid / S] +
                 (int)(ent[u] & (kMaxCellCount - 1));
          o[u] = off[j[u]];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float4 so = slot_tab[ent[u] >> kLocalBits];
          rx[u] = (oi.x - o[u].x) - so.x;
          ry[u] = (oi.y - o[u].y) - so.y;
          if (D == 3) rz[u] = (oi.z - o[u].z) - so.z;
          // past the segment's end: out of the support
          if (u > 0 && p + u >= m_) rx[u] = kBeyond;
        }
        F2 w[2];
#pragma unroll
        for (int u = 0; u < 4; u += 2) {
          const F2 x2 = pack2(rx[u], rx[u + 1]), y2 = pack2(ry[u], ry[u + 1]);
          F2 d2 = fma2(y2, y2, mul2(x2, x2));
          if (D == 3) {
            const F2 z2 = pack2(rz[u], rz[u + 1]);
            d2 = fma2(z2, z2, d2);
          }
          float d2v[2];
          unpack2(d2, d2v[0], d2v[1]);
          w[u / 2] = raw_w2(k, pack2(sqrtf(d2v[0]), sqrtf(d2v[1])));
#pragma unroll
          for (int h = 0; h < 2; ++h)
            if (d2v[h] < k.rc2f) hits |= 1u << (u + h);
        }
        if (mass) {
          // W before the mass: a term is of the density's own size, whatever the
          // units of mass and length (below 1.2e-38 it would be flushed to zero)
          const F2 cw = splat2(k.coeff);
          w[0] = mul2(mul2(cw, w[0]), pack2((float)m[j[0]], (float)m[j[1]]));
          w[1] = mul2(mul2(cw, w[1]), pack2((float)m[j[2]], (float)m[j[3]]));
        }
        // Kahan sums of the two halves; a rejected candidate adds its W of zero
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const F2 y = sub2(w[u], cmp);
          const F2 t = add2(acc, y);
          cmp = sub2(sub2(t, acc), y);
          acc = t;
        }
        if (!up) {
          // two boundary particles: counted, not listed for the force
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (((hits >> u) & 1u) && !interacts(k, si, __float_as_int(o[u].w))) {
              hits &= ~(1u << u);
              ++idle;
            }
        }
        return hits;
      };
      int kept = 0;
      uint4 nx = make_uint4(0, 0, 0, 0);
      if (8 * lane_s < m_) nx = octet(lane_s);
      if (S == 1) {
        QuadTail out;
        auto keep = [&](int p, unsigned wx, unsigned wy) {
          const unsigned e[4] = {wx & 0xffffu, wx >> 16, wy & 0xffffu, wy >> 16};
          const unsigned hits = four(p, e);
          if (in_place && out.count == p && (hits == 15u || p + __popc(hits) == m_))
            out.count += __popc(hits);  // nothing rejected so far: the list holds them
          else
            out.append(nl, up, noct, n, i, make_uint2(wx, wy), hits, s_keep);
        };
#pragma unroll 1
        for (int p0 = 0; p0 < m_; p0 += 8) {
          const uint4 q = nx;
          if (p0 + 8 < m_) nx = octet((p0 >> 3) + 1);
          keep(p0, q.x, q.y);
          if (p0 + 4 < m_) keep(p0 + 4, q.z, q.w);
        }
        if (!(in_place && out.count == m_)) out.finish(nl, up, noct, n, i);
        kept = out.count;
      } else {
#pragma unroll 1
        for (int o0 = 0; 8 * o0 < m_; o0 += S) {
          const int p0 = 8 * (o0 + lane_s);
          const uint4 q = nx;
          if (p0 + 8 * S < m_) nx = octet(o0 + lane_s + S);
          const unsigned e[8] = {q.x & 0xffffu, q.x >> 16, q.y & 0xffffu, q.y >> 16,
                                 q.z & 0xffffu, q.z >> 16, q.w & 0xffffu, q.w >> 16};
          unsigned hits = 0;
          if (p0 < m_) hits = four(p0, e);
          if (p0 + 4 < m_) hits |= four(p0 + 4, e + 4) << 4;
          // the lanes' places: a prefix sum over the group
          const int mine = __popc(hits);
          int incl = mine;
#pragma unroll
          for (int w = 1; w < S; w <<= 1) {
            const int t = __shfl_up_sync(gmask, incl, w, S);
            if (lane_s >= w) incl += t;
          }
          int pos = kept + incl - mine;
          kept += __shfl_sync(gmask, incl, S - 1, S);
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if ((hits >> u) & 1u) {
              if (pos < cap) nl[up ? up_at(pos, n, i) : down_at(pos, cap, n, i)] = (uint16_t)e[u];
              ++pos;
            }
        }
      }
      if (up)
        kff = kept;
      else
        ko = kept;
    }
    join_sums<S>(acc, cmp, gmask, hi, lo);
    if (S > 1) {
#pragma unroll
      for (int w = 1; w < S; w <<= 1) idle += __shfl_xor_sync(gmask, idle, w);
    }
  }
  int my_max = 0;
  unsigned long long my_pairs = 0;
  int fi = i;  // the particle this thread finishes
  bool fin = i < n;
  if (S > 1) {
    constexpr int P = kFinish<S>;
    const int group = tid / S;
    __syncthreads();
    if (lane_s == 0) {
      s_start[group] = __float_as_int(hi);
      s_start[P + group] = __float_as_int(lo);
      s_start[2 * P + group] = kff;
      s_start[3 * P + group] = ko;
      s_start[4 * P + group] = idle;
    }
    __syncthreads();
    fi = blockIdx.x * P + tid;
    fin = tid < P && fi < n;
    if (fin) {
      hi = __int_as_float(s_start[tid]);
      lo = __int_as_float(s_start[P + tid]);
      kff = s_start[2 * P + tid];
      ko = s_start[3 * P + tid];
      idle = s_start[4 * P + tid];
      si = __float_as_int(off[fi].w);
      acc_i = dyn_rho(k, si);
    }
  }
  if (fin) {
    const double sum = widen(hi) + widen(lo);
    const double rho_i = k.rhs_density_type == 1 ? sum : widen(k.coeff) * sum;
    const int kept = kff + ko + idle;
    if (kept > cap) {
      atomicOr(err, kErrNeighOverflow);
      atomicMax(&err[kErrWordNeigh], (unsigned)kept);
      kff = min(kff, cap);
      ko = min(ko, cap - kff);
    }
    ncount[fi] = pack_counts(kff, ko);
    my_max = kept;
    my_pairs = (unsigned long long)kept;
    const double mi = m[fi];
    double rho_out;
    if (acc_i) {
      rho_out = ((k.rhs_density_type == 1) ? k.w0 * mi : k.w0) + rho_i;
    } else {
      rho_out = (k.rhs_density_type == 1) ? k.init_density : k.init_density / mi;
    }
    rho[fi] = rho_out;
    if (!(rho_out > 0.0)) atomicOr(err, kErrZeroDensity);
    if (with_pressure) {
      const double4_32a vi4 =
          (si > 0 && k.ncoll > 0) ? colloid_particle_update<D>(k, fi, si, x[fi], ca) : v[fi];
      write_particle_records<false>(k, fi, rho_out, mi, pid[fi], vi4, pr, nullptr, pcf, vf, nn);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    my_max = max(my_max, __shfl_xor_sync(0xffffffffu, my_max, o));
    my_pairs += __shfl_xor_sync(0xffffffffu, my_pairs, o);
  }
  if ((tid & 31) == 0) {
    atomicMax(&stats[1], my_max);
    atomicAdd(pairs, my_pairs);
  }
}

}  // namespace

int density_list(Handle* h, bool with_pressure, const uint16_t* vl, const int* vcount, int vcap) {
  Consts& k = h->k;
  cudaStream_t s = h->stream;
  const int n = (int)h->n;
  const int S = lanes32(n, k.d);
  const int g = (int)(((int64_t)n * S + kReuseTPB - 1) / kReuseTPB);
#define LAUNCH(DD, SS)                                                                          \
  k_density_list<DD, SS><<<g, kReuseTPB, 0, s>>>(                                              \
      k, h->cell_start, h->cell_of, h->off, h->x, h->v, h->m, h->pid, vl, vcount, vcap, h->nl,     \
      h->ncount, h->neigh_cap, h->rho, h->pr, h->pcf, h->vf, with_pressure ? 1 : 0,             \
      h->d_err, h->d_stats, h->d_pairs, NN{h->ct, h->act, h->vgt, h->qq},                       \
      CollArgs{h->v, h->rxc, h->rxcf})
#define PICK(DD)                     \
  do {                               \
    if (DD == 3 && S == 16) LAUNCH(3, 16); \
    else if (S == 4) LAUNCH(DD, 4);  \
    else LAUNCH(DD, 1);              \
  } while (0)
  if (k.d == 3) PICK(3); else PICK(2);
#undef PICK
#undef LAUNCH
  h->launches++;
  return cuda_check(h, cudaGetLastError(), "density launch") ? MCFG_ECUDA : MCFG_OK;
}

}  // namespace mcfg

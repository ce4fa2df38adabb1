// pair_kernels.cu -- the pair sweeps of the SDPD right-hand side.
//
// Layout: particles sorted by cell (cell_list.cu).
//
// Candidates (k_scan): one warp owns one cell and walks its particles in
// chunks of 32 (lane = particle i) through the 27 (3D) or 9 (2D) neighbour
// cells, an FP32 test on cell offsets; the hits go to a per-particle list of
// 16-bit entries slot<<11 | local index (octets, see pair_common.cuh).  With
// list reuse the list holds the candidates within rc + skin and outlives the
// step, otherwise it is made for this step.
//
// Density (k_density_reuse here for FP64, k_density_list in sweep32.cu for
// FP32-mixed): thread per particle (several lanes each on small systems) over
// the candidates.  The FP64 path re-tests them with the exact FP64 squared
// distance of MCF (so the pair set is MCF's bit for bit); both paths keep the
// step's pairs as the list of the force sweep and sum W.  The epilogue
// evaluates the equation of state and writes the per-particle pair
// coefficients.
//
// Force (k_force32_packed in force32.cu for the common FP32 forms, k_force32 for
// the others, k_force64): walks the step's list and gathers the pair
// accelerations of particle i.  Each pair is evaluated from both sides, so
// there is no scatter, no atomic and the result is deterministic; the random
// term is keyed by the unordered pid pair, so both sides draw the same dW.
// k_force_sym evaluates each pair once (FP64 Newtonian without stress).
//
// Reference: particles_compute_density.F90:369-867, particles_compute_
// interaction.F90:609-900, pp_interaction*.inc, rhs_force_ff_Newtonian*.F90.
#include <algorithm>
#include <type_traits>

#include "mcfg_internal.cuh"
#include "packed.cuh"
#include "pair_common.cuh"
#include "sph.cuh"
#include "sweep_common.cuh"

namespace mcfg {

constexpr int kMaskRows = 32;  // candidate chunks a warp notes between two emissions

// Candidates of every particle with FP32 squared distance below lim, in slot
// order and particle order, into list and count.  With partition (FP32 lists)
// the fluid-fluid candidates form the first segment, the others the second,
// and count = fluid-fluid | other << 16.  EXACT: the separation is formed as
// the density sweep forms it, so that lim decides alike (a step's own FP32
// list); the other lists have slack in lim and save that addition.
// gate: the list is the kept one; return at once when *gate is zero (no rebuild due).
//
// Bound: instruction issue (a 3D particle meets 27 cells of ~28 particles, of
// which ~113 are pairs).  So a chunk of 32 candidates is staged once in shared
// memory as separate coordinates, tested two at a time by packed FP32
// arithmetic against broadcast loads, and leaves one hit bit a candidate (the
// sign of d2 - lim, shifted in): ~6 instructions a test with nothing done a
// hit.  The bits are expanded afterwards, four entries a store.  The next
// chunk is in flight meanwhile.  261,568
// particles: 196 us (tests 113, expansion 83) where writing each hit as it was
// found took 344 us.
template <int D, bool EXACT>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
    k_scan(Consts k, const int* __restrict__ gate, const int* __restrict__ cell_start,
           const float4* __restrict__ off, float lim, uint16_t* __restrict__ list,
           int* __restrict__ count, int cap, int partition, unsigned* __restrict__ err) {
  if (gate && *gate == 0) return;
  constexpr int CENTER = (D == 3) ? 13 : 4;
  __shared__ NbTable tab[kWarpsPerBlock];
  __shared__ __align__(16) float sb[kWarpsPerBlock][2][3][32];
  __shared__ unsigned s_mask[kWarpsPerBlock][kMaskRows][32];
  __shared__ unsigned s_fluid[kWarpsPerBlock][kMaskRows];
  __shared__ int s_ent[kWarpsPerBlock][kMaskRows];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = k.n, ns = k.ns, octets = list_octets(cap, partition != 0);
  const F2 neg_lim = splat2(-lim);
  for (int cell = blockIdx.x * kWarpsPerBlock + wib; cell <= k.ncell;
       cell += gridDim.x * kWarpsPerBlock) {
    NbTable& t = tab[wib];
    build_table<D>(k, cell, cell_start, t);
    const int c0 = t.start[CENTER], c1 = c0 + t.count[CENTER];
    for (int base = c0; base < c1; base += 32) {
      const int i = base + lane;
      const bool active = i < c1;
      const float4 oi = active ? off[i] : make_float4(0.f, 0.f, 0.f, 0.f);
      const bool fluid_i = __float_as_int(oi.w) == 0;
      ListTail ff, other;  // the two segments
      int rows = 0, buf = 0;
      // one segment only: no partition, or all particles met are fluid
      const bool plain0 = !partition || __all_sync(0xffffffffu, fluid_i);
      bool plain = plain0;
      // entries hold 11 bits of local index: a fuller cell is an error
      // already (k_cell_finalize), and only its first 2048 are listed
      int sl = 0, b2 = 0, jn = min(t.count[0], kMaxCellCount);
      while (sl < ns && b2 >= jn) {
        b2 = 0;
        if (++sl < ns) jn = min(t.count[sl], kMaxCellCount);
      }
      const float4 pad = make_float4(0.f, 0.f, 0.f, 0.f);
      float4 nx = (sl < ns && b2 + lane < jn) ? off[t.start[sl] + b2 + lane] : pad;
      while (sl < ns) {
        const int sl_c = sl, b_c = b2, mm = min(32, jn - b2);
        float(*sc)[32] = sb[wib][buf];
        sc[0][lane] = -nx.x;
        sc[1][lane] = -nx.y;
        if (D == 3) sc[2][lane] = -nx.z;
        const unsigned fluid_j = __ballot_sync(0xffffffffu, __float_as_int(nx.w) == 0);
        // the next chunk's offsets, in flight during this one's tests
        b2 += 32;
        while (sl < ns && b2 >= jn) {
          b2 = 0;
          if (++sl < ns) jn = min(t.count[sl], kMaxCellCount);
        }
        __syncwarp();
        nx = (sl < ns && b2 + lane < jn) ? off[t.start[sl] + b2 + lane] : pad;
        const float4 so = t.o[sl_c];
        const F2 px = splat2(EXACT ? oi.x : oi.x - so.x), py = splat2(EXACT ? oi.y : oi.y - so.y),
                 pz = splat2(EXACT ? oi.z : oi.z - so.z);
        const F2 sx = splat2(-so.x), sy = splat2(-so.y), sz = splat2(-so.z);
        unsigned mask = 0;
        int q = 0;
        for (; q < mm; q += 4) {
          const ulonglong2 x4 = *reinterpret_cast<const ulonglong2*>(&sc[0][q]);
          const ulonglong2 y4 = *reinterpret_cast<const ulonglong2*>(&sc[1][q]);
          F2 xa = add2(px, F2{x4.x}), xb = add2(px, F2{x4.y});
          F2 ya = add2(py, F2{y4.x}), yb = add2(py, F2{y4.y});
          if (EXACT) {
            xa = add2(xa, sx);
            xb = add2(xb, sx);
            ya = add2(ya, sy);
            yb = add2(yb, sy);
          }
          F2 da = fma2(ya, ya, mul2(xa, xa)), db = fma2(yb, yb, mul2(xb, xb));
          if (D == 3) {
            const ulonglong2 z4 = *reinterpret_cast<const ulonglong2*>(&sc[2][q]);
            F2 za = add2(pz, F2{z4.x}), zb = add2(pz, F2{z4.y});
            if (EXACT) {
              za = add2(za, sz);
              zb = add2(zb, sz);
            }
            da = fma2(za, za, da);
            db = fma2(zb, zb, db);
          }
          float d0, d1, d2, d3;
          unpack2(add2(da, neg_lim), d0, d1);
          unpack2(add2(db, neg_lim), d2, d3);
          mask = __funnelshift_l(__float_as_uint(d0), mask, 1);
          mask = __funnelshift_l(__float_as_uint(d1), mask, 1);
          mask = __funnelshift_l(__float_as_uint(d2), mask, 1);
          mask = __funnelshift_l(__float_as_uint(d3), mask, 1);
        }
        // candidate c of the chunk at bit 31 - c, the padding's bits cut off
        mask <<= 32 - q;
        mask &= 0xffffffffu << (32 - mm);
        if (sl_c == CENTER) {
          const int self = i - t.start[CENTER] - b_c;
          if (self >= 0 && self < 32) mask &= ~(0x80000000u >> self);
        }
        if (!active) mask = 0;
        if (__any_sync(0xffffffffu, mask != 0)) {
          s_mask[wib][rows][lane] = mask;
          if (lane == 0) {
            s_ent[wib][rows] = (sl_c << kLocalBits) | b_c;
            s_fluid[wib][rows] = __brev(fluid_j);
          }
          if (partition) plain = plain && fluid_j == 0xffffffffu;
          ++rows;
        }
        buf ^= 1;
        if (rows == kMaskRows || sl >= ns) {
          // expand the bits, each lane its own rows in order
          __syncwarp();
          int r = -1, ent0 = 0;
          unsigned m = 0;
          if (plain) {
            for (;;) {
              while (m == 0 && r + 1 < rows) {
                ++r;
                m = s_mask[wib][r][lane];
                ent0 = s_ent[wib][r];
              }
              if (m == 0) break;
              const int c = __clz(m);
              m ^= 0x80000000u >> c;
              ff.push(ent0 + c);
              if (ff.full()) ff.store(list, true, octets, n, i);
            }
          } else {
            for (;;) {
              while (m == 0 && r + 1 < rows) m = s_mask[wib][++r][lane];
              if (m == 0) break;
              const int c = __clz(m);
              m ^= 0x80000000u >> c;
              const unsigned ent = s_ent[wib][r] + c;
              if (fluid_i && ((s_fluid[wib][r] << c) >> 31)) {
                ff.push(ent);
                if (ff.full()) ff.store(list, true, octets, n, i);
              } else {
                other.push(ent);
                if (other.full()) other.store(list, false, octets, n, i);
              }
            }
          }
          plain = plain0;
          __syncwarp();
          rows = 0;
        }
      }
      if (active) {
        ff.finish(list, true, octets, n, i);
        other.finish(list, false, octets, n, i);
        int cnt = ff.count, cnt_o = other.count;
        if (cnt + cnt_o > cap) {
          // the counts are cut to what fits (every entry below them holds a
          // candidate of this particle), the overflow is reported
          atomicOr(err, gate ? kErrKeptOverflow : kErrNeighOverflow);
          atomicMax(&err[gate ? kErrWordKept : kErrWordNeigh], (unsigned)(cnt + cnt_o));
          cnt = min(cnt, cap);
          cnt_o = min(cnt_o, cap - cnt);
        }
        count[i] = partition ? pack_counts(cnt, cnt_o) : cnt;
      }
    }
  }
}

// end of a gated rebuild: count it and lower the flag
__global__ void k_rebuild_done(int* __restrict__ flag) {
  if (flag[0] != 0) flag[1] += 1;
  flag[0] = 0;
}

// FP64 density over the candidate list: the step's exact pair test with
// MCF's FP64 separation, the step's neighbour list for the force sweeps (nhs:
// the first entry of the forward half the symmetric sweep owns), the W sum and
// the per-particle epilogue.  vl and nl may be the same list (a step's own
// candidates, compacted in place: a kept entry never lands behind one still
// to be read).  The FP32 path runs k_density_list (sweep32.cu).
//
// S lanes per particle: the FP64 pipe needs about three warps per scheduler
// (~58k threads) to stay busy, so small systems deal each particle's
// candidates to 4 or 8 lanes; the lanes' sums are added in lane order.
// 4,096 particles in 2D: 19 us with 8 lanes (one warp a cell, the lanes its
// particles, took 50 us).
template <int D, int S>
__global__ void __launch_bounds__(kReuseTPB)
    k_density_reuse(Consts k, const int* __restrict__ cell_start, const int* __restrict__ cell_of,
                    const double4_32a* __restrict__ x, const double4_32a* __restrict__ v,
                    const double* __restrict__ m, const int* __restrict__ sid,
                    const int* __restrict__ pid, const uint16_t* vl, const int* vcount,
                    uint16_t* nl, int* ncount, int* __restrict__ nhs, int cap,
                    double* __restrict__ rho, double* __restrict__ pr,
                    double4_32a* __restrict__ pc, float4* __restrict__ pcf,
                    float4* __restrict__ vf, int with_pressure, unsigned* __restrict__ err,
                    int* __restrict__ stats, unsigned long long* __restrict__ pairs, NN nn,
                    CollArgs ca) {
  constexpr int CENTER = (D == 3) ? 13 : 4;
  __shared__ int s_start[kMaxStencil * kReuseTPB];
  __shared__ __align__(8) int s_shift[kMaxStencil * kReuseTPB];
  const int n = k.n, tid = threadIdx.x;
  const int gt = blockIdx.x * kReuseTPB + tid;
  const int i = gt / S, lane_s = gt % S;
  int my_max = 0;
  unsigned long long my_pairs = 0;
  int si = 0, kept = 0, back = 0;  // back: kept entries before the forward half
  bool acc_i = false;
  double sum = 0.0;
  if (i < n) {
    const int celli = cell_of[i];
    build_lane_table<D, kReuseTPB>(k, celli, cell_start, s_start, s_shift);
    const int li = i - s_start[CENTER * kReuseTPB + tid];
    si = sid[i];
    acc_i = dyn_rho(k, si);
    const int cnt = vcount[i];
    const double4_32a xi4 = x[i];
    const double xi[3] = {xi4.x, xi4.y, xi4.z};
    const int gbase = (tid & 31) & ~(S - 1);
    const unsigned gmask = (S == 32 ? 0xffffffffu : (1u << S) - 1u) << gbase;
    for (int e0 = 0; e0 < cnt; e0 += S) {
      const int e = e0 + lane_s;
      bool in = false, fwd = false;
      int ent = 0;
      if (S == 1 || e < cnt) {
        ent = vl[up_at(e, n, i)];
        const int sl = ent >> kLocalBits, q = ent & (kMaxCellCount - 1);
        const int j = s_start[sl * kReuseTPB + tid] + q;
        const double4_32a xj4 = x[j];
        const double xj[3] = {xj4.x, xj4.y, xj4.z};
        double r[3];
        const double d2 = exact_sep<D>(k, xi, xj, s_shift[sl * kReuseTPB + tid], r);
        in = !beyond(d2, k.rc2);
        fwd = sl > CENTER || (sl == CENTER && q > li);
        if (in && acc_i) {
          const double w = kernel_w<double>(k, root64(d2));
          sum += (k.rhs_density_type == 1) ? w * m[j] : w;
        }
      }
      if (S == 1) {
        if (!in) continue;
        if (kept < cap) nl[up_at(kept, n, i)] = (uint16_t)ent;
        ++kept;
        back += fwd ? 0 : 1;
      } else {
        // the group's ballots place the kept entries in candidate order
        const unsigned bi = (__ballot_sync(gmask, in) & gmask) >> gbase;
        const unsigned bf = (__ballot_sync(gmask, in && !fwd) & gmask) >> gbase;
        const int pos = kept + __popc(bi & ((1u << lane_s) - 1u));
        if (in && pos < cap) nl[up_at(pos, n, i)] = (uint16_t)ent;
        kept += __popc(bi);
        back += __popc(bf);
      }
    }
  }
  int fi = i;  // the particle this thread finishes
  bool fin = i < n;
  if (S > 1) {
    double* s_sum = reinterpret_cast<double*>(s_shift);
    __syncthreads();
    s_sum[tid] = sum;
    if (lane_s == 0) {
      s_start[tid / S] = kept;
      s_start[kFinish<S> + tid / S] = back;
    }
    __syncthreads();
    fi = blockIdx.x * kFinish<S> + tid;
    fin = tid < kFinish<S> && fi < n;
    if (fin) {
      sum = s_sum[tid * S];
#pragma unroll
      for (int q = 1; q < S; ++q) sum += s_sum[tid * S + q];
      kept = s_start[tid];
      back = s_start[kFinish<S> + tid];
      si = sid[fi];
      acc_i = dyn_rho(k, si);
    }
  }
  if (fin) {
    if (kept > cap) {
      atomicOr(err, kErrNeighOverflow);
      atomicMax(&err[kErrWordNeigh], (unsigned)kept);
    }
    my_max = kept;
    kept = min(kept, cap);
    ncount[fi] = kept;
    nhs[fi] = min(back, kept);
    my_pairs = (unsigned long long)kept;
    const double mi = m[fi];
    double rho_out;
    if (acc_i) {
      rho_out = ((k.rhs_density_type == 1) ? k.w0 * mi : k.w0) + sum;
    } else {
      rho_out = (k.rhs_density_type == 1) ? k.init_density : k.init_density / mi;
    }
    rho[fi] = rho_out;
    if (!(rho_out > 0.0)) atomicOr(err, kErrZeroDensity);
    if (with_pressure) {
      const double4_32a vi4 =
          (si > 0 && k.ncoll > 0) ? colloid_particle_update<D>(k, fi, si, x[fi], ca) : v[fi];
      write_particle_records<true>(k, fi, rho_out, mi, pid[fi], vi4, pr, pc, pcf, vf, nn);
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

template <int D, bool FP64>
__global__ void k_pressure(Consts k, const double* __restrict__ rho, const double* __restrict__ m,
                           const int* __restrict__ pid, const double4_32a* __restrict__ v,
                           double* __restrict__ pr, double4_32a* __restrict__ pc,
                           float4* __restrict__ pcf, float4* __restrict__ vf, NN nn,
                           const int* __restrict__ sid, const double4_32a* __restrict__ x,
                           CollArgs ca) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= k.n) return;
  const int si = sid[i];
  const double4_32a vi4 =
      (si > 0 && k.ncoll > 0) ? colloid_particle_update<D>(k, i, si, x[i], ca) : v[i];
  write_particle_records<FP64>(k, i, rho[i], m[i], pid[i], vi4, pr, pc, pcf, vf, nn);
}

// ---------------------------------------------------------------------------
// FP64 force sweep: Oldroyd-B, stress, colloids, Lees-Edwards (k_force_sym has
// the rest).  S lanes per particle take every S-th entry, as in
// k_density_reuse; their sums are added in lane order.  9,216 2D Oldroyd-B
// particles (288 warps for 608 schedulers with one lane each): the adjoint of 20
// steps 9.3 -> 7.6 ms.  The FP64 pipe bounds it, so the particle's own factor and
// the stress's half follow the loop, and W'/d and the velocity's part of L are
// formed once a pair (55 -> 51 us a launch there).
// ---------------------------------------------------------------------------
template <int D, bool NNW, int S>
__global__ void __launch_bounds__(kReuseTPB)
    k_force64(Consts k, const int* __restrict__ cell_start, const int* __restrict__ cell_of,
              const uint16_t* __restrict__ nl,
              const int* __restrict__ ncount, const double4_32a* __restrict__ x,
              const double4_32a* __restrict__ v, const double4_32a* __restrict__ pc,
              const int* __restrict__ sid, const int* __restrict__ pid,
              double4_32a* __restrict__ f, double* __restrict__ st, int fuse_mode, double dt,
              double4_32a* __restrict__ v_out, uint32_t step_arg,
              const int64_t* __restrict__ step_ptr, double inv_sqdt,
              unsigned* __restrict__ err, NN nn, CollArgs ca) {
  constexpr int D2 = D * D;
  using T = double;
  // the Philox counter's step: the argument, or the device step counter
  // when the sweep runs inside a captured graph
  const uint32_t step = step_ptr ? (uint32_t)*step_ptr : step_arg;
  __shared__ __align__(8) int s_tab[2 * kMaxStencil * kReuseTPB];
  int* const s_start = s_tab;
  int* const s_shift = s_tab + kMaxStencil * kReuseTPB;
  const int n = k.n;
  if (n == 0) return;
  const bool noise = k.noise != 0;
  const int gt = blockIdx.x * kReuseTPB + threadIdx.x;
  const int lane_s = gt % S;
  if (S == 1 && gt >= n) return;
  // lanes past the last particle stay for the block's end, with an empty list
  const int i = S == 1 ? gt : min(gt / S, n - 1);
  build_lane_table<D, kReuseTPB>(k, cell_of[i], cell_start, s_start, s_shift);
  const int si = sid[i];
  const int pidi = pid[i];
  const double4_32a xi4 = x[i];
  const double xi[3] = {xi4.x, xi4.y, xi4.z};
  const double4_32a v4i = v[i];
  const double4_32a ci = pc[i];
  constexpr bool nnw = NNW;  // Oldroyd-B terms compiled only when used
  const double* qq = (const double*)nn.qq;
  T qi[1 + D2], L[D2];
#pragma unroll
  for (int cc = 0; cc < D2; ++cc) L[cc] = 0;
  if (nnw) {
#pragma unroll
    for (int cc = 0; cc <= D2; ++cc) qi[cc] = qq[(size_t)cc * n + i];
  }
  T acc[3] = {0, 0, 0};
  T sacc[9];
#pragma unroll
  for (int a = 0; a < 9; ++a) sacc[a] = 0;
  const int cnt = S == 1 || gt / S < n ? ncount[i] : 0;
  for (int e = lane_s; e < cnt; e += S) {
    const int ent = nl[up_at(e, n, i)];
    const int sl = ent >> kLocalBits, q = ent & (kMaxCellCount - 1);
    const int j = s_start[sl * kReuseTPB + threadIdx.x] + q;
    const int sj = sid[j];
    // pp_interaction.inc:63-223: w-w and c-w never interact, c-c only
    // between different colloids with pp_interact_cc
    if (si != 0 && sj != 0 && !(si > 0 && sj > 0 && si != sj && k.pp_cc)) continue;
    const double4_32a xj4 = x[j];
    const double xj[3] = {xj4.x, xj4.y, xj4.z};
    T r[3];
    const int shj = s_shift[sl * kReuseTPB + threadIdx.x];
    const double d2 = exact_sep<D>(k, xi, xj, shj, r);
    // the kernel's argument is MCF's SQRT(DOT_PRODUCT(rij, rij)), correctly
    // rounded: near the cut-off W'(d) ~ (3 - d/h)^4 amplifies any rounding
    // difference of d by 4 d / (3h - d); 1/d only scales well-conditioned terms
    T inv_d;
    const T d = root64<true>(d2, inv_d);
    const double4_32a v4 = v[j];
    T vi[3] = {v4i.x, v4i.y, v4i.z};
    T vj[3] = {v4.x, v4.y, v4.z};
    if (shj >= kLeUp) le_velocity<T>(k, shj, vi, vj);
    const double4_32a cj = pc[j];
    T Ai = ci.x, Aj = cj.x, Bi = ci.y, Bj = cj.y;
    T qj[1 + D2], qie[1 + D2];
    if (nnw) {
#pragma unroll
      for (int cc = 0; cc <= D2; ++cc) {
        qj[cc] = qq[(size_t)cc * n + j];
        qie[cc] = qi[cc];
      }
    }
    if (si < 0 || sj < 0) {
      // fluid-wall pair: wall particle takes the Morris no-slip velocity
      // and the fluid pressure (pp_interaction_fw.inc / _wf.inc); in the
      // Oldroyd-B model also the fluid density and pressure tensor
      const int sw = (sj < 0) ? sj : si;
      const int axis = (-sw - 1) >> 1;
      const double xin = axis == 0 ? xi[0] : axis == 1 ? xi[1] : xi[2];
      const double xjn = axis == 0 ? xj[0] : axis == 1 ? xj[1] : xj[2];
      T vw[3];
      if (sj < 0) {
        wall_noslip<T, D>(k, xin, xjn, vi, sj, vw);
#pragma unroll
        for (int a = 0; a < D; ++a) vj[a] = vw[a];
        if (nnw) {
          Aj = Ai;
          Bj = Bi;
#pragma unroll
          for (int cc = 0; cc <= D2; ++cc) qj[cc] = qi[cc];
        } else {
          Aj = boundary_A<T>(k.rhs_force_type, ci.w, cj.y);
        }
      } else {
        wall_noslip<T, D>(k, xjn, xin, vj, si, vw);
#pragma unroll
        for (int a = 0; a < D; ++a) vi[a] = vw[a];
        if (nnw) {
          Ai = Aj;
          Bi = Bj;
#pragma unroll
          for (int cc = 0; cc <= D2; ++cc) qie[cc] = qj[cc];
        } else {
          Ai = boundary_A<T>(k.rhs_force_type, cj.w, ci.y);
        }
      }
    } else if ((si > 0) != (sj > 0)) {
      // fluid-colloid pair (pp_interaction_fc.inc / _cf.inc): the
      // boundary particle takes the Morris no-slip velocity and the
      // fluid pressure (Oldroyd-B: also its density and pressure tensor)
      if (sj > 0) {
        if (k.coll_noslip == 2) {
          const double4_32a rc4 = ca.rxc[j];
          const T rxc_[3] = {rc4.x, rc4.y, rc4.z};
          T vw[3];
          colloid_noslip<T, D>(k, sj - 1, rxc_, r, vi, vw);
#pragma unroll
          for (int a = 0; a < D; ++a) vj[a] = vw[a];
        }
        if (nnw) {
          Aj = Ai;
          Bj = Bi;
#pragma unroll
          for (int cc = 0; cc <= D2; ++cc) qj[cc] = qi[cc];
        } else {
          Aj = boundary_A<T>(k.rhs_force_type, ci.w, cj.y);
        }
      } else {
        if (k.coll_noslip == 2) {
          const double4_32a rc4 = ca.rxc[i];
          const T rxc_[3] = {rc4.x, rc4.y, rc4.z};
          const T rfc[3] = {-r[0], -r[1], -r[2]};
          T vw[3];
          colloid_noslip<T, D>(k, si - 1, rxc_, rfc, vj, vw);
#pragma unroll
          for (int a = 0; a < D; ++a) vi[a] = vw[a];
        }
        if (nnw) {
          Ai = Aj;
          Bi = Bj;
#pragma unroll
          for (int cc = 0; cc <= D2; ++cc) qie[cc] = qj[cc];
        } else {
          Ai = boundary_A<T>(k.rhs_force_type, cj.w, ci.y);
        }
      }
    }
    const T gw = kernel_gradw<T>(k, d);
    T vij[3];
#pragma unroll
    for (int a = 0; a < D; ++a) vij[a] = vi[a] - vj[a];
    float z[6];
    if (noise) pair_draw<D>(k.rhs_force_type, k.rk, step, pidi, pid[j], z);
    T pa[3];
    pair_force<T, D>(k, r, inv_d, vij, Ai, Bi, Aj, Bj, gw, noise, z, inv_sqdt, pa);
    if (nnw) {
      // polymer part of the pressure-tensor force,
      // rhs_force_ff_non_Newtonian_HuAdams.F90:95-110, and the velocity
      // gradient of pp_vgt_ip.inc
      const T gwu = gw * inv_d;
#pragma unroll
      for (int b = 0; b < D; ++b) {
        T s_ = 0;
#pragma unroll
        for (int a = 0; a < D; ++a) s_ += (qie[1 + a + D * b] + qj[1 + a + D * b]) * r[a];
        pa[b] += gwu * s_;
      }
      const T fac = -gwu * qie[0];
#pragma unroll
      for (int a = 0; a < D; ++a) {
        const T w = vij[a] * fac;
#pragma unroll
        for (int b = 0; b < D; ++b) L[a + D * b] += w * r[b];
      }
    }
    if (k.rhs_force_type == 1) {
#pragma unroll
      for (int a = 0; a < D; ++a) pa[a] *= cj.z;
    }
#pragma unroll
    for (int a = 0; a < D; ++a) acc[a] += pa[a];
    if (k.stress) {
      // pp_interaction_ff.inc:83-93: s_ab += r_a * f_b / 2
#pragma unroll
      for (int b = 0; b < D; ++b)
#pragma unroll
        for (int a = 0; a < D; ++a) sacc[b * D + a] += r[a] * pa[b];
    }
  }
  // the particle's own factor (all forms but Morris'), and the half of
  // the stress
  const T own = k.rhs_force_type == 1 ? T(1) : ci.z;
#pragma unroll
  for (int a = 0; a < D; ++a) acc[a] *= own;
  if (k.stress) {
#pragma unroll
    for (int a = 0; a < D2; ++a) sacc[a] *= T(0.5) * own;
  }
  int fi = i, fsi = si;  // the particle this thread finishes
  double xf[3] = {xi[0], xi[1], xi[2]};
  if (S > 1) {
    // planes of the block's partial sums: acc | L | stress
    static_assert((D + 2 * D2) * 2 <= 2 * kMaxStencil, "partial sums fit over the tables");
    double* s_sum = reinterpret_cast<double*>(s_tab);
    const int tid = threadIdx.x;
    __syncthreads();
#pragma unroll
    for (int a = 0; a < D; ++a) s_sum[a * kReuseTPB + tid] = acc[a];
#pragma unroll
    for (int cc = 0; cc < D2; ++cc) {
      if (nnw) s_sum[(D + cc) * kReuseTPB + tid] = L[cc];
      if (k.stress) s_sum[(D + D2 + cc) * kReuseTPB + tid] = sacc[cc];
    }
    __syncthreads();
    fi = blockIdx.x * kFinish<S> + tid;
    if (tid >= kFinish<S> || fi >= n) return;
    // in lane order
    auto total = [&](int c) {
      const double* part = s_sum + c * kReuseTPB + tid * S;
      double tot = part[0];
#pragma unroll
      for (int q = 1; q < S; ++q) tot += part[q];
      return tot;
    };
#pragma unroll
    for (int a = 0; a < D; ++a) acc[a] = total(a);
#pragma unroll
    for (int cc = 0; cc < D2; ++cc) {
      if (nnw) L[cc] = total(D + cc);
      if (k.stress) sacc[cc] = total(D + D2 + cc);
    }
    fsi = sid[fi];
    const double4_32a xf4 = x[fi];
    xf[0] = xf4.x;
    xf[1] = xf4.y;
    xf[2] = xf4.z;
  }
  if (k.stress) {
#pragma unroll
    for (int a = 0; a < D * D; ++a) st[(size_t)a * n + fi] = sacc[a];
  }
  if (nnw) nn_epilogue<D>(k, nn, fi, L, fuse_mode, dt);
  force_epilogue<D>(k, fi, fsi, xf, acc[0], acc[1], D == 3 ? acc[2] : 0.0, fuse_mode, dt, v,
                    f, v_out, err);
}

// ---------------------------------------------------------------------------
// FP32-mixed force sweep of Oldroyd-B, the Morris and Espanol forms and runs with
// the per-particle stress (the other forms: force32.cu): pair arithmetic in FP32 on cell offsets, Kahan
// sums, the next pair's data loaded while the current one is computed.
// ---------------------------------------------------------------------------
// S lanes per particle (1, or 4 for small systems, where one thread per
// particle leaves most of the GPU idle and each thread's serial pair loop
// sets the time): lane l takes list entries l, l + S, ...; the lanes' sums
// are added in lane order by the thread that runs its epilogue.
// STRESS: the per-particle stress s_i += r_ij (x) a_ij / 2 is accumulated
// (a compile-time switch: its nine sums would otherwise stay live across
// the pair loop of every run).  The 3D Oldroyd-B instances take 4 blocks
// per SM: at 5 (96 registers) they spill the polymer terms.
template <int D, bool NNW, int S, bool STRESS>
__global__ void __launch_bounds__(kReuseTPB, (NNW && D == 3) ? 4 : 5)
    k_force32(Consts k, const int* __restrict__ cell_start, const int* __restrict__ cell_of,
              const uint16_t* __restrict__ nl, const int* __restrict__ ncount, int cap,
              const float4* __restrict__ off,
              const double4_32a* __restrict__ x, const double4_32a* __restrict__ v,
              const float4* __restrict__ vf,
              const float2* __restrict__ wd, double4_32a* __restrict__ f,
              double* __restrict__ st, int fuse_mode, double dt,
              double4_32a* __restrict__ v_out, uint32_t step_arg,
              const int64_t* __restrict__ step_ptr, float inv_sqdt,
              unsigned* __restrict__ err, NN nn, CollArgs ca) {
  constexpr int D2 = D * D;
  using T = float;
  const uint32_t step = step_ptr ? (uint32_t)*step_ptr : step_arg;
  // one thread per particle, whatever its cell: per-thread neighbour-cell
  // tables keep every lane busy (2D cells hold ~9 particles)
  __shared__ int s_start[kMaxStencil * kReuseTPB];
  const int n = k.n;
  if (n == 0) return;
  const bool noise = k.noise != 0;
  const bool walls = k.wall_axis != -1;
  __shared__ float4 s_slot[kSlotTable];
  fill_slot_offsets<D>(k, s_slot);
  __syncthreads();
  const int gt = blockIdx.x * kReuseTPB + threadIdx.x;
  const int lane_s = gt % S;
  if (S == 1 && gt >= n) return;
  // lanes past the last particle stay for the block's end, with an empty list
  const int i = S == 1 ? gt : min(gt / S, n - 1);
  const int celli = cell_of[i];
  build_lane_table<D, kReuseTPB, false>(k, celli, cell_start, s_start, nullptr);
  const float4* slot_tab = slot_table(k, s_slot, celli);
  const float4 oi = off[i];
  const int si = __float_as_int(oi.w);
  float4 v4i, ci;
  load_vc(vf, i, v4i, ci);
  const int pidi = __float_as_int(v4i.w);
  const float2 wdi = (walls && k.wall_axis >= 0) ? wd[i] : make_float2(0.f, 0.f);
  constexpr bool nnw = NNW;  // Oldroyd-B terms compiled only when used
  const float* qq = (const float*)nn.qq;
  T qi[1 + D2], L[D2];
#pragma unroll
  for (int cc = 0; cc < D2; ++cc) L[cc] = 0.f;
  if (nnw) {
#pragma unroll
    for (int cc = 0; cc <= D2; ++cc) qi[cc] = qq[(size_t)cc * n + i];
  }
  T acc[3] = {0.f, 0.f, 0.f}, comp[3] = {0.f, 0.f, 0.f};
  T sacc[9];
#pragma unroll
  for (int a = 0; a < 9; ++a) sacc[a] = 0.f;
  // the list's two segments: fluid-fluid pairs, then the others
  const int nc = S == 1 || gt / S < n ? ncount[i] : 0;
  const int nff = first_count(nc), cnt = nff + second_count(nc);
  JData nxt;
  int ent_n1 = 0;
  if (lane_s < cnt)
    nxt = load_j(s_start, nl[entry_at(lane_s, nff, cap, n, i)], off, vf);
  if (lane_s + S < cnt) ent_n1 = nl[entry_at(lane_s + S, nff, cap, n, i)];
  for (int e = lane_s; e < cnt; e += S) {
    const JData cur = nxt;
    if (e + S < cnt) {
      nxt = load_j(s_start, ent_n1, off, vf);
      if (e + 2 * S < cnt) ent_n1 = nl[entry_at(e + 2 * S, nff, cap, n, i)];
    }
    const int sj = __float_as_int(cur.o.w);
    if (si != 0 && sj != 0 && !(si > 0 && sj > 0 && si != sj && k.pp_cc)) continue;
    const int sl = cur.sl;
    T r[3];
    const float4 so = slot_tab[sl];
    r[0] = (oi.x - cur.o.x) - so.x;
    r[1] = (oi.y - cur.o.y) - so.y;
    r[2] = (D == 3) ? (oi.z - cur.o.z) - so.z : 0.f;
    T d2 = r[0] * r[0] + r[1] * r[1];
    if (D == 3) d2 += r[2] * r[2];
    const T inv_d = rsqrtf(d2);
    const T d = d2 * inv_d;
    T vi[3] = {v4i.x, v4i.y, v4i.z};
    T vj[3] = {cur.v.x + so.w, cur.v.y, cur.v.z};
    T Ai = ci.x, Aj = cur.c.x, Bi = ci.y, Bj = cur.c.y;
    T qj[1 + D2], qie[1 + D2];
    if (nnw) {
#pragma unroll
      for (int cc = 0; cc <= D2; ++cc) {
        qj[cc] = qq[(size_t)cc * n + cur.j];
        qie[cc] = qi[cc];
      }
    }
    if (si < 0 || sj < 0 || (si > 0) != (sj > 0))
      boundary_pair32<D, NNW>(k, i, cur.j, si, sj, r, wdi, wd, x, ca, ci.w, cur.c.w, vi, vj, Ai,
                              Aj, Bi, Bj, qi, qie, qj);
    const T gw = kernel_gradw<T>(k, d);
    T vij[3];
#pragma unroll
    for (int a = 0; a < D; ++a) vij[a] = vi[a] - vj[a];
    float z[6];
    if (noise)
      pair_draw<D>(k.rhs_force_type, k.rk, step, pidi, __float_as_int(cur.v.w), z);
    T pa[3], si_s, sj_s;
    pair_force<T, D>(k, r, inv_d, vij, Ai, Bi, Aj, Bj, gw, noise, z, inv_sqdt, pa);
    if (nnw) {
      // polymer pressure-tensor force and velocity gradient (FP32 pairs)
#pragma unroll
      for (int b = 0; b < D; ++b) {
        T s_ = 0.f;
#pragma unroll
        for (int a = 0; a < D; ++a) s_ += (qie[1 + a + D * b] + qj[1 + a + D * b]) * r[a];
        pa[b] += gw * inv_d * s_;
      }
      const T fac = gw * qie[0] * inv_d;
#pragma unroll
      for (int b = 0; b < D; ++b)
#pragma unroll
        for (int a = 0; a < D; ++a) L[a + D * b] += (vj[a] - vi[a]) * r[b] * fac;
    }
    pair_scales<T>(k.rhs_force_type, ci.z, cur.c.z, si_s, sj_s);
#pragma unroll
    for (int a = 0; a < D; ++a) pa[a] *= si_s;
#pragma unroll
    for (int a = 0; a < D; ++a) {
      const T y = pa[a] - comp[a];
      const T tt = acc[a] + y;
      comp[a] = (tt - acc[a]) - y;
      acc[a] = tt;
    }
    if (STRESS) {
#pragma unroll
      for (int b = 0; b < D; ++b)
#pragma unroll
        for (int a = 0; a < D; ++a) sacc[b * D + a] += r[a] * pa[b] * 0.5f;
    }
  }
  int fi = i, fsi = si;  // the particle this thread finishes
  if (S > 1) {
    // planes of the block's partial sums: acc | L | stress
    static_assert(D + 2 * D2 <= kMaxStencil, "partial sums fit over the table");
    float* s_sum = reinterpret_cast<float*>(s_start);
    const int tid = threadIdx.x;
    __syncthreads();
#pragma unroll
    for (int a = 0; a < D; ++a) s_sum[a * kReuseTPB + tid] = acc[a] - comp[a];
#pragma unroll
    for (int cc = 0; cc < D2; ++cc) {
      if (nnw) s_sum[(D + cc) * kReuseTPB + tid] = L[cc];
      if (STRESS) s_sum[(D + D2 + cc) * kReuseTPB + tid] = sacc[cc];
    }
    __syncthreads();
    fi = blockIdx.x * kFinish<S> + tid;
    if (tid >= kFinish<S> || fi >= n) return;
    // in lane order
    auto total = [&](int c) {
      const float* part = s_sum + c * kReuseTPB + tid * S;
      T tot = part[0];
#pragma unroll
      for (int q = 1; q < S; ++q) tot += part[q];
      return tot;
    };
#pragma unroll
    for (int a = 0; a < D; ++a) acc[a] = total(a);
#pragma unroll
    for (int cc = 0; cc < D2; ++cc) {
      if (nnw) L[cc] = total(D + cc);
      if (STRESS) sacc[cc] = total(D + D2 + cc);
    }
    fsi = __float_as_int(off[fi].w);
  }
  if (STRESS) {
#pragma unroll
    for (int a = 0; a < D * D; ++a) st[(size_t)a * n + fi] = (double)sacc[a];
  }
  const double4_32a xi4 = x[fi];
  const double xi[3] = {xi4.x, xi4.y, xi4.z};
  if (nnw) {
    double Ld[D2];
#pragma unroll
    for (int cc = 0; cc < D2; ++cc) Ld[cc] = (double)L[cc];
    nn_epilogue<D>(k, nn, fi, Ld, fuse_mode, dt);
  }
  force_epilogue<D>(k, fi, fsi, xi, (double)acc[0], (double)acc[1],
                    D == 3 ? (double)acc[2] : 0.0, fuse_mode, dt, v, f, v_out, err);
}

// ---------------------------------------------------------------------------
// Symmetric FP64 force sweep: every pair is evaluated once, by the particle
// whose cell owns it (partner in one of the 13 forward cells, or later in the
// same cell: the half-shell of ppm_neighlist_MkNeighIdx.F90:198-249).  A warp
// takes a cell; the owned pairs of its particles, in owner order, are dealt to
// the lanes in runs of kRun consecutive pairs, so that all lanes work whatever
// the particles' list lengths.  The partner's share is summed per (forward
// slot, partner) in shared memory; lanes that hit the same partner in one
// round are combined with __match_any_sync, in lane order, by the lowest such
// lane.  The owner's share is summed in the lane while its run stays with one
// owner, then over the lanes by a segmented shuffle.  Every sum has a fixed
// order: the result is deterministic without atomics.  The partner sums go to
// planes jp[slot][c][n] that k_force_gather adds up per particle.
//
// Bound: the FP64 pipe (84% busy); what counts is FP64 slots a pair.  Runs of
// 4 spread the owner reduction (15 adds + 3) over 128 pairs; the mass factor
// is left to the gather (not for the Morris form, whose factor is the
// partner's mass).  COOP: a block's warps share one cell, for systems with few
// cells (kCoopCells).  64^3 with noise: 2.64 ms, 86 slots
// a pair, against 3.02 ms and 100 with one pair a round and lane.
// ---------------------------------------------------------------------------
// partners per slot held in shared memory (a fuller cell's sums lie in global
// memory): systems with few cells can afford more
template <int D, bool COOP>
constexpr int kSymCC = (D == 3 && COOP) ? 64 : 32;

// Per-warp dynamic shared memory of k_force_sym (bytes):
// part[NSF][D][CC] | acc[D][32] | ex[33] e0[32] pad | x v pc [32] sid pid [32]
template <int D, bool COOP>
__host__ __device__ constexpr int sym_warp_bytes() {
  constexpr int NSF = (D == 3) ? 14 : 5;
  constexpr int part = NSF * D * kSymCC<D, COOP> * 8;
  constexpr int acc = D * 32 * 8;
  constexpr int idx = 96 * 4;
  constexpr int own = 3 * 32 * 32 + 2 * 32 * 4;
  return (part + acc + idx + own + 31) / 32 * 32;
}

template <int D, bool COOP>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
    k_force_sym(Consts k, const int* __restrict__ cell_start, const uint16_t* __restrict__ nl,
                const int* __restrict__ ncount, const int* __restrict__ nhs,
                const double4_32a* __restrict__ x, const double4_32a* __restrict__ v,
                const double4_32a* __restrict__ pc, const int* __restrict__ sid,
                const int* __restrict__ pid, double* __restrict__ jp, uint32_t step_arg,
                const int64_t* __restrict__ step_ptr, double inv_sqdt) {
  // the Philox counter's step: the argument, or the device step counter
  // when the sweep runs inside a captured graph
  const uint32_t step = step_ptr ? (uint32_t)*step_ptr : step_arg;
  constexpr int CC = kSymCC<D, COOP>;
  constexpr int kRun = (COOP && D == 2) ? 1 : 4;  // consecutive pairs a lane takes in a round
  constexpr int CENTER = (D == 3) ? 13 : 4;
  constexpr int NSF = (D == 3) ? 14 : 5;  // forward slots CENTER..NS-1
  extern __shared__ __align__(32) unsigned char smem_raw[];
  __shared__ NbTable tab[kWarpsPerBlock];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char* wb = smem_raw + (size_t)wib * sym_warp_bytes<D, COOP>();
  double* part = reinterpret_cast<double*>(wb);
  double* acc_s = part + NSF * D * CC;
  int* ex = reinterpret_cast<int*>(acc_s + D * 32);
  int* e0s = ex + 33;
  double4_32a* ox = reinterpret_cast<double4_32a*>(ex + 96);
  int* os = reinterpret_cast<int*>(ox + 96);
  const int n = k.n;
  const bool noise = k.noise != 0;
  const bool scaled = k.rhs_force_type == 1;
  for (int cell = COOP ? blockIdx.x : blockIdx.x * kWarpsPerBlock + wib; cell <= k.ncell;
       cell += gridDim.x * (COOP ? 1 : kWarpsPerBlock)) {
    NbTable& t = tab[wib];
    build_table<D>(k, cell, cell_start, t);
    // shared cells: the warps take rounds in turn, each with sums of its own;
    // sums in global memory (a neighbour cell of more than CC) have one writer
    bool solo = false;
    if (COOP)
      for (int s = 0; s < NSF; ++s) solo = solo || t.count[CENTER + s] > CC;
    // zero the partner sums this cell owns (shared, or global when a cell
    // holds more than CC particles)
    for (int s = 0; s < NSF; ++s) {
      const int cs_ = t.count[CENTER + s], st_ = t.start[CENTER + s];
      for (int q = lane; q < cs_; q += 32)
#pragma unroll
        for (int a = 0; a < D; ++a) {
          if (cs_ <= CC)
            part[(s * D + a) * CC + q] = 0.0;
          else if (!COOP || wib == 0)
            jp[((size_t)s * D + a) * n + st_ + q] = 0.0;
        }
    }
    const int c0 = t.start[CENTER], c1 = c0 + t.count[CENTER];
    for (int base = c0; base < c1; base += 32) {
      const int i = base + lane;
      const bool act = i < c1;
      const int e0 = act ? nhs[i] : 0, e1 = act ? ncount[i] : 0;
      const int len = e1 - e0;
      // owner data and accumulators of this chunk in shared memory
      if (act) {
        ox[lane] = x[i];
        ox[32 + lane] = v[i];
        ox[64 + lane] = pc[i];
        os[lane] = sid[i];
        os[32 + lane] = pid[i];
      }
#pragma unroll
      for (int a = 0; a < D; ++a) acc_s[a * 32 + lane] = 0.0;
      // exclusive prefix of the owned-pair counts
      int incl = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int tt = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += tt;
      }
      const int total = __shfl_sync(0xffffffffu, incl, 31);
      ex[lane] = incl - len;
      e0s[lane] = e0;
      if (lane == 31) ex[32] = total;
      __syncwarp();
      const int turns = (COOP && !solo) ? kWarpsPerBlock : 1;
      const int mine = COOP && solo && wib > 0 ? 0 : total;
      for (int r0 = (turns > 1 ? wib : 0) * 32 * kRun; r0 < mine; r0 += turns * 32 * kRun) {
        // the run's first pair and its owner
        int fidx = r0 + lane * kRun;
        int ow_l = 0;
#pragma unroll
        for (int stp = 16; stp > 0; stp >>= 1)
          if (ex[ow_l + stp] <= fidx) ow_l += stp;
        double vis[3] = {0, 0, 0};  // the share of owner ow_l summed in this lane
#pragma unroll 1
        for (int u = 0; u < kRun; ++u, ++fidx) {
          const bool valid = fidx < total;
          // the run passes into the next owner's pairs: the finished owner's
          // share goes to its sum (at most one lane ends a given owner's pairs)
          const bool next = valid && fidx >= ex[ow_l + 1];
          if (__any_sync(0xffffffffu, next)) {
            if (next) {
#pragma unroll
              for (int a = 0; a < D; ++a) {
                acc_s[a * 32 + ow_l] += vis[a];
                vis[a] = 0.0;
              }
              do ++ow_l;
              while (fidx >= ex[ow_l + 1]);
            }
          }
          bool has = false;
          int keyj = 0, jsl = 0, jq = 0;
          double g[3] = {0, 0, 0}, s_j = 1.0;
          if (valid) {
            const int ii = base + ow_l;
            const int e = e0s[ow_l] + (fidx - ex[ow_l]);
            const int ent = nl[up_at(e, n, ii)];
            jsl = ent >> kLocalBits;
            jq = ent & (kMaxCellCount - 1);
            const int j = t.start[jsl] + jq;
            const int si = os[ow_l], sj = sid[j];
            has = !(si != 0 && sj != 0);  // w-w, c-c, c-w: no interaction here
            if (has) {
              const double4_32a x4 = ox[ow_l], v4 = ox[32 + ow_l], c4 = ox[64 + ow_l];
              const double4_32a xj4 = x[j], vj4 = v[j], cj4 = pc[j];
              const double xi[3] = {x4.x, x4.y, x4.z}, xj[3] = {xj4.x, xj4.y, xj4.z};
              double rr[3] = {0, 0, 0};
              const double d2 = exact_sep<D>(k, xi, xj, t.shift[jsl], rr);
              // MCF's correctly rounded SQRT for the kernel's argument (see
              // k_force64)
              double inv_d;
              const double d = root64<true>(d2, inv_d);
              double vi[3] = {v4.x, v4.y, v4.z}, vj[3] = {vj4.x, vj4.y, vj4.z};
              double Ai = c4.x, Aj = cj4.x;
              if (si < 0 || sj < 0) {
                // fluid-wall pair (pp_interaction_fw.inc / _wf.inc)
                const int sw = (sj < 0) ? sj : si;
                const int axis = (-sw - 1) >> 1;
                const double xa = axis == 0 ? xi[0] : axis == 1 ? xi[1] : xi[2];
                const double xb = axis == 0 ? xj[0] : axis == 1 ? xj[1] : xj[2];
                double vw[3];
                if (sj < 0) {
                  wall_noslip<double, D>(k, xa, xb, vi, sj, vw);
#pragma unroll
                  for (int a = 0; a < D; ++a) vj[a] = vw[a];
                  Aj = boundary_A<double>(k.rhs_force_type, c4.w, cj4.y);
                } else {
                  wall_noslip<double, D>(k, xb, xa, vj, si, vw);
#pragma unroll
                  for (int a = 0; a < D; ++a) vi[a] = vw[a];
                  Ai = boundary_A<double>(k.rhs_force_type, cj4.w, c4.y);
                }
              }
              const double gw = kernel_gradw<double>(k, d);
              double vij[3];
#pragma unroll
              for (int a = 0; a < D; ++a) vij[a] = vi[a] - vj[a];
              float z[6];
              if (noise) pair_draw<D>(k.rhs_force_type, k.rk, step, os[32 + ow_l], pid[j], z);
              pair_force<double, D>(k, rr, inv_d, vij, Ai, c4.y, Aj, cj4.y, gw, noise, z,
                                    inv_sqdt, g);
              if (scaled) {
#pragma unroll
                for (int a = 0; a < D; ++a) vis[a] += g[a] * cj4.z;
                s_j = c4.z;
              } else {
#pragma unroll
                for (int a = 0; a < D; ++a) vis[a] += g[a];
              }
              keyj = (jsl - CENTER) * kMaxCellCount + jq;
            }
          }
          // partner side: lanes with the same partner are summed in lane
          // order by the lowest of them
          const unsigned amask = __ballot_sync(0xffffffffu, has);
          if (has) {
            if (scaled) {
#pragma unroll
              for (int a = 0; a < D; ++a) g[a] *= s_j;
            }
            const unsigned peers = __match_any_sync(amask, keyj);
            double sum[3] = {g[0], g[1], g[2]};
            if (peers != (1u << lane)) {
              sum[0] = sum[1] = sum[2] = 0.0;
              for (unsigned mm = peers; mm; mm &= mm - 1) {
                const int src = __ffs(mm) - 1;
#pragma unroll
                for (int a = 0; a < D; ++a) sum[a] += __shfl_sync(peers, g[a], src);
              }
            }
            if (lane == __ffs(peers) - 1) {
              const int s = jsl - CENTER;
              if (t.count[jsl] <= CC) {
#pragma unroll
                for (int a = 0; a < D; ++a) part[(s * D + a) * CC + jq] -= sum[a];
              } else {
                const size_t b0 = (size_t)t.start[jsl] + jq;
#pragma unroll
                for (int a = 0; a < D; ++a) jp[((size_t)s * D + a) * n + b0] -= sum[a];
              }
            }
          }
          __syncwarp();
        }
        // owner side: the runs lie in owner order, so the lanes whose run ends
        // with one owner are adjacent; five segmented shuffle steps leave their
        // sum in the first of them
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const bool same = __shfl_down_sync(0xffffffffu, ow_l, o) == ow_l && lane + o < 32;
#pragma unroll
          for (int a = 0; a < D; ++a) {
            const double t2 = __shfl_down_sync(0xffffffffu, vis[a], o);
            if (same) vis[a] += t2;
          }
        }
        const int ow_prev = __shfl_up_sync(0xffffffffu, ow_l, 1);
        if (lane == 0 || ow_prev != ow_l) {
#pragma unroll
          for (int a = 0; a < D; ++a) acc_s[a * 32 + ow_l] += vis[a];
        }
        __syncwarp();
      }
      // this warp's sums, or in a shared cell all warps' in warp order
      constexpr int kHop = sym_warp_bytes<D, COOP>() / 8;
      if (COOP) __syncthreads();
      if (act && (!COOP || wib == 0)) {
#pragma unroll
        for (int a = 0; a < D; ++a) {
          double sum = acc_s[a * 32 + lane];
          if (COOP)
#pragma unroll
            for (int w = 1; w < kWarpsPerBlock; ++w) sum += acc_s[w * kHop + a * 32 + lane];
          jp[((size_t)NSF * D + a) * n + i] = sum;
        }
      }
      if (COOP)
        __syncthreads();
      else
        __syncwarp();
    }
    constexpr int kHop = sym_warp_bytes<D, COOP>() / 8;
    const double* part0 = COOP ? reinterpret_cast<const double*>(smem_raw) : part;
    // a shared cell's warps read each other's sums below: those of a cell without
    // particles, which has met no barrier above, are its zeros
    if (COOP)
      __syncthreads();
    else
      __syncwarp();
    for (int s = COOP ? wib : 0; s < NSF; s += COOP ? kWarpsPerBlock : 1) {
      const int cs_ = t.count[CENTER + s], st_ = t.start[CENTER + s];
      if (cs_ > CC) continue;
      for (int q = lane; q < cs_; q += 32)
#pragma unroll
        for (int a = 0; a < D; ++a) {
          double sum = part0[(s * D + a) * CC + q];
          if (COOP)
#pragma unroll
            for (int w = 1; w < kWarpsPerBlock; ++w) sum += part0[w * kHop + (s * D + a) * CC + q];
          jp[((size_t)s * D + a) * n + st_ + q] = sum;
        }
    }
    if (COOP)
      __syncthreads();
    else
      __syncwarp();
  }
}

// Sum of the per-slot partner shares and the owner share of every particle
// (fixed order) times the mass factor, then body force and the second half
// kick.
template <int D>
__global__ void k_force_gather(Consts k, const int* __restrict__ cell_of,
                               const double* __restrict__ jp,
                               const double4_32a* __restrict__ x,
                               const double4_32a* __restrict__ v,
                               const double4_32a* __restrict__ pc, const int* __restrict__ sid,
                               double4_32a* __restrict__ f, int fuse_mode, double dt,
                               double4_32a* __restrict__ v_out, unsigned* __restrict__ err) {
  constexpr int CENTER = (D == 3) ? 13 : 4;
  constexpr int NSF = (D == 3) ? 14 : 5;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = k.n;
  if (j >= n) return;
  const int cj = cell_of[j];
  int cc[3] = {0, 0, 0};
  if (cj < k.ncell) {
    int rem = cj;
#pragma unroll
    for (int a = 0; a < D; ++a) {
      cc[a] = rem % k.nm[a];
      rem /= k.nm[a];
    }
  }
  double acc[3] = {0, 0, 0};
#pragma unroll
  for (int a = 0; a < D; ++a) acc[a] = jp[((size_t)NSF * D + a) * n + j];
  if (cj < k.ncell) {
#pragma unroll
    for (int s = 0; s < NSF; ++s) {
      // the owner cell of plane s is cell(j) - offset(CENTER + s)
      const int sl = CENTER + s;
      const int o[3] = {sl % 3 - 1, (sl / 3) % 3 - 1, sl / 9 - 1};
      bool ok = true;
#pragma unroll
      for (int a = 0; a < D; ++a) {
        const int h = cc[a] - o[a];
        if ((h < 0 || h >= k.nm[a]) && !k.periodic[a]) ok = false;
      }
      if (!ok) continue;
#pragma unroll
      for (int a = 0; a < D; ++a) acc[a] += jp[((size_t)s * D + a) * n + j];
    }
  }
  if (k.rhs_force_type != 1) {
    const double scale = pc[j].z;
#pragma unroll
    for (int a = 0; a < D; ++a) acc[a] *= scale;
  }
  const double4_32a x4 = x[j];
  const double xj[3] = {x4.x, x4.y, x4.z};
  force_epilogue<D>(k, j, sid[j], xj, acc[0], acc[1], D == 3 ? acc[2] : 0.0, fuse_mode, dt, v, f,
                    v_out, err);
}

static int grid_for(Handle* h) {
  const int warps = h->k.ncell + 1;  // + bin of particles without a cell
  int g = (warps + kWarpsPerBlock - 1) / kWarpsPerBlock;
  return g < 1 ? 1 : g;
}

// candidates within sqrt(lim) of every particle into list / count
static int scan_launch(Handle* h, const int* gate, float lim, uint16_t* list, int* count, int cap,
                       bool partition, bool exact) {
  const int g = grid_for(h);
#define LAUNCH_S(DD, EX)                                                                          \
  k_scan<DD, EX><<<g, kWarpsPerBlock * 32, 0, h->stream>>>(h->k, gate, h->cell_start, h->off, lim, \
                                                           list, count, cap, partition ? 1 : 0,    \
                                                           h->d_err)
  if (h->k.d == 3) {
    if (exact) LAUNCH_S(3, true); else LAUNCH_S(3, false);
  } else {
    if (exact) LAUNCH_S(2, true); else LAUNCH_S(2, false);
  }
#undef LAUNCH_S
  h->launches++;
  return cuda_check(h, cudaGetLastError(), "candidate list launch") ? MCFG_ECUDA : MCFG_OK;
}

int verlet_build_gated(Handle* h) {
  const int rc = scan_launch(h, h->d_rebuild, h->k.rv2f, h->vl, h->vcount, h->vcap, h->partitioned,
                             false);
  if (rc) return rc;
  k_rebuild_done<<<1, 1, 0, h->stream>>>(h->d_rebuild);
  h->launches++;
  return cuda_check(h, cudaGetLastError(), "candidate list launch") ? MCFG_ECUDA : MCFG_OK;
}

// Density of the current particle order.  reuse: over the candidate list of
// the last rebuild; otherwise the step's own candidates are listed first, in
// nl, and compacted in place (FP32: within the cut-off by the same test; FP64:
// with the prefilter's slack, the exact test follows).
int compute_density(Handle* h, bool with_pressure, bool reuse) {
  Consts& k = h->k;
  cudaStream_t s = h->stream;
  const int n = (int)h->n;
  if (!h->stats_cleared &&
      (cuda_check(h, cudaMemsetAsync(h->d_stats, 0, sizeof(int) * 4, s), "memset stats") ||
       cuda_check(h, cudaMemsetAsync(h->d_pairs, 0, sizeof(unsigned long long), s),
                  "memset pairs")))
    return MCFG_ECUDA;
  if (n == 0) return MCFG_OK;
  const bool fp64 = h->p.precision == MCFG_PRECISION_FP64;
  const uint16_t* vl = reuse ? h->vl : h->nl;
  const int* vcount = reuse ? h->vcount : h->ncount;
  if (!reuse) {
    const int rc = scan_launch(h, nullptr, fp64 ? k.rc2f_hi : k.rc2f, h->nl, h->ncount,
                               h->neigh_cap, !fp64, !fp64);
    if (rc) return rc;
  }
  if (!fp64) return density_list(h, with_pressure, vl, vcount, reuse ? h->vcap : h->neigh_cap);
  const int S = n < kSplit8Below ? 8 : n < kSplitBelow ? 4 : 1;
  const int gr = (int)(((int64_t)n * S + kReuseTPB - 1) / kReuseTPB);
#define LAUNCH_R(DD, SS)                                                                        \
  k_density_reuse<DD, SS><<<gr, kReuseTPB, 0, s>>>(                                             \
      k, h->cell_start, h->cell_of, h->x, h->v, h->m, h->sid, h->pid, vl, vcount, h->nl,        \
      h->ncount, h->nhs, h->neigh_cap, h->rho, h->pr, h->pc, h->pcf, h->vf,                     \
      with_pressure ? 1 : 0, h->d_err, h->d_stats, h->d_pairs, NN{h->ct, h->act, h->vgt, h->qq}, \
      CollArgs{h->v, h->rxc, h->rxcf})
#define PICK_R(DD)                      \
  do {                                  \
    if (S == 8) LAUNCH_R(DD, 8);        \
    else if (S == 4) LAUNCH_R(DD, 4);   \
    else LAUNCH_R(DD, 1);               \
  } while (0)
  if (k.d == 3) PICK_R(3); else PICK_R(2);
#undef PICK_R
#undef LAUNCH_R
  h->launches++;
  return cuda_check(h, cudaGetLastError(), "density launch") ? MCFG_ECUDA : MCFG_OK;
}

int compute_pressure(Handle* h) {
  const int n = (int)h->n;
  if (n == 0) return MCFG_OK;
  const int tb = 256, gb = (n + tb - 1) / tb;
  const NN nn{h->ct, h->act, h->vgt, h->qq};
  const CollArgs ca{h->v, h->rxc, h->rxcf};
#define LAUNCH_P(DD, PP)                                                                        \
  k_pressure<DD, PP><<<gb, tb, 0, h->stream>>>(h->k, h->rho, h->m, h->pid, h->v, h->pr, h->pc,   \
                                               h->pcf, h->vf, nn, h->sid, h->x, ca)
  if (h->p.precision == MCFG_PRECISION_FP64) {
    if (h->k.d == 3) LAUNCH_P(3, true); else LAUNCH_P(2, true);
  } else {
    if (h->k.d == 3) LAUNCH_P(3, false); else LAUNCH_P(2, false);
  }
#undef LAUNCH_P
  h->launches++;
  if (cuda_check(h, cudaGetLastError(), "pressure launch")) return MCFG_ECUDA;
  return MCFG_OK;
}

// below this many cells the symmetric sweep's warps share cells
// (us a step, own cells / shared: 3D 100 cells 719 / 235, 1,000 896 / 729, 4,913
// 2664 / 2612, 9,261 4446 / 4558; 2D 441 cells 69 / 54, 9,801 350 / 349)
constexpr int kCoopCells = 6000;

int compute_force(Handle* h, int64_t step, int fuse_mode, double dt) {
  Consts& k = h->k;
  cudaStream_t s = h->stream;
  const int g = grid_for(h);
  const bool fp64 = h->p.precision == MCFG_PRECISION_FP64;
  if (k.noise && !(dt > 0.0)) return set_error(h, MCFG_EINVAL, "random force needs dt > 0");
  const double inv_sqdt = (k.noise && dt > 0.0) ? 1.0 / sqrt(dt) : 0.0;
  const int bs = kWarpsPerBlock * 32;
  const NN nn{h->ct, h->act, h->vgt, h->qq};
  const CollArgs ca{h->v, h->rxc, h->rxcf};
  const int gp = std::max(1, ((int)h->n + kReuseTPB - 1) / kReuseTPB);
  const int64_t* step_ptr = h->graph_capturing ? h->d_step : nullptr;
  // small systems: 4 lanes per particle in the FP32 sweep
  const bool split = h->n < kSplitBelow;
  const int gp4 = std::max(1, (int)((h->n * 4 + kReuseTPB - 1) / kReuseTPB));
  if (!k.stress && h->jp && fp64 && k.newtonian && k.ncoll == 0 && !k.le) {
    // symmetric sweep + per-particle gather: halves the FP64 pair work; the
    // FP32 path keeps the two-sided sweep, which is faster there (the
    // symmetric sweep's shared-memory partner sums cap its occupancy)
    const int n = (int)h->n;
    const int gbn = (n + 255) / 256;
    double* jp = (double*)h->jp;
    // the attribute is per device: set it for the handle's (a host call)
#define LAUNCH_SYM(DD, CO)                                                                       \
  do {                                                                                           \
    constexpr int bytes = kWarpsPerBlock * sym_warp_bytes<DD, CO>();                                 \
    cudaFuncSetAttribute(k_force_sym<DD, CO>, cudaFuncAttributeMaxDynamicSharedMemorySize,       \
                         bytes);                                                                 \
    k_force_sym<DD, CO><<<CO ? k.ncell + 1 : g, bs, bytes, s>>>(                                 \
        k, h->cell_start, h->nl, h->ncount, h->nhs, h->x, h->v, h->pc, h->sid, h->pid, jp,       \
        (uint32_t)step, step_ptr, inv_sqdt);                                                     \
    if (n > 0)                                                                                   \
      k_force_gather<DD><<<gbn, 256, 0, s>>>(k, h->cell_of, jp, h->x, h->v, h->pc, h->sid, h->f, \
                                             fuse_mode, dt, h->v2, h->d_err);                    \
  } while (0)
    const bool coop = k.ncell < kCoopCells;
    if (k.d == 3) {
      if (coop) LAUNCH_SYM(3, true); else LAUNCH_SYM(3, false);
    } else {
      if (coop) LAUNCH_SYM(2, true); else LAUNCH_SYM(2, false);
    }
#undef LAUNCH_SYM
    h->launches++;
  } else if (fp64) {
#define LAUNCH_F64(DD, NW, SS)                                                                   \
  k_force64<DD, NW, SS><<<std::max(1, (int)((h->n * SS + kReuseTPB - 1) / kReuseTPB)), kReuseTPB, \
                          0, s>>>(k, h->cell_start, h->cell_of, h->nl, h->ncount, h->x, h->v,    \
                                  h->pc, h->sid, h->pid, h->f, h->st, fuse_mode, dt, h->v2,      \
                                  (uint32_t)step, step_ptr, inv_sqdt, h->d_err, nn, ca)
#define PICK_F64(DD, NW)               \
  do {                                 \
    if (split) LAUNCH_F64(DD, NW, 4);  \
    else LAUNCH_F64(DD, NW, 1);        \
  } while (0)
    if (k.d == 3) {
      if (k.newtonian) PICK_F64(3, false); else PICK_F64(3, true);
    } else {
      if (k.newtonian) PICK_F64(2, false); else PICK_F64(2, true);
    }
#undef PICK_F64
#undef LAUNCH_F64
  } else {
#define LAUNCH_F32(DD, NW, ST)                                                                  \
  do {                                                                                           \
    if (split)                                                                                   \
      k_force32<DD, NW, 4, ST><<<gp4, kReuseTPB, 0, s>>>(                                        \
          k, h->cell_start, h->cell_of, h->nl, h->ncount, h->neigh_cap, h->off, h->x, h->v,      \
          h->vf, h->wd, h->f, h->st, fuse_mode, dt, h->v2, (uint32_t)step, step_ptr,             \
          (float)inv_sqdt, h->d_err, nn, ca);                                                    \
    else                                                                                         \
      k_force32<DD, NW, 1, ST><<<gp, kReuseTPB, 0, s>>>(                                         \
          k, h->cell_start, h->cell_of, h->nl, h->ncount, h->neigh_cap, h->off, h->x, h->v,      \
          h->vf, h->wd, h->f, h->st, fuse_mode, dt, h->v2, (uint32_t)step, step_ptr,             \
          (float)inv_sqdt, h->d_err, nn, ca);                                                    \
  } while (0)
#define PICK_F32_ST(DD, NW)                   \
  do {                                        \
    if (k.stress) LAUNCH_F32(DD, NW, true);   \
    else LAUNCH_F32(DD, NW, false);           \
  } while (0)
    if (force32_packed(h, (uint32_t)step, step_ptr, (float)inv_sqdt, fuse_mode, dt)) {
      // done
    } else if (k.d == 3) {
      if (k.newtonian) PICK_F32_ST(3, false); else PICK_F32_ST(3, true);
    } else {
      if (k.newtonian) PICK_F32_ST(2, false); else PICK_F32_ST(2, true);
    }
#undef PICK_F32_ST
#undef LAUNCH_F32
  }
  h->launches++;
  if (cuda_check(h, cudaGetLastError(), "force launch")) return MCFG_ECUDA;
  if (fuse_mode == kForceBodyKick) std::swap(h->v, h->v2);
  return MCFG_OK;
}

}  // namespace mcfg

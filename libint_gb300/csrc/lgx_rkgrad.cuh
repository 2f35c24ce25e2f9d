// Register-resident gradient kernel: G lanes (1, 2, ..., 32) per contracted
// shell quartet, the primitive quartets split between them as in rk_kernel.
// The density is applied first (gen_grad.py): once per quartet the two
// two-particle densities become weights W over the (e0|f0) set, every
// primitive quartet contracts its VRR values with them, and seven sums per
// density, weighted by the exponents, give the three independent centres;
// no derivative set is formed, transformed or digested.
//
// What bounds it: the FP64 pipe (2 lanes per cycle and SM).  The program
// kernel it replaces runs a class's VRR levels across a warp's lanes, most of
// them idle in the s/p classes, and digests nine derivative sets.  (H2O)12
// cc-pVDZ, serial launches, before -> after: (ss|ss) 352 -> 21 ms, (ss|ps) 321
// -> 52 ms, (ps|ps) 165 -> 30 ms, (pp|dp) 31 -> 10 ms, all classes 1417 -> 285
// ms.  The weights of the larger classes (2 x 144 doubles for (pp|dp)) live in
// local memory, which costs less than the FP64 work they feed.  It ends at
// L = 5: the derivative raises the Boys order to L + 1, and rk_boys is exact
// to m = 6; the classes above take 14 ms of the 285.
#pragma once
#include <algorithm>

#include "gen/grad_classes.cuh"
#include "lgx_rk.cuh"

namespace lgx {

// Sums of one primitive or contracted quartet for one density:
// 2a_A V, 2a_B V, 2a_B S, 2a_D U, 2a_D S.
constexpr int kGradSums = 11;

// Prologue of one FP64 primitive quartet (the screening, Boys values and VRR
// factors of rk_prim); false when screened out.
template <int MMAX>
__device__ __forceinline__ bool rk_prologue(const EriArgs& a, const RkQuartet<double>& q, int ib,
                                            int ik, const PrimScreen& scr, double* F,
                                            rk::Geo<double>& geo) {
  const PrimPairRec& bp = a.pprims[q.bra_pp + ib];
  const PrimPairRec& kp = a.pprims[q.ket_pp + ik];
  if (!ln_kept(a, bp.fln_scr + kp.fln_scr, q.bra_pp + ib, q.ket_pp + ik, scr)) return false;
  const double zeta = bp.zeta, eta = kp.zeta;
  const double2 gpq = rk_gpq(a, bp, kp);
  const double rs = gpq.x, oogpq = gpq.y;
  const double pfac = bp.Kc * kp.Kc * rs;
  if (rk_pfac_dropped<true>(a, q, bp, kp, pfac, scr)) return false;
  const double PQx = bp.P[0] - kp.P[0], PQy = bp.P[1] - kp.P[1], PQz = bp.P[2] - kp.P[2];
  const double ez = eta * oogpq, zz = zeta * oogpq;
  const double T = zeta * ez * fma(PQx, PQx, fma(PQy, PQy, PQz * PQz));
  rk_boys<MMAX>(a.boys_fine, T, pfac, F);
  const double* PA = bp.PA + (q.bsw ? 3 : 0);
  const double* QC = kp.PA + (q.ksw ? 3 : 0);
  geo.PAx = PA[0]; geo.PAy = PA[1]; geo.PAz = PA[2];
  geo.QCx = QC[0]; geo.QCy = QC[1]; geo.QCz = QC[2];
  geo.WPx = -ez * PQx; geo.WPy = -ez * PQy; geo.WPz = -ez * PQz;
  geo.WQx = zz * PQx; geo.WQy = zz * PQy; geo.WQz = zz * PQz;
  geo.oo2z = bp.hoog;
  geo.roz = ez;
  geo.oo2e = kp.hoog;
  geo.roe = zz;
  geo.oo2ze = 0.5 * oogpq;
  return true;
}

template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(128, 2) rk_grad_kernel(EriArgs a) {
  using C = rk::GradCls<LA, LB, LC, LD>;
  constexpr int N0 = C::kN0, N1 = C::kN1, N2 = C::kN2, N3 = C::kN3;
  constexpr int kNsph = N0 * N1 * N2 * N3;
  // (ss|ss): both densities weight the same integrals, so one unweighted set
  constexpr int kSets = C::kNacc == 1 ? 1 : 2;
  const int G = a.group;
  const int lane = threadIdx.x & 31;
  const int g = lane & (G - 1);
  const unsigned gmask = G == 32 ? 0xffffffffu : (((1u << G) - 1u) << (lane & ~(G - 1)));
  const int per_warp = 32 / G;
  const long long warp_id = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  const long long first = a.bin.first, total = a.bin.total;
  const size_t copy = size_t(blockIdx.x % a.gcopies) * a.gstride;
  unsigned long long my_prims = 0;
  PrimScreen scr;
  scr.prec = a.precision;
  scr.ln_prec = a.ln_prec;
  scr.fprec = a.fprecision;
  scr.fln_prec = a.fln_prec;
  RkChunks<true> ch(a, total, per_warp, warp_id, nwarps);
  for (; ch.left(); ch.next(lane)) {
    ch.fetch(a, lane);
    const long long c0 = first + ch.at(1) * per_warp;
    const long long qi = c0 + (lane / G);
    // segment of each quartet of the chunk (see rk_kernel)
    const int seg0 = bin_segment(a.bin, c0);
    const int kseg = seg0 + 1 + lane;
    const long long mseg = (kseg <= a.bin.nseg ? a.bin.seg_start[kseg] : c0 + 64) - c0;
    const unsigned starts = __reduce_or_sync(0xffffffffu, mseg < per_warp ? 1u << mseg : 0u);
    const int seg = seg0 + __popc(starts & ((2u << (lane / G)) - 1u));
    if (qi >= first + total) continue;
    const int bpair = a.bin.bra_pairs[a.bin.seg_bra[seg]];
    const int kpair = a.bin.ket_pairs[int(qi - a.bin.seg_start[seg]) + a.bin.seg_j0[seg]];
    RkQuartet<double> q;
    rk_load<double>(a, bpair, kpair, a.pair_swap[bpair] != 0, a.pair_swap[kpair] != 0, q);
    const int nbf = a.nbf;
    const size_t o0 = a.basis.bf_off[q.sh[0]], o1 = a.basis.bf_off[q.sh[1]];
    const size_t o2 = a.basis.bf_off[q.sh[2]], o3 = a.basis.bf_off[q.sh[3]];
    const double* D = a.D;
    // the two-particle densities of the quartet
    auto gamma = [&](double* GJ, double* GK) {
#pragma unroll
      for (int i = 0; i < N0; ++i)
#pragma unroll
        for (int j = 0; j < N1; ++j)
#pragma unroll
          for (int k = 0; k < N2; ++k)
#pragma unroll
            for (int l = 0; l < N3; ++l) {
              const int e = ((i * N1 + j) * N2 + k) * N3 + l;
              GJ[e] = __ldg(D + (o0 + i) * nbf + o1 + j) * __ldg(D + (o2 + k) * nbf + o3 + l);
              GK[e] = 0.5 * fma(__ldg(D + (o0 + i) * nbf + o2 + k),
                                __ldg(D + (o1 + j) * nbf + o3 + l),
                                __ldg(D + (o0 + i) * nbf + o3 + l) *
                                    __ldg(D + (o1 + j) * nbf + o2 + k));
            }
    };
    double WJ[C::kNacc], WK[C::kNacc];
    if constexpr (kSets == 1) {
      WJ[0] = WK[0] = 1.0;
    } else {
      double GJ[kNsph], GK[kNsph];
      gamma(GJ, GK);
      C::template weights<double>(GJ, q.AB, q.CD, WJ);
      C::template weights<double>(GK, q.AB, q.CD, WK);
    }
    double acc[kSets][kGradSums];
#pragma unroll
    for (int x = 0; x < kSets; ++x)
#pragma unroll
      for (int i = 0; i < kGradSums; ++i) acc[x][i] = 0.0;
    double I[C::kNI];
#pragma unroll
    for (int i = 0; i < C::kNI; ++i) I[i] = 0.0;
    const int nq = q.nbpp * q.nkpp;
    int kept = 0;
    int ib = g / q.nkpp, ik = g - ib * q.nkpp;
    const int gb = G / q.nkpp, gk = G - gb * q.nkpp;
    for (int p = g; p < nq; p += G) {
      double F[C::kMmax + 1];
      rk::Geo<double> geo;
      if (rk_prologue<C::kMmax>(a, q, ib, ik, scr, F, geo)) {
        ++kept;
        double s[14];
        C::template prim<double>(F, geo, WJ, WK, s, I);
        const PrimPairRec& bp = a.pprims[q.bra_pp + ib];
        const PrimPairRec& kp = a.pprims[q.ket_pp + ik];
        const double wa = (q.bsw ? bp.ta2 : bp.ta1), wb = (q.bsw ? bp.ta1 : bp.ta2);
        const double wd = (q.ksw ? kp.ta1 : kp.ta2);
#pragma unroll
        for (int x = 0; x < kSets; ++x) {
          const double* sx = s + 7 * x;
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            acc[x][i] = fma(wa, sx[1 + i], acc[x][i]);
            acc[x][3 + i] = fma(wb, sx[1 + i], acc[x][3 + i]);
            acc[x][7 + i] = fma(wd, sx[4 + i], acc[x][7 + i]);
          }
          acc[x][6] = fma(wb, sx[0], acc[x][6]);
          acc[x][10] = fma(wd, sx[0], acc[x][10]);
        }
      }
      ib += gb;
      ik += gk;
      if (ik >= q.nkpp) {
        ik -= q.nkpp;
        ++ib;
      }
    }
    for (int o = G >> 1; o > 0; o >>= 1) {
#pragma unroll
      for (int x = 0; x < kSets; ++x)
#pragma unroll
        for (int i = 0; i < kGradSums; ++i)
          acc[x][i] += rk_shfl_xor<double>(gmask, acc[x][i], o, G);
      if constexpr (C::kTail)
#pragma unroll
        for (int i = 0; i < C::kNI; ++i) I[i] += rk_shfl_xor<double>(gmask, I[i], o, G);
      kept += __shfl_xor_sync(gmask, kept, o, G);
    }
    if (g == 0) my_prims += (unsigned long long)kept;
    if (kept == 0) continue;
    double GJ[kNsph], GK[kNsph];
    if constexpr (kSets == 1 || C::kTail) gamma(GJ, GK);
    const double deg = double((q.sh[0] == q.sh[1] ? 1 : 2) * (q.sh[2] == q.sh[3] ? 1 : 2) *
                              (bpair == kpair ? 1 : 2));
    const int at[4] = {a.basis.atom[q.sh[0]], a.basis.atom[q.sh[1]], a.basis.atom[q.sh[2]],
                       a.basis.atom[q.sh[3]]};
    int slot = 0;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const double* sx = acc[kSets == 1 ? 0 : x];
      const double f = (x == 0 ? 0.5 : -0.25) * deg * (kSets == 1 ? (x == 0 ? GJ[0] : GK[0]) : 1.0);
      double lo[3] = {0, 0, 0}, dab[3] = {0, 0, 0}, dcd[3] = {0, 0, 0};
      if constexpr (C::kTail)
        C::template tail<double>(I, x == 0 ? GJ : GK, x == 0 ? WJ : WK, q.AB, q.CD, lo, dab, dcd);
      double* out = (x == 0 ? a.gJ : a.gK) + copy;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        double gA = sx[i], gB = fma(q.AB[i], sx[6], sx[3 + i]), gD = fma(q.CD[i], sx[10], sx[7 + i]);
        if constexpr (LA > 0) gA -= lo[i];
        if constexpr (C::kBraHrr) {
          gA += dab[i];
          gB -= dab[i];
        }
        if constexpr (C::kKetHrr) gD -= dcd[i];
        const double gC = -(gA + gB + gD);
        const double gv[4] = {gA, gB, gC, gD};
#pragma unroll
        for (int t = 0; t < 4; ++t, ++slot)
          if ((slot & (G - 1)) == g) atomicAdd(out + 3 * at[t] + i, f * gv[t]);
      }
    }
  }
  if (a.prim_count && my_prims) atomicAdd(a.prim_count, my_prims);
}

// Stores the twelve derivative sets of one quartet from its accumulators, the
// elements split between G lanes.
template <class C>
__device__ __forceinline__ void rk_store_deriv(const EriArgs& a, const QuartetItem& it,
                                               const RkQuartet<double>& q, const double* I, int G,
                                               int g) {
  constexpr int N0 = C::kN0, N1 = C::kN1, N2 = C::kN2, N3 = C::kN3, N = C::kNsph;
  double v[9 * N];
  C::template sets<double>(I, q.AB, q.CD, v);
  const int fl = it.flags >> 2;
  const bool sbk = fl & 1, stb = (fl >> 1) & 1, stk = (fl >> 2) & 1;
  // canonical position -> caller position, and the strides there
  const int perm[4] = {sbk ? (stk ? 3 : 2) : (stb ? 1 : 0), sbk ? (stk ? 2 : 3) : (stb ? 0 : 1),
                       sbk ? (stb ? 1 : 0) : (stk ? 3 : 2), sbk ? (stb ? 0 : 1) : (stk ? 2 : 3)};
  const int dims[4] = {N0, N1, N2, N3};
  int str[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    str[t] = 1;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (perm[u] > perm[t]) str[t] *= dims[u];
  }
  double* o = a.out + it.out;
#pragma unroll
  for (int e = 0; e < N; ++e) {
    if ((e & (G - 1)) != g) continue;
    double* oe = o + (e / (N1 * N2 * N3)) * str[0] + ((e / (N2 * N3)) % N1) * str[1] +
                 ((e / N3) % N2) * str[2] + (e % N3) * str[3];
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      const double dA = v[s * N + e], dB = v[(3 + s) * N + e], dD = v[(6 + s) * N + e];
      oe[(size_t)(perm[0] * 3 + s) * N] = dA;
      oe[(size_t)(perm[1] * 3 + s) * N] = dB;
      oe[(size_t)(perm[2] * 3 + s) * N] = -(dA + dB + dD);
      oe[(size_t)(perm[3] * 3 + s) * N] = dD;
    }
  }
}

// First-derivative shell sets of an explicit list, G lanes per quartet: the
// accumulators of gen_grad.py's DerivCls in registers, the twelve sets written
// in the caller's order (centre C by translational invariance).
//
// What bounds it: the FP64 pipe; the program kernel it replaces left most lanes
// of a level idle in these classes, whose primitive quartets are the many (a
// water dimer in cc-pVDZ: 8 of 10 ms).  It ends at L = 3: from (pp|pp) on the
// accumulators (540 there) no longer fit the registers, and few primitive
// quartets are left.
template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(128, 2) rk_deriv_kernel(EriArgs a) {
  using C = rk::DerivCls<LA, LB, LC, LD>;
  const int G = a.group;
  const int lane = threadIdx.x & 31;
  const int g = lane & (G - 1);
  const unsigned gmask = G == 32 ? 0xffffffffu : (((1u << G) - 1u) << (lane & ~(G - 1)));
  const long long first = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / G;
  const long long step = ((long long)gridDim.x * blockDim.x) / G;
  PrimScreen scr;
  scr.prec = a.precision;
  scr.ln_prec = a.ln_prec;
  scr.fprec = a.fprecision;
  scr.fln_prec = a.fln_prec;
  for (long long qi = first; qi < a.nitems; qi += step) {
    const QuartetItem it = a.items[qi];
    RkQuartet<double> q;
    rk_load<double>(a, it.bra_pair, it.ket_pair, it.flags & 1, (it.flags >> 1) & 1, q);
    double I[C::kNacc];
#pragma unroll
    for (int i = 0; i < C::kNacc; ++i) I[i] = 0.0;
    const int nq = q.nbpp * q.nkpp;
    int kept = 0;
    int ib = g / q.nkpp, ik = g - ib * q.nkpp;
    const int gb = G / q.nkpp, gk = G - gb * q.nkpp;
    for (int p = g; p < nq; p += G) {
      double F[C::kMmax + 1];
      rk::Geo<double> geo;
      if (rk_prologue<C::kMmax>(a, q, ib, ik, scr, F, geo)) {
        ++kept;
        const PrimPairRec& bp = a.pprims[q.bra_pp + ib];
        const PrimPairRec& kp = a.pprims[q.ket_pp + ik];
        const double w[3] = {(q.bsw ? bp.ta2 : bp.ta1), (q.bsw ? bp.ta1 : bp.ta2),
                             (q.ksw ? kp.ta1 : kp.ta2)};
        C::template prim<double>(F, geo, w, I);
      }
      ib += gb;
      ik += gk;
      if (ik >= q.nkpp) {
        ik -= q.nkpp;
        ++ib;
      }
    }
    for (int o = G >> 1; o > 0; o >>= 1) {
#pragma unroll
      for (int i = 0; i < C::kNacc; ++i) I[i] += rk_shfl_xor<double>(gmask, I[i], o, G);
      kept += __shfl_xor_sync(gmask, kept, o, G);
    }
    if (a.is_null && g == 0) a.is_null[it.pad] = kept == 0 ? 1 : 0;
    if (kept == 0) continue;
    rk_store_deriv<C>(a, it, q, I, G, g);
  }
}

// One quartet over several blocks: every thread takes its own primitive
// quartets, a block adds its threads' accumulators through shared memory and puts
// the sums to a.gscratch; the block that comes last (the ticket a.counter counts
// blocks and is left at zero) adds the blocks' sums, transforms and stores.
//
// What bounds it: one scheduler's FP64 rate, 64 cycles a warp instruction, so a
// single warp needed 77 us for the 81 primitive quartets of a (pp|pp) set and 40%
// of that went into the shuffled sums.  One warp a scheduler and a column of the
// accumulators per thread afterwards: 4 warps a block, as many blocks as give each
// thread one primitive quartet (16 at most): that set 35 us, the call 121 -> 83 us.
template <int LA, int LB, int LC, int LD, int DERIV>
__global__ void __launch_bounds__(128, 1) rk_one_kernel(EriArgs a) {
  using Cd = rk::DerivCls<DERIV ? LA : 0, DERIV ? LB : 0, DERIV ? LC : 0, DERIV ? LD : 0>;
  using Ce = rk::Cls<LA, LB, LC, LD>;
  constexpr int NA = DERIV ? Cd::kNacc : Ce::kNacc;
  constexpr int MM = DERIV ? Cd::kMmax : Ce::kMmax;
  extern __shared__ double s_acc[];  // [rows][NA + 1]
  __shared__ int s_kept;
  __shared__ unsigned s_last;
  const int tid = threadIdx.x;
  const QuartetItem it = a.items[0];
  RkQuartet<double> q;
  rk_load<double>(a, it.bra_pair, it.ket_pair, it.flags & 1, (it.flags >> 1) & 1, q);
  PrimScreen scr;
  scr.prec = a.precision;
  scr.ln_prec = a.ln_prec;
  scr.fprec = a.fprecision;
  scr.fln_prec = a.fln_prec;
  if (tid == 0) s_kept = 0;
  __syncthreads();
  double I[NA];
#pragma unroll
  for (int i = 0; i < NA; ++i) I[i] = 0.0;
  const int nq = q.nbpp * q.nkpp;
  int kept = 0;
  for (int p = blockIdx.x * 128 + tid; p < nq; p += gridDim.x * 128) {
    const int ib = p / q.nkpp, ik = p - ib * q.nkpp;
    if constexpr (DERIV) {
      double F[MM + 1];
      rk::Geo<double> geo;
      if (rk_prologue<MM>(a, q, ib, ik, scr, F, geo)) {
        ++kept;
        const PrimPairRec& bp = a.pprims[q.bra_pp + ib];
        const PrimPairRec& kp = a.pprims[q.ket_pp + ik];
        const double w[3] = {q.bsw ? bp.ta2 : bp.ta1, q.bsw ? bp.ta1 : bp.ta2,
                             q.ksw ? kp.ta1 : kp.ta2};
        Cd::template prim<double>(F, geo, w, I);
      }
    } else {
      kept += rk_prim<Ce, false, true>(a, q, ib, ik, scr, I) ? 1 : 0;
    }
  }
  const int rows = min(128, nq);
  if (tid < rows) {
#pragma unroll
    for (int i = 0; i < NA; ++i) s_acc[tid * (NA + 1) + i] = I[i];
  }
  if (kept) atomicAdd(&s_kept, kept);
  __syncthreads();
  double* part = reinterpret_cast<double*>(a.gscratch);
  for (int i = tid; i < NA; i += 128) {
    // four running sums: the chain of dependent additions is what takes time
    double s0 = 0, s1 = 0, s2 = 0, s3 = 0;
    int r = 0;
    for (; r + 4 <= rows; r += 4) {
      s0 += s_acc[r * (NA + 1) + i];
      s1 += s_acc[(r + 1) * (NA + 1) + i];
      s2 += s_acc[(r + 2) * (NA + 1) + i];
      s3 += s_acc[(r + 3) * (NA + 1) + i];
    }
    for (; r < rows; ++r) s0 += s_acc[r * (NA + 1) + i];
    part[(size_t)blockIdx.x * (NA + 1) + i] = (s0 + s1) + (s2 + s3);
  }
  if (tid == 0) part[(size_t)blockIdx.x * (NA + 1) + NA] = double(s_kept);
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(a.counter, 1ull) == gridDim.x - 1 ? 1u : 0u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  if (tid == 0) *a.counter = 0;
  for (int i = tid; i <= NA; i += 128) {
    double s = 0;
    for (unsigned b = 0; b < gridDim.x; ++b) s += __ldcg(part + (size_t)b * (NA + 1) + i);
    s_acc[i] = s;
  }
  __syncthreads();
  if (tid >= 32) return;
  const bool null = !(s_acc[NA] > 0.0);
  if (a.is_null && tid == 0) a.is_null[it.pad] = null ? 1 : 0;
  if (null) return;
#pragma unroll
  for (int i = 0; i < NA; ++i) I[i] = s_acc[i];
  if constexpr (DERIV) {
    rk_store_deriv<Cd>(a, it, q, I, 32, tid);
  } else {
    double cart[Ce::kNcart];
    Ce::template hrr<double>(I, q.AB, q.CD, cart);
    double v[Ce::kNsph];
    Ce::template sph<double>(cart, v);
    rk_store_set<Ce>(a, it.flags, it.out, v, 32, tid);
  }
}

template <int LA, int LB, int LC, int LD, int DERIV>
cudaError_t rk_one_launch_one(const EriArgs& a, int blocks, cudaStream_t st) {
  constexpr int NA = DERIV ? rk::DerivCls<DERIV ? LA : 0, DERIV ? LB : 0, DERIV ? LC : 0,
                                          DERIV ? LD : 0>::kNacc
                           : rk::Cls<LA, LB, LC, LD>::kNacc;
  static_assert(128 * (NA + 1) * sizeof(double) <= 227 * 1024, "accumulators of one block");
  auto k = rk_one_kernel<LA, LB, LC, LD, DERIV>;
  const size_t smem = size_t(128) * (NA + 1) * sizeof(double);
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k<<<blocks, 128, smem, st>>>(a);
  return cudaGetLastError();
}

template <class K>
cudaError_t rk_deriv_launch_any(K k, const EriArgs& a, long long work, int nsm, cudaStream_t st) {
  const int block = 128;
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, block, 0) != cudaSuccess || occ < 1)
    occ = 1;
  const long long need = (work * a.group + block - 1) / block;
  const long long grid = std::max(1LL, std::min((long long)nsm * occ, need));
  k<<<(unsigned)grid, block, 0, st>>>(a);
  return cudaGetLastError();
}

template <int LA, int LB, int LC, int LD>
cudaError_t rk_grad_launch_one(const EriArgs& a, long long work, int nsm, cudaStream_t st) {
  return rk_deriv_launch_any(rk_grad_kernel<LA, LB, LC, LD>, a, work, nsm, st);
}

template <int LA, int LB, int LC, int LD>
cudaError_t rk_deriv_launch_one(const EriArgs& a, long long work, int nsm, cudaStream_t st) {
  return rk_deriv_launch_any(rk_deriv_kernel<LA, LB, LC, LD>, a, work, nsm, st);
}

}  // namespace lgx

// Grouped class kernel of the plain FP64 J/K builds: one warp per task, a
// task = up to 32 ket pairs (one per lane or lane group, fixed for the task)
// and a run of bra pairs that share their first shell a.
//
// Two things bounded the one-bra-per-task kernel (eri_class_kernel): scattered
// FP64 atomics (180e9 adds/s on random addresses, 5 to 69 of them per shell
// quartet) and Boys-function divergence (87% of the primitive quartets of a
// water cluster are at large T, but 77% of a warp's steps had a lane that was
// not, so that nearly every step ran both branches).  Here
//   * the ket of a lane and the shell a stay fixed over the run of bras, so
//     J_cd, K_ac and K_ad accumulate in registers and are added to memory once
//     per task; per quartet only K_bc and K_bd (b is the small shell) remain;
//   * a plan-time kernel (group_masks_kernel) marks per bra and ket whether
//     every primitive quartet is far (T >= far_T).  The far loop has no Boys
//     table, no exponential, one reciprocal square root and no divergence.  A
//     bra's quartets that are not far are spread over the whole warp (32 / their
//     number lanes each) for the general loop, and their blocks handed back to
//     the kets' lanes through shared memory;
//   * what the task needs of its bras (masks, primitive ranges, A-B, D_ab) is
//     read by the lanes side by side at its start, and the next bra's primitive
//     pairs are prefetched: per bra the one-bra kernel walked a chain of five
//     dependent loads;
//   * ket primitive pairs come field by field from the blocked list (a row of
//     the warp's lanes per field instead of one cache line per lane).
// Per (H2O)32 / 6-31G* build, classes one after another, before and now:
// (ps|ss) 4.36 -> 3.05 ms, (ss|ss) 2.70 -> 1.85, (ds|ps) 2.17 -> 1.83, (ds|ss)
// 1.97 -> 1.42, (ps|ps) 1.77 -> 1.57, (dp|ss) 1.06 -> 0.79.  (ps|ss) now issues on
// 47% of the cycles (26% before), with the FP64 pipe at 31% and the L1 data pipe
// at 62%; it waits on L1 misses (2.8 of 8.0 warps per issue) and fixed latencies
// (2.2).  Switched off in
// turn there, the near loop takes 1.4 ms, the far loop 1.3 ms and the digestion
// 0.35 ms.
#pragma once

#include <atomic>

#include "eri_kernels.cuh"

namespace hfg {

// One ket primitive pair of a lane, from the blocked list (KetBlocks).
template <bool TRANSFER>
struct FarKet {
  double Qx, Qy, Qz, Kf, ie, bx, by, bz;
  __device__ __forceinline__ void load(const double *__restrict__ k) {
    Qx = __ldg(k + kKetPx * 32);
    Qy = __ldg(k + (kKetPx + 1) * 32);
    Qz = __ldg(k + (kKetPx + 2) * 32);
    Kf = __ldg(k + kKetKf * 32);
    if constexpr (TRANSFER) {
      ie = __ldg(k + kKetInvZeta * 32);
      bx = __ldg(k + kKetBAB * 32);
      by = __ldg(k + (kKetBAB + 1) * 32);
      bz = __ldg(k + (kKetBAB + 2) * 32);
    } else {
      ie = bx = by = bz = 0.0;
    }
  }
};

// Far primitive quartets: with theta^(m) = rho^m [..]^(m) the vertical
// recursion keeps its form with W-P -> -(P-Q)/zeta and rho/zeta -> 1/zeta, and
// rho^m F_m K_ab K_cd / sqrt(zeta + eta) = (2m-1)!!/(2R^2)^m Kf_ab Kf_cd / R:
// no zeta + eta, no rho, one reciprocal square root (Kf: PrimPair).
template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ void far_primitive(const PrimPair *__restrict__ pb, const FarKet<(LC + LD > 0)> &k,
                                              double *acc) {
  constexpr int LTOT = LA + LB + LC + LD;
  const double PQx = pb->Px - k.Qx, PQy = pb->Py - k.Qy, PQz = pb->Pz - k.Qz;
  const double R2 = PQx * PQx + PQy * PQy + PQz * PQz;
  const double r = rsqrt(R2);
  double F[LTOT + 1];
  F[0] = pb->Kf * k.Kf * r;
  if constexpr (LTOT == 0) {
    acc[0] += F[0];
  } else {
    const double h = 0.5 * r * r;
#pragma unroll
    for (int m = 0; m < LTOT; ++m) F[m + 1] = (2 * m + 1) * h * F[m];
    const double iz = pb->inv_zeta;
    double d0 = 0, d1 = 0, d2 = 0, zoe = 0, oo2e = 0;
    if constexpr (LC + LD > 0) {
      d0 = -(pb->bABx + k.bx) * k.ie;
      d1 = -(pb->bABy + k.by) * k.ie;
      d2 = -(pb->bABz + k.bz) * k.ie;
      zoe = pb->zeta * k.ie;
      oo2e = 0.5 * k.ie;
    }
    EriClass<LA, LB, LC, LD, false>::template prim<double>(acc, F, pb->PAx, pb->PAy, pb->PAz, -iz * PQx, -iz * PQy,
                                                           -iz * PQz, 0.5 * iz, iz, d0, d1, d2, zoe, oo2e);
  }
}

// Any primitive quartet (the Boys function of accumulate_primitives); k: the
// ket primitive pair in the blocked list.
template <bool TRANSFER>
struct NearKet {
  double Qx, Qy, Qz, eta, K, ie, bx, by, bz;
  __device__ __forceinline__ void load(const double *__restrict__ k) {
    Qx = __ldg(k + kKetPx * 32);
    Qy = __ldg(k + (kKetPx + 1) * 32);
    Qz = __ldg(k + (kKetPx + 2) * 32);
    eta = __ldg(k + kKetZeta * 32);
    K = __ldg(k + kKetK * 32);
    if constexpr (TRANSFER) {
      ie = __ldg(k + kKetInvZeta * 32);
      bx = __ldg(k + kKetBAB * 32);
      by = __ldg(k + (kKetBAB + 1) * 32);
      bz = __ldg(k + (kKetBAB + 2) * 32);
    } else {
      ie = bx = by = bz = 0.0;
    }
  }
};
template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ void near_primitive(const PrimPair *__restrict__ pb, const NearKet<(LC + LD > 0)> &k,
                                               const BoysShared tab, double *acc) {
  constexpr int LTOT = LA + LB + LC + LD;
  const double rs = rsqrt(pb->zeta + k.eta);
  const double rho = pb->zeta * k.eta * (rs * rs);
  const double PQx = pb->Px - k.Qx, PQy = pb->Py - k.Qy, PQz = pb->Pz - k.Qz;
  const double T = rho * (PQx * PQx + PQy * PQy + PQz * PQz);
  double F[LTOT + 1];
  boys_eval<LTOT>(F, T, pb->K * k.K * rs, tab);
  const double roz = rho * pb->inv_zeta;
  double d0 = 0, d1 = 0, d2 = 0, zoe = 0, oo2e = 0;
  if constexpr (LC + LD > 0) {
    d0 = -(pb->bABx + k.bx) * k.ie;
    d1 = -(pb->bABy + k.by) * k.ie;
    d2 = -(pb->bABz + k.bz) * k.ie;
    zoe = pb->zeta * k.ie;
    oo2e = 0.5 * k.ie;
  }
  EriClass<LA, LB, LC, LD, false>::template prim<double>(acc, F, pb->PAx, pb->PAy, pb->PAz, -roz * PQx, -roz * PQy,
                                                         -roz * PQz, 0.5 * pb->inv_zeta, roz, d0, d1, d2, zoe, oo2e);
}

template <int N>
__device__ __forceinline__ void sum_lane_groups(double *acc, int lg) {
  for (int o = 1; o < (1 << lg); o <<= 1)
#pragma unroll
    for (int x = 0; x < N; ++x) acc[x] += __shfl_xor_sync(0xffffffffu, acc[x], o);
}

// What a task needs of one of its bras, in the warp's shared memory.
template <int NAB>
struct BraMeta {
  int off, np, ao, bp;
  unsigned on, near;
  double AB[3], D[NAB];  // A - B; 2 D_ab
};

__device__ __forceinline__ void prefetch_line(const void *p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// Shared memory of a block: the Boys slice, then per warp the blocks of a bra's
// quartets that are not far [kAcc][32], the bras' records and the J_ab sums.
template <int LA, int LB, int LC, int LD>
struct GroupShape {
  static constexpr int kWarps = group_warps(LA, LB, LC, LD);
  static constexpr int kAcc = EriClass<LA, LB, LC, LD, false>::kAcc;
  static constexpr int NAB = ncart(LA) * ncart(LB);
  using Meta = BraMeta<NAB>;
  static constexpr int kMetaDoubles = kGroupMaxBras * sizeof(Meta) / sizeof(double);
  static_assert(NAB <= 32, "one lane per bra component");
  static constexpr int kParts = NAB > 16 ? 1 : NAB > 8 ? 2 : NAB > 4 ? 4 : NAB > 2 ? 8 : 32;
  static constexpr int kRed = NAB > 1 ? NAB * 33 : 0;
  static constexpr int kStage = kAcc * 32;
  static constexpr int kWarpDoubles = kStage + kMetaDoubles + kRed;
  static constexpr size_t kBytes = sizeof(double) * (kBoysFoldedSize + kWarps * kWarpDoubles) + kWarps * 32;
  static_assert(kBytes <= 227 * 1024, "shared memory of one block");
};

template <int LA, int LB, int LC, int LD, int MODE>
__global__ void __launch_bounds__(32 * group_warps(LA, LB, LC, LD), 1)
    eri_group_kernel(const EngineView v, const ClassLaunch cl) {
  using Cls = EriClass<LA, LB, LC, LD, false>;
  constexpr int LTOT = LA + LB + LC + LD;
  constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
  constexpr int N = NA * NB * NC * ND;
  constexpr bool kUhf = MODE == kJkUhf;
  constexpr int NS = kUhf ? 2 : 1;
  using S = GroupShape<LA, LB, LC, LD>;
  constexpr int W = S::kWarps;
  extern __shared__ __align__(16) double group_sh[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double *stage = group_sh + kBoysFoldedSize + warp * S::kWarpDoubles;
  typename S::Meta *meta = reinterpret_cast<typename S::Meta *>(stage + S::kStage);
  [[maybe_unused]] double *jred = stage + S::kStage + S::kMetaDoubles;
  unsigned char *queue = reinterpret_cast<unsigned char *>(group_sh + kBoysFoldedSize + W * S::kWarpDoubles) + warp * 32;
  stage_boys<LTOT>(group_sh, v.boys_table);
  const BoysShared tab{group_sh};
  const int ntasks = launch_ntasks(cl);
  int t = first_task(cl, blockIdx.x * W + warp);
  Task raw_next{};
  if (t < ntasks) raw_next = launch_task(cl, t);
  for (int tn; t < ntasks; t = tn) {
    const GroupTask task = group_task(raw_next);
    tn = next_task(cl, t, gridDim.x * W);
    if (tn < ntasks) raw_next = launch_task(cl, tn);
    const int lg = task.lg, gl = lane & ((1 << lg) - 1), kl = lane >> lg;
    const int bp0 = cl.bra_list[task.bra_start];
    const MolView mv = task_molecule(v, bp0);
    if (mv.skip) continue;  // warp-uniform
    const int n = mv.n;
    const double *Dm[2] = {cl.Da + mv.base, kUhf ? cl.Db + mv.base : nullptr};
    const double *DJ = kUhf ? cl.Dt + mv.base : Dm[0];
    double *Jm = cl.J + mv.base;
    double *Km[2] = {cl.Ka + mv.base, kUhf ? cl.Kb + mv.base : nullptr};
    // the lane's ket (lanes past the task's kets repeat the last one, masked)
    const int kpos = task.ket_start + min(kl, task.nket - 1);
    const int kp = cl.ket_list[kpos];
    const int npk = v.pair_nprim[kp];
    const long long koff = (long long)cl.ket_block_off[kpos >> 5] * kKetStride + (kpos & 31);
    const double *ket = cl.ket_blocks + koff;
    const int aoc = v.pair_ao_a[kp], aod = v.pair_ao_b[kp];
    const bool kdiag = v.pair_sa[kp] == v.pair_sb[kp];
    const double Y0 = v.pair_AB[3 * kp], Y1 = v.pair_AB[3 * kp + 1], Y2 = v.pair_AB[3 * kp + 2];
    const int aoa = v.pair_ao_a[bp0], sa = v.pair_sa[bp0];
    for (int b = lane; b < task.nbra; b += 32) {
      const uint2 m = cl.masks[task.mask_off + b];
      const int bp = cl.bra_list[task.bra_start + b];
      typename S::Meta &r = meta[b];
      r.on = m.x;
      r.near = m.y;
      r.off = v.pair_prim_off[bp];
      r.np = v.pair_nprim[bp];
      r.ao = v.pair_ao_b[bp];
      r.bp = sa == v.pair_sb[bp] ? ~bp : bp;  // complemented: both shells the same
#pragma unroll
      for (int x = 0; x < 3; ++x) r.AB[x] = v.pair_AB[3 * bp + x];
#pragma unroll
      for (int x = 0; x < NA * NB; ++x) r.D[x] = 2.0 * __ldg(&DJ[(aoa + x / NB) * n + r.ao + x % NB]);
    }

    double jcd[NC * ND], kac[NS][NA * NC], kad[NS][NA * ND];
#pragma unroll
    for (int x = 0; x < NC * ND; ++x) jcd[x] = 0.0;
#pragma unroll
    for (int sp = 0; sp < NS; ++sp) {
#pragma unroll
      for (int x = 0; x < NA * NC; ++x) kac[sp][x] = 0.0;
#pragma unroll
      for (int x = 0; x < NA * ND; ++x) kad[sp][x] = 0.0;
    }
    __syncwarp();
    const int npmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)npk);
    for (int b = 0; b < task.nbra; ++b) {
      const typename S::Meta &r = meta[b];
      const unsigned mon = r.on, nm = r.near;
      if (!mon) continue;  // warp-uniform
      if (b + 1 < task.nbra && lane < meta[b + 1].np) prefetch_line(v.prim + meta[b + 1].off + lane);
      const PrimPair *pb = v.prim + r.off;
      const int np = r.np;
      double acc[Cls::kAcc];
#pragma unroll
      for (int x = 0; x < Cls::kAcc; ++x) acc[x] = 0.0;
      // far pass over all lanes, also those whose quartet is not far (replaced
      // below) or not of the build (left out of the digestion).  The lanes of
      // a group split the bra primitives, or the ket ones where those are too few.
      if (mon & ~nm) {
        const int G = 1 << lg;
        const bool bras = np >= G;
        const int dik = bras ? 1 : G, ib0 = bras ? gl : 0, dib = bras ? G : 1;
        const int ik0 = bras ? 0 : gl;
        FarKet<(LC + LD > 0)> next;  // the loads run one ket primitive pair ahead
        next.load(ket + min(ik0, npmax - (npmax > 0)) * kKetStride);
        for (int ik = ik0; ik < npmax; ik += dik) {
          const FarKet<(LC + LD > 0)> k = next;
          next.load(ket + min(ik + dik, npmax - 1) * kKetStride);
#pragma unroll far_unroll(LA, LB, LC, LD)
          for (int ib = ib0; ib < np; ib += dib) far_primitive<LA, LB, LC, LD>(pb + ib, k, acc);
        }
        sum_lane_groups<Cls::kAcc>(acc, lg);
      }
      if (nm) {
        // g = 2^gs lanes for each of the bra's near quartets: gk of them over
        // its ket primitives, g / gk over the bra's
        const int cnt = __popc(nm), gs = 5 - (32 - __clz(cnt - 1)) * (cnt > 1), e = lane >> gs;
        if (gl == 0 && ((nm >> kl) & 1u)) queue[__popc(nm & ((1u << kl) - 1u))] = (unsigned char)lane;
        __syncwarp();
        const bool act = e < cnt;
        const int owner = act ? queue[e] : 0;
        const int npn = __shfl_sync(0xffffffffu, npk, owner);
        const double *kn = cl.ket_blocks + __shfl_sync(0xffffffffu, koff, owner);
        const int gks = min(gs, npmax > 1 ? 31 - __clz(npmax) : 0), sub = lane & ((1 << gs) - 1);
        double one[Cls::kAcc];
#pragma unroll
        for (int x = 0; x < Cls::kAcc; ++x) one[x] = 0.0;
        for (int ik = sub & ((1 << gks) - 1); ik < (act ? npn : 0); ik += 1 << gks) {
          NearKet<(LC + LD > 0)> k;
          k.load(kn + ik * kKetStride);
          for (int ib = sub >> gks; ib < np; ib += 1 << (gs - gks))
            near_primitive<LA, LB, LC, LD>(pb + ib, k, tab, one);
        }
        __syncwarp();
        sum_lane_groups<Cls::kAcc>(one, gs);
        if (act && sub == 0) {
#pragma unroll
          for (int x = 0; x < Cls::kAcc; ++x) stage[x * 32 + owner] = one[x];
        }
        __syncwarp();
        if ((nm >> kl) & 1u) {
#pragma unroll
          for (int x = 0; x < Cls::kAcc; ++x) acc[x] = stage[x * 32 + (lane & ~((1 << lg) - 1))];
        }
        __syncwarp();
      }
      const bool on = gl == 0 && ((mon >> kl) & 1u);
      const int aob = r.ao;
      double dbc[NS][NB * NC], dbd[NS][NB * ND];
#pragma unroll
      for (int sp = 0; sp < NS; ++sp)
#pragma unroll
        for (int bb = 0; bb < NB; ++bb) {
#pragma unroll
          for (int c = 0; c < NC; ++c) dbc[sp][bb * NC + c] = __ldg(&Dm[sp][(aob + bb) * n + aoc + c]);
#pragma unroll
          for (int d = 0; d < ND; ++d) dbd[sp][bb * ND + d] = __ldg(&Dm[sp][(aob + bb) * n + aod + d]);
        }

      double out[N];
      Cls::template hrr<double>(out, acc, r.AB[0], r.AB[1], r.AB[2], Y0, Y1, Y2);
      const bool bdiag = r.bp < 0;
      // degeneracy of the unique quartet among its 8 permutations; 0 where
      // the lane has none
      const double s = on ? (bdiag ? 0.5 : 1.0) * (kdiag ? 0.5 : 1.0) * ((bdiag ? ~r.bp : r.bp) == kp ? 0.5 : 1.0) : 0.0;
      double jab[NA * NB];
#pragma unroll
      for (int x = 0; x < NA * NB; ++x) jab[x] = 0.0;
      // a lane without a quartet of the build adds nothing, not even zero
      // times a density entry that is not finite
      if (s != 0.0) {
#pragma unroll
        for (int a = 0; a < NA; ++a)
#pragma unroll
          for (int bb = 0; bb < NB; ++bb) {
            const double nab = s * comp_norm<LA>(a) * comp_norm<LB>(bb);
            const double dij = r.D[a * NB + bb];
            double ja = 0.0;
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
              for (int d = 0; d < ND; ++d) {
                const int x = ((a * NB + bb) * NC + c) * ND + d;
                out[x] *= nab * comp_norm<LC>(c) * comp_norm<LD>(d);
                ja += out[x] * __ldg(&DJ[(aoc + c) * n + aod + d]);
                jcd[c * ND + d] += out[x] * dij;
              }
            jab[a * NB + bb] = 2.0 * ja;
          }
#pragma unroll
        for (int sp = 0; sp < NS; ++sp) {
          double *K = Km[sp];
          // K_ac += (ab|cd) D_bd, K_ad += (ab|cd) D_bc
#pragma unroll
          for (int bb = 0; bb < NB; ++bb) {
#pragma unroll
            for (int d = 0; d < ND; ++d) {
              const double x = dbd[sp][bb * ND + d];
#pragma unroll
              for (int a = 0; a < NA; ++a)
#pragma unroll
                for (int c = 0; c < NC; ++c) kac[sp][a * NC + c] += out[((a * NB + bb) * NC + c) * ND + d] * x;
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              const double x = dbc[sp][bb * NC + c];
#pragma unroll
              for (int a = 0; a < NA; ++a)
#pragma unroll
                for (int d = 0; d < ND; ++d) kad[sp][a * ND + d] += out[((a * NB + bb) * NC + c) * ND + d] * x;
            }
          }
          // K_bc += (ab|cd) D_ad, K_bd += (ab|cd) D_ac
          double kbc[NB * NC], kbd[NB * ND];
#pragma unroll
          for (int x = 0; x < NB * NC; ++x) kbc[x] = 0.0;
#pragma unroll
          for (int x = 0; x < NB * ND; ++x) kbd[x] = 0.0;
#pragma unroll
          for (int a = 0; a < NA; ++a) {
#pragma unroll
            for (int d = 0; d < ND; ++d) {
              const double x = __ldg(&Dm[sp][(aoa + a) * n + aod + d]);
#pragma unroll
              for (int bb = 0; bb < NB; ++bb)
#pragma unroll
                for (int c = 0; c < NC; ++c) kbc[bb * NC + c] += out[((a * NB + bb) * NC + c) * ND + d] * x;
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              const double x = __ldg(&Dm[sp][(aoa + a) * n + aoc + c]);
#pragma unroll
              for (int bb = 0; bb < NB; ++bb)
#pragma unroll
                for (int d = 0; d < ND; ++d) kbd[bb * ND + d] += out[((a * NB + bb) * NC + c) * ND + d] * x;
            }
          }
#pragma unroll
          for (int bb = 0; bb < NB; ++bb) {
#pragma unroll
            for (int c = 0; c < NC; ++c) atomicAdd(&K[(aob + bb) * n + aoc + c], kbc[bb * NC + c]);
#pragma unroll
            for (int d = 0; d < ND; ++d) atomicAdd(&K[(aob + bb) * n + aod + d], kbd[bb * ND + d]);
          }
        }
      }
      // the warp shares the bra pair: its J block is summed over the lanes,
      // kParts lanes per entry over shared memory (one entry: shuffles)
      if constexpr (NA * NB == 1) {
        double x = jab[0];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) atomicAdd(&Jm[aoa * n + aob], x);
      } else {
        constexpr int kParts = S::kParts;
#pragma unroll
        for (int x = 0; x < NA * NB; ++x) jred[x * 33 + lane] = jab[x];
        __syncwarp();
        const int e = lane / kParts, part = lane % kParts;
        double x = 0.0;
        if (e < NA * NB) {
#pragma unroll
          for (int y = 0; y < 32 / kParts; ++y) x += jred[e * 33 + part + y * kParts];
        }
#pragma unroll
        for (int o = kParts / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (e < NA * NB && part == 0) atomicAdd(&Jm[(aoa + e / NB) * n + aob + e % NB], x);
        __syncwarp();
      }
    }
    __syncwarp();  // the next task rewrites the bras' records
    if (gl == 0 && kl < task.nket) {
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int d = 0; d < ND; ++d) atomicAdd(&Jm[(aoc + c) * n + aod + d], jcd[c * ND + d]);
#pragma unroll
      for (int sp = 0; sp < NS; ++sp)
#pragma unroll
        for (int a = 0; a < NA; ++a) {
#pragma unroll
          for (int c = 0; c < NC; ++c) atomicAdd(&Km[sp][(aoa + a) * n + aoc + c], kac[sp][a * NC + c]);
#pragma unroll
          for (int d = 0; d < ND; ++d) atomicAdd(&Km[sp][(aoa + a) * n + aod + d], kad[sp][a * ND + d]);
        }
    }
  }
}

// Host: launch one grouped class kernel.
template <int LA, int LB, int LC, int LD, int MODE>
void launch_group(const EngineView &v, const ClassLaunch &cl, int grid, cudaStream_t s) {
  using S = GroupShape<LA, LB, LC, LD>;
  static std::atomic<unsigned> sized{0};  // one bit per device
  int dev = 0;
  cudaGetDevice(&dev);
  const unsigned bit = 1u << (dev & 31);
  if (!(sized.load() & bit)) {
    cudaFuncSetAttribute(eri_group_kernel<LA, LB, LC, LD, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::kBytes);
    sized.fetch_or(bit);
  }
  eri_group_kernel<LA, LB, LC, LD, MODE><<<grid, 32 * S::kWarps, S::kBytes, s>>>(v, cl);
}

}  // namespace hfg

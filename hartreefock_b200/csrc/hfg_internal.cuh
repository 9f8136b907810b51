// Internal definitions shared by the class kernels and the host context.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace hfg {

constexpr int kMaxL = 2;                      // compiled shells: s, p, d
constexpr int kMaxLtot = 4 * kMaxL;           // highest Boys order used
constexpr int kBoysTaylor = 7;                // Taylor terms around a grid point
constexpr double kBoysStep = 0.05;            // grid spacing in T
constexpr double kBoysTmax = 36.0;            // above: asymptotic F_0 + upward recursion
constexpr int kBoysGrid = 721;                // 36 / 0.05 + 1 grid points
constexpr int kBoysOrders = kMaxLtot + kBoysTaylor;  // orders 0 .. 14 tabulated
// staged row: 7 Taylor terms and exp(-T_i), 8 doubles, read as four 16-byte
// words.  Word j of row i is stored at j ^ ((i >> 1) & 3) within the row: rows
// start on one of two halves of the banks only, and the swizzle spreads one
// word of 8 consecutive rows (the lanes of one 16-byte access phase) over all
// banks.
constexpr int kBoysRow = kBoysTaylor + 1;
__host__ __device__ constexpr int boys_swizzle(int i, int k) { return i * kBoysRow + (k ^ (i & 6)); }
// Per-order rows ready for evaluation, after the e^-T tail of the table:
// table L (L = 0 .. kMaxLtot) holds in each grid row F_{L+k}(T_i) / k!
// (k < kBoysTaylor) and e^-T_i, unswizzled.
constexpr int kBoysFoldedOff = kBoysGrid * kBoysOrders + kBoysGrid;
constexpr int kBoysFoldedSize = kBoysGrid * kBoysRow;
// the same rows as a staged slice holds them (swizzled), for block-wide copies
constexpr int kBoysStagedOff = kBoysFoldedOff + (kMaxLtot + 1) * kBoysFoldedSize;

constexpr int kWarpsPerBlock = 4;
constexpr int kThreads = 32 * kWarpsPerBlock;
__host__ __device__ constexpr int ncart(int L) { return (L + 1) * (L + 2) / 2; }

// Warps per block of the fused class kernel.  The staged Boys table (46 KB)
// admits 4 blocks per SM: the light classes (<= 9 integrals per quartet,
// <= ~120 registers) run 8 warps per block so that the table is shared by
// more warps; the register-heavy ones keep 4, where the register file, not
// the table, sets the residency.
__host__ __device__ constexpr int fused_warps(int la, int lb, int lc, int ld) {
  return ncart(la) * ncart(lb) * ncart(lc) * ncart(ld) <= 9 ? 8 : 4;
}
// Resident blocks per SM the compiler must allow (1: the register
// allocation is free).  A 64-register cap (four 8-warp blocks per SM) fits
// (ss|ss) and (ps|ss) without spills but made (ps|ss) 20% slower alone
// (1.20 -> 1.43 ms per (H2O)16 launch) for a change within noise in the
// concurrent build; the other light classes spill under it.
__host__ __device__ constexpr int fused_min_blocks(int, int, int, int) { return 1; }
// Unroll factor of the inner (bra) primitive loop of the thread-per-quartet
// kernels (two primitive quartets in flight per lane).  Measured per class on
// the (H2O)32 / 6-31G* build: unrolling by 2 takes (ds|ps) from 2.68 to
// 2.14 ms and (ps|ss) from 4.44 to 4.34 ms, but slows (ss|ss) (2.59 -> 3.80)
// and (ps|ps) (1.75 -> 2.22), so it is per class.
__host__ __device__ constexpr int prim_unroll(int la, int lb, int lc, int ld) {
  return (la == 2 && lb == 0 && lc == 1 && ld == 0) || (la == 1 && lb == 0 && lc == 0 && ld == 0) ||
                 (la == 2 && lb == 0 && lc == 0 && ld == 0)
             ? 2
             : 1;
}
// Where a class kernel reads its Boys slice: staged into shared memory
// (46 KB per block, which also caps an SM at four such blocks over all the
// classes running at once) or straight from the per-order rows in global
// memory through L1 (kBoysFoldedOff; no shared memory).  Measured per class
// on the (H2O)32 / 6-31G* build, classes one after another: from global
// memory (ss|ss) 3.13 -> 2.66 ms, (pp|pp) 0.25 -> 0.21, (dd|ss) 0.33 -> 0.30,
// (ds|ds) 0.68 -> 0.66, (ds|pp) 0.61 -> 0.59, but (ps|ss) 4.35 -> 4.58 and
// (ds|ps), (ds|ss) 1-2% slower.
__host__ __device__ constexpr bool boys_from_global(int la, int lb, int lc, int ld) {
  return (la == 0 && lb == 0 && lc == 0 && ld == 0) || (la == 1 && lb == 1 && lc == 1 && ld == 1) ||
         (la == 2 && lb == 2 && lc == 0 && ld == 0) || (la == 2 && lb == 0 && lc == 2 && ld == 0) ||
         (la == 2 && lb == 0 && lc == 1 && ld == 1);
}
// Fused class kernels whose warps load their next task record while they
// work on the current one (every class but (ss|ss): with its Boys slice in
// global memory the prefetch made it slower, 2.66 -> 3.15 ms per (H2O)32
// build; without the prefetch the class is 4% slower with the staged slice
// and 15% faster with the global one).
__host__ __device__ constexpr bool task_prefetch(int la, int lb, int lc, int ld) {
  return la + lb + lc + ld > 0;
}
// The same choice for the split path's primitive kernel: from global memory
// (dp|ds) 1.78 -> 1.33 ms, (dp|pp) 0.95 -> 0.74, (dd|ps) 1.15 -> 0.90, (dp|dp)
// 0.87 -> 0.77, (dd|ds) 0.81 -> 0.71, (dd|pp) 0.55 -> 0.50; (dd|dp) 0.91 ->
// 2.13 ms, so it keeps the staged slice, as does (dd|dd).
__host__ __device__ constexpr bool boys_from_global_split(int la, int lb, int lc, int ld) {
  return !(la == 2 && lb == 2 && lc == 2 && (ld == 1 || ld == 2));
}

// T from which a primitive quartet of total angular momentum L counts as far:
// there the asymptotic F_m = (2m-1)!!/(2T)^m sqrt(pi/T)/2 without the e^-T
// terms is within 1.2e-16 relative, about half an ulp, of F_m for every m <= L
// (what is missing is the regularised upper incomplete gamma function
// Q(m + 1/2, T): 2e-17 at L = 1, T = 40.5; 1.0e-16 at L = 4, T = 48; at most
// 1.13e-16, at L = 5 and 6; 9e-17 at L = 8, T = 58).
__host__ __device__ constexpr double far_T(int L) { return 38.0 + 2.5 * L; }
// Unroll factor of the grouped kernel's far loop over bra primitives.
__host__ __device__ constexpr int far_unroll(int la, int lb, int lc, int ld) {
  return ncart(la) * ncart(lb) * ncart(lc) * ncart(ld) <= 9 ? 2 : 1;
}
// Warps per block of the grouped kernel: one block per SM, so that its warps
// share one staged Boys slice and L1 keeps the rest of the SM's memory.
__host__ __device__ constexpr int group_warps(int la, int lb, int lc, int ld) {
  const int n = ncart(la) * ncart(lb) * ncart(lc) * ncart(ld);
  return n == 1 ? 24 : n <= 9 ? 16 : n == 18 ? 12 : 8;
}
// Primitive quartets of a large class up to which its builds run the
// warp-cooperative kernel, a quartet per warp, instead of the split path, a
// quartet per thread: the thread takes 50 to 300 us over one quartet however
// few there are, the warp a fraction of that, until there are enough to fill
// the GPU with threads.  us per J/K build, warp kernel against split path, at
// the primitive quartets of (H2O)1 to (H2O)24 / 6-31G* and C2H6 to C9H20:
//   (dd|dp)  43/264 at 4, 66/309 at 2,106, 127/356 at 6,078, 228/405 at 12,186,
//            273/432 at 16,640, 437/551 at 28,666, level at 40,104: 16,000 is
//            below where they meet
//   (dd|pp)  50/87 at 13, 93/128 at 4,844, 146/159 at 9,506, 162/166 at 14,313,
//            269/173 at 36,401
//   (dd|ds)  37/48 at 18, 50/77 at 2,405, 78/81 at 3,866, 93/88 at 8,367
//   (dp|pp)  78/89 at 52, 80/96 at 1,994, 109/98 at 4,836
//   (dd|ps)  52/49 at 72, 56/54 at 550, level at 1,014 and 2,167, 54/57 at 5,169,
//            82/58 at 8,514; the one launch instead of two decides it in whole
//            builds on class streams: 170/204 at 184 (CH3), 265/280 at 1,014
//            (C2H6), 277/288 at 2,167 ((H2O)3), 382/311 at 5,169 ((H2O)4)
//   (dp|ds)  60/57 at 72, 70/65 at 3,574, 89/65 at 8,730: the split path
// (dd|dd) is faster here at every size (0.24 against 0.82 ms at (H2O)16, before
// its recursions became tables).  (dp|dp) would gain too (56 against 161 at
// (H2O)2), but this kernel is 3.1e-12 off the reference on two cancelling
// elements of O2 / 6-31G* (1.3e-12 on the split path; adding the transfer terms
// one by one as the per-thread code does changes nothing), so it stays there.
__host__ __device__ constexpr long long warp_prim_limit(int la, int lb, int lc, int ld) {
  const int ket = 10 * lc + ld;
  if (la == 2 && lb == 2)
    return ket == 22 ? (1ll << 62) : ket == 21 ? 16000 : ket == 11 ? 9000 : ket == 20 ? 5000 : ket == 10 ? 4500 : 0;
  return ket == 11 ? 2500 : 0;
}

enum Mode { kStorePacked = 0, kJkRhf = 1, kJkUhf = 2, kSchwarz = 3, kBlock = 4 };

// Density screening and precision of a J/K launch.  kScreenNone: every
// Schwarz-surviving quartet in FP64.  kScreenFp64 / kScreenMixed: quartets
// whose density-weighted bound Q_ab Q_cd max|D| falls below the launch's
// density threshold are skipped.  kScreenFp64 evaluates the rest in FP64;
// kScreenMixed decides per task (one bra pair, <= 32 kets, a warp-uniform
// test): FP64 when the task's largest bound reaches the mixed cutoff, else
// FP32 primitive pairs, geometry, Boys interpolation and recursions (the
// Boys function's edges in FP64) with the J/K digestion in FP64.
enum Screen { kScreenNone = 0, kScreenFp64 = 1, kScreenMixed = 2 };

// One primitive pair of a shell pair (first shell A with exponent a, second
// B with exponent b): zeta = a+b, P = (aA+bB)/zeta, PA = P-A,
// bAB = b(A-B) and K = N_a c_a N_b c_b exp(-ab/zeta |AB|^2) sqrt(2) pi^(5/4) / zeta,
// so that the quartet prefactor 2 pi^(5/2) / (zeta eta sqrt(zeta+eta))
// exp(...) of GaussianTwoElectrons.cpp:44-45 is K_ab K_cd / sqrt(zeta+eta).
// Kf = K (pi^(1/4) / sqrt 2) / sqrt(zeta) is the prefactor of far quartets
// (eri_group.cuh).  128 B: one cache line per primitive pair, in the order of
// use, so that an s-s pair reads two of its sectors.
struct __align__(128) PrimPair {
  double Px, Py, Pz, zeta;
  double K, Kf, inv_zeta, PAx;
  double PAy, PAz, bABx, bABy;
  double bABz, pad[3];
};
// FP32 copy of a PrimPair for the mixed-precision kernels (48 B)
struct __align__(16) PrimPairF {
  float zeta, Px, Py, Pz, PAx, PAy, PAz, bABx, bABy, bABz, K, inv_zeta;
};

// Device view of one context's tables.
struct EngineView {
  const PrimPair *prim;       // all primitive pairs, pair-major
  const PrimPairF *primf;     // the same in FP32
  const int *pair_prim_off;   // per pair
  const int *pair_nprim;
  const int *pair_sa;         // first shell (higher L; higher index on ties)
  const int *pair_sb;
  const int *pair_ao_a;       // first AO of each shell of the pair
  const int *pair_ao_b;
  const double *pair_AB;      // [3*npairs] A - B
  const double *pair_Q;       // Schwarz bound
  const float *shell_dmax;    // [nshells][nshells] max |D| over each shell block (density screening)
  int nshells;
  const double *boys_table;   // [kBoysGrid][kBoysOrders] F_m(T_i), e^-T_i, then the per-order rows
  int nbf;
  int reference_convention;   // 1: reproduce the reference's (dd|dd) ET rows
  // batched contexts (many molecules, one launch per class); null otherwise
  const int *pair_mol;             // molecule of each shell pair
  const int *mol_nbf;              // basis functions per molecule
  const long long *mol_off;        // offset of each molecule's n x n matrices
  const unsigned char *mol_active; // 0: skip the molecule in this build
};

// The molecule a task belongs to (its bra pair's): its size, the offset of
// its matrices in the batch buffers, and whether this build skips it.
struct MolView {
  int n;
  long long base;
  bool skip;
};
__device__ __forceinline__ MolView task_molecule(const EngineView &v, int bp) {
  if (!v.pair_mol) return MolView{v.nbf, 0, false};
  const int m = v.pair_mol[bp];
  return MolView{v.mol_nbf[m], v.mol_off[m], v.mol_active != nullptr && v.mol_active[m] == 0};
}

// One unit of work: a bra pair position in the class's pair list and a
// range of at most 32 ket positions (kets of one primitive-count bucket).
// lg: the thread-per-quartet kernels give each quartet 2^lg lanes, which
// split its primitive quartets and sum them with warp shuffles (tasks with
// fewer kets than lanes, and long contractions); 0 = one lane per quartet.
struct __align__(16) Task {
  int bra_pos;
  int ket_start;
  int ket_end;
  int lg = 0;
};

// The same 16 bytes as the grouped kernel (eri_group.cuh) reads them: nbra
// consecutive bras of its bra list from bra_start (all with one first shell),
// nket kets from ket_start, 2^lg lanes per ket, and per bra a pair of ket
// masks from mask_off on: x = quartets of the build, y = those of them with a
// primitive quartet that is not far.
struct GroupTask {
  int bra_start, ket_start, nket, nbra, lg;
  unsigned mask_off;
};
constexpr int kGroupMaxBras = 16;
// primitive quartets per lane a grouped task is kept below
constexpr int kGroupTaskSteps = 256;
// Tasks of a class (one bra, up to 32 kets) per SM from which its plain J/K
// builds run the grouped kernel, whose blocks fill an SM each; twice as many on
// concurrent class streams, where below it the one-bra-per-task kernel, whose
// small blocks share the SMs with the other classes, is as fast or faster.  With
// every class grouped: (H2O)32 / 6-31G* (80,000 to 958,000 tasks a class) 25.5 ->
// 22.1 ms one after another and 25.2 -> 22.1 on streams, (H2O)16 (14,000 to
// 153,000) 6.26 -> 5.83 and 4.99 -> 4.88, C9H20 / 6-31+G** (23,000 to 211,000)
// 8.79 -> 8.55 but 6.94 -> 7.30, UHF C10H22 / 6-31G* (below 100,000) 5.03 -> 4.91
// but 3.23 -> 3.57.  Shards take the line of concurrent streams whatever the
// context's (each walks a part of the tasks, and every rank the same list).
constexpr int kGroupMinTasks = 750;

// Ket primitive pairs by list position: block `pos >> 5` of a pair class's list
// starts at record off[pos >> 5], record ik of it holds primitive pair ik of
// its 32 pairs, field by field (kKetFields x 32 doubles), so that a warp's
// lanes read a field of 32 neighbouring kets as one row.
enum KetField { kKetPx = 0, kKetKf = 3, kKetInvZeta = 4, kKetBAB = 5, kKetZeta = 8, kKetK = 9, kKetFields = 10 };
constexpr int kKetStride = kKetFields * 32;
__host__ __device__ __forceinline__ Task pack_group_task(int bra_start, int ket_start, int nket, int nbra, int lg,
                                                         unsigned mask_off) {
  return Task{bra_start, ket_start, (int)mask_off, lg | nket << 8 | nbra << 16};
}
__host__ __device__ __forceinline__ GroupTask group_task(const Task &t) {
  return GroupTask{t.bra_pos, t.ket_start, (t.lg >> 8) & 0xff, (t.lg >> 16) & 0xff, t.lg & 0xff, (unsigned)t.ket_end};
}

struct ClassLaunch {
  const int *bra_list;   // pair indices of the bra class, sorted by Q desc
  const int *ket_list;   // pair indices of the ket class, sorted by Q desc
  const Task *tasks;
  int ntasks;            // tasks of this launch (of this shard)
  int task_offset;       // shard: launch task t is tasks[task_offset + t * task_stride]
  int task_stride;
  const uint2 *masks;    // grouped launches: ket masks of the tasks
  const double *ket_blocks;  // grouped launches: ket primitive pairs (KetField)
  const int *ket_block_off;
  int same_class;        // bra class == ket class
  double threshold;
  // outputs by mode
  double *packed;        // kStorePacked
  const double *Da, *Db; // kJk*: densities (Db for UHF)
  const double *Dt;      // total density for J in UHF
  double *J, *Ka, *Kb;   // accumulators (n x n)
  double *Qout;          // kSchwarz: per pair
  // density screening (kScreenFp64 / kScreenMixed launches)
  float dens_threshold;  // skip quartets whose density-weighted bound is below
  float mixed_cutoff;    // tasks whose largest bound is below run in FP32
  unsigned long long *counters;  // [0] FP64, [1] FP32 quartets evaluated
  // device work queue (batched builds without host synchronisation): the
  // task count lives in device memory (written by the compaction of the
  // active molecules' tasks) and warps take the next task from an atomic
  // counter that starts at 0; null = ntasks above, static grid-stride order
  const int *ntasks_dev;
  int *queue;
};

// task t of a launch (shards take every task_stride-th task of the class)
__device__ __forceinline__ Task launch_task(const ClassLaunch &cl, int t) {
  return cl.tasks[cl.task_offset + (long long)t * cl.task_stride];
}

// Tasks of the launch: the device count when the queue is on.
__device__ __forceinline__ int launch_ntasks(const ClassLaunch &cl) {
  return cl.ntasks_dev ? *cl.ntasks_dev : cl.ntasks;
}
// A warp's first task and its next one after t: the grid-stride order
// (start, start + stride, ...) or, with the queue, one atomic per warp.
__device__ __forceinline__ int warp_fetch(int *queue, int step) {
  int t = 0;
  if ((threadIdx.x & 31) == 0) t = atomicAdd(queue, step);
  return __shfl_sync(0xffffffffu, t, 0);
}
__device__ __forceinline__ int first_task(const ClassLaunch &cl, int start) {
  return cl.queue ? warp_fetch(cl.queue, 1) : start;
}
__device__ __forceinline__ int next_task(const ClassLaunch &cl, int t, int stride) {
  return cl.queue ? warp_fetch(cl.queue, 1) : t + stride;
}

// One chunk of a split-path class launch (see eri_split.cuh): scratch for
// the contracted [e0|f0] blocks of `ntasks` tasks starting at `task0`.
struct SplitChunk {
  double *scr_fwd;   // [kAcc][slots]: block with bra = task's bra pair
  double *scr_rev;   // [kAcc][slots]: reference-convention (dd|dd) only, bra = ket pair
  long long stride;  // slots in the chunk (ntasks * 32)
  int task0;         // first task of the chunk
  int ntasks;
};

// component normalisation f(l,m,n) = 1/sqrt((2l-1)!!(2m-1)!!(2n-1)!!) in the
// canonical component order; the L-dependent part of the primitive
// normalisation sits in the contraction coefficients
template <int L>
__device__ __forceinline__ double comp_norm(int c);
template <>
__device__ __forceinline__ double comp_norm<0>(int) { return 1.0; }
template <>
__device__ __forceinline__ double comp_norm<1>(int) { return 1.0; }
template <>
__device__ __forceinline__ double comp_norm<2>(int c) {
  // xx xy xz yy yz zz
  return (c == 0 || c == 3 || c == 5) ? 0.57735026918962576451 : 1.0;
}

// Packed 8-fold index (IntegralsRepository.h:151-162)
__device__ __forceinline__ long long tri(long long a, long long b) {
  return a < b ? b * (b + 1) / 2 + a : a * (a + 1) / 2 + b;
}

// Nearest Boys grid point of 0 <= T < kBoysTmax: index i = round(T / step)
// and dT = i * step - T.  The integer comes out of the low mantissa bits of
// T / step + 1.5 * 2^52 (the sum rounds to an integer there), so no
// float-integer conversion is issued either way.
struct BoysGridPoint {
  int i;
  double dt;
};
__device__ __forceinline__ BoysGridPoint boys_grid_point(double T) {
  constexpr double kShift = 6755399441055744.0;  // 1.5 * 2^52
  const double y = fma(T, 1.0 / kBoysStep, kShift);
  return {__double2loint(y), (y - kShift) * kBoysStep - T};
}

// e^-T for T >= kBoysTmax (36), to ~1.2e-7 relative: there e^-T enters F_m
// only through the upward recursion below, where it is under 1e-6 of
// (2m+1) F_m for m <= 8, so single precision in this factor moves F_m by less
// than 1e-13 relative.  2^y with y = -T log2(e) in FP64: the integer part
// goes into the exponent field, the fraction through exp2f (underflows to
// ~2^-1022 and below, far under anything that survives the recursion).
__device__ __forceinline__ double exp_neg_far(double T) {
  const double y = -T * 1.4426950408889634074;  // log2(e)
  const double n = floor(y);
  const int ni = max((int)n, -1022);
  return (double)exp2f((float)(y - n)) * __hiloint2double((ni + 1023) << 20, 0);
}

// A class's Boys slice, staged in shared memory (swizzled rows) or as the
// per-order rows in global memory (plain rows of 64 bytes: four 16-byte loads).
struct BoysShared {
  const double *p;
  __device__ __forceinline__ void row(int i, double *c) const {
    const double2 *t = reinterpret_cast<const double2 *>(p + i * kBoysRow);
    const int sw = (i >> 1) & 3;
#pragma unroll
    for (int j = 0; j < kBoysRow / 2; ++j) {
      const double2 x = t[j ^ sw];
      c[2 * j] = x.x;
      c[2 * j + 1] = x.y;
    }
  }
};
struct BoysGlobal {
  const double *p;
  __device__ __forceinline__ void row(int i, double *c) const {
    const double2 *t = reinterpret_cast<const double2 *>(p + i * kBoysRow);
#pragma unroll
    for (int k = 0; k < kBoysRow / 2; ++k) {
      const double2 x = __ldg(t + k);
      c[2 * k] = x.x;
      c[2 * k + 1] = x.y;
    }
  }
};

// Boys function F_0..F_M at T.  Below kBoysTmax: 7-term Taylor expansion of
// F_M about the nearest grid point, F_M(T) = sum_k F_{M+k}(T_i) (-dT)^k / k!,
// from the shared-memory slice tab[i][k] = F_{M+k}(T_i)/k! (k < 7), then the
// downward recursion F_m = (2T F_{m+1} + e^-T) / (2m+1) (BoysFunctions.cpp:17-20)
// with e^-T = e^-T_i * e^(T_i - T), tab[i][7] = e^-T_i and the second factor
// from its 8-term Taylor series (|T_i - T| <= 0.025: truncation < 4e-18);
// both polynomials evaluated in Estrin's scheme.
// Above: F_0 = sqrt(pi/T)/2 (erfc(sqrt T) < 3e-17 there) and the upward
// recursion F_{m+1} = ((2m+1) F_m - e^-T) / (2T), 1/T as rsqrt(T)^2 and e^-T
// from exp_neg_far.  The scale folds the quartet prefactor into every order.
// e^-T is left out from far_T(M) on, where it is below the rounding of F_m.
template <int M, class R, class Tab>
__device__ __forceinline__ void boys_eval(R *F, double T, double scale, const Tab tab) {
  if (T < kBoysTmax) {
    const BoysGridPoint gp = boys_grid_point(T);
    const int i = gp.i;
    const double dt = gp.dt;  // -(T - T_i)
    double t[kBoysRow];
    tab.row(i, t);
    // both polynomials in Estrin's scheme (pairs, then powers dt^2 and dt^4):
    // three dependent multiply-adds instead of six and seven in Horner's
    const double d2 = dt * dt, d4 = d2 * d2;
    const double p01 = fma(t[1], dt, t[0]), p23 = fma(t[3], dt, t[2]);
    const double p45 = fma(t[5], dt, t[4]);
    double fm[M + 1];
    fm[M] = fma(fma(t[6], d2, p45), d4, fma(p23, d2, p01));
    if (M > 0) {
      const double a01 = 1.0 + dt, a23 = fma(dt, 1.0 / 6.0, 0.5);
      const double a45 = fma(dt, 1.0 / 120.0, 1.0 / 24.0), a67 = fma(dt, 1.0 / 5040.0, 1.0 / 720.0);
      const double x = fma(fma(a67, d2, a45), d4, fma(a23, d2, a01));
      const double e = t[7] * x;
      const double t2 = 2.0 * T;
#pragma unroll
      for (int m = M - 1; m >= 0; --m) fm[m] = fma(t2, fm[m + 1], e) * (1.0 / (2 * m + 1));
    }
#pragma unroll
    for (int m = 0; m <= M; ++m) F[m] = (R)(fm[m] * scale);
  } else {
    const double r = rsqrt(T);
    double f = 0.88622692545275801365 * r;  // sqrt(pi)/2 / sqrt(T)
    F[0] = (R)(f * scale);
    if (M > 0) {
      const double e = T < far_T(M) ? exp_neg_far(T) : 0.0;
      const double h = 0.5 * r * r;
#pragma unroll
      for (int m = 0; m < M; ++m) {
        f = ((2 * m + 1) * f - e) * h;
        F[m + 1] = (R)(f * scale);
      }
    }
  }
}

}  // namespace hfg

// Real-space r-RESPA shell kernel: the B200 counterpart of ORAC's `force`
// (src/force.f:1-917).
//
// One warp owns one i-group (a charge group, <= ORAC_MAXG atoms, staged in
// shared memory) and its neighbour-list row.  Per partner group it
//   1. forms the group-centre minimum image in FP64 scaled coordinates and
//      classifies the pair into ORAC's bands (non-switched [rinn0, rout),
//      switched S on [rout, rout0), 1-S on [rinn, rinn0)), src/force.f:265-333;
//   2. writes the next inner shell's list entry (order preserved with a warp
//      ballot), src/force.f:279-286;
//   3. evaluates every atom pair of the two groups in FP32 -- LJ
//      ecc12/r^12 - ecc6/r^6 and q q erfc_AS(alpha r)/r with the A&S 7.1.26
//      polynomial ORAC uses -- skipping excluded pairs through the list
//      entry's mask, src/force.f:396-731;
//   4. for switched pairs adds the S'(R) V_ij term distributed by mass
//      fraction, src/force.f:754-817.
// Steps 1-2 run a lane per list entry; steps 3-4 a lane per in-band entry,
// queued in shared memory (k_pair below).  Forces go to
// 64-bit fixed-point accumulators with atomics, so the sum is independent
// of the order of the atomics.
// The molecular virial is assembled without per-pair work: ORAC's
// sum_pairs f (x) (Rm_i - Rm_j - img) equals sum_atoms F_a (x) Rm_a (done in
// the finalize kernel) plus, for pairs that cross the box, G_ij (x) co.img
// where G_ij is the pair's total force on the j group (done here).
#include <type_traits>

#include "common.cuh"

namespace {

// warps per block: 4; 2 for groups of more than 4 atoms, whose lanes keep
// more in shared memory
__host__ __device__ constexpr int warps_per_block(int mg) { return mg > 4 ? 2 : 4; }
constexpr float AS_A1 = 0.2548296f, AS_A2 = -0.28449674f, AS_A3 = 1.4214137f;
constexpr float AS_A4 = -1.453152f, AS_A5 = 1.0614054f, AS_QP = 0.3275911f;

__device__ __forceinline__ long long to_fix(float v) { return __float2ll_rn(v * (float)ORAC_FSCALE); }

__device__ __forceinline__ void fix_add(unsigned long long* p, float v) {
  long long q = __float2ll_rn(v * (float)ORAC_FSCALE);
  if (q != 0) atomicAdd(p, (unsigned long long)q);
}

// The force path's products and sums with their rounding spelled out: every
// build of the kernel (with energies or without, any lanes per row) then gives
// the same forces bit for bit, and an energy step or a restart does not change
// a trajectory.  The soft-core pair (alch_pair_f32) leaves the contraction of
// its products to the compiler, which has treated its builds alike; the tests
// hold the builds of every group size and variant to the same bits.
__device__ __forceinline__ float fm(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float mu(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float ad(float a, float b) { return __fadd_rn(a, b); }

// 2^x by the hardware instruction
__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ double warp_sumd(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Pair energies in FP64 from the FP64 centre distance, the stored atom
// offsets, FP64 charges and FP64 LJ parameters: used only when energies are
// requested (EN), so the FP32 force path is the same in both modes.
__device__ __forceinline__ void pair_energy_fp64(const PairArgs& A, double rx, double ry, double rz, double2 L,
                                                 bool ljon, double qq, double* conf, double* coul) {
  const double r2 = rx * rx + ry * ry + rz * rz;
  const double rsqi = 1.0 / r2;
  *conf = 0.0;
  *coul = 0.0;
  if (ljon) {
    const double r6 = rsqi * rsqi * rsqi;
    *conf = L.x * r6 * r6 - L.y * r6;
  }
  if (!A.lskip) {
    const double rsp = sqrt(r2);
    const double ar = A.alphad * rsp;
    const double qt = 1.0 / (1.0 + 0.3275911 * ar);
    const double erfcst =
        ((((1.0614054 * qt - 1.453152) * qt + 1.4214137) * qt - 0.28449674) * qt + 0.2548296) * qt * exp(-ar * ar);
    *coul = qq * erfcst / rsp;
  } else if (!A.ewald) {
    *coul = qq / sqrt(r2);
  }
}

// seg_select, src/rem.f90:631-645: 0 either atom in the segment, 1 both,
// 2 exactly one
__device__ __forceinline__ bool seg_sel(int kind, int fa, int fb) {
  const bool ra = (fa & VF_REM) != 0, rb = (fb & VF_REM) != 0;
  return kind == 0 ? (ra || rb) : (kind == 1 ? (ra && rb) : (ra != rb));
}

// Soft-core pair of force_alchemy (src/force_alchemy.f:441-531) in FP32:
// qf is the force over r, conf/coul the scaled energies that enter the S'V
// sum.  t indexes the tables (ss_i + ss_j + 4).
__device__ __forceinline__ void alch_pair_f32(const PairArgs& A, const float (*af)[9], const float (*afq)[9], float r2,
                                              int t, float rmi, float rmj, float eps4, float qq, float* qf,
                                              float* conf, float* coul) {
  if (A.at.shifted) {
    // force_ALCHEMY_shift (src/force_alchemy_shifted.f:466-520): LJ at the
    // shifted distance rl, Coulomb erfc(alpha r) over the shifted rq
    const float ir = rsqrtf(r2), r = r2 * ir;
    float f = 0.f, uc = 0.f, uq = 0.f;
    if (eps4 > 1e-12f) {
      const float sig = A.at.opls ? 2.f * sqrtf(rmi * rmj) : rmi + rmj;
      const float rl = r + A.ljshift_s * sig * af[0][t];
      const float irl = __fdividef(1.f, rl);
      const float s2 = sig * sig * irl * irl, x = s2 * s2 * s2;
      const float sc = af[1][t] * eps4;
      f = sc * (12.f * x * x - 6.f * x) * ir * irl;
      uc = sc * (x * x - x);
    }
    const float irq = __fdividef(1.f, r + A.qshift * afq[0][t]);
    if (!A.lskip) {
      const float ar = A.alphal * r;
      const float qt = __fdividef(1.0f, 1.0f + AS_QP * ar);
      const float ex = __expf(-ar * ar);
      const float erfcst = ((((AS_A5 * qt + AS_A4) * qt + AS_A3) * qt + AS_A2) * qt + AS_A1) * qt * ex;
      const float furpar = afq[1][t] * qq;
      uq = furpar * erfcst * irq;
      // -dU/dr / r of erfc(alpha r) / rq: erfc / (r rq^2) + 2 alpha / sqrt(pi) e / (r rq)
      f += furpar * (erfcst * irq + A.twrtpi * ar * ex * ir) * irq * ir;
    } else if (!A.ewald) {
      uq = afq[1][t] * qq * irq;
      f += uq * irq * ir;
    }
    *qf = f;
    *conf = uc;
    *coul = uq;
    return;
  }
  const float auxa = rsqrtf(r2);
  const float fq1 = afq[0][t];
  const float auxaa = rsqrtf(A.qsoft * fq1 * fq1 + r2);
  float f = 0.f, uc = 0.f, uq = 0.f;
  if (eps4 > 1e-12f) {
    const float sig = A.at.opls ? 2.f * sqrtf(rmi * rmj) : rmi + rmj;
    const float s2 = sig * sig;
    const float r6 = __fdividef(r2 * r2 * r2, s2 * s2 * s2);
    const float gp1 = __fdividef(1.f, A.ljsoft * af[0][t] + r6);
    const float gp2 = gp1 * gp1;
    const float sc = af[1][t] * eps4;
    f = sc * (2.f * gp1 * gp2 - gp2) * 6.f * r6 * auxa * auxa;
    uc = sc * (gp2 - gp1);
  }
  if (!A.lskip) {
    const float rsp = r2 * auxa;
    const float ar = A.alphal * rsp;
    const float qt = __fdividef(1.0f, 1.0f + AS_QP * ar);
    const float ex = __expf(-ar * ar);
    const float erfcst = ((((AS_A5 * qt + AS_A4) * qt + AS_A3) * qt + AS_A2) * qt + AS_A1) * qt * ex;
    const float furpar = afq[1][t] * qq;
    uq = furpar * erfcst * auxaa;
    f += uq * auxaa * auxaa + furpar * A.twrtpi * ar * ex * auxa * auxa * auxaa;
  } else if (!A.ewald) {
    uq = afq[1][t] * qq * auxaa;
    f += uq * auxaa * auxaa;
  }
  *qf = f;
  *conf = uc;
  *coul = uq;
}

// The same pair in FP64 for the energy outputs: LJ and Coulomb at lambda,
// their sum at lambda0, and dU/dlambda of the control lambda (chain rule
// through the alch_fact tables).
__device__ __forceinline__ void alch_energy_fp64(const PairArgs& A, double rx, double ry, double rz, double2 si,
                                                 double2 sj, double qq, int t, double* cd, double* qd,
                                                 double* c0, double* q0, double* du) {
  const AlchTables& T = A.at;
  const AlchDyn& D = *A.ad;
  const double rsq = rx * rx + ry * ry + rz * rz;
  if (T.shifted) {
    // force_ALCHEMY_shift's energies at lambda and lambda0, and dU/dlambda
    // through the tables: rl = r + c f0, x = (sigma/rl)^6, U = f1 e (x^2 - x),
    // dx/dlambda = -6 x c df0 / rl; Coulomb f1 g / rq, rq = r + qshift f0
    const double r = sqrt(rsq);
    const double epsmin = 4.0 * sqrt(si.y * sj.y);
    *cd = *qd = *c0 = *q0 = *du = 0.0;
    if (epsmin > 1.0e-12) {
      const double sigma = T.opls ? 2.0 * sqrt(si.x * sj.x) : si.x + sj.x;
      const double c = T.ljshift_s * sigma;
      const double rl = r + c * D.f[0][t], rl0 = r + c * D.f0[0][t];
      const double s1 = sigma / rl, s0 = sigma / rl0;
      const double x = s1 * s1 * s1 * s1 * s1 * s1, x0 = s0 * s0 * s0 * s0 * s0 * s0;
      *cd = D.f[1][t] * epsmin * (x * x - x);
      *c0 = D.f0[1][t] * epsmin * (x0 * x0 - x0);
      *du = D.df[1][t] * epsmin * (x * x - x) +
            D.f[1][t] * epsmin * (2.0 * x - 1.0) * (-6.0 * x / rl) * c * D.df[0][t];
    }
    double g = 0.0;
    if (!A.lskip) {
      const double ar = A.alphad * r;
      const double qt = 1.0 / (1.0 + 0.3275911 * ar);
      g = qq * ((((1.0614054 * qt - 1.453152) * qt + 1.4214137) * qt - 0.28449674) * qt + 0.2548296) * qt *
          exp(-ar * ar);
    } else if (!A.ewald) {
      g = qq;
    }
    if (g != 0.0) {
      const double rq = r + T.qshift * D.fq[0][t], rq0 = r + T.qshift * D.fq0[0][t];
      *qd = D.fq[1][t] * g / rq;
      *q0 = D.fq0[1][t] * g / rq0;
      *du += D.dfq[1][t] * g / rq - D.fq[1][t] * g / (rq * rq) * T.qshift * D.dfq[0][t];
    }
    return;
  }
  const double auxa = 1.0 / sqrt(rsq);
  const double fq = D.fq[0][t], fq0 = D.fq0[0][t];
  const double auxaa = 1.0 / sqrt(T.qsoft * (fq * fq) + rsq);
  const double auxa0 = 1.0 / sqrt(T.qsoft * (fq0 * fq0) + rsq);
  const double epsmin = 4.0 * sqrt(si.y * sj.y);
  *cd = *qd = *c0 = *q0 = *du = 0.0;
  if (epsmin > 1.0e-12) {
    const double sigma = T.opls ? 2.0 * sqrt(si.x * sj.x) : si.x + sj.x;
    const double s2 = sigma * sigma;
    const double r6 = rsq * rsq * rsq / (s2 * s2 * s2);
    const double gp1 = 1.0 / (T.ljsoft * D.f[0][t] + r6);
    const double gp2 = gp1 * gp1;
    const double gp10 = 1.0 / (T.ljsoft * D.f0[0][t] + r6);
    const double gp20 = gp10 * gp10;
    const double auxc = epsmin * (gp2 - gp1);
    *cd = D.f[1][t] * auxc;
    *c0 = D.f0[1][t] * epsmin * (gp20 - gp10);
    *du = D.df[1][t] * auxc + D.f[1][t] * epsmin * (gp2 - 2.0 * gp1 * gp2) * T.ljsoft * D.df[0][t];
  }
  double g = 0.0;  // charge-pair kernel without its scale and soft core
  if (!A.lskip) {
    const double ar = A.alphad / auxa;
    const double qt = 1.0 / (1.0 + 0.3275911 * ar);
    g = qq * ((((1.0614054 * qt - 1.453152) * qt + 1.4214137) * qt - 0.28449674) * qt + 0.2548296) * qt *
        exp(-ar * ar);
  } else if (!A.ewald) {
    g = qq;
  }
  if (g != 0.0) {
    *qd = D.fq[1][t] * g * auxaa;
    *q0 = D.fq0[1][t] * g * auxa0;
    *du += D.dfq[1][t] * g * auxaa - D.fq[1][t] * g * T.qsoft * fq * D.dfq[0][t] * auxaa * auxaa * auxaa;
  }
}


// Entry queue of one i group: at most LPG - 1 entries left over from the
// chunks before plus LPG new ones.
template <int LPG>
struct Queue {
  static constexpr int N = 2 * LPG;
};

// LPG lanes own one i group for a whole list row (two groups per warp at 16).
//
// Phase 1 (a lane per list entry, LPG entries per chunk): FP64 minimum image
// and band of the group pair, the next shell's list entry (order kept by
// ballots), and, for an in-band entry with a pair to evaluate, its geometry
// (FP32 centre distance, S, S', and in FP64 what the energies need) and the
// bits of its atom pairs into the row's queue in shared memory.
//
// Phase 2 (a lane per queued entry, full passes of LPG entries and one for
// the row's rest): the lane evaluates every atom pair of its two groups, the
// i atoms from shared memory (a broadcast), the j atoms from memory once.
// Forces of both groups and V sum in the lane in a fixed order, so neither
// LPG nor the order of the passes changes a result; the S'(R) V term needs no
// exchange between lanes.  The j atoms leave by one fixed-point atomic per
// component and entry; the i atoms are added in fixed point over the row's
// passes and leave by one reduction over the lanes at the end of the row.
//
// Within an entry the sums are FP32 on both sides (an i atom's over up to MG
// pairs and its S'V share, where the lane-per-j-atom form before added each
// pair in fixed point).  Forces against 64 bits, relative, that form -> this
// one, shells M, L, H: 3,000 waters 8.1e-7 1.27e-6 5.5e-7 -> 8.0e-7 8.0e-7
// 5.4e-7; protein 5.8e-7 1.14e-6 6.2e-7 -> 5.8e-7 7.6e-7 5.8e-7; chains in
// groups of 4 6.8e-7 8.1e-7 4.7e-7 -> 7.0e-7 6.0e-7 4.5e-7, of 8 7.0e-7 8.4e-7
// 6.1e-7 -> 7.1e-7 8.3e-7 6.4e-7 (means of six systems, standard errors 3e-8 M,
// 1e-7 L, 2e-7 H).  Adding pair by pair here moved groups of 5 and 8 by no more
// than 0.3%, 1.2% and 7%, either way.
//
// What bounds it: on one system latency (a row is one pass of the M shell,
// two of the L shell), with the device full the issue of the pair arithmetic.
// A lane per entry keeps the pair arithmetic free of queue bookkeeping: the
// lane-per-j-atom form before it spent 4.4 M warp instructions on the M shell
// of 3,000 waters, two thirds of them on slots, shuffles and reductions.
//
// MINB: resident blocks per SM the forces-only build is compiled for (5, 6
// or 8, and 3, 4 or 5 with the work terms; fewer registers per thread the more
// blocks).
template <int MG, bool EN, int VAR, int LPG, int MINB>
__global__ void __launch_bounds__(warps_per_block(MG) * 32, MINB) k_pair(const PairArgs A) {
  constexpr int WPB = warps_per_block(MG);
  // the alchemy variant, and its build that also sums force_alchemy's dwrk
  constexpr bool ALCH = VAR == VAR_ALCH || VAR == VAR_ALCHW;
  constexpr int SEG = 32 / LPG;  // groups per warp
  constexpr int QE = Queue<LPG>::N;
  constexpr int NQ = WPB * SEG;  // groups per block
  constexpr unsigned FULL = 0xffffffffu;
  // pair bits: a * 8 + b, as the list's masks have them; four atoms a group
  // fit the low word
  using Bits = typename std::conditional<(MG > 4), unsigned long long, unsigned>::type;
  constexpr Bits COLS = (Bits)0x0101010101010101ull;
  __shared__ float4 s_ai[NQ][MG];
  __shared__ int s_ti[NQ][MG];  // the i atom's row of the LJ tables (type * ntype)
  __shared__ float s_pm[NQ][MG];
  __shared__ double4 s_gi[NQ];
  __shared__ double s_qd[NQ][EN ? MG : 1];
  __shared__ int s_fi[NQ][VAR != VAR_STD ? MG : 1];
  __shared__ float2 s_sf[NQ][ALCH ? MG : 1];
  // entry queue: centre distance and S; first j atom, j group metadata, S';
  // pair bits; FP64 distance and S and the Cartesian image for the energies
  __shared__ float4 s_edc[NQ][QE];
  __shared__ int4 s_emeta[NQ][QE];
  __shared__ float s_edsw[NQ][QE];
  __shared__ Bits s_ebits[NQ][QE];
  __shared__ double4 s_ecd[EN ? NQ : 1][EN ? QE : 1];
  __shared__ double4 s_eimg[EN ? NQ : 1][EN ? QE : 1];
  // the i atoms' forces of each lane's entries, in fixed point (a row of
  // lanes per value; the padding puts the values a lane apart in the banks)
  __shared__ long long s_fiq[3 * MG][WPB * 32 + 2];
  __shared__ double s_red[EN ? WPB : 1][18];
  __shared__ unsigned s_cnt[WPB][3];
  __shared__ float s_af[ALCH ? 2 : 1][9], s_afq[ALCH ? 2 : 1][9];

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane / LPG, sl = lane % LPG, q = warp * SEG + sub;
  const unsigned below = (1u << sl) - 1u;  // lanes of this segment below this one
  const int seg0 = sub * LPG;              // first lane of this segment
  const float2* __restrict__ lj = A.lj;
  // the row and its first entries: with list_old they are older than the
  // kernel before this one, and read before the wait for it
  if (!A.list_old) pdl_enter();
  const int i = (blockIdx.x * WPB + warp) * SEG + sub;
  const bool gvalid = i < A.ngrp;
  const int4 mi = gvalid ? A.gmeta[i] : make_int4(0, 0, 0, 0);
  const int row = gvalid ? A.off[i] : 0, m = gvalid ? A.cnt[i] : 0;
  int jnext = 0;  // the lane's entry of the chunk to come
  unsigned long long mnext = 0ull;
  if (sl < m) {
    jnext = A.lj_[row + sl];
    mnext = A.lmask[row + sl];
  }
  if (A.list_old) pdl_enter();
  pdl_release(A.early);
  if constexpr (ALCH) {  // the current lambda tables
    if (threadIdx.x < 18) {
      s_af[threadIdx.x / 9][threadIdx.x % 9] = A.ad->af[threadIdx.x / 9][threadIdx.x % 9];
      s_afq[threadIdx.x / 9][threadIdx.x % 9] = A.ad->afq[threadIdx.x / 9][threadIdx.x % 9];
    }
    __syncthreads();
  }
  // under lskip_ewald only pairs of atoms with LJ are evaluated
  const bool ljonly = A.lskip && A.ewald;
  const float remf = VAR == VAR_REM ? __ldg(A.remf) : 1.f;  // rem_factor(3)
  const float asqp = AS_QP * A.alphal;                      // A&S: t = 1 / (1 + p alpha r)
  const float a2l2 = -A.alphal * A.alphal * 1.44269504f;    // exp(-(alpha r)^2) as a power of two
  const float twa = A.twrtpi * A.alphal;
  // this segment's bits of a warp ballot
  auto segbits = [&](unsigned b) -> unsigned { return SEG == 1 ? b : (b >> seg0) & 0xffffu; };

  double ec0 = 0, ec1 = 0, ec2 = 0, eq0 = 0, eq1 = 0, eq2 = 0;
  double ex0 = 0, ex1 = 0, ex2 = 0;  // variant sums (ACC_X)
  // image term of the molecular virial (stress only)
  double vimg[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  // force_alchemy's dwrk of a forces-only launch under a schedule (A.dwrk):
  // U(lambda) - U(lambda0) of the alchemical pairs, FP64 on the FP32 pair
  // geometry (the other pairs' terms are equal at lambda and lambda0)
  double wk = 0.0;
  unsigned npairs = 0, nscan = 0, nkept = 0;

  // every lane of a warp runs the same trip counts, so the warp-wide ballots
  // and shuffles stay convergent
  {
    const int ifirst = mi.x, ni = mi.y & 15, typei = (mi.y >> 4) & 15, ljmi = (mi.y >> 8) & 0xff;
    if (sl == 0) s_gi[q] = gvalid ? A.gpos[i] : make_double4(0.0, 0.0, 0.0, 0.0);
    int mmax = m;
    if (SEG == 2) mmax = max(mmax, __shfl_xor_sync(FULL, m, 16));
    if (sl < MG) {  // (slots beyond the group's atoms: zeros, type 0)
      const bool in = sl < ni;
      const int at = ifirst + sl;
      s_ai[q][sl] = in ? A.aoff[at] : make_float4(0.f, 0.f, 0.f, 0.f);
      s_ti[q][sl] = in ? A.atype[at] * A.ntype : 0;
      s_pm[q][sl] = in ? A.apm[at] : 0.f;
      if (EN) s_qd[q][sl] = in ? A.qd[at] : 0.0;
      if (VAR != VAR_STD) s_fi[q][sl] = in ? A.vflag[at] : 0;
      if (ALCH) s_sf[q][sl] = in ? A.soft[at] : make_float2(0.f, 0.f);
    }
    Bits irows = 0;  // the i atoms to evaluate, a byte each
#pragma unroll
    for (int a = 0; a < MG; a++)
      if (a < ni && (!ljonly || ((ljmi >> a) & 1))) irows |= (Bits)0xff << (8 * a);
    __syncwarp();
    // the i atoms' forces are added over the lane's entries in fixed point,
    // in shared memory: integer sums are exact, so the row's total does not
    // depend on which lane took which entry
    bool started = false;  // a pass of this row has run

    int nout = 0;
    int qh = 0, qn = 0;  // entry queue: head, entries pending
    for (int base = 0; base < mmax; base += LPG) {
      // ---- phase 1: geometry of list entry k (src/force.f:265-333)
      const int k = base + sl;
      const bool valid = k < m;
      const int j = jnext;
      const unsigned long long msk = mnext;
      if (k + LPG < m) {
        jnext = A.lj_[row + k + LPG];
        mnext = A.lmask[row + k + LPG];
      }
      int4 mj = make_int4(0, 0, 0, 0);
      double drj = 1e300, cx = 0.0, cy = 0.0, cz = 0.0, imx = 0.0, imy = 0.0, imz = 0.0;
      if (valid) {
        const double4 gj = A.gpos[j];
        mj = A.gmeta[j];
        const double4 gi = s_gi[q];
        double dx = gi.x - gj.x, dy = gi.y - gj.y, dz = gi.z - gj.z;
        imx = 2.0 * round(0.5 * dx);
        imy = 2.0 * round(0.5 * dy);
        imz = 2.0 * round(0.5 * dz);
        dx -= imx;
        dy -= imy;
        dz -= imz;
        cx = __fma_rn(A.c13, dz, __fma_rn(A.c12, dy, __dmul_rn(A.c11, dx)));
        cy = __fma_rn(A.c23, dz, __dmul_rn(A.c22, dy));
        cz = __dmul_rn(A.c33, dz);
        drj = __fma_rn(cz, cz, __fma_rn(cy, cy, __dmul_rn(cx, cx)));
      }
      if (A.next_on) {  // the next inner shell's list, order kept (src/force.f:279-286)
        const bool keep = valid && drj < A.r2neigh;
        const unsigned bal = segbits(__ballot_sync(FULL, keep));
        if (keep) {
          const int pos = nout + __popc(bal & below);
          A.j_out[row + pos] = j;
          A.mask_out[row + pos] = msk;
        }
        nout += __popc(bal);
      }
      nscan += valid ? 1u : 0u;
      if (!A.forces_on) continue;
      // band: non-switched [rinn0, rout), S on [rout, rout0), 1-S on [rinn, rinn0)
      Bits bits = 0;
      float sw = 1.f, dsw = 0.f;
      double swd = 1.0;
      if (valid) {
        const bool sw_out = drj >= A.r2out && drj < A.r2out0;
        const bool sw_in = drj >= A.r2inn && drj < A.r2inn0;
        if ((drj >= A.r2inn0 && drj < A.r2out) || sw_out || sw_in) {
          const unsigned cols = ljonly ? (unsigned)(mj.y >> 8) & 0xffu : (1u << (mj.y & 15)) - 1u;
          bits = ~(Bits)msk & irows & ((Bits)cols * COLS);
        }
        if (sw_out || sw_in) {
          // S(R) of src/force.f:311-317 for the forces: FP32 arithmetic on
          // the two factors taken in FP64, the distance to the band edge
          // (edge - R) and auxa (ars1 + 2R, where -3 r and 2R cancel to under
          // a tenth of their size): FP32 R would leave both with 1e-5
          // relative error.  R in FP64 from an FP32 reciprocal square root
          // and one Newton step (relative error ~1e-14); the outer band
          // gives S = auxa auxb^2, the inner one 1 - auxa auxb^2, both from
          // the same code with the band's constants.  FP64 where S enters
          // the energies.
          const double edge = sw_out ? A.rout0 : A.rinn0;
          const double ars1 = sw_out ? A.arsout1 : A.arsinn1;
          const double iars2 = sw_out ? A.diarsout2 : A.diarsinn2;
          const float iars2f = sw_out ? A.iarsout2 : A.iarsinn2;
          const float sgn = sw_out ? 1.f : -1.f;
          double y = (double)rsqrtf((float)drj);
          y = __dmul_rn(y, __fma_rn(__dmul_rn(-0.5 * drj, y), y, 1.5));
          const double rspd = __dmul_rn(drj, y);
          const float auxa = (float)__dmul_rn(__fma_rn(2.0, rspd, ars1), iars2);
          const float auxb = (float)__dsub_rn(edge, rspd);
          const float s3 = mu(mu(auxa, auxb), auxb);
          sw = sw_out ? s3 : ad(1.0f, -s3);
          dsw = mu(mu(sgn, mu(2.0f * auxb, fm(auxb, iars2f, -auxa))), (float)y);
          if (EN) {
            const double auxbd = edge - rspd;
            const double s3d = (ars1 + 2.0 * rspd) * iars2 * auxbd * auxbd;
            swd = sw_out ? s3d : 1.0 - s3d;
          }
        }
      }
      // Entries with alchemical or fixed-mass atoms are queued a j atom at a
      // time (V and the S'V term are sums over the pairs): their pairs are
      // evaluated one after another, with FP64 work terms along a schedule,
      // and a lane with a whole entry of them would hold up its warp.
      const bool special = ALCH && ((mi.y | mj.y) & GM_SPECIAL);
      bool more = true;
      for (int part = 0; more; part++) {
        const Bits push = special ? bits & (COLS << part) : (part ? (Bits)0 : bits);
        const Bits rest = special ? bits & ~(Bits)(COLS * ((2u << part) - 1u)) : (Bits)0;
        more = ALCH && __any_sync(FULL, rest != 0);
        const unsigned bq = segbits(__ballot_sync(FULL, push != 0));
        if (push != 0) {
          const int e = (qh + qn + __popc(bq & below)) & (QE - 1);
          s_edc[q][e] = make_float4((float)cx, (float)cy, (float)cz, sw);
          s_emeta[q][e] = make_int4(mj.x, mj.y, mj.z, mj.w);
          s_edsw[q][e] = dsw;
          s_ebits[q][e] = push;
          if constexpr (EN) {
            s_ecd[q][e] = make_double4(cx, cy, cz, swd);
            if (A.stress)  // j sits at its image xpg_j + img: its virial arm gains co.img
              s_eimg[q][e] = make_double4(A.c11 * imx + A.c12 * imy + A.c13 * imz, A.c22 * imy + A.c23 * imz,
                                          A.c33 * imz, 0.0);
          }
        }
        qn += __popc(bq);
        __syncwarp();

        // ---- phase 2: a lane per queued entry
        const bool last = base + LPG >= m && !more;
        for (;;) {
          const int take = qn >= LPG ? LPG : (last ? qn : 0);
          if (!__any_sync(FULL, take > 0)) break;
          if (sl < take) {
            const int e = (qh + sl) & (QE - 1);
            const float4 dcs = s_edc[q][e];
            const int4 me = s_emeta[q][e];
            const Bits pb = s_ebits[q][e];
            const int jf = me.x, nj = me.y & 15;
            const float dswe = s_edsw[q][e];
            double4 cd = make_double4(0.0, 0.0, 0.0, 1.0);
            if (EN) cd = s_ecd[q][e];
            float fi[MG][3], fj[MG <= 4 ? MG : 1][3];
            double gjx = 0.0, gjy = 0.0, gjz = 0.0;  // the j group's force (image virial)
#pragma unroll
            for (int a = 0; a < MG; a++) fi[a][0] = fi[a][1] = fi[a][2] = 0.f;
#pragma unroll
            for (int b = 0; b < (MG <= 4 ? MG : 1); b++) fj[b][0] = fj[b][1] = fj[b][2] = 0.f;
            float V = 0.f;
            double pconf = 0.0, pcoul = 0.0, px0 = 0.0, px1 = 0.0, px2 = 0.0;
            // the straight path: every pair of the two groups without a branch,
            // so that the pairs' chains of dependent instructions overlap; pairs
            // that are not to be evaluated take part with coefficients 0.  Three
            // pairs share one test for LJ (in water only the oxygens have it).
            // Not for pairs of LJ alone (one in nine of water's) nor for groups
            // with alchemical or fixed-mass atoms.
            bool straight = MG <= 4 && !A.lskip && !(ALCH && ((mi.y | me.y) & GM_SPECIAL));
            if constexpr (MG <= 4) {
              if (straight) {
                float4 ob[MG];
#pragma unroll
                for (int b = 0; b < MG; b++)
                  ob[b] = b < nj ? A.aoff[jf + b] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int b = 0; b < MG; b++) {
                  const float bx = ad(dcs.x, -ob[b].x), by = ad(dcs.y, -ob[b].y), bz = ad(dcs.z, -ob[b].z);
                  float rx[MG], ry[MG], rz[MG], rsqi[MG], qf[MG], u[MG];
#pragma unroll
                  for (int a = 0; a < MG; a++) {
                    const float4 ai = s_ai[q][a];  // a broadcast read
                    const bool on = ((unsigned)pb >> (a * 8 + b)) & 1u;
                    rx[a] = ad(ai.x, bx);
                    ry[a] = ad(ai.y, by);
                    rz[a] = ad(ai.z, bz);
                    const float r2 = fm(rz[a], rz[a], fm(ry[a], ry[a], mu(rx[a], rx[a])));
                    const float qq = on ? mu(ai.w, ob[b].w) : 0.f;
                    // 1/r from the hardware reciprocal square root, exp from ex2
                    // and an approximate reciprocal: a few ulp, far below the
                    // pair's FP32 rounding budget
                    const float rinv = rsqrtf(r2);
                    rsqi[a] = mu(rinv, rinv);
                    const float qt = __fdividef(1.0f, fm(asqp, mu(r2, rinv), 1.0f));
                    const float qe = mu(qq, ex2f(mu(a2l2, r2)));
                    const float poly = fm(fm(fm(fm(AS_A5, qt, AS_A4), qt, AS_A3), qt, AS_A2), qt, AS_A1);
                    u[a] = mu(mu(mu(poly, qt), qe), rinv);
                    qf[a] = fm(twa, qe, u[a]);
                  }
                  if ((me.y >> (8 + b)) & 1) {  // the j atom has LJ
                    const int tb = b < 2 ? (me.z >> (16 * b)) & 0xffff : (me.w >> (16 * (b - 2))) & 0xffff;
#pragma unroll
                    for (int a = 0; a < MG; a++) {
                      const bool on = ((unsigned)pb >> (a * 8 + b)) & 1u;
                      float u12, u6;
                      if constexpr (ALCH) {  // two normal atoms: full strength, force_alchemy's sigma and epsilon
                        const float2 sa = s_sf[q][a], sb = A.soft[jf + b];
                        const float eps4 = on && sa.y * sb.y > 1e-12f ? sa.y * sb.y : 0.f;
                        const float sig = A.at.opls ? 2.f * sqrtf(mu(sa.x, sb.x)) : ad(sa.x, sb.x);
                        const float s2 = mu(mu(sig, sig), rsqi[a]);
                        const float x = mu(mu(s2, s2), s2);
                        u6 = mu(eps4, x);
                        u12 = mu(u6, x);
                      } else {
                        const float2 L = __ldg(lj + s_ti[q][a] + tb);
                        const float r6 = on ? mu(mu(rsqi[a], rsqi[a]), rsqi[a]) : 0.f;
                        u6 = mu(L.y, r6);
                        u12 = mu(mu(L.x, r6), r6);
                      }
                      qf[a] = fm(12.0f, u12, fm(-6.0f, u6, qf[a]));
                      u[a] = ad(u[a], ad(u12, -u6));
                    }
                  }
                  float fbx = 0.f, fby = 0.f, fbz = 0.f;
#pragma unroll
                  for (int a = 0; a < MG; a++) {
                    // force_rem (src/force_REM.f:491-495,634-678): selected pairs
                    // scale their force and their share of the S'V sum
                    float w = dcs.w;
                    bool sel = false;
                    if constexpr (VAR == VAR_REM) {
                      const bool ra = (mi.y >> (GM_REM + a)) & 1, rb = (me.y >> (GM_REM + b)) & 1;
                      sel = A.rem_kind == 0 ? (ra || rb) : (A.rem_kind == 1 ? (ra && rb) : (ra != rb));
                      w = sel ? mu(w, remf) : w;
                      V = sel ? fm(u[a], remf, V) : ad(V, u[a]);
                    } else {
                      V = ad(V, u[a]);
                    }
                    const float f = mu(mu(qf[a], rsqi[a]), w);
                    fi[a][0] = fm(f, rx[a], fi[a][0]);
                    fi[a][1] = fm(f, ry[a], fi[a][1]);
                    fi[a][2] = fm(f, rz[a], fi[a][2]);
                    fbx = fm(-f, rx[a], fbx);
                    fby = fm(-f, ry[a], fby);
                    fbz = fm(-f, rz[a], fbz);
                  }
                  fj[b][0] = fbx;
                  fj[b][1] = fby;
                  fj[b][2] = fbz;
                  if (EN) {
                    gjx += fbx;
                    gjy += fby;
                    gjz += fbz;
                  }
                }
                // V is no number where a coordinate is none or infinite (every pair's
                // distance enters it, also of the pairs that are not to be evaluated,
                // with coefficient 0), or where such a pair has no distance at all.
                // Their forces would then be NaN too, and those of the slots beyond a
                // group's atoms belong to other atoms or to none: the entry is
                // evaluated pair by pair instead.
                if (V == V) {
                  npairs += __popc((unsigned)pb);
                } else {
                  straight = false;
                  V = 0.f;
                  gjx = gjy = gjz = 0.0;
#pragma unroll
                  for (int a = 0; a < MG; a++)
#pragma unroll
                    for (int c = 0; c < 3; c++) fi[a][c] = fj[a][c] = 0.f;
                }
              }
            }
            if (!straight) {
              if (!ljonly && !ALCH) npairs += MG > 4 ? __popcll(pb) : __popc((unsigned)pb);
#pragma unroll 1
              for (int b = 0; b < MG; b++) {
                const Bits col = (pb >> b) & COLS;  // the i atoms of this j atom's pairs
                if (!col) continue;
                float fbx = 0.f, fby = 0.f, fbz = 0.f;
                const int jat = jf + b;
                const float4 ob = A.aoff[jat];
                const int tb = A.atype[jat];
                const int fjb = (VAR != VAR_STD) ? (int)A.vflag[jat] : 0;
                const float2 sfb = ALCH ? A.soft[jat] : make_float2(0.f, 0.f);
                const float bx = ad(dcs.x, -ob.x), by = ad(dcs.y, -ob.y), bz = ad(dcs.z, -ob.z);
#pragma unroll
                for (int a = 0; a < MG; a++) {
                  if (!((col >> (a * 8)) & 1)) continue;
                  const float4 ai = s_ai[q][a];  // a broadcast read
                  const float rx = ad(ai.x, bx), ry = ad(ai.y, by), rz = ad(ai.z, bz);
                  const float r2 = fm(rz, rz, fm(ry, ry, mu(rx, rx)));
                  float qf = 0.f, conf = 0.f, coul = 0.f;
                  if constexpr (ALCH) {
                    // src/force_alchemy.f:412-451: exclusions and fixed-mass pairs
                    // are always skipped; no LJ and no Coulomb skips the pair
                    const int fia = s_fi[q][a];
                    if (fia & fjb & VF_MINF) continue;
                    const float2 sa = s_sf[q][a];
                    const float eps4 = sa.y * sfb.y;
                    if (eps4 < 1e-12f && ljonly) continue;
                    npairs++;
                    alch_pair_f32(A, s_af, s_afq, r2, (fia >> VF_SSHIFT) + (fjb >> VF_SSHIFT) - 4, sa.x, sfb.x, eps4,
                                  ai.w * ob.w, &qf, &conf, &coul);
                  } else {
                    const float2 Lp = __ldg(lj + s_ti[q][a] + tb);
                    const bool ljon = Lp.y != 0.f;
                    if (ljonly) {  // src/force.f:416-417
                      if (!ljon) continue;
                      npairs++;
                    }
                    const float rinv = rsqrtf(r2);
                    const float rsqi = mu(rinv, rinv);
                    if (ljon) {
                      const float r6 = mu(mu(rsqi, rsqi), rsqi);
                      const float u6 = mu(Lp.y, r6), u12 = mu(mu(Lp.x, r6), r6);
                      qf = fm(12.0f, u12, mu(-6.0f, u6));
                      conf = ad(u12, -u6);
                    }
                    if (!A.lskip) {
                      const float qt = __fdividef(1.0f, fm(asqp, mu(r2, rinv), 1.0f));
                      const float qe = mu(mu(ai.w, ob.w), ex2f(mu(a2l2, r2)));
                      const float poly = fm(fm(fm(fm(AS_A5, qt, AS_A4), qt, AS_A3), qt, AS_A2), qt, AS_A1);
                      coul = mu(mu(mu(poly, qt), qe), rinv);
                      qf = ad(qf, fm(twa, qe, coul));
                    } else if (!A.ewald) {
                      coul = mu(mu(ai.w, ob.w), rinv);
                      qf = ad(qf, coul);
                    }
                    qf = mu(qf, rsqi);
                  }
                  // force_rem (src/force_REM.f:491-495,634-678): selected pairs scale
                  // their force and their share of the S'V sum
                  const bool sel = (VAR == VAR_REM) && seg_sel(A.rem_kind, s_fi[q][a], fjb);
                  V = sel ? fm(ad(conf, coul), remf, V) : ad(V, ad(conf, coul));
                  qf = mu(qf, dcs.w);
                  if (sel) qf = mu(qf, remf);
                  fi[a][0] = fm(qf, rx, fi[a][0]);
                  fi[a][1] = fm(qf, ry, fi[a][1]);
                  fi[a][2] = fm(qf, rz, fi[a][2]);
                  fbx = fm(-qf, rx, fbx);
                  fby = fm(-qf, ry, fby);
                  fbz = fm(-qf, rz, fbz);
                }
                if constexpr (MG <= 4) {
#pragma unroll
                  for (int c = 0; c < MG; c++)
                    if (c == b) {
                      fj[c][0] = fbx;
                      fj[c][1] = fby;
                      fj[c][2] = fbz;
                    }
                } else {
                  fix_add(A.ffix + jat, fbx);
                  fix_add(A.ffix + A.natom + jat, fby);
                  fix_add(A.ffix + 2 * A.natom + jat, fbz);
                }
                if (EN) {
                  gjx += fbx;
                  gjy += fby;
                  gjz += fbz;
                }
              }
            }
            // along a schedule, force_alchemy's dwrk of an entry with alchemical
            // atoms (one j atom): U(lambda) - U(lambda0) of its pairs
            if constexpr (VAR == VAR_ALCHW) {
              if ((mi.y | me.y) & GM_SPECIAL) {
                const int b = MG > 4 ? (__ffsll((long long)pb) - 1) & 7 : (__ffs((int)pb) - 1) & 7;
                const int jat = jf + b;
                const float4 ob = A.aoff[jat];
                const float bx = ad(dcs.x, -ob.x), by = ad(dcs.y, -ob.y), bz = ad(dcs.z, -ob.z);
                const int fjb = A.vflag[jat];
                const double2 sj = A.softd[jat];
                const double qj = A.qd[jat];
                const float yj = A.soft[jat].y;
#pragma unroll
                for (int a = 0; a < MG; a++) {
                  if (!((pb >> (a * 8 + b)) & 1)) continue;
                  const int fia = s_fi[q][a], tal = (fia >> VF_SSHIFT) + (fjb >> VF_SSHIFT) - 4;
                  if (tal == 6 || (fia & fjb & VF_MINF)) continue;  // 6: two normal atoms
                  if (s_sf[q][a].y * yj < 1e-12f && ljonly) continue;
                  const float4 ai = s_ai[q][a];
                  double cdd, qdd, c0, q0, du;
                  alch_energy_fp64(A, (double)ad(ai.x, bx), (double)ad(ai.y, by), (double)ad(ai.z, bz),
                                   A.softd[ifirst + a], sj, A.qd[ifirst + a] * qj, tal, &cdd, &qdd, &c0, &q0, &du);
                  wk += ((cdd + qdd) - (c0 + q0)) * (double)dcs.w;
                }
              }
            }
            // the FP64 pair energies: one rolled loop over the entry's pairs
            if constexpr (EN) {
#pragma unroll 1
              for (Bits rest = pb; rest; rest &= rest - 1) {
                const int bit = MG > 4 ? __ffsll((long long)rest) - 1 : __ffs((int)rest) - 1;
                const int a = bit >> 3, jat = jf + (bit & 7);
                const float4 ai = s_ai[q][a], ob = A.aoff[jat];
                const double erx = cd.x + ((double)ai.x - (double)ob.x);
                const double ery = cd.y + ((double)ai.y - (double)ob.y);
                const double erz = cd.z + ((double)ai.z - (double)ob.z);
                double cdd, qdd;
                if constexpr (ALCH) {
                  const int fia = s_fi[q][a], fjb = A.vflag[jat];
                  if (fia & fjb & VF_MINF) continue;
                  if (s_sf[q][a].y * A.soft[jat].y < 1e-12f && ljonly) continue;
                  double c0, q0, du;
                  alch_energy_fp64(A, erx, ery, erz, A.softd[ifirst + a], A.softd[jat], s_qd[q][a] * A.qd[jat],
                                   (fia >> VF_SSHIFT) + (fjb >> VF_SSHIFT) - 4, &cdd, &qdd, &c0, &q0, &du);
                  px0 += c0;
                  px1 += q0;
                  px2 += du;
                } else {
                  const double2 L = A.ljd[s_ti[q][a] + A.atype[jat]];
                  if (ljonly && L.y == 0.0) continue;
                  pair_energy_fp64(A, erx, ery, erz, L, L.y != 0.0, s_qd[q][a] * A.qd[jat], &cdd, &qdd);
                  if (VAR == VAR_REM && seg_sel(A.rem_kind, s_fi[q][a], A.vflag[jat])) px0 += cdd + qdd;  // seg_ene
                }
                pconf += cdd;
                pcoul += qdd;
              }
            }
            // S'(R) V term of a switched entry (src/force.f:754-817): X = -dS/dR / R
            // V R_vec distributed by mass fraction over both groups' atoms
            if (dswe != 0.f) {
              const float sv = mu(-dswe, V);
              const float sx = mu(sv, dcs.x), sy = mu(sv, dcs.y), sz = mu(sv, dcs.z);
              if constexpr (MG <= 4) {
#pragma unroll
                for (int b = 0; b < MG; b++) {
                  if (b >= nj) continue;
                  const float pm = A.apm[jf + b];
                  fj[b][0] = fm(-pm, sx, fj[b][0]);
                  fj[b][1] = fm(-pm, sy, fj[b][1]);
                  fj[b][2] = fm(-pm, sz, fj[b][2]);
                }
              } else {
                for (int b = 0; b < nj; b++) {
                  const float pm = A.apm[jf + b];
                  fix_add(A.ffix + jf + b, -pm * sx);
                  fix_add(A.ffix + A.natom + jf + b, -pm * sy);
                  fix_add(A.ffix + 2 * A.natom + jf + b, -pm * sz);
                }
              }
#pragma unroll
              for (int a = 0; a < MG; a++) {
                const float pmi = s_pm[q][a];
                fi[a][0] = fm(pmi, sx, fi[a][0]);
                fi[a][1] = fm(pmi, sy, fi[a][1]);
                fi[a][2] = fm(pmi, sz, fi[a][2]);
              }
              if (EN) {
                gjx -= sx;
                gjy -= sy;
                gjz -= sz;
              }
            }
            if constexpr (MG <= 4) {
#pragma unroll
              for (int b = 0; b < MG; b++) {  // (zero beyond the group's atoms, whatever the coordinates)
                fix_add(A.ffix + jf + b, fj[b][0]);
                fix_add(A.ffix + A.natom + jf + b, fj[b][1]);
                fix_add(A.ffix + 2 * A.natom + jf + b, fj[b][2]);
              }
            }
#pragma unroll
            for (int c = 0; c < 3 * MG; c++) {
              const long long add = to_fix(fi[c / 3][c % 3]);
              s_fiq[c][threadIdx.x] = started ? s_fiq[c][threadIdx.x] + add : add;
            }
            if constexpr (EN) {
              const int tt = typei + ((me.y >> 4) & 15) - 2;  // 0 slt-slt, 1 slt-slv, 2 slv-slv
              pconf *= cd.w;
              pcoul *= cd.w;
              if (tt == 0) {
                ec0 += pconf;
                eq0 += pcoul;
              } else if (tt == 1) {
                ec1 += pconf;
                eq1 += pcoul;
              } else {
                ec2 += pconf;
                eq2 += pcoul;
              }
              ex0 += px0 * cd.w;
              ex1 += px1 * cd.w;
              ex2 += px2 * cd.w;
              if (A.stress) {
                const double4 im = s_eimg[q][e];
                const double g3[3] = {gjx, gjy, gjz}, i3[3] = {im.x, im.y, im.z};
#pragma unroll
                for (int c = 0; c < 9; c++) vimg[c] += g3[c / 3] * i3[c % 3];
              }
            }
          }
          if (take > 0 && take < LPG && !started && sl >= take) {
#pragma unroll
            for (int c = 0; c < 3 * MG; c++) s_fiq[c][threadIdx.x] = 0ll;
          }
          started = started || take > 0;
          qh += take;
          qn -= take;
          __syncwarp();
        }
      }
    }
    if (A.next_on && sl == 0 && gvalid) {
      A.cnt_out[i] = nout;
      nkept += (unsigned)nout;
    }
    // i atoms: a lane sums one value over the row's lanes (of a whole-warp row, half
    // of the lanes each) and adds it
    constexpr int PARTS = (LPG == 32 && 3 * MG <= 16) ? 2 : 1;
    const int val = sl % (LPG / PARTS), part = sl / (LPG / PARTS);
    long long sum = 0ll;
    if (started && val < 3 * ni) {
      const long long* src = &s_fiq[val][warp * 32 + seg0 + part * (LPG / PARTS)];
#pragma unroll 8
      for (int k = 0; k < LPG / PARTS; k++) sum += src[k];
    }
    if (PARTS == 2) sum += __shfl_xor_sync(FULL, sum, 16);
    if (part == 0 && sum != 0ll)
      atomicAdd(A.ffix + (val % 3) * A.natom + ifirst + val / 3, (unsigned long long)sum);
  }
  {
    // work counters: one atomic per block and counter, over WCNT_SLOTS copies
    // (a single copy's atomics of a launch wait for one another at the L2)
    nscan = __reduce_add_sync(FULL, nscan);
    nkept = __reduce_add_sync(FULL, nkept);
    npairs = __reduce_add_sync(FULL, npairs);
    if (lane < 3) s_cnt[warp][lane] = lane == 0 ? nscan : (lane == 1 ? nkept : npairs);
  }
  // energies and the image virial: the EN build only (a stress request
  // selects it, pair_launch)
  constexpr int NV = (VAR != VAR_STD) ? 18 : 15;
  if constexpr (EN) {
    const double vals[18] = {ec0, ec1, ec2, eq0, eq1, eq2, vimg[0], vimg[1], vimg[2],
                             vimg[3], vimg[4], vimg[5], vimg[6], vimg[7], vimg[8], ex0, ex1, ex2};
#pragma unroll
    for (int c = 0; c < NV; c++) {
      const double sred = warp_sumd(vals[c]);
      if (lane == 0) s_red[warp][c] = sred;
    }
  }
  if constexpr (VAR == VAR_ALCHW) {
    const double w = warp_sumd(wk);
    if (lane == 0 && w != 0.0) atomicAdd(A.dwrk, w);
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    unsigned s = 0;
#pragma unroll
    for (int w = 0; w < WPB; w++) s += s_cnt[w][threadIdx.x];
    const int slot = threadIdx.x < 2 ? (int)threadIdx.x : (A.lskip ? 3 : 2);
    if (s) atomicAdd(A.wcnt + 4 * (blockIdx.x % WCNT_SLOTS) + slot, (unsigned long long)s);
  }
  if constexpr (EN) {
    if (A.forces_on && threadIdx.x < NV) {
      double sacc = 0;
      for (int w = 0; w < WPB; w++) sacc += s_red[w][threadIdx.x];
      // slots 0..14 = ACC_CONF..ACC_VIMG+8, then ACC_X..ACC_X+2
      const int acc_slot = threadIdx.x < 15 ? (int)threadIdx.x : ACC_X + (int)threadIdx.x - 15;
      if (sacc != 0.0) atomicAdd(A.acc + acc_slot, sacc);
    }
  }
}

// group centres as double4 and atom offsets from their group centre
__global__ void k_prep(int N, int G, const double* __restrict__ xyz,
                       const double* __restrict__ grp,
                       const int* __restrict__ agrp,
                       const float* __restrict__ aq, double c11, double c12,
                       double c13, double c22, double c23, double c33,
                       double4* __restrict__ gpos, float4* __restrict__ aoff,
                       unsigned long long* __restrict__ ffix) {
  pdl_enter();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < G) gpos[t] = make_double4(grp[t], grp[G + t], grp[2 * G + t], 0.0);
  if (t < N) {
    const int g = agrp[t];
    const double dx = xyz[t] - grp[g];
    const double dy = xyz[N + t] - grp[G + g];
    const double dz = xyz[2 * N + t] - grp[2 * G + g];
    aoff[t] = make_float4((float)(c11 * dx + c12 * dy + c13 * dz),
                          (float)(c22 * dy + c23 * dz), (float)(c33 * dz),
                          aq[t]);
    ffix[t] = 0ull;
    ffix[N + t] = 0ull;
    ffix[2 * N + t] = 0ull;
  }
}

// fixed point -> double forces (accumulated into fout) and the atom part of
// the molecular virial: sum_a F_a (x) co.Rm_a
__global__ void k_finalize(int N, const unsigned long long* __restrict__ ffix,
                           const double* __restrict__ mol, int P,
                           const int* __restrict__ amol, double c11, double c12,
                           double c13, double c22, double c23, double c33,
                           double* __restrict__ fout, double* __restrict__ acc) {
  pdl_enter();
  __shared__ double s_red[8][9];
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (!mol) {  // forces only; the condition is uniform over the grid
    if (t < N) {
      fout[t] += (double)(long long)ffix[t] * ORAC_FSCALE_INV;
      fout[N + t] += (double)(long long)ffix[N + t] * ORAC_FSCALE_INV;
      fout[2 * N + t] += (double)(long long)ffix[2 * N + t] * ORAC_FSCALE_INV;
    }
    return;
  }
  double st[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  if (t < N) {
    const double fx = (double)(long long)ffix[t] * ORAC_FSCALE_INV;
    const double fy = (double)(long long)ffix[N + t] * ORAC_FSCALE_INV;
    const double fz = (double)(long long)ffix[2 * N + t] * ORAC_FSCALE_INV;
    fout[t] += fx;
    fout[N + t] += fy;
    fout[2 * N + t] += fz;
    const int p = amol[t];
    const double sx = mol[p], sy = mol[P + p], sz = mol[2 * P + p];
    const double rx = c11 * sx + c12 * sy + c13 * sz;
    const double ry = c22 * sy + c23 * sz;
    const double rz = c33 * sz;
    st[0] = fx * rx;
    st[1] = fx * ry;
    st[2] = fx * rz;
    st[3] = fy * rx;
    st[4] = fy * ry;
    st[5] = fy * rz;
    st[6] = fz * rx;
    st[7] = fz * ry;
    st[8] = fz * rz;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 9; q++) {
    const double s = warp_sumd(st[q]);
    if (lane == 0) s_red[warp][q] = s;
  }
  __syncthreads();
  if (threadIdx.x < 9) {
    double s = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += s_red[w][threadIdx.x];
    atomicAdd(acc + ACC_STR + threadIdx.x, s);
  }
}

}  // namespace

int pair_launch(orac_gpu_ctx* ctx, const PairArgs& a, int maxg) {
  if (maxg > ORAC_MAXG)
    return ctx_fail(ctx, ORAC_ERR_PARAM, "charge group of %d atoms exceeds %d", maxg, ORAC_MAXG);
  if (a.variant < VAR_STD || a.variant > VAR_ALCH) return ctx_fail(ctx, ORAC_ERR_PARAM, "variant %d", a.variant);
  // the alchemy build that sums force_alchemy's dwrk (forces only)
  const int var = (a.variant == VAR_ALCH && a.dwrk && !a.energy && !a.stress) ? VAR_ALCHW : a.variant;
  // atoms-per-group bound of the instantiation: 3 (waters, and chains cut
  // in threes), 4, or 8; half-warp groups and the occupancy classes only
  // for the two small bounds
  const int mgk = maxg <= 3 ? 0 : (maxg <= 4 ? 1 : 2);
  const bool half = mgk < 2 && a.lpg == 16;
  const int wpb = warps_per_block(mgk == 2 ? 8 : 4);
  const int gpb = wpb * (half ? 2 : 1);  // groups per block
  int nb = (a.ngrp + gpb - 1) / gpb;
  if (nb < 1) nb = 1;
  int slot = -1;
  if (int rc = prof_begin(ctx, &slot)) return rc;
  const bool en = a.energy || a.stress;  // the forces-only build keeps no sums
  // occupancy class of the forces-only build: 0, 1, 2 = 5, 6, 8 blocks per SM
  const int occ = (en || mgk == 2) ? 0 : (a.minb <= 5 ? 0 : (a.minb <= 7 ? 1 : 2));
  switch ((((mgk * 4 + var) * 2 + (en ? 1 : 0)) * 2 + (half ? 1 : 0)) * 3 + occ) {
#define ORAC_KP(MGK, MG, VAR, EN, LPG, OCC, MINB)                                               \
  case (((MGK * 4 + VAR) * 2 + (EN ? 1 : 0)) * 2 + (LPG == 16 ? 1 : 0)) * 3 + OCC:             \
    orac_launch(k_pair<MG, EN, VAR, LPG, MINB>, nb, wpb * 32, 0, ctx->stream, a);            \
    break;
#define ORAC_KP_L(MGK, MG, VAR, LPG)       \
  ORAC_KP(MGK, MG, VAR, false, LPG, 0, 5) \
  ORAC_KP(MGK, MG, VAR, false, LPG, 1, 6)  \
  ORAC_KP(MGK, MG, VAR, false, LPG, 2, 8)  \
  ORAC_KP(MGK, MG, VAR, true, LPG, 0, 1)
#define ORAC_KP_V(MGK, MG, VAR) \
  ORAC_KP_L(MGK, MG, VAR, 32)   \
  ORAC_KP_L(MGK, MG, VAR, 16)
// (the FP64 work terms of its alchemical rows are the launch's longest chain:
// registers before occupancy)
#define ORAC_KP_W(MGK, MG)                         \
  ORAC_KP(MGK, MG, VAR_ALCHW, false, 32, 0, 3)     \
  ORAC_KP(MGK, MG, VAR_ALCHW, false, 32, 1, 4)     \
  ORAC_KP(MGK, MG, VAR_ALCHW, false, 32, 2, 5)     \
  ORAC_KP(MGK, MG, VAR_ALCHW, false, 16, 0, 3)     \
  ORAC_KP(MGK, MG, VAR_ALCHW, false, 16, 1, 4)     \
  ORAC_KP(MGK, MG, VAR_ALCHW, false, 16, 2, 5)
    ORAC_KP_V(0, 3, VAR_STD)
    ORAC_KP_V(0, 3, VAR_REM)
    ORAC_KP_V(0, 3, VAR_ALCH)
    ORAC_KP_V(1, 4, VAR_STD)
    ORAC_KP_V(1, 4, VAR_REM)
    ORAC_KP_V(1, 4, VAR_ALCH)
    ORAC_KP(2, 8, VAR_STD, false, 32, 0, 1)
    ORAC_KP(2, 8, VAR_STD, true, 32, 0, 1)
    ORAC_KP(2, 8, VAR_REM, false, 32, 0, 1)
    ORAC_KP(2, 8, VAR_REM, true, 32, 0, 1)
    ORAC_KP(2, 8, VAR_ALCH, false, 32, 0, 1)
    ORAC_KP(2, 8, VAR_ALCH, true, 32, 0, 1)
    ORAC_KP_W(0, 3)
    ORAC_KP_W(1, 4)
    ORAC_KP(2, 8, VAR_ALCHW, false, 32, 0, 1)
#undef ORAC_KP_W
#undef ORAC_KP_V
#undef ORAC_KP_L
#undef ORAC_KP
    default:
      return ctx_fail(ctx, ORAC_ERR_PARAM, "no pair-kernel build for %d atoms per group, lpg %d, %d blocks per SM",
                      maxg, a.lpg, a.minb);
  }
  CKL();
  return prof_end(ctx, slot);
}

// Inside a stream capture an event must be recorded as an external event
// node to be a real, timed record when the graph replays.
static int prof_record(orac_gpu_ctx* ctx, cudaEvent_t ev) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  CK(cudaStreamIsCapturing(ctx->stream, &cs));
  if (cs == cudaStreamCaptureStatusActive)
    CK(cudaEventRecordWithFlags(ev, ctx->stream, cudaEventRecordExternal));
  else
    CK(cudaEventRecord(ev, ctx->stream));
  return ORAC_OK;
}

int prof_begin(orac_gpu_ctx* ctx, int* slot, int family) {
  *slot = -1;
  if (!(ctx->prof & (1 << family))) return ORAC_OK;
  if (2 * (ctx->prof_next + 1) > (int)ctx->prof_ev.size()) return ORAC_OK;  // pool exhausted: not profiled
  *slot = ctx->prof_next++;
  ctx->prof_fam[*slot] = family;
  return prof_record(ctx, ctx->prof_ev[2 * *slot]);
}

int prof_end(orac_gpu_ctx* ctx, int slot) {
  if (slot < 0) return ORAC_OK;
  return prof_record(ctx, ctx->prof_ev[2 * slot + 1]);
}

int prof_collect(orac_gpu_ctx* ctx, int a, int b) {
  for (int s = a; s < b; s++) {
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, ctx->prof_ev[2 * s], ctx->prof_ev[2 * s + 1]) != cudaSuccess) {
      cudaGetLastError();  // not sticky: mark the measurement invalid, keep running
      ctx->prof_bad = true;
      continue;
    }
    const int f = ctx->prof_fam[s];
    ctx->prof_ms[f] += ms;
    ctx->prof_n[f]++;
  }
  return ORAC_OK;
}

int prep_launch(orac_gpu_ctx* ctx, const double* xyz, const double* grp) {
  const int n = ctx->N > ctx->G ? ctx->N : ctx->G;
  const double* c = ctx->co;
  orac_launch(k_prep, (n + 255) / 256, 256, 0, ctx->stream, 
      ctx->N, ctx->G, xyz, grp, ctx->d_agrp, ctx->d_aq, c[0], c[3], c[6], c[4], c[7], c[8], ctx->d_gpos,
      ctx->d_aoff, ctx->d_ffix);
  CKL();
  return ORAC_OK;
}

int finalize_launch(orac_gpu_ctx* ctx, const double* mol, double* fout, int stress) {
  const double* c = ctx->co;
  orac_launch(k_finalize, (ctx->N + 255) / 256, 256, 0, ctx->stream, ctx->N, ctx->d_ffix, stress ? mol : nullptr, ctx->P,
                                                            ctx->d_amol, c[0], c[3], c[6], c[4], c[7], c[8], fout,
                                                            ctx->d_acc);
  CKL();
  return ORAC_OK;
}

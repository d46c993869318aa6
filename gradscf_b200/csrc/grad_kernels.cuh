// Coordinate VJP of J/K: sum over canonical screened quartets of
//   dE = sum_abcd d(ab|cd)/dR * Gamma_abcd,
// Gamma = the eight-permutation symmetrisation (times the degeneracy scale
// s of load_quartet) of  Jbar_ab D_cd + Kbar_ac D_bd  (the reference's
// transposed contraction, csrc/direct_jk_geometry.cc:68-84, which runs over
// all n^4 entries instead).  Derivatives recomputed, never stored:
//   d/dA_x phi_a = 2 alpha phi_{a+1x} - a_x phi_{a-1x}  (same for B, C),
//   d/dD = -(d/dA + d/dB + d/dC)  (translational invariance).
// Three kernels by block size: grad_reg_kernel and grad_lane_kernel (one lane
// per quartet), grad_unit_kernel (a warp or a block per quartet).
#pragma once
#include "jk_kernels.cuh"

namespace b200jk {

// Roots of a first-derivative quartet.
template <int LA, int LB, int LC, int LD>
struct GradCfg {
  static constexpr int NROOT = (LA + LB + LC + LD + 1) / 2 + 1;
};

// Raw Cartesian Gamma of one AO quartet (a, b, c, d), summed over batches.
__device__ __forceinline__ double gamma_abcd(const JKArgs& args, long long base, int n, int a, int b,
                                             int c, int d) {
  double gsum = 0.0;
  for (int e = 0; e < args.gnb; ++e) {
    const double* D = args.dens + e * args.dstride + base;
    const double* J = args.cot_j ? args.cot_j + e * args.dstride + base : nullptr;
    const double* K = args.cot_k ? args.cot_k + e * args.dstride + base : nullptr;
#define M_(X, i, j) X[(long long)(i) * n + (j)]
    if (J)
      gsum += (M_(J, a, b) + M_(J, b, a)) * (M_(D, c, d) + M_(D, d, c)) +
              (M_(J, c, d) + M_(J, d, c)) * (M_(D, a, b) + M_(D, b, a));
    if (K)
      gsum += M_(K, a, c) * M_(D, b, d) + M_(K, c, a) * M_(D, d, b) + M_(K, b, c) * M_(D, a, d) +
              M_(K, c, b) * M_(D, d, a) + M_(K, a, d) * M_(D, b, c) + M_(K, d, a) * M_(D, c, b) +
              M_(K, b, d) * M_(D, a, c) + M_(K, d, b) * M_(D, c, a);
#undef M_
  }
  return gsum;
}

// Ket range of a coordinate-VJP work item for the requested precision slice
// (split_mode 1: the kets before the item's FP32 boundary, 2: from it on).
__device__ __forceinline__ void grad_ket_range(const JKArgs& args, int item, const int4 w, int& kb, int& ke) {
  kb = w.y;
  ke = w.z;
  if (args.split_mode != 0) {
    const int s = args.split[item];
    if (args.split_mode == 1) ke = min(ke, s);
    else kb = max(kb, s);
  }
}

// One primitive quartet's scalars in precision R (FP32 quartets: the pair
// data stored relative to A and C, centre differences formed in FP64).
template <typename R>
__device__ __forceinline__ void grad_prim(const JKArgs& args, const QuartetGeom& g, int i, int j, PrimQ<R>& s) {
  const float3 ac = make_float3(float(g.ax - g.cx), float(g.ay - g.cy), float(g.az - g.cz));
  prim_any<R>(g, ac, PrimData<R>::a(args, i), PrimData<R>::b(args, i), PrimData<R>::a(args, j),
              PrimData<R>::b(args, j), s);
}

}  // namespace b200jk

namespace b200jk {

// Register-path coordinate VJP for small classes: one lane per ket of a
// work item (warp-granular items as the J/K register path), the raised 2D
// integrals of one root in registers, nine derivative partials per lane;
// the bra-centre partials (A, B fixed per warp) are warp-reduced.
template <int LA, int LB, int LC, int LD>
struct GradReg {
  using CI = ClassInfo<LA, LB, LC, LD>;
  static constexpr int NGR = (LA + 2) * (LB + 2) * (LC + 2) * (LD + 1);
#ifndef B200JK_GRAD_REG_LIMIT
#define B200JK_GRAD_REG_LIMIT 96  // measured: (H2O)8 cc-pVTZ gradient 510 -> 479 ms
#endif
  static constexpr bool OK = 3 * NGR + CI::NOUT <= B200JK_GRAD_REG_LIMIT;
};

template <int LA, int LB, int LC, int LD, typename R>
__global__ void __launch_bounds__(128, 3) grad_reg_kernel(JKArgs args) {
  using CI = ClassInfo<LA, LB, LC, LD>;
  using GC = GradCfg<LA, LB, LC, LD>;
  using GI = GIdx<LA + 1, LB + 1, LC + 1, LD>;
  constexpr int N = GC::NROOT;
  constexpr int NGR = GradReg<LA, LB, LC, LD>::NGR;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int item = blockIdx.x * 4 + warp;
  if (item >= args.nwork) return;
  const int4 w = args.work[item];
  const int bra = args.bra_pairs[w.x];
  double bA[3] = {0, 0, 0}, bB[3] = {0, 0, 0};
  int atA = 0, atB = 0;
  int kb, ke;
  grad_ket_range(args, item, w, kb, ke);
  if (kb >= ke) return;
  // few kets in the item: groups of lanes share each quartet's primitives
  const LaneSplit ls = lane_split(lane, ke - kb, args.pair_info[bra].w, args.pair_info[args.ket_pairs[kb]].w);
  const int slot = lane / ls.t;
  for (int k0 = kb; k0 < ke; k0 += 32 / ls.t) {
    const bool active = k0 + slot < ke;
    const int k = active ? k0 + slot : ke - 1;
    QuartetGeom g;
    load_quartet(args, bra, args.ket_pairs[k], g);
    atA = args.ws_atm[g.A];
    atB = args.ws_atm[g.B];
    const long long base = args.mol_base[g.mol];
    const int n = args.mol_n[g.mol];
    R gam[CI::NOUT];
    static_for<0, CI::NOUT>([&](auto O) {
      constexpr int o = decltype(O)::value;
      constexpr int id = o % CI::ND, ic = (o / CI::ND) % CI::NC;
      constexpr int ib = (o / CI::NCD) % CI::NB, ia = o / (CI::NCD * CI::NB);
      gam[o] = active ? R(g.scale * gamma_abcd(args, base, n, g.aoA + ia, g.aoB + ib, g.aoC + ic, g.aoD + id)) : R(0);
    });
    R dA[3] = {0, 0, 0}, dB[3] = {0, 0, 0}, dC[3] = {0, 0, 0};
    for (int i = g.ppa + ls.si; i < g.ppa + g.npa; i += ls.ti) {
      const R alpha = R(args.pp_exp[i].x), beta = R(args.pp_exp[i].y);
      for (int j = g.ppc + ls.sj; j < g.ppc + g.npc; j += ls.tj) {
        PrimQ<R> s;
        grad_prim<R>(args, g, i, j, s);
        const R gamma_c = R(args.pp_exp[j].x);
        R x[N], wt[N];
        rys_roots<N, R>(s.t, x, wt, args.tb);
#pragma unroll
        for (int r = 0; r < N; ++r) {
          RootCoef<R> rc;
          root_coef<R>(s, x[r], rc);
          R G[3][NGR];
          build_g<LA + 1, LB + 1, LC + 1, LD, R>(rc.c00[0], rc.c0p[0], rc.b10, rc.b01, rc.b00, R(1), R(g.abx),
                                                 R(g.cdx), G[0]);
          build_g<LA + 1, LB + 1, LC + 1, LD, R>(rc.c00[1], rc.c0p[1], rc.b10, rc.b01, rc.b00, R(1), R(g.aby),
                                                 R(g.cdy), G[1]);
          build_g<LA + 1, LB + 1, LC + 1, LD, R>(rc.c00[2], rc.c0p[2], rc.b10, rc.b01, rc.b00, wt[r] * s.pref,
                                                 R(g.abz), R(g.cdz), G[2]);
          static_for<0, CI::NOUT>([&](auto O) {
            constexpr int o = decltype(O)::value;
            constexpr int id = o % CI::ND, ic = (o / CI::ND) % CI::NC;
            constexpr int ib = (o / CI::NCD) % CI::NB, ia = o / (CI::NCD * CI::NB);
            R v[3], fa[3], fb[3], fc[3];
            static_for<0, 3>([&](auto X) {
              constexpr int ax = decltype(X)::value;
              constexpr int a = ax == 0 ? cart_lx(LA, ia) : ax == 1 ? cart_ly(LA, ia) : cart_lz(LA, ia);
              constexpr int b = ax == 0 ? cart_lx(LB, ib) : ax == 1 ? cart_ly(LB, ib) : cart_lz(LB, ib);
              constexpr int c = ax == 0 ? cart_lx(LC, ic) : ax == 1 ? cart_ly(LC, ic) : cart_lz(LC, ic);
              constexpr int d = ax == 0 ? cart_lx(LD, id) : ax == 1 ? cart_ly(LD, id) : cart_lz(LD, id);
              v[ax] = G[ax][GI::idx(a, b, c, d)];
              fa[ax] = R(2) * alpha * G[ax][GI::idx(a + 1, b, c, d)];
              fb[ax] = R(2) * beta * G[ax][GI::idx(a, b + 1, c, d)];
              fc[ax] = R(2) * gamma_c * G[ax][GI::idx(a, b, c + 1, d)];
              if constexpr (a > 0) fa[ax] -= R(a) * G[ax][GI::idx(a - 1, b, c, d)];
              if constexpr (b > 0) fb[ax] -= R(b) * G[ax][GI::idx(a, b - 1, c, d)];
              if constexpr (c > 0) fc[ax] -= R(c) * G[ax][GI::idx(a, b, c - 1, d)];
            });
            const R gq = gam[o];
            const R yz = v[1] * v[2], xz = v[0] * v[2], xy = v[0] * v[1];
            dA[0] += gq * fa[0] * yz; dA[1] += gq * fa[1] * xz; dA[2] += gq * fa[2] * xy;
            dB[0] += gq * fb[0] * yz; dB[1] += gq * fb[1] * xz; dB[2] += gq * fb[2] * xy;
            dC[0] += gq * fc[0] * yz; dC[1] += gq * fc[1] * xz; dC[2] += gq * fc[2] * xy;
          });
        }
      }
    }
    lane_sum<3>(dA, ls);
    lane_sum<3>(dB, ls);
    lane_sum<3>(dC, ls);
    if (active && ls.sub == 0) {
      double* gC = args.grad + 3LL * args.ws_atm[g.C];
      double* gD = args.grad + 3LL * args.ws_atm[g.D];
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        atomicAdd(gC + x, double(dC[x]));
        atomicAdd(gD + x, -(double(dA[x]) + double(dB[x]) + double(dC[x])));
        bA[x] += double(dA[x]);
        bB[x] += double(dB[x]);
      }
    }
  }
#pragma unroll
  for (int x = 0; x < 3; ++x)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      bA[x] += __shfl_down_sync(0xffffffffu, bA[x], off);
      bB[x] += __shfl_down_sync(0xffffffffu, bB[x], off);
    }
  if (lane == 0) {
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      atomicAdd(args.grad + 3LL * atA + x, bA[x]);
      atomicAdd(args.grad + 3LL * atB + x, bB[x]);
    }
  }
}

// Four derivative-table values (G, f_A, f_B, f_C) stored side by side: one
// 16-byte access in FP32, two in FP64.
template <typename R> struct Quad;
template <> struct Quad<double> {
  static __device__ __forceinline__ void st(double* p, double a, double b, double c, double d) {
    reinterpret_cast<double2*>(p)[0] = make_double2(a, b);
    reinterpret_cast<double2*>(p)[1] = make_double2(c, d);
  }
  static __device__ __forceinline__ void ld(const double* p, double& a, double& b, double& c, double& d) {
    const double2 x = reinterpret_cast<const double2*>(p)[0], y = reinterpret_cast<const double2*>(p)[1];
    a = x.x; b = x.y; c = y.x; d = y.y;
  }
};
template <> struct Quad<float> {
  static __device__ __forceinline__ void st(float* p, float a, float b, float c, float d) {
    *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
  }
  static __device__ __forceinline__ void ld(const float* p, float& a, float& b, float& c, float& d) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    a = x.x; b = x.y; c = x.z; d = x.w;
  }
};

// ---------------------------------------------------------------------------
// Raised 2D tables of one (root, axis) in memory, in two stages: the vertical
// recursion (columns in registers) with the ket transfer, one thread per
// table; then the bra transfer, independent for every ket pair (c, d), one
// thread per (table, c, d).  RA, RB, RC are the raised shells; the table is
// G[((a (RB+1) + b)(RC+1) + c)(LD+1) + d], `w` holds raised_scratch values.
// ---------------------------------------------------------------------------
template <int RA, int RB, int RC, int LD>
__host__ __device__ constexpr int raised_scratch() { return (RA + RB + 1) * (RC + LD + 1) * (LD + 1); }

template <int RA, int RB, int RC, int LD, typename R>
__device__ __forceinline__ void raised_vertical(R c00, R c0p, R b10, R b01, R b00, R g00, R cd, R* w) {
  constexpr int LAB = RA + RB, LCD = RC + LD;
  auto W = [&](int e, int c, int d) -> R& { return w[(e * (LCD + 1) + c) * (LD + 1) + d]; };
  R prev[LAB + 1], cur[LAB + 1];
  cur[0] = g00;
  cur[1] = c00 * g00;
#pragma unroll
  for (int e = 1; e < LAB; ++e) cur[e + 1] = c00 * cur[e] + R(e) * b10 * cur[e - 1];
#pragma unroll
  for (int e = 0; e <= LAB; ++e) {
    W(e, 0, 0) = cur[e];
    prev[e] = R(0);
  }
#pragma unroll 1
  for (int f = 0; f < LCD; ++f) {
    R next[LAB + 1];
    const R fb = R(f) * b01;
#pragma unroll
    for (int e = 0; e <= LAB; ++e) {
      R val = c0p * cur[e] + fb * prev[e];
      if (e > 0) val += R(e) * b00 * cur[e - 1];
      next[e] = val;
    }
#pragma unroll
    for (int e = 0; e <= LAB; ++e) {
      prev[e] = cur[e];
      cur[e] = next[e];
      W(e, f + 1, 0) = next[e];
    }
  }
  if constexpr (LD > 0) {
#pragma unroll 1
    for (int e = 0; e <= LAB; ++e)
#pragma unroll
      for (int d = 1; d <= LD; ++d)
#pragma unroll
        for (int c = 0; c <= LCD - d; ++c) W(e, c, d) = W(e, c + 1, d - 1) + cd * W(e, c, d - 1);
  }
}

// `q` = c (LD+1) + d, c <= RC.
template <int RA, int RB, int RC, int LD, typename R>
__device__ __forceinline__ void raised_bra(R ab, const R* w, int q, R* G) {
  constexpr int LAB = RA + RB, KET = (RC + LD + 1) * (LD + 1), ROW = (RC + 1) * (LD + 1);
  R y[LAB + 1];
#pragma unroll
  for (int e = 0; e <= LAB; ++e) y[e] = w[e * KET + q];
#pragma unroll
  for (int b = 0; b <= RB; ++b) {
#pragma unroll
    for (int a = 0; a <= RA; ++a) G[(a * (RB + 1) + b) * ROW + q] = y[a];
    if (b < RB) {
#pragma unroll
      for (int a = 0; a + b < LAB; ++a) y[a] = y[a + 1] + ab * y[a];
    }
  }
}

// ---------------------------------------------------------------------------
// Coordinate VJP of every class off the register and lane kernels: a team (a
// warp, or the block of 128 threads for the large blocks) takes one quartet
// and in it batches of RB (primitive quartet, root) units.  Per batch the team
// builds the raised tables (raised_vertical, raised_bra), turns them into
// (value, d/dA, d/dB, d/dC) per (unit, axis, unraised index tuple) -- four
// values side by side, one or two 16-byte loads -- and sums the nine centre
// partials over the (unit, element) pairs; Gamma stays in shared memory per
// quartet.  What bounds it is shared memory: three quads (96 bytes in FP64) feed
// fifteen operations of a (unit, element) pair.  Under ncu, (H2O)4 cc-pVTZ FP64
// (22|10) has the L1 data stage 82% busy (44% of the shared wavefronts are bank
// conflicts) beside 15% of the FP64 pipe.  The forms this replaces built one
// primitive quartet's tables on 3 N threads at a time and recomputed each
// element's derivative factors from the table.
// (H2O)4 cc-pVTZ split VJP 42.2 -> 33.9 ms (serial class times 70 -> 40).
// ---------------------------------------------------------------------------
template <int LA, int LB, int LC, int LD, typename R>
struct GradUnit {
  using CI = ClassInfo<LA, LB, LC, LD>;
  static constexpr int THREADS = 128;
#ifndef B200JK_GRAD_TEAM_NOUT
#define B200JK_GRAD_TEAM_NOUT 400
#endif
  static constexpr int TEAM = CI::NOUT <= B200JK_GRAD_TEAM_NOUT ? 32 : THREADS, TEAMS = THREADS / TEAM;
  static constexpr int N = (CI::L + 1) / 2 + 1;
  static constexpr int B1 = LB + 2, C1 = LC + 2, D1 = LD + 1;
  static constexpr int NG = (((LA + 2) * B1 * C1 * D1) + 3) / 4 * 4;   // 16-byte multiples keep the quads aligned
  static constexpr int NW = raised_scratch<LA + 1, LB + 1, LC + 1, LD>();
  static constexpr int NGU = CI::NG;
  static constexpr int SIDE = ((NW > 4 * NGU ? NW : 4 * NGU) + 3) / 4 * 4;   // scratch, then the quads
  static constexpr int TS = NG + SIDE, UNIT = 3 * TS;
  static constexpr int NEL = (CI::NOUT + 3) / 4 * 4;
#ifndef B200JK_GRAD_UNIT_KB
#define B200JK_GRAD_UNIT_KB 72
#endif
  static constexpr int FIT = (int)((B200JK_GRAD_UNIT_KB * 1024 / sizeof(R) / TEAMS - NEL) / UNIT);
  static constexpr int CAP = TEAM == 32 ? 10 : 42;   // 3 tables per unit fill the team
  static constexpr int RB =
      (int)(B200JK_GRAD_UNIT_KB * 1024 / sizeof(R) / TEAMS) < NEL + UNIT ? 1 : (FIT > CAP ? CAP : FIT);
  static constexpr int TEAM_ELEMS = NEL + RB * UNIT;
  static constexpr size_t bytes() { return (size_t)TEAMS * TEAM_ELEMS * sizeof(R); }
  static_assert(bytes() <= 220 * 1024, "gradient batch exceeds shared memory");
};

template <int LA, int LB, int LC, int LD, typename R>
__global__ void __launch_bounds__(128) grad_unit_kernel(JKArgs args) {
  using CI = ClassInfo<LA, LB, LC, LD>;
  using GU = GradUnit<LA, LB, LC, LD, R>;
  constexpr int TEAM = GU::TEAM, TEAMS = GU::TEAMS, N = GU::N, NGU = GU::NGU, RB = GU::RB, NO = CI::NOUT;
  constexpr int GRP = NO >= TEAM ? 1 : (TEAM / NO < RB ? TEAM / NO : RB);   // threads sharing an element
  constexpr int NCMP = CI::NA + CI::NB + CI::NC + CI::ND;
  extern __shared__ __align__(16) unsigned char gu_raw[];
  __shared__ R s_ex[TEAMS][RB][3];
  __shared__ double red[9][4];
  __shared__ int tup[3][NCMP];
  const int team = threadIdx.x / TEAM, tid = threadIdx.x % TEAM;
  R* gam = reinterpret_cast<R*>(gu_raw) + (size_t)team * GU::TEAM_ELEMS;
  R* units = gam + GU::NEL;
  R(*ex)[3] = s_ex[team];
  auto sync = [] {
    if constexpr (TEAM == 32) __syncwarp();
    else __syncthreads();
  };
  // an element's unraised tuple along each axis is a sum over its four components
  for (int t = threadIdx.x; t < NCMP; t += GU::THREADS) {
    const int which = t < CI::NA ? 0 : t < CI::NA + CI::NB ? 1 : t < CI::NA + CI::NB + CI::NC ? 2 : 3;
    const int c = t - (which > 0 ? CI::NA : 0) - (which > 1 ? CI::NB : 0) - (which > 2 ? CI::NC : 0);
    const int l = which == 0 ? LA : which == 1 ? LB : which == 2 ? LC : LD;
    const int stride = which == 0 ? (LB + 1) * (LC + 1) * (LD + 1)
                                  : which == 1 ? (LC + 1) * (LD + 1) : which == 2 ? (LD + 1) : 1;
    tup[0][t] = cart_lx(l, c) * stride;
    tup[1][t] = cart_ly(l, c) * stride;
    tup[2][t] = cart_lz(l, c) * stride;
  }
  __syncthreads();
  const int4 w = args.work[blockIdx.x];
  const int bra = args.bra_pairs[w.x];
  int kb, ke;
  grad_ket_range(args, blockIdx.x, w, kb, ke);
  for (int k = kb + team; k < ke; k += TEAMS) {
    QuartetGeom g;
    load_quartet(args, bra, args.ket_pairs[k], g);
    const long long base = args.mol_base[g.mol];
    const int n = args.mol_n[g.mol];
    for (int o = tid; o < NO; o += TEAM) {
      const int id = o % CI::ND, ic = (o / CI::ND) % CI::NC, ib = (o / CI::NCD) % CI::NB, ia = o / (CI::NCD * CI::NB);
      gam[o] = R(g.scale * gamma_abcd(args, base, n, g.aoA + ia, g.aoB + ib, g.aoC + ic, g.aoD + id));
    }
    R dA[3] = {0, 0, 0}, dB[3] = {0, 0, 0}, dC[3] = {0, 0, 0};
    const int nunit = g.npa * g.npc * N;
    for (int u0 = 0; u0 < nunit; u0 += RB) {
      const int nu = min(RB, nunit - u0);
      sync();   // the previous batch's quads are no longer read
      for (int t = tid; t < 3 * nu; t += TEAM) {
        const int u = t / 3, ax = t - 3 * u;
        const int p = (u0 + u) / N, r = (u0 + u) - p * N;
        const int i = g.ppa + p / g.npc, j = g.ppc + p % g.npc;
        PrimQ<R> s;
        grad_prim<R>(args, g, i, j, s);
        RootCoef<R> rc;
        root_coef<R>(s, rys_one<N, R>(s.t, r, args.tb), rc);
        const R cdd = R(ax == 0 ? g.cdx : (ax == 1 ? g.cdy : g.cdz));
        const R c00 = ax == 0 ? rc.c00[0] : (ax == 1 ? rc.c00[1] : rc.c00[2]);
        const R c0p = ax == 0 ? rc.c0p[0] : (ax == 1 ? rc.c0p[1] : rc.c0p[2]);
        const R g00 = ax == 2 ? rys_one<N, R>(s.t, N + r, args.tb) * s.pref : R(1);
        raised_vertical<LA + 1, LB + 1, LC + 1, LD, R>(c00, c0p, rc.b10, rc.b01, rc.b00, g00, cdd,
                                                       units + t * GU::TS + GU::NG);
        ex[u][ax] = R(2) * R(ax == 0 ? args.pp_exp[i].x : ax == 1 ? args.pp_exp[i].y : args.pp_exp[j].x);
      }
      sync();
      for (int t = tid; t < 3 * nu * GU::C1 * GU::D1; t += TEAM) {
        const int ua = t / (GU::C1 * GU::D1), q = t - ua * (GU::C1 * GU::D1), ax = ua % 3;
        const R abd = R(ax == 0 ? g.abx : (ax == 1 ? g.aby : g.abz));
        raised_bra<LA + 1, LB + 1, LC + 1, LD, R>(abd, units + ua * GU::TS + GU::NG, q, units + ua * GU::TS);
      }
      sync();
      for (int t = tid; t < 3 * nu * NGU; t += TEAM) {
        const int ua = t / NGU, q = t - ua * NGU, u = ua / 3;
        const int d = q % (LD + 1), c = (q / (LD + 1)) % (LC + 1);
        const int b = (q / ((LD + 1) * (LC + 1))) % (LB + 1), a = q / ((LD + 1) * (LC + 1) * (LB + 1));
        const R* G = units + ua * GU::TS + ((a * GU::B1 + b) * GU::C1 + c) * GU::D1 + d;
        R fa = ex[u][0] * G[GU::B1 * GU::C1 * GU::D1], fb = ex[u][1] * G[GU::C1 * GU::D1], fc = ex[u][2] * G[GU::D1];
        if (a) fa -= R(a) * G[-GU::B1 * GU::C1 * GU::D1];
        if (b) fb -= R(b) * G[-GU::C1 * GU::D1];
        if (c) fc -= R(c) * G[-GU::D1];
        Quad<R>::st(units + ua * GU::TS + GU::NG + 4 * q, G[0], fa, fb, fc);
      }
      sync();
      for (int t = tid; t < GRP * NO; t += TEAM) {
        const int grp = t / NO, o = t - grp * NO;
        const R gq = gam[o];
        if (gq == R(0)) continue;
        const int id = o % CI::ND, ic = (o / CI::ND) % CI::NC, ib = (o / CI::NCD) % CI::NB, ia = o / (CI::NCD * CI::NB);
        int tx[3];
#pragma unroll
        for (int x = 0; x < 3; ++x)
          tx[x] = GU::NG + x * GU::TS +
                  4 * (tup[x][ia] + tup[x][CI::NA + ib] + tup[x][CI::NA + CI::NB + ic] +
                       tup[x][CI::NA + CI::NB + CI::NC + id]);
#pragma unroll 2
        for (int u = grp; u < nu; u += GRP) {
          const R* U = units + u * GU::UNIT;
          R vx, ax, bx, cx, vy, ay, by, cy, vz, az, bz, cz;
          Quad<R>::ld(U + tx[0], vx, ax, bx, cx);
          Quad<R>::ld(U + tx[1], vy, ay, by, cy);
          Quad<R>::ld(U + tx[2], vz, az, bz, cz);
          const R yz = gq * vy * vz, xz = gq * vx * vz, xy = gq * vx * vy;
          dA[0] += ax * yz; dA[1] += ay * xz; dA[2] += az * xy;
          dB[0] += bx * yz; dB[1] += by * xz; dB[2] += bz * xy;
          dC[0] += cx * yz; dC[1] += cy * xz; dC[2] += cz * xy;
        }
      }
    }
    double part[9] = {double(dA[0]), double(dA[1]), double(dA[2]), double(dB[0]), double(dB[1]),
                      double(dB[2]), double(dC[0]), double(dC[1]), double(dC[2])};
#pragma unroll
    for (int q = 0; q < 9; ++q)
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) part[q] += __shfl_down_sync(0xffffffffu, part[q], off);
    if constexpr (TEAM != 32) {
      if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int q = 0; q < 9; ++q) red[q][threadIdx.x >> 5] = part[q];
      }
      __syncthreads();
      if (tid == 0) {
#pragma unroll
        for (int q = 0; q < 9; ++q) part[q] = red[q][0] + red[q][1] + red[q][2] + red[q][3];
      }
    }
    if (tid == 0) {
      double* gA = args.grad + 3LL * args.ws_atm[g.A];
      double* gB = args.grad + 3LL * args.ws_atm[g.B];
      double* gC = args.grad + 3LL * args.ws_atm[g.C];
      double* gD = args.grad + 3LL * args.ws_atm[g.D];
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        atomicAdd(gA + x, part[x]);
        atomicAdd(gB + x, part[3 + x]);
        atomicAdd(gC + x, part[6 + x]);
        atomicAdd(gD + x, -(part[x] + part[3 + x] + part[6 + x]));
      }
    }
    sync();   // Gamma (and red) are rewritten by the next quartet
  }
}

// Per-lane coordinate VJP for the mid-size classes (NOUT <= 90): one lane
// per ket of a work item as the register path, Gamma of the lane's quartet
// in a private column of shared memory (conflict-free: element-major,
// lane-minor), and per root the derivative tables of one centre at a time
// in registers -- raised in a for d/dA, in b for d/dB, in c for d/dC (three
// smaller tables instead of one raised in all three, so a table set fits
// the registers).  Every index is a compile-time constant.
template <int LA, int LB, int LC, int LD>
struct GradLane {
  using CI = ClassInfo<LA, LB, LC, LD>;
  static constexpr int NGA = (LA + 2) * (LB + 1) * (LC + 1) * (LD + 1);
  static constexpr int NGB = (LA + 1) * (LB + 2) * (LC + 1) * (LD + 1);
  static constexpr int NGC = (LA + 1) * (LB + 1) * (LC + 2) * (LD + 1);
  static constexpr int NGMAX = NGA > NGB ? (NGA > NGC ? NGA : NGC) : (NGB > NGC ? NGB : NGC);
  static constexpr int THREADS = 128;
  static constexpr size_t bytes() { return (size_t)CI::NOUT * THREADS * sizeof(double); }   // FP64; FP32 half
#ifndef B200JK_GRAD_LANE_TABLES
#define B200JK_GRAD_LANE_TABLES 90   // doubles of one centre's three tables
#endif
  // (H2O)8 cc-pVTZ FP64 class times, this kernel against grad_unit_kernel: all
  // eleven classes inside the line are faster here, from (11|11) 3.0 against
  // 5.2 ms and (20|11) 6.3 / 21.2 to (31|00) 1.6 / 6.7 (the whole VJP 269 / 348 ms,
  // split 236 / 281).  With the line at 110 elements and 162 doubles (30|11)
  // 4.5 -> 3.1 ms and (22|10) 11.4 -> 10.5, but (30|30) 1.13 -> 1.30, the whole VJP
  // unchanged and the split one 236 -> 242 ms: the line stays.  Classes that fit
  // the register kernel were slower here (0.83-0.87x, (H2O)16 cc-pVTZ).
  static constexpr bool OK = !GradReg<LA, LB, LC, LD>::OK && CI::NOUT <= 90 && 3 * NGMAX <= B200JK_GRAD_LANE_TABLES;
};

// One shared-memory load the compiler keeps in place: each centre pass
// re-reads Gamma instead of holding NOUT values live across the passes.
__device__ __forceinline__ double lds_keep(const double* p) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"((unsigned)__cvta_generic_to_shared(p)));
  return v;
}
__device__ __forceinline__ float lds_keep(const float* p) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"((unsigned)__cvta_generic_to_shared(p)));
  return v;
}

// d/dX of one centre (X = 0: A, 1: B, 2: C) for every element of the lane's
// quartet at one root: tables raised in X's index, Gamma from the lane's
// shared-memory column, partials into d[3].
template <int LA, int LB, int LC, int LD, int X, typename R>
__device__ __forceinline__ void grad_lane_centre(const RootCoef<R>& rc, R g00, const QuartetGeom& g, R expo,
                                                 const R* __restrict__ gam, R* d) {
  using CI = ClassInfo<LA, LB, LC, LD>;
  constexpr int RA = LA + (X == 0), RB = LB + (X == 1), RC = LC + (X == 2);
  using GI = GIdx<RA, RB, RC, LD>;
  constexpr int NGX = (RA + 1) * (RB + 1) * (RC + 1) * (LD + 1);
  R G[3][NGX];
  build_g<RA, RB, RC, LD, R>(rc.c00[0], rc.c0p[0], rc.b10, rc.b01, rc.b00, R(1), R(g.abx), R(g.cdx), G[0]);
  build_g<RA, RB, RC, LD, R>(rc.c00[1], rc.c0p[1], rc.b10, rc.b01, rc.b00, R(1), R(g.aby), R(g.cdy), G[1]);
  build_g<RA, RB, RC, LD, R>(rc.c00[2], rc.c0p[2], rc.b10, rc.b01, rc.b00, g00, R(g.abz), R(g.cdz), G[2]);
  const R e2 = R(2) * expo;
  // compile-time element indices: the tables stay in registers
  static_for_n<CI::NOUT>([&](auto O) {
    constexpr int o = decltype(O)::value;
    constexpr int id = o % CI::ND, ic = (o / CI::ND) % CI::NC;
    constexpr int ib = (o / CI::NCD) % CI::NB, ia = o / (CI::NCD * CI::NB);
    R v[3], f[3];
    static_for_n<3>([&](auto AX) {
      constexpr int ax = decltype(AX)::value;
      constexpr int a = ax == 0 ? cart_lx(LA, ia) : ax == 1 ? cart_ly(LA, ia) : cart_lz(LA, ia);
      constexpr int b = ax == 0 ? cart_lx(LB, ib) : ax == 1 ? cart_ly(LB, ib) : cart_lz(LB, ib);
      constexpr int c = ax == 0 ? cart_lx(LC, ic) : ax == 1 ? cart_ly(LC, ic) : cart_lz(LC, ic);
      constexpr int dd = ax == 0 ? cart_lx(LD, id) : ax == 1 ? cart_ly(LD, id) : cart_lz(LD, id);
      constexpr int n = X == 0 ? a : X == 1 ? b : c;   // the raised index
      v[ax] = G[ax][GI::idx(a, b, c, dd)];
      f[ax] = e2 * G[ax][GI::idx(a + (X == 0), b + (X == 1), c + (X == 2), dd)];
      if constexpr (n > 0) f[ax] -= R(n) * G[ax][GI::idx(a - (X == 0), b - (X == 1), c - (X == 2), dd)];
    });
    const R gq = lds_keep(gam + o * GradLane<LA, LB, LC, LD>::THREADS);
    d[0] += gq * f[0] * (v[1] * v[2]);
    d[1] += gq * f[1] * (v[0] * v[2]);
    d[2] += gq * f[2] * (v[0] * v[1]);
  });
}

template <int LA, int LB, int LC, int LD, typename R>
__global__ void __launch_bounds__(128) grad_lane_kernel(JKArgs args) {
  using CI = ClassInfo<LA, LB, LC, LD>;
  using GC = GradCfg<LA, LB, LC, LD>;
  using GL = GradLane<LA, LB, LC, LD>;
  constexpr int N = GC::NROOT;
  extern __shared__ __align__(16) unsigned char s_gam_raw[];   // [NOUT][THREADS]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int item = blockIdx.x * (GL::THREADS / 32) + warp;
  if (item >= args.nwork) return;
  R* gam = reinterpret_cast<R*>(s_gam_raw) + threadIdx.x;
  const int4 w = args.work[item];
  const int bra = args.bra_pairs[w.x];
  double bA[3] = {0, 0, 0}, bB[3] = {0, 0, 0};
  int atA = 0, atB = 0;
  int kb, ke;
  grad_ket_range(args, item, w, kb, ke);
  if (kb >= ke) return;
  // few kets in the item: groups of lanes share each quartet's primitives
  const LaneSplit ls = lane_split(lane, ke - kb, args.pair_info[bra].w, args.pair_info[args.ket_pairs[kb]].w);
  const int slot = lane / ls.t;
  for (int k0 = kb; k0 < ke; k0 += 32 / ls.t) {
    const bool active = k0 + slot < ke;
    const int k = active ? k0 + slot : ke - 1;
    QuartetGeom g;
    load_quartet(args, bra, args.ket_pairs[k], g);
    atA = args.ws_atm[g.A];
    atB = args.ws_atm[g.B];
    const long long base = args.mol_base[g.mol];
    const int n = args.mol_n[g.mol];
    for (int o = 0; o < CI::NOUT; ++o) {
      const int id = o % CI::ND, ic = (o / CI::ND) % CI::NC;
      const int ib = (o / CI::NCD) % CI::NB, ia = o / (CI::NCD * CI::NB);
      gam[o * GL::THREADS] =
          active ? R(g.scale * gamma_abcd(args, base, n, g.aoA + ia, g.aoB + ib, g.aoC + ic, g.aoD + id)) : R(0);
    }
    R dA[3] = {0, 0, 0}, dB[3] = {0, 0, 0}, dC[3] = {0, 0, 0};
    for (int i = g.ppa + ls.si; i < g.ppa + g.npa; i += ls.ti) {
      const R alpha = R(args.pp_exp[i].x), beta = R(args.pp_exp[i].y);
      for (int j = g.ppc + ls.sj; j < g.ppc + g.npc; j += ls.tj) {
        PrimQ<R> s;
        grad_prim<R>(args, g, i, j, s);
        const R gamma_c = R(args.pp_exp[j].x);
        R x[N], wt[N];
        rys_roots<N, R>(s.t, x, wt, args.tb);
        // one (root, centre) pass per iteration, not unrolled: one centre's
        // tables are live at a time
#pragma unroll 1
        for (int tsk = 0; tsk < 3 * N; ++tsk) {
          const int r = tsk / 3, cx = tsk - 3 * r;
          RootCoef<R> rc;
          root_coef<R>(s, x[r], rc);
          const R g00 = wt[r] * s.pref;
          if (cx == 0) grad_lane_centre<LA, LB, LC, LD, 0, R>(rc, g00, g, alpha, gam, dA);
          else if (cx == 1) grad_lane_centre<LA, LB, LC, LD, 1, R>(rc, g00, g, beta, gam, dB);
          else grad_lane_centre<LA, LB, LC, LD, 2, R>(rc, g00, g, gamma_c, gam, dC);
        }
      }
    }
    lane_sum<3>(dA, ls);
    lane_sum<3>(dB, ls);
    lane_sum<3>(dC, ls);
    if (active && ls.sub == 0) {
      double* gC = args.grad + 3LL * args.ws_atm[g.C];
      double* gD = args.grad + 3LL * args.ws_atm[g.D];
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        atomicAdd(gC + x, double(dC[x]));
        atomicAdd(gD + x, -(double(dA[x]) + double(dB[x]) + double(dC[x])));
        bA[x] += double(dA[x]);
        bB[x] += double(dB[x]);
      }
    }
  }
#pragma unroll
  for (int x = 0; x < 3; ++x)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      bA[x] += __shfl_down_sync(0xffffffffu, bA[x], off);
      bB[x] += __shfl_down_sync(0xffffffffu, bB[x], off);
    }
  if (lane == 0) {
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      atomicAdd(args.grad + 3LL * atA + x, bA[x]);
      atomicAdd(args.grad + 3LL * atB + x, bB[x]);
    }
  }
}

}  // namespace b200jk

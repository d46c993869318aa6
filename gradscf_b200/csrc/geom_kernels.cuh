// Coordinate products of J/K beyond the gradient: the directional JVP of
// order 1 and 2 and the order-2 VJP (Hessian-vector product), replacing the
// reference's gradscf_direct_jk_geometry_{jvp_cpu_v1, vjp_cpu_v2} with order
// 1 and 2 (csrc/direct_jk_geometry.cc:8-99 over the entries of
// csrc/eri_geometry_entries.h:6-31 and csrc/geometry_contraction.h:7-53).
//
// With u, v coordinate directions (one 3-vector per atm row) and, for one
// canonical quartet with centres A, B, C, D, the translation-invariant
// reductions u~_P = u_P - u_D (P = A, B, C), the kernels evaluate
//   W1 = (u~ . d)(ab|cd),   W2 = (u~ . d)(v~ . d)(ab|cd)
// -- the first and second directional derivatives of the ERI block, which
// keep its eight-fold permutational symmetry, so the JVPs digest W1 / W2
// into J and K exactly as the J/K build digests (ab|cd) -- and, for the VJP,
//   T_{P,x} = sum_abcd Gamma_abcd d/dP_x (u~ . d)(ab|cd),  P = A, B, C,
//   T_{D,x} = -(T_{A,x} + T_{B,x} + T_{C,x}),
// Gamma the eight-permutation contraction of the cotangents with D (as in
// the gradient kernel).  Derivatives act on the 2D Rys integrals with the
// primitive exponents (d/dA_x phi_a = 2 alpha phi_{a+1} - a phi_{a-1}, twice
// for the second derivatives), computed from one table raised by two on A, B
// and C; nothing is stored.
//
// What bounds these products is latency: a small molecule has few quartets
// with up to 1296 (6-31G*) or 4096 (cc-pVDZ) primitive quartets each.  So a
// block of 128 threads works on one quartet, and in it on a batch of RB
// (primitive quartet, root) units: a thread builds the raised table of one
// (unit, axis), then the threads turn the tables into derivative values per
// (unit, axis, unraised index tuple), then they take the (unit, element)
// pairs.  The batch fills about 64 KB of shared memory (three blocks an SM); where
// one unit beside the accumulators is more, a block takes that: (32|32) and
// (33|22) 69 KB, (33|32) 100 (two blocks), (33|33) 150 (one).  Under ncu the
// (00|00) and (10|00) launches of (H2O)2 6-31G* have 2 to 3 warps a scheduler, waiting on the batch's barriers
// and on fixed latencies, the FP64 pipe 20 to 23% busy.
// (H2O)2 6-31G* Hessian-vector product: 120.9 -> 1.55 ms.
#pragma once
#include "grad_kernels.cuh"

namespace b200jk {

constexpr int kGeoThreads = 128;
constexpr int kGeoValues = 8;   // derivative values per (axis, tuple)

template <int LA, int LB, int LC, int LD>
struct GeoCfg {
  using CI = ClassInfo<LA, LB, LC, LD>;
  static constexpr int N = (CI::L + 2) / 2 + 1;
  static constexpr int B2 = LB + 3, C2 = LC + 3, D1 = LD + 1;
  static constexpr int NG = (LA + 3) * B2 * C2 * D1;                      // raised table of one axis
  static constexpr int LAB = LA + LB + 4, LCD = LC + LD + 2;
  static constexpr int NW = (LAB + 1) * (LCD + 1) * D1;                   // recursion scratch
  static constexpr int NGU = CI::NG;                                      // unraised tuples
  static constexpr int SIDE = NW > kGeoValues * NGU ? NW : kGeoValues * NGU;   // scratch, then derivative values
  static constexpr int TS = (NG + SIDE) | 1;                              // per (unit, axis); odd: no bank conflicts
  static constexpr int UNIT = 3 * TS;
  static constexpr int NEL = CI::NOUT > kGeoThreads ? CI::NOUT : kGeoThreads;  // Gamma or block accumulators
  static constexpr int FIT = (64 * 1024 / 8 - NEL) / UNIT;
  static constexpr int RB = FIT < 1 ? 1 : (FIT > 42 ? 42 : FIT);          // 42 units x 3 axes fill the block
  static constexpr size_t bytes() { return (size_t)(NEL + RB * UNIT) * sizeof(double); }
  static_assert(bytes() <= 220 * 1024, "geometry batch exceeds shared memory");
};

// The raised 2D table of one (unit, axis) (build_g with A, B and C raised by
// two): vertical recursion column by column in registers, transfers in the
// scratch `w`; runtime loops over f, c and d keep the code small.
template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ void geo_table(double c00, double c0p, double b10, double b01, double b00, double g00,
                                          double ab, double cd, double* G, double* w) {
  using GC = GeoCfg<LA, LB, LC, LD>;
  constexpr int LAB = GC::LAB, LCD = GC::LCD;
  auto W = [&](int e, int c, int d) -> double& { return w[(e * (LCD + 1) + c) * GC::D1 + d]; };
  double prev[LAB + 1], cur[LAB + 1];
  cur[0] = g00;
  cur[1] = c00 * g00;
#pragma unroll
  for (int e = 1; e < LAB; ++e) cur[e + 1] = c00 * cur[e] + e * b10 * cur[e - 1];
#pragma unroll
  for (int e = 0; e <= LAB; ++e) {
    W(e, 0, 0) = cur[e];
    prev[e] = 0.0;
  }
#pragma unroll 1
  for (int f = 0; f < LCD; ++f) {
    double next[LAB + 1];
    const double fb = f * b01;
#pragma unroll
    for (int e = 0; e <= LAB; ++e) {
      double val = c0p * cur[e] + fb * prev[e];
      if (e > 0) val += e * b00 * cur[e - 1];
      next[e] = val;
    }
#pragma unroll
    for (int e = 0; e <= LAB; ++e) {
      prev[e] = cur[e];
      cur[e] = next[e];
      W(e, f + 1, 0) = next[e];
    }
  }
#pragma unroll 1
  for (int e = 0; e <= LAB; ++e)
#pragma unroll
    for (int d = 1; d <= LD; ++d)
#pragma unroll
      for (int c = 0; c <= LCD - d; ++c) W(e, c, d) = W(e, c + 1, d - 1) + cd * W(e, c, d - 1);
#pragma unroll 1
  for (int cdi = 0; cdi < GC::C2 * GC::D1; ++cdi) {
    double y[LAB + 1];
#pragma unroll
    for (int e = 0; e <= LAB; ++e) y[e] = w[e * (LCD + 1) * GC::D1 + cdi];
#pragma unroll
    for (int b = 0; b < GC::B2; ++b) {
#pragma unroll
      for (int a = 0; a < LA + 3; ++a) G[(a * GC::B2 + b) * GC::C2 * GC::D1 + cdi] = y[a];
      if (b + 1 < GC::B2) {
#pragma unroll
        for (int a = 0; a + b < LAB; ++a) y[a] = y[a + 1] + ab * y[a];
      }
    }
  }
}

// mode 0: JVP order 1, 1: JVP order 2, 2: VJP order 2.
// JKArgs: dens (raw Cartesian D), vj/vk accumulators (JVP), cot_j/cot_k +
// gnb (VJP), grad (VJP output), geo_u / geo_v (atm rows x 3).
template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(kGeoThreads) geom_kernel(JKArgs args, int mode) {
  using CI = ClassInfo<LA, LB, LC, LD>;
  using GC = GeoCfg<LA, LB, LC, LD>;
  constexpr int N = GC::N, NGU = GC::NGU, RB = GC::RB, NO = CI::NOUT;
  // (unit, element) pairs: with few elements, GRP threads share one and
  // split the batch's units
  constexpr int GRP = NO >= kGeoThreads ? 1 : (kGeoThreads / NO < RB ? kGeoThreads / NO : RB);
  extern __shared__ __align__(16) double geo_sm[];
  double* el = geo_sm;              // Gamma (VJP) or block accumulators (JVP)
  double* units = geo_sm + GC::NEL;
  __shared__ double ex[RB][3], su[3][3], sv[3][3], red[9][kGeoThreads / 32];
  __shared__ int tup[3][CI::NA + CI::NB + CI::NC + CI::ND];
  const int tid = threadIdx.x;
  // an element's unraised tuple along each axis is a sum over its four components
  for (int t = tid; t < CI::NA + CI::NB + CI::NC + CI::ND; t += kGeoThreads) {
    const int which = t < CI::NA ? 0 : t < CI::NA + CI::NB ? 1 : t < CI::NA + CI::NB + CI::NC ? 2 : 3;
    const int c = t - (which > 0 ? CI::NA : 0) - (which > 1 ? CI::NB : 0) - (which > 2 ? CI::NC : 0);
    const int l = which == 0 ? LA : which == 1 ? LB : which == 2 ? LC : LD;
    const int stride = which == 0 ? (LB + 1) * (LC + 1) * (LD + 1)
                                  : which == 1 ? (LC + 1) * (LD + 1) : which == 2 ? (LD + 1) : 1;
    tup[0][t] = cart_lx(l, c) * stride;
    tup[1][t] = cart_ly(l, c) * stride;
    tup[2][t] = cart_lz(l, c) * stride;
  }
  const int4 w = args.work[blockIdx.x];
  const int bra = args.bra_pairs[w.x];
  for (int k = w.y + blockIdx.y; k < w.z; k += gridDim.y) {
    QuartetGeom g;
    load_quartet(args, bra, args.ket_pairs[k], g);
    const long long mbase = args.mol_base[g.mol];
    const int n = args.mol_n[g.mol];
    const int at[4] = {args.ws_atm[g.A], args.ws_atm[g.B], args.ws_atm[g.C], args.ws_atm[g.D]};
    __syncthreads();   // the previous quartet's shared values are no longer read
    if (tid < 9) {     // reduced directions [axis][P]
      const int x = tid / 3, P = tid % 3;
      su[x][P] = args.geo_u[3 * at[P] + x] - args.geo_u[3 * at[3] + x];
      sv[x][P] = mode == 1 ? args.geo_v[3 * at[P] + x] - args.geo_v[3 * at[3] + x] : 0.0;
    }
    for (int o = tid; o < GC::NEL; o += kGeoThreads) {
      double v = 0.0;
      if (mode == 2 && o < NO) {
        const int id = o % CI::ND, ic = (o / CI::ND) % CI::NC, ib = (o / CI::NCD) % CI::NB,
                  ia = o / (CI::NCD * CI::NB);
        v = g.scale * gamma_abcd(args, mbase, n, g.aoA + ia, g.aoB + ib, g.aoC + ic, g.aoD + id);
      }
      el[o] = v;
    }
    double T[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};   // VJP: [P][axis]
    const int nunit = g.npa * g.npc * N;
    for (int u0 = 0; u0 < nunit; u0 += RB) {
      const int nu = min(RB, nunit - u0);
      __syncthreads();   // the previous batch's values are no longer read
      for (int t = tid; t < 3 * nu; t += kGeoThreads) {
        const int u = t / 3, ax = t - 3 * u;
        const int p = (u0 + u) / N, r = (u0 + u) - p * N;
        const int i = g.ppa + p / g.npc, j = g.ppc + p % g.npc;
        PrimQ<double> s;
        prim_setup<double>(g, args.pp_data[i], args.pp_aux[i], args.pp_data[j], args.pp_aux[j], s);
        RootCoef<double> rc;
        root_coef<double>(s, rys_one<N, double>(s.t, r, args.tb), rc);
        const double abd = ax == 0 ? g.abx : (ax == 1 ? g.aby : g.abz);
        const double cdd = ax == 0 ? g.cdx : (ax == 1 ? g.cdy : g.cdz);
        const double c00 = ax == 0 ? rc.c00[0] : (ax == 1 ? rc.c00[1] : rc.c00[2]);
        const double c0p = ax == 0 ? rc.c0p[0] : (ax == 1 ? rc.c0p[1] : rc.c0p[2]);
        const double g00 = ax == 2 ? rys_one<N, double>(s.t, N + r, args.tb) * s.pref : 1.0;
        double* G = units + (u * 3 + ax) * GC::TS;
        geo_table<LA, LB, LC, LD>(c00, c0p, rc.b10, rc.b01, rc.b00, g00, abd, cdd, G, G + GC::NG);
        ex[u][ax] = ax == 0 ? args.pp_exp[i].x : ax == 1 ? args.pp_exp[i].y : args.pp_exp[j].x;
      }
      __syncthreads();
      // derivative values per (unit, axis, unraised tuple), over the scratch
      for (int t = tid; t < 3 * nu * NGU; t += kGeoThreads) {
        const int ua = t / NGU, q = t - ua * NGU, u = ua / 3, x = ua - 3 * u;
        const int d = q % (LD + 1), c = (q / (LD + 1)) % (LC + 1);
        const int b = (q / ((LD + 1) * (LC + 1))) % (LB + 1), a = q / ((LD + 1) * (LC + 1) * (LB + 1));
        const double* G = units + ua * GC::TS;
        double* D = units + ua * GC::TS + GC::NG + q * kGeoValues;
        const double al = ex[u][0], be = ex[u][1], ga = ex[u][2];
        auto gat = [&](int p, int r, int s) { return G[((p * GC::B2 + r) * GC::C2 + s) * GC::D1 + d]; };
        const double I = gat(a, b, c);
        // d/dP of the value at (p, r, s): 2 e f(+1) - n f(-1)
        auto dA = [&](int p, int r, int s) { return 2.0 * al * gat(p + 1, r, s) - (p ? p * gat(p - 1, r, s) : 0.0); };
        auto dB = [&](int p, int r, int s) { return 2.0 * be * gat(p, r + 1, s) - (r ? r * gat(p, r - 1, s) : 0.0); };
        auto dC = [&](int p, int r, int s) { return 2.0 * ga * gat(p, r, s + 1) - (s ? s * gat(p, r, s - 1) : 0.0); };
        const double vA = dA(a, b, c), vB = dB(a, b, c), vC = dC(a, b, c);
        const double uA = su[x][0], uB = su[x][1], uC = su[x][2];
        D[0] = I;
        D[1] = uA * vA + uB * vB + uC * vC;
        if (mode == 0) continue;
        const double AA = 2.0 * al * dA(a + 1, b, c) - (a ? a * dA(a - 1, b, c) : 0.0);
        const double AB = 2.0 * al * dB(a + 1, b, c) - (a ? a * dB(a - 1, b, c) : 0.0);
        const double AC = 2.0 * al * dC(a + 1, b, c) - (a ? a * dC(a - 1, b, c) : 0.0);
        const double BB = 2.0 * be * dB(a, b + 1, c) - (b ? b * dB(a, b - 1, c) : 0.0);
        const double BC = 2.0 * be * dC(a, b + 1, c) - (b ? b * dC(a, b - 1, c) : 0.0);
        const double CC = 2.0 * ga * dC(a, b, c + 1) - (c ? c * dC(a, b, c - 1) : 0.0);
        const double PA = uA * AA + uB * AB + uC * AC, PB = uA * AB + uB * BB + uC * BC,
                     PC = uA * AC + uB * BC + uC * CC;
        if (mode == 1) {
          D[2] = sv[x][0] * vA + sv[x][1] * vB + sv[x][2] * vC;
          D[3] = sv[x][0] * PA + sv[x][1] * PB + sv[x][2] * PC;
        } else {
          D[2] = vA; D[3] = vB; D[4] = vC;
          D[5] = PA; D[6] = PB; D[7] = PC;
        }
      }
      __syncthreads();
      for (int t = tid; t < GRP * NO; t += kGeoThreads) {
        const int grp = t / NO, o = t - grp * NO;
        const double gq = mode == 2 ? el[o] : 0.0;
        if (mode == 2 && gq == 0.0) continue;
        const int id = o % CI::ND, ic = (o / CI::ND) % CI::NC, ib = (o / CI::NCD) % CI::NB,
                  ia = o / (CI::NCD * CI::NB);
        int tx[3];
#pragma unroll
        for (int x = 0; x < 3; ++x)
          tx[x] = GC::NG + x * GC::TS +
                  kGeoValues * (tup[x][ia] + tup[x][CI::NA + ib] + tup[x][CI::NA + CI::NB + ic] +
                                tup[x][CI::NA + CI::NB + CI::NC + id]);
        double sum = 0.0;
        for (int u = grp; u < nu; u += GRP) {
          const double* U = units + u * GC::UNIT;
          const double *X = U + tx[0], *Y = U + tx[1], *Z = U + tx[2];
          const double x0 = X[0], y0 = Y[0], z0 = Z[0], x1 = X[1], y1 = Y[1], z1 = Z[1];
          if (mode == 0) {
            sum += x1 * y0 * z0 + x0 * y1 * z0 + x0 * y0 * z1;
          } else if (mode == 1) {
            const double x2 = X[2], y2 = Y[2], z2 = Z[2];
            sum += X[3] * y0 * z0 + x0 * Y[3] * z0 + x0 * y0 * Z[3] + (x1 * y2 + x2 * y1) * z0 +
                   (x1 * z2 + x2 * z1) * y0 + (y1 * z2 + y2 * z1) * x0;
          } else {
            // d/dP_x (u~ . d): the x factor takes dP, the others their plain / directional value
            const double px = gq * y0 * z0, py = gq * x0 * z0, pz = gq * x0 * y0;
            const double rx = gq * (y1 * z0 + y0 * z1), ry = gq * (x1 * z0 + x0 * z1), rz = gq * (x1 * y0 + x0 * y1);
#pragma unroll
            for (int P = 0; P < 3; ++P) {
              T[P][0] += X[5 + P] * px + X[2 + P] * rx;
              T[P][1] += Y[5 + P] * py + Y[2 + P] * ry;
              T[P][2] += Z[5 + P] * pz + Z[2 + P] * rz;
            }
          }
        }
        if (mode != 2) el[t] += sum;
      }
    }
    __syncthreads();
    if (mode == 2) {
#pragma unroll
      for (int q = 0; q < 9; ++q) {
        double v = T[q / 3][q % 3];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
        if ((tid & 31) == 0) red[q][tid >> 5] = v;
      }
      __syncthreads();
      if (tid < 12) {   // [P][axis], P = A, B, C, D
        const int P = tid / 3, x = tid % 3;
        double v = 0.0;
        for (int q = (P == 3 ? 0 : P); q < (P == 3 ? 3 : P + 1); ++q)
          for (int wi = 0; wi < kGeoThreads / 32; ++wi) v += red[3 * q + x][wi];
        const int row = P == 0 ? at[0] : P == 1 ? at[1] : P == 2 ? at[2] : at[3];
        atomicAdd(args.grad + 3LL * row + x, P == 3 ? -v : v);
      }
    } else {
      // the derivative block has the ERI's permutational symmetry, so it
      // enters J/K as (ab|cd) does
      const double sc = g.scale;
      for (int o = tid; o < NO; o += kGeoThreads) {
        double v = 0.0;
        for (int q = 0; q < GRP; ++q) v += el[q * NO + o];
        const int id = o % CI::ND, ic = (o / CI::ND) % CI::NC, ib = (o / CI::NCD) % CI::NB,
                  ia = o / (CI::NCD * CI::NB);
        const int a = g.aoA + ia, b = g.aoB + ib, c = g.aoC + ic, d = g.aoD + id;
        for (int e = 0; e < args.ndm; ++e) {
          const double* dm = args.dens + e * args.dstride + mbase;
          if (args.with_j && e < args.nsym) {
            double* vj = args.vj + e * args.dstride + mbase;
            atomicAdd(vj + (long long)a * n + b, 2.0 * sc * v * dm[(long long)c * n + d]);
            atomicAdd(vj + (long long)c * n + d, 2.0 * sc * v * dm[(long long)a * n + b]);
          }
          if (args.with_k) {
            double* vk = args.vk + e * args.dstride + mbase;
            atomicAdd(vk + (long long)a * n + c, sc * v * dm[(long long)b * n + d]);
            atomicAdd(vk + (long long)a * n + d, sc * v * dm[(long long)b * n + c]);
            atomicAdd(vk + (long long)b * n + c, sc * v * dm[(long long)a * n + d]);
            atomicAdd(vk + (long long)b * n + d, sc * v * dm[(long long)a * n + c]);
          }
        }
      }
    }
  }
}

}  // namespace b200jk

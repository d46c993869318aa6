// Contracted [e0|f0] integrals by the Obara-Saika vertical recursion and the
// horizontal recursion on the contracted block (Obara & Saika, J. Chem. Phys.
// 84, 3963 (1986); Head-Gordon & Pople, J. Chem. Phys. 89, 5777 (1988)).
//
// Why beside Rys quadrature: for total angular momentum L the auxiliary
// integrals need F_0..F_L alone -- no roots (a quadratic or cubic with five to
// ten dependent reciprocals and square roots) -- and the transfer to (ab|cd)
// leaves the primitive loop.  Everything is indexed at compile time, so the
// recursion's values live in registers.
#pragma once
#include "common.cuh"

namespace b200jk {

__host__ __device__ constexpr int cart_l(int axis, int l, int i) {
  return axis == 0 ? cart_lx(l, i) : axis == 1 ? cart_ly(l, i) : cart_lz(l, i);
}
// Components of the shells below l, and the index of component (lx, ., lz) of shell l.
__host__ __device__ constexpr int cart_below(int l) { return l * (l + 1) * (l + 2) / 6; }
__host__ __device__ constexpr int cart_at(int l, int lx, int lz) { return (l - lx) * (l - lx + 1) / 2 + lz; }
// Component i of shell l moved by `by` quanta along `axis`.
__host__ __device__ constexpr int cart_move(int l, int i, int axis, int by) {
  return cart_at(l + by, cart_lx(l, i) + (axis == 0 ? by : 0), cart_lz(l, i) + (axis == 2 ? by : 0));
}
// The axis a component is built along: its smallest nonzero exponent, so the
// fewest components carry the term of the shell two below.
__host__ __device__ constexpr int cart_axis(int l, int i) {
  int best = -1, n = 99;
  for (int x = 0; x < 3; ++x) {
    const int e = cart_l(x, l, i);
    if (e > 0 && e < n) { n = e; best = x; }
  }
  return best;
}

template <int LA, int LB, int LC, int LD>
struct OsInfo {
  static constexpr int LAB = LA + LB, LCD = LC + LD, L = LAB + LCD;
  static constexpr int NE = cart_below(LAB + 1) - cart_below(LA), NF = cart_below(LCD + 1) - cart_below(LC);
  static constexpr int NACC = NE * NF;   // contracted [e0|f0], e = LA..LAB, f = LC..LCD
  // lowest bra shell kept at ket shell f, and the auxiliary orders m kept there
  __host__ __device__ static constexpr int emin(int f) { return f == 0 ? 0 : (LA - (LCD - f) > 0 ? LA - (LCD - f) : 0); }
  __host__ __device__ static constexpr int orders(int e, int f) { return f == 0 ? L - e + 1 : LCD - f + 1; }
  __host__ __device__ static constexpr int off(int e, int f) {
    int o = 0;
    for (int ff = 0; ff <= LCD; ++ff)
      for (int ee = emin(ff); ee <= LAB; ++ee) {
        if (ff == f && ee == e) return o;
        o += ncart(ee) * ncart(ff) * orders(ee, ff);
      }
    return o;
  }
  static constexpr int TOTAL = off(LAB + 1, LCD);   // not found: the sum of all
  __host__ __device__ static constexpr int at(int e, int f, int ce, int cf, int m) {
    return off(e, f) + (ce * ncart(f) + cf) * orders(e, f) + m;
  }
};

// One primitive quartet's scalars for the recursion.
template <typename R>
struct OsPrim {
  R pa[3], wp[3], qc[3], wq[3];
  R inv2p, inv2q, inv2pq, q_pq, p_pq;
};

// The [e0|f0] of one primitive quartet from f[m] = prefactor F_m (m = 0..L):
// `put(index, value)` for every element e >= LA, f >= LC (index < NACC).
template <int LA, int LB, int LC, int LD, typename R, typename Put>
__device__ __forceinline__ void os_vertical(const OsPrim<R>& s, const R* f, Put&& put) {
  using I = OsInfo<LA, LB, LC, LD>;
  constexpr int LAB = I::LAB, LCD = I::LCD, L = I::L;
  R v[I::TOTAL];
  static_for_n<L + 1>([&](auto M) { v[I::at(0, 0, 0, 0, decltype(M)::value)] = f[decltype(M)::value]; });
  // bra: [e+1 0|00]^m
  static_for_n<LAB>([&](auto E) {
    constexpr int e = decltype(E)::value;
    static_for_n<ncart(e + 1)>([&](auto C) {
      constexpr int c = decltype(C)::value, x = cart_axis(e + 1, c), p = cart_move(e + 1, c, x, -1);
      constexpr int n = cart_l(x, e + 1, c) - 1;
      static_for_n<I::orders(e + 1, 0)>([&](auto M) {
        constexpr int m = decltype(M)::value;
        R val = s.pa[x] * v[I::at(e, 0, p, 0, m)] + s.wp[x] * v[I::at(e, 0, p, 0, m + 1)];
        if constexpr (n > 0) {
          constexpr int g = cart_move(e, p, x, -1);
          val += R(n) * (s.inv2p * (v[I::at(e - 1, 0, g, 0, m)] - s.q_pq * v[I::at(e - 1, 0, g, 0, m + 1)]));
        }
        v[I::at(e + 1, 0, c, 0, m)] = val;
      });
    });
  });
  // ket: [e0|f+1 0]^m
  static_for_n<LCD>([&](auto F) {
    constexpr int f0 = decltype(F)::value, e0 = I::emin(f0 + 1);
    static_for_n<LAB + 1 - e0>([&](auto E) {
      constexpr int e = e0 + decltype(E)::value;
      static_for_n<ncart(e)>([&](auto CE) {
        constexpr int ce = decltype(CE)::value;
        static_for_n<ncart(f0 + 1)>([&](auto C) {
          constexpr int c = decltype(C)::value, x = cart_axis(f0 + 1, c), p = cart_move(f0 + 1, c, x, -1);
          constexpr int n = cart_l(x, f0 + 1, c) - 1, k = cart_l(x, e, ce);
          static_for_n<I::orders(e, f0 + 1)>([&](auto M) {
            constexpr int m = decltype(M)::value;
            R val = s.qc[x] * v[I::at(e, f0, ce, p, m)] + s.wq[x] * v[I::at(e, f0, ce, p, m + 1)];
            if constexpr (n > 0) {
              constexpr int g = cart_move(f0, p, x, -1);
              val += R(n) * (s.inv2q * (v[I::at(e, f0 - 1, ce, g, m)] - s.p_pq * v[I::at(e, f0 - 1, ce, g, m + 1)]));
            }
            if constexpr (k > 0) {
              constexpr int d = cart_move(e, ce, x, -1);
              val += R(k) * (s.inv2pq * v[I::at(e - 1, f0, d, p, m + 1)]);
            }
            v[I::at(e, f0 + 1, ce, c, m)] = val;
          });
        });
      });
    });
  });
  static_for_n<LAB + 1 - LA>([&](auto E) {
    constexpr int e = LA + decltype(E)::value;
    static_for_n<ncart(e)>([&](auto CE) {
      constexpr int ce = decltype(CE)::value;
      static_for_n<LCD + 1 - LC>([&](auto F) {
        constexpr int ff = LC + decltype(F)::value;
        static_for_n<ncart(ff)>([&](auto CF) {
          constexpr int cf = decltype(CF)::value;
          constexpr int o = (cart_below(e) - cart_below(LA) + ce) * I::NF + cart_below(ff) - cart_below(LC) + cf;
          put(std::integral_constant<int, o>{}, v[I::at(e, ff, ce, cf, 0)]);
        });
      });
    });
  });
}

// One horizontal transfer: x[shell a = L1..L1+L2, components] (stride S) ->
// y[(a component) ncart(L2) + b component] (stride 1), with
// (a b+1_i) = (a+1_i b) + AB_i (a b); L2 <= 2.
template <int L1, int L2, int S, typename R>
__device__ __forceinline__ void os_transfer(const R* x, const R* ab, R* y) {
  static_assert(L2 <= 2, "transfers up to d shells");
  auto src = [](int l, int c) constexpr { return (cart_below(l) - cart_below(L1) + c) * S; };
  if constexpr (L2 == 0) {
    static_for_n<ncart(L1)>([&](auto C) { y[decltype(C)::value] = x[src(L1, decltype(C)::value)]; });
  } else if constexpr (L2 == 1) {
    static_for_n<ncart(L1)>([&](auto C) {
      constexpr int c = decltype(C)::value;
      static_for_n<3>([&](auto X) {
        constexpr int i = decltype(X)::value;
        y[c * 3 + i] = x[src(L1 + 1, cart_move(L1, c, i, 1))] + ab[i] * x[src(L1, c)];
      });
    });
  } else {
    R t0[ncart(L1) * 3], t1[ncart(L1 + 1) * 3];
    os_transfer<L1, 1, S, R>(x, ab, t0);
    os_transfer<L1 + 1, 1, S, R>(x + ncart(L1) * S, ab, t1);
    static_for_n<ncart(L1)>([&](auto C) {
      constexpr int c = decltype(C)::value;
      static_for_n<6>([&](auto D) {
        constexpr int d = decltype(D)::value, i = cart_axis(2, d), q = cart_move(2, d, i, -1);
        y[c * 6 + d] = t1[cart_move(L1, c, i, 1) * 3 + q] + ab[i] * t0[c * 3 + q];
      });
    });
  }
}

// Contracted [e0|f0] -> (ab|cd), out[((a NB + b) NC + c) ND + d].
template <int LA, int LB, int LC, int LD, typename R>
__device__ __forceinline__ void os_horizontal(const R* acc, const R* ab, const R* cd, R* out) {
  using I = OsInfo<LA, LB, LC, LD>;
  constexpr int NAB = ncart(LA) * ncart(LB), NCD = ncart(LC) * ncart(LD);
  if constexpr (LB == 0 && LD == 0) {
    static_for_n<I::NACC>([&](auto O) { out[decltype(O)::value] = acc[decltype(O)::value]; });
  } else if constexpr (LD == 0) {
    static_for_n<I::NF>([&](auto K) {
      constexpr int k = decltype(K)::value;
      R y[NAB];
      os_transfer<LA, LB, I::NF, R>(acc + k, ab, y);
      static_for_n<NAB>([&](auto O) { out[decltype(O)::value * NCD + k] = y[decltype(O)::value]; });
    });
  } else {
    R y[NAB * I::NF];
    static_for_n<I::NF>([&](auto K) {
      constexpr int k = decltype(K)::value;
      R t[NAB];
      os_transfer<LA, LB, I::NF, R>(acc + k, ab, t);
      static_for_n<NAB>([&](auto O) { y[decltype(O)::value * I::NF + k] = t[decltype(O)::value]; });
    });
    static_for_n<NAB>([&](auto O) {
      constexpr int o = decltype(O)::value;
      os_transfer<LC, LD, 1, R>(y + o * I::NF, cd, out + o * NCD);
    });
  }
}

}  // namespace b200jk
